"""Epilogue of the tensor-core GEMM: eight warps, 32 columns at a time.  Column counts that end inside a group, inside a 16-byte unit and inside a
tile, rows that end inside a warp's 32, more tiles than SMs; both formats, every combination of operands that the lean and the full form
take, rows of the residual on and off the 16-byte grid."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _act(v, act):
    return torch.relu(v) if act == 1 else v * torch.sigmoid(1.702 * v) if act == 6 else v


@pytest.mark.parametrize("M,N,K,block_n", [(1, 8, 64, 128), (33, 40, 64, 256), (130, 264, 72, 128), (257, 328, 200, 256), (40000, 136, 64, 128), (300, 96, 512, 256)])
@pytest.mark.parametrize("opts", [dict(), dict(bias="f32"), dict(bias="lp", act=1), dict(bias="f32", res=0, relu=True), dict(res=3), dict(bias="f32", act=6, aux=True),
                                  dict(out32=True, bias="f32"), dict(alpha=0.5, bias="lp"), dict(res=0, res_act=6)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_matches_fp64(M, N, K, block_n, opts, dtype):
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)      # noqa: E731
    a, b = rnd(M, K), (rnd(N, K).float() * K ** -0.5).to(dtype).t()
    bias = {None: None, "f32": torch.randn(N, device="cuda", generator=g), "lp": rnd(N)}[opts.get("bias")]
    res = rnd(M, N + opts["res"])[:, opts["res"]:] if "res" in opts else None      # 3: rows off the 16-byte grid
    aux = torch.empty(M, N, device="cuda", dtype=dtype) if opts.get("aux") else None
    act = opts.get("act", 0)
    out = native.gemm_raw(a, b, bias=bias, act=act | (1 << 16 if opts.get("relu") else 0), aux=aux, residual=res, alpha=opts.get("alpha", 1.0), block_n=block_n,
                          out_dtype=torch.float32 if opts.get("out32") else None, res_act=opts.get("res_act", 0))
    torch.cuda.synchronize()
    native.check_status()
    ref = a.double() @ b.double() * opts.get("alpha", 1.0) + (bias.double() if bias is not None else 0.0)
    eps = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    if aux is not None:
        assert float((aux.double() - ref).norm() / ref.norm()) < 1.3 * eps
    ref = _act(ref, act)
    if opts.get("res_act"):
        z = res.double().requires_grad_(True)
        (d,) = torch.autograd.grad(_act(z, 6).sum(), z)
        ref = ref * d
    elif res is not None:
        ref = ref + res.double()
    if opts.get("relu"):
        ref = torch.relu(ref)
    # one rounding of an fp32 result (fp32 output: none); GELU and its derivative through tanh.approx, 2 ** -11
    tol = 2e-6 if opts.get("out32") else 1.3 * eps
    assert float((out.double() - ref).norm() / ref.norm()) < tol + (6e-4 if act == 6 or opts.get("res_act") else 0.0)
