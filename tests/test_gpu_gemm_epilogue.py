"""Epilogue of the tensor-core GEMM: eight warps, 32 columns at a time.  Column counts that end inside a group, inside a 16-byte unit and inside a
tile, rows that end inside a warp's 32, more tiles than SMs, tiles of a pair of CTAs (512); both formats, every combination of operands that
the lean and the full form take, rows of the residual on and off the 16-byte grid."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _act(v, act):
    return torch.relu(v) if act == 1 else v * torch.sigmoid(1.702 * v) if act == 6 else v


@pytest.mark.parametrize("M,N,K,block_n", [(1, 8, 64, 128), (33, 40, 64, 256), (130, 264, 72, 128), (257, 328, 200, 256), (40000, 136, 64, 128), (300, 96, 512, 256),
                                           (1, 8, 64, 512), (130, 264, 72, 512), (257, 328, 1000, 512), (40000, 520, 64, 512)])
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


@pytest.mark.parametrize("M,N,K", [(8, 264, 16000), (304, 520, 9000), (264, 1000, 4608), (1000, 768, 30528)])
def test_long_reductions_on_pairs(M, N, K):
    """Weight gradients (both operands MN-major, parts added into fp32) on CTA pairs, and data gradients whose long reduction is split."""
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + N)
    dz, x = (torch.randn(K, c, device="cuda", generator=g).bfloat16() for c in (M, N))
    ref = dz.double().t() @ x.double()
    for s in (1, 2, 5):
        out = torch.ones(M, N, device="cuda")
        native.gemm_raw(dz.t(), x, out=out, atomic=True, splits=s, pair=True)
        # exact products; the tensor core truncates its fp32 accumulator once per 16 of K: at most 2 ** -23 of it each time
        assert float((out.double() - 1 - ref).norm() / ref.norm()) < K / s / 16 * 2.0 ** -23 + 1e-6
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(N, K, device="cuda", generator=g).bfloat16().t()
    y = native._dgrad_gemm(a, b)
    torch.cuda.synchronize()
    native.check_status()
    ref = a.double() @ b.double()
    assert float((y.double() - ref).norm() / ref.norm()) < 1.3 * 2.0 ** -9         # one rounding
