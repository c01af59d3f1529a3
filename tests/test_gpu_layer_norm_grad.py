"""Layer-norm gradient kernel against fp64 autograd: tile edges, odd widths, misaligned rows, few and many rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.bfloat16, 4e-3), (torch.float16, 5e-4)])
@pytest.mark.parametrize("rows,C", [(1, 1), (3, 8), (5, 17), (9, 256), (700, 264), (2500, 513), (40, 768), (5000, 1024), (33, 1025), (900, 2048),
                                    (17, 2049), (300, 4096), (7, 4104), (5, 8191), (6, 8192), (4, 8200)])
def test_gradient_matches_fp64(rows, C, dtype, tol):
    """dx is rounded once to the data type (half a unit of 2^-8 / 2^-11; fp32: sums of up to 8192 terms); dgain / dbias are fp32 sums."""
    from deeplearning4j_b200.nd.nd4j import Nd4j
    g = torch.Generator(device="cuda").manual_seed(rows * 10007 + C)
    x = (torch.randn(rows, C, generator=g, device="cuda") + 0.5).to(dtype)
    dy = torch.randn(rows, C, generator=g, device="cuda").to(dtype)
    gain, bias = 1 + 0.1 * torch.randn(C, generator=g, device="cuda"), torch.randn(C, generator=g, device="cuda")
    got = [t.t.double() for t in Nd4j.exec("layer_norm_bp", x, gain, bias, dy)]
    x64, g64, b64 = (t.double().requires_grad_(True) for t in (x, gain, bias))
    want = torch.autograd.grad(torch.nn.functional.layer_norm(x64, (C,), g64, b64, 1e-5), (x64, g64, b64), dy.double())
    scale = (dy.double() * gain.double()).norm() * torch.rsqrt(x.double().var(1, unbiased=False) + 1e-5).max()
    assert (got[0] - want[0]).norm() <= tol * scale + 1e-12
    sum_tol = 2e-6 if C <= 8192 else max(tol, 2e-6)               # wider rows: the general path, whose sums come back in x's type
    for a, b in zip(got[1:], want[1:]):
        assert (a - b).norm() <= sum_tol * (b.norm() + dy.double().norm())


def test_misaligned_rows_and_other_axes_take_the_general_path():
    from deeplearning4j_b200.nd.nd4j import Nd4j
    base = torch.randn(64 * 256 + 1, device="cuda").bfloat16()
    x = base[1:].view(64, 256)                                   # two bytes off the 16-byte grid
    dy, gain, bias = torch.randn(64, 256, device="cuda").bfloat16(), torch.rand(256, device="cuda"), torch.rand(256, device="cuda")
    a = Nd4j.exec("layer_norm_bp", x, gain, bias, dy)
    b = Nd4j.exec("layer_norm_bp", x.clone(), gain, bias, dy)
    for u, v in zip(a, b):
        assert torch.allclose(u.t.float(), v.t.float(), rtol=1e-2, atol=1e-3)
    y = torch.randn(6, 10, 5, device="cuda")
    dx, dg, db = Nd4j.exec("layer_norm_bp", y, torch.ones(10, device="cuda"), torch.zeros(10, device="cuda"), torch.randn_like(y),
                           dimensions=[1])
    assert dx.t.shape == y.shape and dg.t.shape == (10,) and db.t.shape == (10,)
    assert len(Nd4j.exec("layer_norm_bp", x, gain, dy)) == 2       # no bias


@pytest.mark.parametrize("rows", [1, 8, 2000])
def test_training_backward_adds_into_the_gradient(rows):
    from deeplearning4j_b200.ops import native
    x = torch.randn(rows, 768, device="cuda").bfloat16().requires_grad_(True)
    g, b = torch.rand(768, device="cuda", requires_grad=True), torch.rand(768, device="cuda", requires_grad=True)
    g.grad, b.grad = torch.ones(768, device="cuda"), torch.full((768,), 2.0, device="cuda")
    dy = torch.randn(rows, 768, device="cuda").bfloat16()
    native.layer_norm(x, g, b, 1e-5).backward(dy)
    x64, g64, b64 = (t.detach().double().requires_grad_(True) for t in (x, g, b))
    want = torch.autograd.grad(torch.nn.functional.layer_norm(x64, (768,), g64, b64, 1e-5), (x64, g64, b64), dy.double())
    assert torch.allclose(g.grad.double(), want[1] + 1, rtol=1e-4, atol=1e-4 * rows ** 0.5)
    assert torch.allclose(b.grad.double(), want[2] + 2, rtol=1e-4, atol=1e-4 * rows ** 0.5)
    assert (x.grad.double() - want[0]).norm() <= 6e-3 * want[0].norm() + 1e-9
