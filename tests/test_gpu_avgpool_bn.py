"""Global average pooling on channels-last activations, and batch norm at row counts off the unrolled tiles, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -11)])
@pytest.mark.parametrize("N,C,H,W", [(1, 8, 1, 1), (3, 72, 5, 7), (2, 64, 32, 4), (5, 256, 19, 19), (2, 2048, 7, 7)])
def test_global_average_pooling(N, C, H, W, dtype, tol):
    from deeplearning4j_b200.nn.conf.base import PoolingType
    from deeplearning4j_b200.nn.layers.conv import GlobalPoolingLayer
    from deeplearning4j_b200.ops import native
    x = torch.randn(N, C, H, W, device="cuda").to(dtype).contiguous(memory_format=torch.channels_last).requires_grad_(True)
    before = native.LAUNCHES
    y = GlobalPoolingLayer(PoolingType.AVG).forward({}, x, True)
    dy = torch.randn(N, C, device="cuda").to(dtype)
    dx, = torch.autograd.grad(y, x, dy)
    assert native.LAUNCHES - before == 2 and dx.is_contiguous(memory_format=torch.channels_last)
    want = x.detach().double().mean((2, 3))
    assert ((y.double() - want).abs() <= tol * want.abs() + 1e-6).all()          # one rounding
    assert ((dx.double() - (dy.double() / (H * W))[:, :, None, None]).abs() <= tol * dy.double().abs()[:, :, None, None] / (H * W) + 1e-7).all()
    z = GlobalPoolingLayer(PoolingType.AVG).forward({}, x.detach().contiguous(), True)          # NCHW: the general path
    assert torch.allclose(z.float(), y.float(), rtol=2 * tol, atol=1e-5)


@pytest.mark.parametrize("rows,C", [(1, 8), (5, 2048), (127, 64), (148 * 4 * 32 + 1, 256), (9999, 16)])
@pytest.mark.parametrize("relu,with_res", [(False, False), (True, False), (True, True), (False, True)])
def test_batch_norm_rows(rows, C, relu, with_res):
    """2-D activations [rows, C]; a large mean makes the statistics' cancellation visible."""
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(rows + C)
    x = (torch.randn(rows, C, generator=g, device="cuda") + 2.0).bfloat16().requires_grad_(True)
    res = torch.randn(rows, C, generator=g, device="cuda").bfloat16().requires_grad_(True) if with_res else None
    gamma, beta = (1 + 0.2 * torch.randn(C, generator=g, device="cuda")).requires_grad_(True), torch.randn(C, generator=g, device="cuda").requires_grad_(True)
    dy = torch.randn(rows, C, generator=g, device="cuda").bfloat16()
    y = native.bn_act_train(x, res, gamma, beta, torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda"), True, 0.9, 1e-3, relu)
    leaves = [t for t in (x, gamma, beta, res) if t is not None]
    got = torch.autograd.grad(y, leaves, dy)
    l64 = [t.detach().double().requires_grad_(True) for t in leaves]
    m, v = l64[0].mean(0), l64[0].var(0, unbiased=False)
    z = (l64[0] - m) * torch.rsqrt(v + 1e-3) * l64[1] + l64[2] + (l64[3] if with_res else 0)
    keep = (y.detach() > 0).double() if relu else torch.ones_like(z)              # the kernel's own mask: ties at zero are rounding
    want = torch.autograd.grad(z * keep, l64, dy.double())
    assert (y.double() - torch.relu(z) if relu else y.double() - z).norm() <= 6e-3 * z.norm()
    for a, b in zip(got, want):
        assert (a.double() - b).norm() <= 6e-3 * b.norm() + 2e-3 * dy.double().norm() * (1 if rows < 10 else 0.1)
