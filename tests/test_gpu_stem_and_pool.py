"""Convolutions over a few channels as a product of patches, max pooling, folded batch norm of every kernel size."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,O,k,stride,pad,dil,layout", [
    ((3, 3, 19, 17), 32, (3, 3), (1, 1), (1, 1), (1, 1), "nchw"), ((2, 1, 28, 28), 64, (7, 7), (1, 1), (3, 2), (1, 1), "nchw"),
    ((1, 7, 9, 30), 64, (3, 3), (1, 2), (0, 1), (1, 1), "nhwc"), ((5, 3, 33, 20), 40, (3, 4), (3, 1), (2, 0), (2, 3), "view"),
    ((2, 4, 1, 1), 40, (3, 3), (1, 1), (1, 1), (1, 1), "nchw"), ((130, 3, 12, 12), 264, (2, 2), (1, 1), (0, 0), (1, 1), "expand")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_few_channels_match_fp64(shape, O, k, stride, pad, dil, layout, dtype):
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    if layout == "view":                                  # odd strides, off the 16-byte grid
        x = torch.randn(shape[0], shape[1], shape[2] + 1, shape[3] + 3, device="cuda", generator=g).to(dtype)[:, :, 1:, 3:]
    elif layout == "expand":
        x = torch.randn(1, *shape[1:], device="cuda", generator=g).to(dtype).expand(shape)
    else:
        x = torch.randn(shape, device="cuda", generator=g).to(dtype)
        x = x.contiguous(memory_format=torch.channels_last) if layout == "nhwc" else x
    W = (torch.randn(O, shape[1], *k, device="cuda", generator=g) * (shape[1] * k[0] * k[1]) ** -0.5).requires_grad_(True)
    b = torch.randn(O, device="cuda", generator=g).requires_grad_(True)
    y = native.conv_few_channels(x, W, b, stride, pad, dil)
    assert y is not None and y.dtype == dtype
    dy = torch.randn(y.shape, device="cuda", generator=g).to(dtype)
    dW, db = torch.autograd.grad(y, (W, b), dy)
    torch.cuda.synchronize()
    native.check_status()
    Wr, br = W.detach().to(dtype).double().requires_grad_(True), b.detach().double().requires_grad_(True)
    yr = F.conv2d(x.double(), Wr, br, stride, pad, dil)
    dWr, dbr = torch.autograd.grad(yr, (Wr, br), dy.double())
    eps = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert float((y.double() - yr).norm() / yr.norm()) < 1.3 * eps          # one rounding of an fp32 sum
    assert float((dW.double() - dWr).norm() / dWr.norm()) < 1e-5            # fp32 gradients
    assert float((db.double() - dbr).norm() / dbr.norm()) < 1e-5


def test_few_channels_leaves_the_rest_to_others():
    from deeplearning4j_b200.ops import native
    x = torch.randn(2, 3, 8, 8, device="cuda").bfloat16()
    W = torch.randn(32, 3, 3, 3, device="cuda")
    one = (1, 1)
    assert native.conv_few_channels(x.clone().requires_grad_(True), W, None, one, one, one) is None          # gradient into the image
    assert native.conv_few_channels(x, torch.randn(36, 3, 3, 3, device="cuda"), None, one, one, one) is None  # channels off the 8 grid
    assert native.conv_few_channels(x, torch.randn(64, 3, 5, 5, device="cuda"), None, one, one, one) is None  # 75 values per patch
    assert native.conv_few_channels(x, torch.randn(24, 3, 3, 3, device="cuda"), None, one, one, one) is None  # patches larger than the output
    assert native.conv_few_channels(x.float(), W, None, one, one, one) is None
    assert native.conv_few_channels(x, torch.randn(32, 4, 3, 3, device="cuda"), None, one, one, one) is None


@pytest.mark.parametrize("k,s,p", [((3, 3), (2, 2), (0, 0)), ((3, 3), (1, 2), (1, 1)), ((2, 2), (2, 2), (0, 0)), ((2, 2), (1, 1), (1, 0)), ((3, 2), (2, 1), (1, 1))])
def test_max_pool_values_and_gradient(k, s, p):
    from deeplearning4j_b200.ops import native
    x = torch.randint(-4, 5, (3, 24, 13, 10), device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)      # ties: the first window position wins
    x[0, 3, 4, 4] = float("-inf")
    x.requires_grad_(True)
    y = native._MaxPoolFn.apply(x, k, s, p)
    dy = torch.randn(y.shape, device="cuda").bfloat16()
    (dx,) = torch.autograd.grad(y, x, dy)
    xr = x.detach().double().requires_grad_(True)
    yr = F.max_pool2d(xr, k, s, p)
    (dxr,) = torch.autograd.grad(yr, xr, dy.double())
    assert torch.equal(y.double(), yr)
    assert float((dx.double() - dxr).abs().max()) <= 2.0 ** -8 * float(dxr.abs().max())


@pytest.mark.parametrize("O,I,k", [(5, 8, 1), (9, 7, 1), (3, 130, 3), (6, 129, 3), (2, 64, 7), (2, 3, 34), (1, 2048, 1), (4, 300, 2)])
def test_fold_matches_fp64(O, I, k):
    """Odd and even channel counts, several staging rounds, and kernels of more taps than a round holds."""
    import ctypes
    import struct
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(O + I)
    S = k * k
    w = torch.randn(O, I, S, device="cuda", generator=g)
    vec = [torch.randn(O, device="cuda", generator=g) for _ in range(4)]
    var = torch.rand(O, device="cuda", generator=g) + 0.1
    params = torch.cat([w.reshape(-1)] + vec + [var])
    n = w.numel()
    entry = struct.pack("<8q4i3fi", n * 0, n, n + O, n + 2 * O, n + 3 * O, n + 4 * O, 0, 0, O, I, S, 0, 1e-5, 1.0, 0.0, 0)
    table = torch.frombuffer(bytearray(entry), dtype=torch.uint8).cuda()
    blocks = torch.zeros(O, dtype=torch.int32, device="cuda")
    wo, bo = torch.full((O, S, I), 9.0, device="cuda").bfloat16(), torch.empty(O, device="cuda")
    native.bn_fold(table, blocks, params, wo, bo)
    torch.cuda.synchronize()
    b, gamma, beta, mean = (t.double() for t in vec)
    s = gamma / (var.double() + 1e-5).sqrt()
    ref = w.double().permute(0, 2, 1) * s[:, None, None]
    assert float(((wo.double() - ref).abs() / ref.abs().clamp_min(1e-3)).max()) < 2 ** -8
    rb = (b - mean) * s + beta
    assert float((bo.double() - rb).abs().max()) < 2e-5 * float(rb.abs().max() + 1)
