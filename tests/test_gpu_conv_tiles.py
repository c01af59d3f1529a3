"""Per-tap convolution kernel at the sizes where its tile width changes: few pixels (64 columns), a wave of 128-column tiles, many (256),
with channel counts that leave the last tile part empty; forward and data gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,C,O", [(1, 7, 64, 512), (32, 7, 128, 512), (8, 14, 64, 264), (32, 14, 64, 256), (60, 14, 64, 256), (130, 14, 64, 256), (1, 3, 64, 72),
                                     (32, 28, 64, 136)])
def test_forward_and_data_gradient(N, H, C, O):
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(N + H)
    x = torch.randn(N, C, H, H, device="cuda", generator=g).bfloat16().contiguous(memory_format=torch.channels_last).requires_grad_(True)
    w = (torch.randn(O, C, 3, 3, device="cuda", generator=g) * (9 * C) ** -0.5).bfloat16()
    b = torch.randn(O, device="cuda", generator=g)
    dy = torch.randn(N, O, H, H, device="cuda", generator=g).bfloat16().contiguous(memory_format=torch.channels_last)
    y = native.conv2d(x, w, b, (1, 1), (1, 1), path="tap")
    (dx,) = torch.autograd.grad(y, x, dy)
    torch.cuda.synchronize()
    native.check_status()
    xr = x.detach().double().requires_grad_(True)
    yr = torch.nn.functional.conv2d(xr, w.double(), b.double(), padding=1)
    (dxr,) = torch.autograd.grad(yr, xr, dy.double())
    for got, ref in ((y, yr), (dx, dxr)):             # fp32 sums, one rounding to bf16 (2 ** -9)
        assert float((got.double() - ref).norm() / ref.norm()) < 2.5e-3
        assert float((got.double() - ref).abs().max() / ref.abs().max()) < 2 ** -8
