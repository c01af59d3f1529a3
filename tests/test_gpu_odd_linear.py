"""Dense layers of widths off the 8-element grid and long-reduction data gradients, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,wdtype", [(torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16)])
@pytest.mark.parametrize("M,K,N", [(256, 77, 10), (257, 64, 1), (300, 1, 9), (512, 768, 1001), (1000, 131, 264), (256, 13, 30522)])
@pytest.mark.parametrize("f_order", [False, True])
@pytest.mark.parametrize("act", [None, "relu", "gelu"])
def test_forward_and_gradients(M, K, N, dtype, wdtype, f_order, act):
    """Operands are exact in the compute type; one rounding of the result (and of dz where there is an activation)."""
    from deeplearning4j_b200.nn.activations import ActivationGELU, ActivationReLU
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype).requires_grad_(True)
    W = (torch.randn(K, N, generator=g, device="cuda") / K ** 0.5).to(dtype).to(wdtype)
    W = (W.t().contiguous().t() if f_order else W).requires_grad_(True)
    b = torch.randn(N, generator=g, device="cuda").to(wdtype).requires_grad_(True)
    dy = torch.randn(M, N, generator=g, device="cuda").to(dtype)
    a = {None: None, "relu": ActivationReLU(), "gelu": ActivationGELU(True)}[act]
    y = native.linear(x, W, b, a)
    assert y is not None and y.shape == (M, N)
    got = torch.autograd.grad(y, (x, W, b), dy)
    native.check_status()
    x64, W64, b64 = (t.detach().double().requires_grad_(True) for t in (x, W, b))
    z = x64 @ W64 + b64
    ref = {None: lambda v: v, "relu": torch.relu, "gelu": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act](z)
    want = torch.autograd.grad(ref, (x64, W64, b64), dy.double())
    tol = 6e-3 if dtype == torch.bfloat16 else 1e-3
    assert (y.double() - ref).norm() <= tol * ref.norm()
    for u, v, p in zip(got, want, (x, W, b)):
        assert u.shape == p.shape and u.dtype == p.dtype
        assert (u.double() - v).norm() <= 2 * tol * v.norm() + 1e-6 * dy.double().norm()


def test_gradient_of_a_view_without_its_padding():
    """An upstream gradient whose last row ends at the end of its storage must not be read past it."""
    from deeplearning4j_b200.ops import native
    x = torch.randn(256, 16, device="cuda").bfloat16().requires_grad_(True)
    W = torch.randn(16, 13, device="cuda").bfloat16().requires_grad_(True)
    y = native.linear(x, W, None, None)
    store = torch.randn(255 * 16 + 13, device="cuda").bfloat16()
    dy = store.as_strided((256, 13), (16, 1))
    dx, dW = torch.autograd.grad(y, (x, W), dy)
    assert (dx.double() - dy.double() @ W.double().t()).norm() <= 6e-3 * dx.double().norm()
    assert (dW.double() - x.double().t() @ dy.double()).norm() <= 6e-3 * dW.double().norm()


@pytest.mark.parametrize("M,N,K", [(2456, 768, 30522), (100, 256, 4096), (128, 12, 2048), (300, 264, 5000), (2456, 770, 9000)])
def test_long_reduction_splits_keep_the_precision(M, N, K):
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(K)
    a = torch.randn(M, (K + 7) // 8 * 8, generator=g, device="cuda").bfloat16()[:, :K]
    b = torch.randn(N, (K + 7) // 8 * 8, generator=g, device="cuda").bfloat16()[:, :K].t()
    got = native._dgrad_gemm(a, b, out=None if N % 8 == 0 else native._pitched(M, N, torch.bfloat16, a.device))
    plain = native.gemm_raw(a, b, out=native._pitched(M, N, torch.bfloat16, a.device))
    want = a.double() @ b.double()
    assert (got.double() - want).norm() <= 1.05 * (plain.double() - want).norm()


@pytest.mark.parametrize("C", [8, 2048, 8191, 8192, 8200, 30522])
@pytest.mark.parametrize("sparse", [True, False])
def test_cross_entropy_rows_with_infinities(C, sparse):
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(C)
    base = torch.randn(9, (C + 7) // 8 * 8, generator=g, device="cuda").bfloat16() * 4
    z = base[:, :C].detach()
    z[1, 1:] = float("-inf")
    z[2, : C // 2] = float("-inf")
    z[3, 0] = float("-inf")
    lab = torch.randint(C // 2, C, (9,), generator=g, device="cuda")
    lab[1] = 0
    dense = torch.nn.functional.one_hot(lab, C).to(z.dtype)
    z.requires_grad_(True)
    if sparse:
        loss = native.softmax_xent(z, lab, True)
        want = torch.nn.functional.cross_entropy(z.double(), lab, reduction="none")
        assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5)
    else:
        z2 = z.detach()[4:].requires_grad_(True)
        loss = native.softmax_xent(z2, dense[4:], False)
        want = torch.nn.functional.cross_entropy(z2.double(), lab[4:], reduction="none")
        assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5)
        z = z2
    grad = torch.autograd.grad(loss.sum(), z)[0]
    p = torch.softmax(z.detach().double(), -1) - torch.nn.functional.one_hot(lab if sparse else lab[4:], C)
    assert (grad.double() - p).abs().max() <= 2 ** -8


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(2456, 768, 30522), (1, 4, 2048), (130, 260, 4100), (300, 264, 2500), (7, 1000, 9001)])
def test_split_reductions_repeat_bit_for_bit(M, N, K, dtype):
    """Partial results are added in order: every call gives the same bits, and splits that get no part of K add zero."""
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(K)
    P = (K + 7) // 8 * 8
    a, b = torch.randn(M, P, generator=g, device="cuda").to(dtype)[:, :K], torch.randn(N, P, generator=g, device="cuda").to(dtype)[:, :K].t()
    want = a.double() @ b.double()
    for s in (2, 7, 16, 30):
        out = native._pitched(M, N, dtype, a.device)
        first = native._split_gemm(a, b, s, out).clone()
        assert (first.double() - want).norm() <= (4e-3 if dtype == torch.bfloat16 else 5e-4) * want.norm()
        for _ in range(4):
            assert torch.equal(native._split_gemm(a, b, s), first)
    x = torch.randn(300, 768, generator=g, device="cuda").to(dtype).requires_grad_(True)
    W = (torch.randn(768, 9001, generator=g, device="cuda") * 0.03).requires_grad_(True)
    dy = torch.randn(300, 9001, generator=g, device="cuda").to(dtype)
    grads = [torch.autograd.grad(native.linear(x, W, None, None), x, dy)[0] for _ in range(5)]
    assert all(torch.equal(grads[0], t) for t in grads)
    native.check_status()


def test_bias_is_the_parameter_not_its_shadow():
    """256.5 is not a bf16 number: what is left after the product's -256 shows the bits of the bias; a change in place is seen at once."""
    from deeplearning4j_b200 import DataType, nn
    from deeplearning4j_b200.nn.layers.core import DenseLayer, OutputLayer
    net = nn.MultiLayerNetwork(nn.NeuralNetConfiguration.Builder().computeDataType(DataType.BFLOAT16).list()
                               .layer(DenseLayer(nIn=8, nOut=10, activation="IDENTITY"))
                               .layer(OutputLayer("MSE", nIn=10, nOut=8, activation="IDENTITY")).build())
    net.device = torch.device("cuda")
    net.init()
    p = net.paramTable()
    p["0_W"].t.fill_(-32.0)
    p["0_b"].t.fill_(256.5)
    p["1_W"].t.zero_()
    p["1_W"].t[0, 0] = 1.0
    p["1_b"].t.zero_()
    x = torch.ones(300, 8, device="cuda")
    net.setParams(net.params().t.clone())                     # the shadows are up to date
    assert (net.output(x).t[:, 0] == 0.5).all()
    net.paramTable()["0_b"].t.fill_(257.25)
    assert (net.output(x).t[:, 0] == 1.25).all()
