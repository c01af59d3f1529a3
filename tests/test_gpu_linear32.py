"""Small fp32 dense layers on the cluster-split product, against fp64, and the autograd forms they must not break."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(M, K, N, f_order, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, generator=g, device="cuda")
    W = torch.randn(K, N, generator=g, device="cuda") / K ** 0.5
    W = W.t().contiguous().t() if f_order else W
    return x, W, torch.randn(N, generator=g, device="cuda"), torch.randn(M, N, generator=g, device="cuda")


@pytest.mark.parametrize("M,K,N", [(1, 1, 1), (3, 5, 7), (64, 32, 64), (65, 33, 63), (128, 784, 512), (128, 512, 10), (17, 1000, 129),
                                   (200, 300, 777), (1000, 64, 64), (2, 4096, 2)])
@pytest.mark.parametrize("f_order", [False, True])
@pytest.mark.parametrize("act", [None, "relu", "tanh"])
def test_forward_and_gradients(M, K, N, f_order, act):
    """fp32 sums of at most 4096 terms: a few units of 2^-24 times the square root of the count."""
    from deeplearning4j_b200.nn.activations import ActivationReLU, ActivationTanH
    from deeplearning4j_b200.ops import native, nnops
    x, W, b, dy = _case(M, K, N, f_order, M + K + N)
    leaves = [t.detach().requires_grad_(True) for t in (x, W, b)]
    before = native.LAUNCHES
    y = nnops.linear(*leaves, {None: None, "relu": ActivationReLU(), "tanh": ActivationTanH()}[act])
    assert (native.LAUNCHES > before) == native._sgemm_wins(M, N, K, act == "relu", True)
    got = torch.autograd.grad(y, leaves, dy)
    ref_leaves = [t.detach().double().requires_grad_(True) for t in (x, W, b)]
    z = ref_leaves[0] @ ref_leaves[1] + ref_leaves[2]
    ref = {None: lambda v: v, "relu": torch.relu, "tanh": torch.tanh}[act](z)
    want = torch.autograd.grad(ref, ref_leaves, dy.double())
    assert (y.double() - ref).norm() <= 2e-6 * (z.norm() + ref.norm())
    size = dy.double().norm()
    for u, v, p in zip(got, want, leaves):
        assert u.shape == p.shape and (u.double() - v).norm() <= 3e-6 * (v.norm() + size)
    # the parameter's own gradient is added to
    for t in leaves:
        t.grad = torch.ones_like(t)
    nnops.linear(*leaves, ActivationReLU() if act == "relu" else None).backward(dy if act != "tanh" else torch.zeros_like(dy))
    if act != "tanh":
        for t, v in zip(leaves, want):
            assert (t.grad.double() - 1 - v).norm() <= 3e-6 * (v.norm() + size + t.numel() ** 0.5)


@pytest.mark.parametrize("M,N", [(1, 8), (2, 4096), (15, 64), (16, 64), (63, 512), (64, 64), (64, 4096), (64, 4160)])
@pytest.mark.parametrize("K", [255, 256, 257, 1024, 1025, 4096, 4097])
def test_both_sides_of_the_rule(M, N, K):
    """The edges in rows, units and length of the sum, with the kernel itself at each of them."""
    from deeplearning4j_b200.nn.activations import ActivationReLU
    from deeplearning4j_b200.ops import native, nnops
    x, W, b, dy = _case(M, K, N, True, M + K + N)
    for grad in (True, False):
        before = native.LAUNCHES
        y = nnops.linear(x, W.detach().requires_grad_(grad), b, ActivationReLU()).detach()
        assert (native.LAUNCHES > before) == (M * N <= 64 * 4096 and K <= (256 if M < 16 and not grad else 1024 if M < 64 else 4096))
    want = torch.relu(x.double() @ W.double() + b.double())
    direct = native._sgemm(x, W, torch.empty(M, N, device="cuda"), bias=b, act=1)
    for u in (y, direct):
        assert (u.double() - want).norm() <= 2e-6 * (want.norm() + x.double().norm() * W.double().norm() / K ** 0.5)
    dx = native._sgemm(dy, W.t(), torch.empty(M, K, device="cuda"))
    want = dy.double() @ W.double().t()
    assert (dx.double() - want).norm() <= 2e-6 * want.norm()


def test_hooks_create_graph_and_transforms():
    from deeplearning4j_b200.nn.activations import ActivationReLU
    from deeplearning4j_b200.ops import nnops
    x, W, b, dy = _case(64, 300, 16, False, 3)
    Wl = W.detach().requires_grad_(True)
    Wl.grad = torch.zeros_like(W)
    seen = []
    Wl.register_hook(lambda g: seen.append(g.clone()))
    nnops.linear(x, Wl, b, None).backward(dy)
    assert len(seen) == 1 and torch.allclose(Wl.grad, x.t() @ dy, atol=1e-5)
    # second derivatives
    xl = x.detach().requires_grad_(True)
    gx = torch.autograd.grad((nnops.linear(xl, W, b, ActivationReLU()) ** 2).sum(), xl, create_graph=True)[0]
    ggx = torch.autograd.grad(gx.sum(), xl)[0]
    x2 = x.detach().double().requires_grad_(True)
    g2 = torch.autograd.grad((torch.relu(x2 @ W.double() + b.double()) ** 2).sum(), x2, create_graph=True)[0]
    assert torch.allclose(ggx.double(), torch.autograd.grad(g2.sum(), x2)[0], rtol=1e-4, atol=1e-4)
    # transforms and forward mode go through torch operators
    v = torch.func.vmap(lambda r: nnops.linear(r[None], W, b, None)[0])(x)
    assert torch.allclose(v, x @ W + b, atol=1e-5)
    with torch.autograd.forward_ad.dual_level():
        d = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
        t = torch.autograd.forward_ad.unpack_dual(nnops.linear(d, W, b, None)).tangent
    assert torch.allclose(t, torch.ones_like(x) @ W, atol=1e-5)


@pytest.mark.parametrize("M,K,N", [(64, 8, 8), (70, 40, 24), (64, 8, 5)])
def test_nan_and_inf_pass(M, K, N):
    """Values and gradients have NaN and infinities of either sign where the library's operators have them."""
    from deeplearning4j_b200.nn.activations import ActivationReLU
    from deeplearning4j_b200.ops import native, nnops
    x, W, b, dy = _case(M, K, N, True, 1)
    x[0, 0] = float("nan")
    x[1, 0], x[2, 0] = float("inf"), float("-inf")
    dy[3, 1], dy[4, 2], dy[5, 3] = float("inf"), float("-inf"), float("nan")
    dy[0, 4] = float("inf")

    def same(u, v):
        assert torch.equal(torch.isnan(u), torch.isnan(v)) and torch.equal(torch.isposinf(u), torch.isposinf(v)) \
            and torch.equal(torch.isneginf(u), torch.isneginf(v))
        fin = torch.isfinite(v)
        assert torch.allclose(u[fin], v[fin], rtol=1e-4, atol=1e-4)
    for create in (False, True):
        leaves = [t.detach().requires_grad_(True) for t in (x, W, b)]
        before = native.LAUNCHES
        y = nnops.linear(*leaves, ActivationReLU())
        assert native.LAUNCHES > before
        ref = [t.detach().requires_grad_(True) for t in (x, W, b)]
        z = torch.relu(ref[0] @ ref[1] + ref[2])
        same(y.detach(), z.detach())
        for u, v in zip(torch.autograd.grad(y, leaves, dy, create_graph=create), torch.autograd.grad(z, ref, dy)):
            same(u.detach(), v)


@pytest.mark.parametrize("M,K,N", [(1, 8, 8), (31, 5, 24), (128, 784, 512), (128, 512, 10), (257, 64, 63), (4096, 16, 64), (1000, 33, 200)])
@pytest.mark.parametrize("relu", [True, False])
def test_gradients_repeat_bit_for_bit(M, K, N, relu):
    """Every sum of an fp32 layer has one order; the bias gradient is exact to a few units of the column's absolute sum."""
    from deeplearning4j_b200.nn.activations import ActivationReLU
    from deeplearning4j_b200.ops import native, nnops
    x, W, b, dy = _case(M, K, N, True, M + N)
    leaves = [t.detach().requires_grad_(True) for t in (x, W, b)]

    def run():
        before = native.LAUNCHES
        y = nnops.linear(*leaves, ActivationReLU() if relu else None)
        g = torch.autograd.grad(y, leaves, dy)
        assert native.LAUNCHES > before or not native._sgemm_wins(M, N, K, relu, True)
        return (y.detach(), *g)
    first = run()
    for _ in range(10):
        assert all(torch.equal(a, c) for a, c in zip(first, run()))
    dz = dy.double() * (first[0] > 0) if relu else dy.double()
    assert ((first[3].double() - dz.sum(0)).abs() <= 1e-6 * dz.abs().sum(0) + 1e-30).all()


@pytest.mark.parametrize("M,K,N", [(16, 24, 32), (5, 7, 3)])
def test_autograd_grad_with_preallocated_gradients(M, K, N):
    """``.grad`` belongs to the caller: only a trainer's own backward pass is added to behind autograd's back."""
    from deeplearning4j_b200.nn.activations import ActivationReLU
    from deeplearning4j_b200.ops import native, nnops
    x, W, b, dy = _case(M, K, N, True, 9)
    x, W, b = (t.detach().requires_grad_(True) for t in (x, W, b))
    W.grad, b.grad = torch.full_like(W, 7.0), torch.full_like(b, 7.0)
    ref = torch.autograd.grad(torch.relu(x.double() @ W.double() + b.double()), (x, W, b), dy.double())
    call = lambda: nnops.linear(x, W, b, ActivationReLU())
    for got, want in zip(torch.autograd.grad(call(), (x, W, b), dy), ref):
        assert torch.allclose(got.double(), want.double(), rtol=1e-4, atol=1e-4)
    assert torch.allclose(torch.autograd.grad(call(), x, dy)[0].double(), ref[0].double(), rtol=1e-4, atol=1e-4)
    with native.TrainingStep() as step:
        y = call()
        inner = torch.autograd.grad(y, (W, b), dy, retain_graph=True)         # a layer's own gradient inside the forward pass
        assert torch.allclose(inner[0].double(), ref[1].double(), rtol=1e-4, atol=1e-4)
        assert (W.grad == 7).all() and (b.grad == 7).all()
        step.backward((y * dy).sum())
    for p, want in ((W, ref[1]), (b, ref[2])):
        assert torch.allclose(p.grad.double(), want.double() + 7, rtol=1e-4, atol=1e-4)
    got = torch.autograd.grad(call(), (W, b), dy)
    assert torch.allclose(got[0].double(), ref[1].double(), rtol=1e-4, atol=1e-4)


def test_a_network_trains_into_its_flat_gradient(monkeypatch):
    """fit and computeGradientAndScore keep adding in place: autograd is handed no gradient for the dense parameters."""
    from deeplearning4j_b200 import nn
    from deeplearning4j_b200.nn.layers.core import DenseLayer, OutputLayer
    from deeplearning4j_b200.ops import native
    net = nn.MultiLayerNetwork(nn.NeuralNetConfiguration.Builder().seed(1).updater(nn.Sgd(0.1)).list().layer(DenseLayer(nIn=8, nOut=16, activation="RELU"))
                               .layer(OutputLayer("MCXENT", nIn=16, nOut=4, activation="SOFTMAX")).build())
    net.device = torch.device("cuda")
    net.init()
    seen, backward = [], native._Linear32Fn.backward
    monkeypatch.setattr(native._Linear32Fn, "backward", staticmethod(lambda ctx, dy: seen.append(backward(ctx, dy)) or seen[-1]))
    x, y = torch.randn(32, 8, device="cuda"), torch.eye(4, device="cuda")[torch.arange(32, device="cuda") % 4]
    net.computeGradientAndScore(x, y)
    assert len(seen) == 2 and all(g[1] is None and g[2] is None for g in seen)
