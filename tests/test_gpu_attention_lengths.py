"""Fused attention at lengths and head sizes off the tile grid, causal and masked, against fp64; routes against the general path."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B, H, Tq, Tk, D, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = lambda T: torch.randn(B, T, H, D, generator=g, device="cuda").bfloat16().permute(0, 2, 1, 3)
    return t(Tq), t(Tk), t(Tk), t(Tq), g


def _ref(q, k, v, scale, mask, causal):
    s = q @ k.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    if mask is not None:
        s = s.masked_fill(mask[:, None, None, :] == 0, float("-inf"))
    return torch.softmax(s, -1) @ v


@pytest.mark.parametrize("Tq,Tk", [(1, 1), (7, 5), (16, 127), (128, 128), (129, 129), (200, 200), (256, 255), (257, 384), (500, 130), (1000, 1000)])
@pytest.mark.parametrize("D", [8, 32, 40, 64])
@pytest.mark.parametrize("masked,causal", [(False, False), (True, False), (False, True), (True, True)])
def test_forward_and_gradients(Tq, Tk, D, masked, causal):
    """bf16 rounds P, dS and the results once each (2^-9 relative): 1e-2 of the norm leaves a factor of two."""
    from deeplearning4j_b200.nd.nd4j import Nd4j
    from deeplearning4j_b200.ops import native
    B, H = 2, 3
    q, k, v, do, g = _inputs(B, H, Tq, Tk, D, Tq * 1000 + Tk + D)
    mask = None
    if masked:
        mask = (torch.rand(B, Tk, generator=g, device="cuda") > 0.3).float()
        mask[:, 0] = 1.0
    scale = D ** -0.5
    q64, k64, v64 = (t.double().requires_grad_(True) for t in (q, k, v))
    want = _ref(q64, k64, v64, scale, mask, causal)
    dq, dk, dv = torch.autograd.grad(want, (q64, k64, v64), do.double())
    got = Nd4j.exec("dot_product_attention_v2", q, v, k, None, None, mask, scale=scale, useCausalMask=causal).t
    gq, gv, gk = (a.t for a in Nd4j.exec("dot_product_attention_v2_bp", q, v, k, do, vMask=mask, scale=scale, useCausalMask=causal))
    # ... and through autograd
    ql, kl, vl = (t.detach().requires_grad_(True) for t in (q, k, v))
    from deeplearning4j_b200.ops import attention_native as an
    aq, ak, av = torch.autograd.grad(an.attention(ql, kl, vl, mask, scale, causal=causal), (ql, kl, vl), do)
    torch.cuda.synchronize()
    native.check_status()
    assert (got.double() - want).norm() <= 1e-2 * want.norm()
    # with one visible key P is exactly 1 and dq, dk vanish: compare against the size of the terms that cancel
    size = do.double().norm() * scale
    for a, b in ((gq, dq), (gk, dk), (aq, dq), (ak, dk)):
        assert (a.double() - b).norm() <= 1e-2 * (b.norm() + size)
    for a, b in ((gv, dv), (av, dv)):
        assert (a.double() - b).norm() <= 1e-2 * b.norm()


@pytest.mark.parametrize("T,causal,zero", [(256, False, True), (200, False, True), (201, False, False), (130, True, False)])
def test_rows_without_keys(T, causal, zero):
    """Zero where the native kernels always served the length, NaN where the softmax over -inf did."""
    from deeplearning4j_b200.nd.nd4j import Nd4j
    q, k, v, do, _ = _inputs(2, 2, T, T, 64, T)
    mask = torch.ones(2, T, device="cuda")
    if causal:
        mask[1, :3] = 0                                     # the first three queries of example 1 see nothing
    else:
        mask[1] = 0
    out = Nd4j.exec("dot_product_attention_v2", q, v, k, None, None, mask, scale=0.125, useCausalMask=causal).t
    dq, dv, dk = (a.t for a in Nd4j.exec("dot_product_attention_v2_bp", q, v, k, do, vMask=mask, scale=0.125, useCausalMask=causal))
    bad = out[1, :, :3] if causal else out[1]
    assert torch.isfinite(out[0]).all() and torch.isfinite(dv[0]).all()
    if zero:
        assert (bad == 0).all() and (dv[1] == 0).all()
    else:
        assert torch.isnan(bad).all() and torch.isnan(dv[1]).all()
    assert (dq[1, :, :3] == 0).all() and torch.isfinite(dk).all()


def test_three_dimensional_and_misaligned_inputs():
    from deeplearning4j_b200.nd.nd4j import Nd4j
    base = torch.randn(3 * 50 * 24 + 3, device="cuda").bfloat16()
    q = base[3:].view(3, 50, 24)                            # off the 16-byte grid
    k, v = torch.randn(3, 33, 24, device="cuda").bfloat16(), torch.randn(3, 33, 24, device="cuda").bfloat16()
    out = Nd4j.exec("dot_product_attention_v2", q, v, k, scale=0.2).t
    want = _ref(q.double()[:, None], k.double()[:, None], v.double()[:, None], 0.2, None, False)[:, 0]
    assert out.shape == (3, 50, 24) and (out.double() - want).norm() <= 1e-2 * want.norm()
    dq, dv, dk = Nd4j.exec("dot_product_attention_v2_bp", q, v, k, torch.ones_like(q), scale=0.2)
    assert dq.t.shape == q.shape and dk.t.shape == k.shape and dv.t.shape == v.shape


@pytest.mark.parametrize("T,masked,causal", [(201, True, False), (100, False, True), (1032, False, False), (104, False, False), (256, True, True)])
def test_second_derivatives_forward_mode_and_vmap(T, masked, causal):
    """What the calls gave through torch operators: a gradient penalty, a tangent, a mapped call."""
    from deeplearning4j_b200.nd.nd4j import Nd4j
    B, H, D, scale = 2, 2, 64, 0.125
    q, k, v, do, g = _inputs(B, H, T, T, D, T)
    mask = None
    if masked:
        mask = (torch.rand(B, T, generator=g, device="cuda") > 0.3).float()
        mask[:, 0] = 1.0

    def call(a, b, c):
        from deeplearning4j_b200.ops.impl_nn import dot_product_attention_v2
        return dot_product_attention_v2(a, c, b, vMask=mask, scale=scale, useCausalMask=causal)[0]
    # second derivatives, of views that the kernels copy as well
    for lay in (lambda t: t, lambda t: t.transpose(-1, -2).contiguous().transpose(-1, -2)):
        ql, kl, vl = (lay(t.detach()).requires_grad_(True) for t in (q, k, v))
        gq = torch.autograd.grad(call(ql, kl, vl), ql, do, create_graph=True)[0]
        second = torch.autograd.grad((gq.float() ** 2).sum(), (ql, kl, vl))
        q6, k6, v6 = (t.detach().double().requires_grad_(True) for t in (q, k, v))
        gq6 = torch.autograd.grad(_ref(q6, k6, v6, scale, mask, causal), q6, do.double(), create_graph=True)[0]
        want = torch.autograd.grad((gq6 ** 2).sum(), (q6, k6, v6))
        assert (gq.double() - gq6).norm() <= 1e-2 * gq6.norm()
        for a, b in zip(second, want):
            assert (a.double() - b).norm() <= 4e-2 * b.norm()
    with torch.autograd.forward_ad.dual_level():
        d = torch.autograd.forward_ad.make_dual(q, do)
        t = torch.autograd.forward_ad.unpack_dual(call(d, k, v)).tangent
    q6 = q.double()
    want = torch.func.jvp(lambda a: _ref(a, k.double(), v.double(), scale, mask, causal), (q6,), (do.double(),))[1]
    assert t is not None and (t.double() - want).norm() <= 3e-2 * want.norm()
    if mask is None:
        got = torch.func.vmap(lambda a: call(a, k, v))(torch.stack([q, q.flip(0)]))
        assert (got[0].double() - _ref(q6, k.double(), v.double(), scale, None, causal)).norm() <= 1e-2 * got[0].double().norm()


@pytest.mark.parametrize("T,causal", [(201, False), (64, False), (256, False), (130, True), (1032, False)])
@pytest.mark.parametrize("scale", [-0.125, -8.0])
def test_negative_scale(T, causal, scale):
    """Scores are scaled before the row maximum is taken: large ones of the other sign do not overflow."""
    from deeplearning4j_b200.nd.nd4j import Nd4j
    q, k, v, do, _ = _inputs(2, 2, T, T, 64, T)
    q = q * 4
    q6, k6, v6 = (t.double().requires_grad_(True) for t in (q, k, v))
    want = _ref(q6, k6, v6, scale, None, causal)
    grads = torch.autograd.grad(want, (q6, k6, v6), do.double())
    out = Nd4j.exec("dot_product_attention_v2", q, v, k, scale=scale, useCausalMask=causal).t
    dq, dv, dk = (a.t for a in Nd4j.exec("dot_product_attention_v2_bp", q, v, k, do, scale=scale, useCausalMask=causal))
    # the operator path rounds the scores to bf16, 2^-9 of them, and that error goes into the exponent: scores to 16 and to 1000
    tol = 4e-2 if abs(scale) < 1 else 0.5
    assert torch.isfinite(out).all() and (out.double() - want).norm() <= tol * want.norm()
    for a, b in zip((dq, dk, dv), grads):
        assert torch.isfinite(a).all() and (a.double() - b).norm() <= 3 * tol * (b.norm() + abs(scale) * do.double().norm())


@pytest.mark.parametrize("kshape,vshape", [((1, 2, 64, 64), (1, 2, 64, 64)), ((2, 1, 64, 64), (2, 1, 64, 64)), ((2, 2, 64, 64), (2, 2, 64, 32))])
def test_operands_that_broadcast(kshape, vshape):
    from deeplearning4j_b200.nd.nd4j import Nd4j
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((2, 2, 64, 64), kshape, vshape))
    out = Nd4j.exec("dot_product_attention_v2", q, v, k, scale=0.1).t
    want = _ref(q.double(), k.double(), v.double(), 0.1, None, False)
    assert out.shape == want.shape and (out.double() - want).norm() <= 1e-2 * want.norm()


@pytest.mark.parametrize("T,causal", [(201, False), (100, True), (130, True), (1032, False)])
@pytest.mark.parametrize("where", ["q", "k"])
def test_nan_reaches_the_gradients(T, causal, where):
    """A NaN query makes its own row and dk, dv NaN; a NaN key makes every row that sees it NaN: as the operators have it (which under a
    causal mask spread it to keys that the row does not see as well)."""
    from deeplearning4j_b200.nd.nd4j import Nd4j
    q, k, v, do, _ = _inputs(2, 2, T, T, 64, T)
    bad = q if where == "q" else k
    bad[1, 0, 3, 5] = float("nan")
    q6, k6, v6 = (t.double().requires_grad_(True) for t in (q, k, v))
    want = _ref(q6, k6, v6, 0.125, None, causal)
    grads = torch.autograd.grad(want, (q6, k6, v6), do.double())
    out = Nd4j.exec("dot_product_attention_v2", q, v, k, scale=0.125, useCausalMask=causal).t
    dq, dv, dk = (a.t for a in Nd4j.exec("dot_product_attention_v2_bp", q, v, k, do, scale=0.125, useCausalMask=causal))
    for a, b in zip((out, dq, dk, dv), (want, *grads)):
        assert torch.equal(torch.isnan(a).any(-1).any(-1), torch.isnan(b).any(-1).any(-1))       # the same heads
        if not causal or a is out:
            assert (torch.isnan(a) >= torch.isnan(b)).all()                                      # nothing hidden


@pytest.mark.parametrize("Tq,Tk,causal", [(400, 400, False), (1000, 1000, False), (512, 512, True), (300, 700, True), (700, 300, True), (129, 1032, False)])
@pytest.mark.parametrize("D,masked", [(64, False), (40, True)])
def test_gradients_repeat_bit_for_bit(Tq, Tk, causal, D, masked):
    """The parts of dq from several key blocks are added in one order (a key mask that hides key 0 visits every causal block)."""
    from deeplearning4j_b200.nd.nd4j import Nd4j
    q, k, v, do, g = _inputs(2, 3, Tq, Tk, D, Tq + Tk)
    mask = None
    if masked:
        mask = (torch.rand(2, Tk, generator=g, device="cuda") > 0.3).float()
        mask[0, 0], mask[1, 0] = 0.0, 1.0

    def run():
        return [a.t for a in Nd4j.exec("dot_product_attention_v2_bp", q, v, k, do, vMask=mask, scale=0.125, useCausalMask=causal)]
    first = run()
    torch.empty(2 * 9 * 3 * 1100 * 64, device="cuda").fill_(float("nan"))          # what the next buffers are made of
    for _ in range(8):
        assert all(torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0)) for a, b in zip(first, run()))
    q6, k6, v6 = (t.double().requires_grad_(True) for t in (q, k, v))
    want = torch.autograd.grad(_ref(q6, k6, v6, 0.125, mask, causal), (q6, k6, v6), do.double())
    size = do.double().norm() * 0.125
    ok = slice(1, 2) if masked and causal else slice(None)                          # example 0 has rows without keys there
    for a, b in zip((first[0], first[2]), want[:2]):
        assert (a.double() - b)[ok].norm() <= 1e-2 * (b[ok].norm() + size)


@pytest.mark.parametrize("Tq,Tk", [(1, 1), (1, 37), (33, 33), (128, 128)])
def test_expanded_and_oddly_pitched_operands(Tq, Tk):
    """One key head for all query heads, and single rows cut from a buffer of an odd pitch."""
    from deeplearning4j_b200.nd.nd4j import Nd4j
    g = torch.Generator(device="cuda").manual_seed(Tk)
    t = lambda H, T: torch.randn(1, H, T, 35, generator=g, device="cuda").bfloat16()[..., :32]
    H = 1 if Tq == Tk == 1 else 4
    q, k, v, do = t(H, Tq), t(1, Tk).expand(1, H, Tk, 32), t(1, Tk).expand(1, H, Tk, 32), t(H, Tq)
    q6, k6, v6 = (a.double().requires_grad_(True) for a in (q, k, v))
    want = _ref(q6, k6, v6, 0.2, None, False)
    grads = torch.autograd.grad(want, (q6, k6, v6), do.double())
    out = Nd4j.exec("dot_product_attention_v2", q, v, k, scale=0.2).t
    assert (out.double() - want).norm() <= 1e-2 * want.norm()
    dq, dv, dk = (a.t for a in Nd4j.exec("dot_product_attention_v2_bp", q, v, k, do, scale=0.2))
    size = do.double().norm() * 0.2
    for a, b in zip((dq, dk, dv), grads):
        assert a.shape == b.shape and (a.double() - b).norm() <= 1e-2 * (b.norm() + size)
