"""Whole-sequence LSTM kernels whose batch is split over the chip (``csrc/lstm_split.cu``): edges of the row groups (multiples of 8, a
last group of one row, 40 and 48 rows: two items per thread), of the k-blocks (1, 4, 5, 19: more than one round of loader warps) and of the
limits (what no longer fits runs on the ring kernels), both directions, with and without gradients of the initial state."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(T, mb, n, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    zx = (torch.randn(T, mb, 4 * n, device="cuda", generator=g) * 0.5).bfloat16().requires_grad_(True)
    rw = (torch.randn(4 * n, n, device="cuda", generator=g) * n ** -0.5).bfloat16().t().requires_grad_(True)
    h0 = (torch.randn(mb, n, device="cuda", generator=g) * 0.3).bfloat16().requires_grad_(True)
    c0 = (torch.randn(mb, n, device="cuda", generator=g) * 0.3).requires_grad_(True)
    return zx, rw, h0, c0, torch.randn(T, mb, n, device="cuda", generator=g)


def _reference(zx, rw, h0, c0, w, reverse):
    zx, rw, h0, c0 = (t.detach().double().requires_grad_(True) for t in (zx, rw, h0, c0))
    T, n = zx.shape[0], rw.shape[0]
    h, c, outs = h0, c0, [None] * T
    for t in (range(T - 1, -1, -1) if reverse else range(T)):
        z = zx[t] + h @ rw
        a, f, o, g = torch.tanh(z[:, :n]), torch.sigmoid(z[:, n:2 * n]), torch.sigmoid(z[:, 2 * n:3 * n]), torch.sigmoid(z[:, 3 * n:])
        c = f * c + g * a
        h = o * torch.tanh(c)
        outs[t] = h
    out = torch.stack(outs)
    return (out.detach(), h.detach(), c.detach()) + torch.autograd.grad((out * w.double()).sum(), (zx, rw, h0, c0))


def _run(native, zx, rw, h0, c0, w, reverse):
    hs, h, c = native.lstm_seq(zx, rw, h0, c0, reverse)
    return (hs.detach(), h.detach(), c.detach()) + torch.autograd.grad((hs.float() * w).sum(), (zx, rw, h0, c0))


@pytest.mark.parametrize("T,mb,n,reverse", [(1, 8, 64, False), (2, 1, 64, True), (5, 9, 128, False), (4, 33, 320, True), (5, 64, 512, False), (3, 50, 768, True),
                                            (5, 64, 1024, False), (3, 80, 768, False), (3, 128, 768, True), (3, 90, 1024, False), (3, 24, 1216, False), (2, 25, 1216, True)])
def test_matches_fp64(T, mb, n, reverse):
    """h, gates and dz are rounded to bf16 once per step (2 ** -9 each) and the non-linearities are tanh.approx (2 ** -11): relative 2-norm
    errors of a few 1e-3 that do not grow over a handful of steps."""
    from deeplearning4j_b200.ops import native
    a = _case(T, mb, n)
    ref, got = _reference(*a, reverse), _run(native, *a, reverse)
    again = _run(native, *a, reverse)
    torch.cuda.synchronize()
    native.check_status()
    for name, x, y, z in zip(("hs", "h", "c", "dzx", "drw", "dh0", "dc0"), got, ref, again):
        assert float((x.double() - y).norm() / y.norm()) < 8e-3, name
        assert torch.equal(x, z), name


def test_nan_and_infinite_inputs_pass_and_nothing_waits_for_them():
    """A step's values are handed over with an all-ones word as "not written yet"; NaN results are a different word."""
    from deeplearning4j_b200.ops import native
    zx, rw, h0, c0, w = _case(4, 16, 128)
    with torch.no_grad():
        zx[1, 3] = float("nan")
        zx[2, 7, :64] = float("inf")
        h0.view(torch.int16)[5] = -1                       # the mark itself, as a NaN of the caller's
    out = _run(native, zx, rw, h0, c0, w, False)
    torch.cuda.synchronize()
    native.check_status()
    bad = out[0].float().isnan().any(2)
    assert bad[:, 5].all() and bad[1:, 3].all() and not bad[0, 3]
    ok = [b for b in range(16) if b not in (3, 5)]
    assert not bad[:, ok].any() and not out[3].float()[:, ok].isnan().any()


def test_two_streams():
    from deeplearning4j_b200.ops import native
    a, b = _case(20, 40, 512, 1), _case(20, 40, 512, 2)
    want = [_run(native, *t, False) for t in (a, b)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for t, s in zip((a, b), streams):
        with torch.cuda.stream(s):
            got.append(_run(native, *t, False))
    torch.cuda.synchronize()
    native.check_status()
    for x, y in zip(want, got):
        for p, q in zip(x, y):
            assert torch.equal(p, q)
