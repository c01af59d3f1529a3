"""Upstream gradients off the 16-byte grid: a one-row slice of a concatenation's gradient counts as contiguous wherever it starts."""
import ctypes

import pytest
import torch


def test_one_row_slice_is_copied_to_the_grid():
    from deeplearning4j_b200.ops.native import _dense16
    d = torch.randn(1, 11)[:, 3:]
    assert d.is_contiguous() and d.data_ptr() % 16 != 0
    c = _dense16(d)
    assert c.data_ptr() % 16 == 0 and torch.equal(c, d)


class _Recorder:
    """Stands in for the native library: every entry returns 0 and notes its pointer arguments."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append((name, [a.value for a in args if isinstance(a, ctypes.c_void_p)]))
            return 0
        setattr(self, name, entry)
        return entry


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_backward_hands_over_aligned_pointers(monkeypatch, dtype):
    from deeplearning4j_b200.ops import native
    rec = _Recorder()
    monkeypatch.setattr(native, "require", lambda: rec)
    monkeypatch.setattr(native, "_stream", lambda: None)
    monkeypatch.setattr(native, "num_sms", lambda: 148)
    x = torch.randn(1, 16).to(dtype)
    W, b = torch.randn(16, 8).t().contiguous().t().requires_grad_(True), torch.randn(8, requires_grad=True)
    a = torch.randn(1, 3, requires_grad=True)
    if dtype == torch.float32:
        y = native._Linear32Fn.apply(x, W, b, True)
    else:
        y = native._LinearFn.apply(x, W, b, 1, W.detach().to(dtype))
    torch.cat([a.to(dtype), y], 1).backward(torch.ones(1, 11, dtype=dtype))
    ptrs = [p for n, args in rec.calls if n == "dl4j_bias_act_bwd" for p in args[:3]]
    assert ptrs and all(p % 16 == 0 for p in ptrs)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 3e-6), (torch.bfloat16, 8e-3)])
@pytest.mark.parametrize("act", [None, "relu"])
def test_merged_dense_layers_of_one_row(dtype, tol, act):
    """Two dense layers of 3 and 8 units, concatenated: the second one's gradient starts at column 3."""
    from deeplearning4j_b200.nn.activations import ActivationReLU
    from deeplearning4j_b200.ops import nnops
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(1, 16, generator=g, device="cuda").to(dtype)
    leaves = [(torch.randn(*s, generator=g, device="cuda")).requires_grad_(True) for s in ((16, 3), (3,), (16, 8), (8,))]
    dy = torch.randn(1, 11, generator=g, device="cuda").to(dtype)
    a = ActivationReLU() if act else None
    y = torch.cat([nnops.linear(x, leaves[0], leaves[1], a), nnops.linear(x, leaves[2], leaves[3], a)], 1)
    got = torch.autograd.grad(y, leaves, dy)
    ref = [t.detach().double().requires_grad_(True) for t in leaves]
    f = torch.relu if act else (lambda v: v)
    want = torch.autograd.grad(torch.cat([f(x.double() @ ref[0] + ref[1]), f(x.double() @ ref[2] + ref[3])], 1), ref, dy.double())
    for u, v in zip(got, want):
        assert (u.double() - v).norm() <= tol * (v.norm() + dy.double().norm())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [(1, 0, 0), (0, 3, 0), (0, 0, 5), (1, 1, 1), (0, 0, 0)])
def test_entry_takes_any_alignment(dtype, off):
    from deeplearning4j_b200.ops import native
    rows, C = 5, 24
    base = [torch.randn(rows * C + 16, device="cuda").to(dtype) for _ in range(3)]
    dy, z, dz = (b[o:o + rows * C].view(rows, C) for b, o in zip(base, off))
    acc = torch.zeros(C, device="cuda")
    rc = native.require().dl4j_bias_act_bwd(native._ptr(dy), native._ptr(z), native._ptr(dz), native._ptr(acc), rows, C, 1, native._DT[dtype],
                                            native._stream())
    assert rc == 0
    want = dy * (z > 0).to(dtype)
    assert torch.equal(dz, want)
    assert torch.allclose(acc, want.float().sum(0), atol=1e-5)
