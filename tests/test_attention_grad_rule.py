"""The operator form of the fused attention gradient (second derivatives) against autograd, on the CPU."""
import pytest
import torch

from deeplearning4j_b200.ops.attention_native import _grad_in_ops


def _hidden(mask, causal, T):
    h = (mask == 0)[:, None, None, :].expand(2, 1, T, T)
    return h | torch.ones(T, T, dtype=torch.bool).triu(1) if causal else h


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("empty", [None, 0, float("nan")])
def test_matches_autograd(causal, empty):
    T = 5
    g = torch.Generator().manual_seed(3)
    q, k, v, do = (torch.randn(2, 2, T, 8, generator=g) for _ in range(4))
    mask = torch.ones(2, T)
    mask[0, 1:3] = 0
    if empty is not None:
        mask[1] = 0
    flags = int(causal) | (2 if empty != 0 else 0)
    hid = _hidden(mask, causal, T)
    none = hid.all(-1, keepdim=True)
    ql, kl, vl = (t.clone().requires_grad_(True) for t in (q, k, v))
    s = (ql @ kl.transpose(-1, -2) * 0.3).masked_fill(hid, float("-inf"))
    p = torch.softmax(s.masked_fill(none, 0.0), -1).masked_fill(none, 0.0 if empty == 0 else float("nan"))
    want = torch.autograd.grad(p @ vl, (ql, kl, vl), do)
    got = _grad_in_ops(q, k, v, do, mask, 0.3, flags)
    for a, b in zip(got, want):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-5, equal_nan=True), (a - b).abs().max()


def test_is_differentiable():
    q, k, v, do = (torch.randn(1, 1, 3, 8, dtype=torch.float64, requires_grad=True) for _ in range(4))
    out = _grad_in_ops(q, k, v, do, None, 0.3, 1)
    assert all(t is not None for t in torch.autograd.grad([(o ** 2).sum() for o in out], (q, k, v, do)))


@pytest.mark.parametrize("make", [
    lambda: torch.randn(1, 1, 1, 33)[..., :32],                                     # one row: any pitch counts as contiguous
    lambda: torch.randn(2, 1, 5, 32).expand(2, 3, 5, 32),                           # one head for all
    lambda: torch.randn(1, 1, 1, 32).expand(2, 3, 5, 32),
    lambda: torch.randn(2, 3, 5, 36)[..., :32],
    lambda: torch.randn(2 * 3 * 5 * 32 + 1)[1:].view(2, 3, 5, 32),
    lambda: torch.randn(2, 3, 32, 5).transpose(-1, -2),
])
def test_operands_are_laid_out_for_the_tensor_map(make):
    from deeplearning4j_b200.ops.attention_native import _ok_view, _prep
    t = make()
    p = _prep(t)
    assert torch.equal(p, t) and _ok_view(p) and p.is_contiguous()
    ok = torch.randn(2, 5, 3, 32).permute(0, 2, 1, 3)
    assert _prep(ok) is ok
