"""Fused attention with more work items (batch x heads x query or key blocks) than resident CTAs: each CTA takes several items of one or of
different lengths, with the key mask, the causal mask, ragged query and key counts, and keys that no query sees."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Tq,Tk,D,mask,causal", [(75, 4, 128, 128, 64, False, False), (40, 8, 129, 129, 64, False, True), (20, 8, 300, 300, 32, True, True),
                                                     (37, 5, 257, 70, 64, True, False), (10, 16, 384, 640, 64, False, False)])
def test_matches_fp64(B, H, Tq, Tk, D, mask, causal):
    from deeplearning4j_b200.nd.nd4j import Nd4j
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(B + Tq)
    q, k, v = (torch.randn(B, H, T, D, device="cuda", generator=g).bfloat16() for T in (Tq, Tk, Tk))
    m = None
    if mask:
        lens = torch.randint(1, Tk + 1, (B,), device="cuda", generator=g)
        m = (torch.arange(Tk, device="cuda")[None] < lens[:, None]).float()
    out = Nd4j.exec("dot_product_attention_v2", q, v, k, None, None, m, scale=D ** -0.5, useCausalMask=causal).t
    torch.cuda.synchronize()
    native.check_status()
    for b in range(B):
        s = q[b].double() @ k[b].double().transpose(-1, -2) * D ** -0.5
        if causal:
            s = s.masked_fill(torch.ones(Tq, Tk, dtype=torch.bool, device="cuda").triu(1), -math.inf)
        if m is not None:
            s = s.masked_fill(m[b][None, None] == 0, -math.inf)
        ref = torch.softmax(s, -1) @ v[b].double()
        # weights and output rounded to bf16 (2 ** -9 each), sums in fp32
        assert float((out[b].double() - ref).norm() / ref.norm()) < 6e-3, b


@pytest.mark.parametrize("B,H,Tq,Tk,D,mask,causal", [(40, 4, 128, 128, 64, False, False), (30, 8, 129, 257, 64, False, True), (12, 8, 300, 300, 32, True, True),
                                                     (37, 5, 257, 70, 64, True, False), (60, 4, 100, 400, 64, False, True)])
def test_gradients_match_fp64(B, H, Tq, Tk, D, mask, causal):
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(B + Tq)
    q, k, v = (torch.randn(B, H, T, D, device="cuda", generator=g).bfloat16().requires_grad_(True) for T in (Tq, Tk, Tk))
    m = None
    if mask:
        lens = torch.randint(1, Tk + 1, (B,), device="cuda", generator=g)
        m = (torch.arange(Tk, device="cuda")[None] < lens[:, None]).float()
    out = native.attention(q, k, v, m, D ** -0.5, causal=causal)
    dy = torch.randn(out.shape, device="cuda", generator=g).bfloat16()
    got = torch.autograd.grad(out, (q, k, v), dy)
    torch.cuda.synchronize()
    native.check_status()
    num, den = torch.zeros(3, dtype=torch.float64), torch.zeros(3, dtype=torch.float64)
    for b in range(B):
        qd, kd, vd = (t[b].detach().double().requires_grad_(True) for t in (q, k, v))
        s = qd @ kd.transpose(-1, -2) * D ** -0.5
        if causal:
            s = s.masked_fill(torch.ones(Tq, Tk, dtype=torch.bool, device="cuda").triu(1), -math.inf)
        if m is not None:
            s = s.masked_fill(m[b][None, None] == 0, -math.inf)
        ref = torch.autograd.grad(torch.softmax(s, -1) @ vd, (qd, kd, vd), dy[b].double())
        for i, (a, r) in enumerate(zip(got, ref)):
            assert torch.isfinite(a[b]).all()
            num[i] += float((a[b].double() - r).square().sum())
            den[i] += float(r.square().sum())
    # P, dS and the results are rounded to bf16 (2 ** -9 each), D = sum(dO * O) from a rounded O, sums in fp32.  The norms go over the batch: an
    # example with a single key has dQ = dK = 0, where the rounding of O is all there is
    assert float((num / den).sqrt().max()) < 1.2e-2
