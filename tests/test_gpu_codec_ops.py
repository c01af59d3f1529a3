"""Gradient codec ops out of place, at tile edges, off the 16-byte grid and with a capacity, against the CPU codec (exact)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(n, shift):
    g = torch.Generator().manual_seed(n + shift)
    base = torch.randn(n + shift, generator=g) * 1e-3
    return base, base.cuda()[shift:], base[shift:]


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 15, 16, 511, 512, 513, 8191, 8192, 8193, 1_000_003])
def test_threshold_ops(n, shift):
    from deeplearning4j_b200.nd.nd4j import Nd4j
    from deeplearning4j_b200.ops import native
    from deeplearning4j_b200.parallel import codec
    _, x, ref = _case(n, shift)
    keep, r_cpu = x.clone(), ref.clone()
    m_cpu = codec.threshold_encode(r_cpu, 1.5e-3)
    r, m = (a.t for a in Nd4j.exec("encode_threshold", x, threshold=1.5e-3))
    k = int(m_cpu[0])
    assert torch.equal(x, keep) and torch.equal(r.cpu(), r_cpu)
    assert m[:4].cpu().tolist() == m_cpu[:4].tolist()
    assert torch.equal(torch.sort(m[4:4 + k].cpu()).values, torch.sort(m_cpu[4:4 + k]).values)
    cap = max(1, k // 2)
    y = x.clone()
    m2 = codec.threshold_encode(y, 1.5e-3, cap)
    z = torch.empty_like(x)
    m3 = native.threshold_encode(x, 1.5e-3, cap, residual=z)
    assert int(m3[0]) == k and torch.equal(x, keep)
    back3 = torch.zeros(n, device="cuda")
    codec.threshold_decode(m3, back3)
    assert int((back3 != 0).sum()) == min(k, cap) and torch.equal(z[back3 == 0], x[back3 == 0]) and torch.allclose(back3 + z, x, atol=1e-9)
    back = torch.zeros(n, device="cuda")
    codec.threshold_decode(m2, back)
    assert int((back != 0).sum()) == min(k, cap) and torch.allclose(back + y, x, atol=1e-9)


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 15, 16, 511, 512, 513, 8193, 1_000_003])
def test_bitmap_ops(n, shift):
    from deeplearning4j_b200.nd.nd4j import Nd4j
    from deeplearning4j_b200.parallel import codec
    _, x, ref = _case(n, shift)
    keep, r_cpu = x.clone(), ref.clone()
    m_cpu = codec.bitmap_encode(r_cpu, 1e-3)
    r, m, count = (a.t for a in Nd4j.exec("encode_bitmap", x, threshold=1e-3))
    assert torch.equal(x, keep) and torch.equal(r.cpu(), r_cpu) and torch.equal(m.cpu(), m_cpu) and int(count) == int(m_cpu[0])
    t = torch.rand(n, device="cuda")
    want = t.cpu().clone()
    codec.bitmap_decode(m_cpu, want)
    t0 = t.clone()
    assert torch.equal(Nd4j.exec("decode_bitmap", t, m).t.cpu(), want) and torch.equal(t, t0)
    codec.bitmap_decode(m, t)                                    # in place
    assert torch.equal(t.cpu(), want)
