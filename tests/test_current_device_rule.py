"""The native library launches on the current device: tensors of another one, or of the host, take the general path."""
import pytest
import torch


class _On:
    def __init__(self, d): self.d = d
    def get_device(self): return self.d


def test_rule(monkeypatch):
    from deeplearning4j_b200.ops import native
    monkeypatch.setattr(native, "_current_device", lambda: 1)
    assert native.on_current_device(_On(1), None, _On(1))
    assert not native.on_current_device(_On(1), _On(0)) and not native.on_current_device(torch.zeros(2))


@pytest.mark.gpu
def test_routes_decline_tensors_of_another_device(monkeypatch):
    from deeplearning4j_b200.ops import attention_native as an
    from deeplearning4j_b200.ops import impl_misc, native
    bf = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    f = lambda *s: torch.randn(*s, device="cuda")
    q = bf(1, 2, 30, 64)
    with torch.no_grad():
        calls = {
            "linear32": lambda: native.linear32(f(8, 16), f(16, 8), f(8), True),
            "layer_norm_grad": lambda: native.layer_norm_grad(f(4, 33), f(33), f(33), f(4, 33), 1e-5),
            "linear_small": lambda: native.linear_small(bf(2, 24), f(10, 24).t(), f(10)),
            "lstm_step": lambda: native.lstm_step_supported(bf(1, 2, 24), f(32, 24).t(), f(32, 8).t(), 8, 2) or None,
            "avgpool": lambda: native.global_avgpool(bf(2, 8, 4, 4).contiguous(memory_format=torch.channels_last)),
            "attention": lambda: an.attention(q, q, q, None, 0.1, causal=True),
            "attention_grad": lambda: an.attention_grad(q, q, q, None, 0.1, q),
            "odd": lambda: native.linear(bf(256, 24), f(24, 10), f(10), None),
            "codec": lambda: impl_misc._out_of_place_codec(f(64)),
        }
        for n, c in calls.items():
            assert c() is not None, n
        monkeypatch.setattr(native, "_current_device", lambda: 1)
        for n, c in calls.items():
            assert c() is None, n


@pytest.mark.gpu
@pytest.mark.parametrize("T,causal", [(201, False), (128, False), (1032, False), (64, True), (64, False)])
def test_host_operands_are_refused(T, causal):
    from deeplearning4j_b200.nd.nd4j import Nd4j
    q, k, v, do = (torch.randn(2, 2, T, 64, device="cuda").bfloat16() for _ in range(4))
    mask = torch.ones(2, T)
    with pytest.raises(RuntimeError):
        Nd4j.exec("dot_product_attention_v2", q, v, k, None, None, mask, scale=0.1, useCausalMask=causal)
    with pytest.raises(RuntimeError):
        Nd4j.exec("dot_product_attention_v2_bp", q, v, k, do, vMask=mask, scale=0.1, useCausalMask=causal)
    with pytest.raises(RuntimeError):
        Nd4j.exec("dot_product_attention_v2", q, v.cpu(), k, scale=0.1, useCausalMask=causal)
    x, g = torch.randn(4, 33, device="cuda"), torch.ones(33, device="cuda")
    with pytest.raises(RuntimeError):
        Nd4j.exec("layer_norm_bp", x, g.cpu(), g, x)
