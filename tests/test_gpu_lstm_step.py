"""Hidden sizes off the 64 grid on the sequence kernels and the one-launch inference step, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(n_in, n, layers, bf16=True, dtype=None):
    from deeplearning4j_b200 import DataType, nn
    from deeplearning4j_b200.nn.layers.core import RnnOutputLayer
    from deeplearning4j_b200.nn.layers.recurrent import LSTM
    b = nn.NeuralNetConfiguration.Builder().seed(n).updater(nn.Sgd(0.1))
    if bf16:
        b = b.computeDataType(DataType.BFLOAT16)
    lb, i = b.list(), n_in
    for _ in range(layers):
        lb.layer(LSTM(nIn=i, nOut=n, activation="TANH"))
        i = n
    lb.layer(RnnOutputLayer("MCXENT", nIn=i, nOut=n_in, activation="SOFTMAX"))
    net = nn.MultiLayerNetwork(lb.build())
    net.device = torch.device("cuda")
    return net.init()


def _ref(net, x, layers, n):
    """[T, mb, n_in] -> logits, states, in fp64 with gradients to the parameters."""
    ps = [{k: v.detach().double().requires_grad_(True) for k, v in net.param_views[str(i)].items()} for i in range(layers + 1)]
    out, states = x, []
    for p in ps[:-1]:
        h = c = torch.zeros(x.shape[1], n, dtype=torch.float64, device="cuda")
        hs = []
        for t in range(x.shape[0]):
            z = out[t] @ p["W"] + p["b"].reshape(-1) + h @ p["RW"]
            c = torch.sigmoid(z[:, n:2 * n]) * c + torch.sigmoid(z[:, 3 * n:]) * torch.tanh(z[:, :n])
            h = torch.sigmoid(z[:, 2 * n:3 * n]) * torch.tanh(c)
            hs.append(h)
        out = torch.stack(hs)
        states.append((h, c))
    return out @ ps[-1]["W"] + ps[-1]["b"].reshape(-1), states, ps


@pytest.mark.parametrize("n,mb,T", [(8, 3, 4), (20, 5, 7), (63, 1, 3), (72, 17, 5), (200, 32, 9), (1270, 2, 3)])
def test_padded_hidden_sizes_train(n, mb, T):
    """bf16 hidden state and gates over T steps: 2^-9 per rounding, a few per step."""
    from deeplearning4j_b200.ops import native
    n_in = 16
    net = _net(n_in, n, 2)
    g = torch.Generator(device="cuda").manual_seed(n)
    idx = torch.randint(0, n_in, (2, mb, T), generator=g, device="cuda")
    x, y = (torch.nn.functional.one_hot(i, n_in).float().permute(0, 2, 1) for i in idx)
    before = native.LAUNCHES
    grad, score = net.computeGradientAndScore(x, y)
    assert native.LAUNCHES - before < 60                       # not one launch per step and layer
    logits, _, ps = _ref(net, x.permute(2, 0, 1).double(), 2, n)
    loss = -(y.permute(2, 0, 1).double() * torch.log_softmax(logits, -1)).sum() / mb
    loss.backward()
    native.check_status()
    assert abs(score - float(loss)) <= 4e-3 * abs(float(loss))
    for i, p in enumerate(ps):
        for k, t in p.items():
            got = grad.gradientForVariable()[f"{i}_{k}"].t.double().reshape(t.shape)
            assert (got - t.grad).norm() <= 3e-2 * t.grad.norm() + 1e-6, (i, k)


@pytest.mark.parametrize("n,mb,n_in", [(1, 1, 1), (8, 2, 5), (33, 9, 77), (256, 1, 77), (200, 64, 98), (512, 33, 16), (1024, 32, 40)])
def test_one_step_matches_fp64(n, mb, n_in):
    """Three consecutive steps: h is rounded to bf16 once per layer and step, nothing else is."""
    from deeplearning4j_b200.ops import native
    net = _net(n_in, n, 2)
    g = torch.Generator(device="cuda").manual_seed(mb)
    x = torch.randn(3, mb, n_in, generator=g, device="cuda").bfloat16().float()
    before = native.LAUNCHES
    for t in range(3):
        out = net.rnnTimeStep(x[t]).t
    if mb * n <= native.LSTM_STEP_MAX:
        assert native.LAUNCHES - before <= 3 * 3
    with torch.no_grad():
        logits, states, _ = _ref(net, x.double(), 2, n)
    assert (out.double() - torch.softmax(logits[-1], -1)).norm() <= 1.5e-2 * torch.softmax(logits[-1], -1).norm()
    for i, (h, c) in enumerate(states):
        gh, gc = net.rnnGetPreviousState(i)
        assert (gh.double() - h).norm() <= 1e-2 * h.norm() and (gc.double() - c).norm() <= 1e-2 * c.norm()
    net.paramTable()["0_W"].t.zero_()                           # a change of the parameters is seen at once
    net.rnnClearPreviousState()
    a = net.rnnTimeStep(x[0]).t
    net.rnnClearPreviousState()
    assert torch.equal(a, net.rnnTimeStep(torch.zeros_like(x[0])).t)


@pytest.mark.parametrize("n,mb", [(64, 5), (256, 128), (1024, 64)])
def test_sequence_kernels_repeat_bit_for_bit(n, mb):
    """h and dz pass from one block to the others through memory at every step: a reader that came too early would change the bits."""
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(1)
    T = 40
    zx = (torch.randn(T, mb, 4 * n, generator=g, device="cuda") * 0.5).bfloat16()
    rw = torch.randn(n, 4 * n, generator=g, device="cuda") * n ** -0.5
    h0, c0 = torch.zeros(mb, n, device="cuda", dtype=torch.bfloat16), torch.zeros(mb, n, device="cuda")

    def run():
        z = zx.clone().requires_grad_(True)
        out = native.lstm_seq(z, rw, h0, c0)[0]
        out.float().square().sum().backward()
        return out.detach(), z.grad
    want = run()
    for _ in range(20):
        got = run()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    native.check_status()


@pytest.mark.parametrize("n,mb,T,seq", [(300, 120, 1, False), (300, 120, 2, True), (320, 120, 1, True), (1000, 40, 1, False)])
def test_route_of_a_single_step(monkeypatch, n, mb, T, seq):
    """One step of a size off the 64 grid takes the general path, two take the padded sequence kernel; same values either way."""
    from deeplearning4j_b200.ops import native
    calls, apply = [], native._LstmSeqFn.apply
    monkeypatch.setattr(native._LstmSeqFn, "apply", lambda *a: calls.append(1) or apply(*a))
    net = _net(16, n, 1)
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(T, mb, 16, generator=g, device="cuda").bfloat16().float()
    out = net.output(x.permute(1, 2, 0)).t
    with torch.no_grad():
        logits, _, _ = _ref(net, x.double(), 1, n)
    want = torch.softmax(logits, -1).permute(1, 2, 0)
    assert (len(calls) > 0) == seq and (out.double() - want).norm() <= 1.5e-2 * want.norm()


@pytest.mark.parametrize("M,K,N", [(1, 1, 1), (3, 24, 77), (8, 77, 10), (9, 256, 5), (32, 131, 33)])
@pytest.mark.parametrize("wdtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bias", [True, False])
def test_small_dense_layers_without_a_gradient(M, K, N, wdtype, bias):
    """A few rows on the parameters themselves, in either type they are held in: one rounding of the result."""
    from deeplearning4j_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    base = torch.randn(M * K + 1, generator=g, device="cuda").bfloat16()
    W = torch.randn(N, K, generator=g, device="cuda").to(wdtype).t()
    b = torch.randn(1, N, generator=g, device="cuda") if bias else None
    with torch.no_grad():
        for x in (base[:M * K].view(M, K), base[1:].view(M, K)):
            y = native.linear_small(x, W, b)
            want = x.double() @ W.double() + (b.double() if bias else 0.0)
            assert y.dtype == torch.bfloat16 and (y.double() - want).norm() <= 2 ** -8 * want.norm()
