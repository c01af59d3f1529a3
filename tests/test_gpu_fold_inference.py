"""Inference with batch norm folded into the convolutions against the layer-by-layer executor in fp32 on the CPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(cin, hw, width, layers, has_bias=True, log_std=True, lock=False, residual=True):
    from deeplearning4j_b200 import DataType, nn
    from deeplearning4j_b200.nn.conf.base import ConvolutionMode, InputType, PoolingType
    from deeplearning4j_b200.nn.conf.graphconf import ElementWiseVertex
    from deeplearning4j_b200.nn.graph import ComputationGraph
    from deeplearning4j_b200.nn.layers.conv import BatchNormalization, ConvolutionLayer, GlobalPoolingLayer
    from deeplearning4j_b200.nn.layers.core import ActivationLayer, OutputLayer

    def build(compute):
        b = nn.NeuralNetConfiguration.Builder().seed(3).activation("IDENTITY").convolutionMode(ConvolutionMode.Same)
        if compute:
            b = b.computeDataType(DataType.BFLOAT16)
        gb = b.graphBuilder()
        gb.addInputs("in").setInputTypes(InputType.convolutional(hw, hw + 3, cin))
        prev, first = "in", None
        for i, (k, s, n) in enumerate(layers):
            gb.addLayer(f"c{i}", ConvolutionLayer([k, k], [s, s], nOut=n, hasBias=has_bias), prev)
            gb.addLayer(f"n{i}", BatchNormalization(useLogStd=log_std, lockGammaBeta=lock, gamma=1.5, beta=0.25), f"c{i}")
            prev = f"n{i}"
            if i + 1 < len(layers) or not residual:
                gb.addLayer(f"a{i}", ActivationLayer("RELU"), prev)
                prev = f"a{i}"
            if i == 0:
                first = prev
        if residual:
            gb.addVertex("add", ElementWiseVertex("Add"), prev, first)
            gb.addLayer("ra", ActivationLayer("RELU"), "add")
            prev = "ra"
        gb.addLayer("pool", GlobalPoolingLayer(PoolingType.AVG), prev)
        gb.addLayer("out", OutputLayer("MCXENT", nOut=10, activation="SOFTMAX"), "pool")
        return ComputationGraph(gb.setOutputs("out").build())
    gpu, cpu = build(True), build(False)
    gpu.device = torch.device("cuda")
    gpu.init(), cpu.init()
    g = torch.Generator().manual_seed(5)
    p = torch.empty(cpu.numParams())
    for e in cpu.entries:
        seg = p[e.offset:e.end]
        if e.spec.kind == "weight" and len(e.spec.shape) >= 2 and min(e.spec.shape) > 1:
            fan = e.spec.numel / (e.spec.shape[0] if len(e.spec.shape) == 4 else e.spec.shape[1])
            seg.normal_(0, (1.0 / fan) ** 0.5, generator=g)
        else:
            seg.normal_(0, 0.1, generator=g)
            if e.spec.name == "gamma" or e.spec.name == "var":
                seg.add_(1.0)
    gpu.setParams(p), cpu.setParams(p)
    return gpu, cpu


@pytest.mark.parametrize("layers,opts", [
    ([(3, 1, 16), (1, 1, 8), (3, 1, 8), (1, 1, 16)], {}),                                  # bottleneck, residual in the GEMM epilogue
    ([(3, 1, 24), (3, 1, 24)], {}),                                                        # basic block: residual after a k x k convolution
    ([(7, 2, 16), (1, 2, 40), (5, 1, 8)], {"residual": False}),                            # stem, strided 1x1, 5x5
    ([(3, 2, 16), (3, 1, 12), (1, 1, 16)], {"residual": False, "has_bias": False, "log_std": False}),   # 12 channels: not on the 8 grid
    ([(1, 1, 16), (1, 1, 16)], {"lock": True}),
])
@pytest.mark.parametrize("cin,hw,n", [(3, 12, 2), (16, 9, 1), (8, 17, 5)])
def test_folded_output_matches_fp32(layers, opts, cin, hw, n):
    gpu, cpu = _net(cin, hw, 16, layers, **opts)
    x = torch.randn(n, cin, hw, hw + 3, generator=torch.Generator().manual_seed(n))
    want = cpu.output(x)[0].t
    for xin in (x.cuda(), x.cuda().to(memory_format=torch.channels_last)):
        got = gpu.output(xin)[0].t.cpu()
        # bf16 weights and activations: 2^-9 per rounding, at most 2 roundings per layer, on logits of order one
        assert (got - want).norm() <= 2 ** -8 * (2 * len(layers)) ** 0.5 * want.norm() * 2
    got2 = gpu.output(x.cuda(), train=False)[0].t.cpu()
    acts = gpu.feedForward(x.cuda())                                  # the unfused executor still exposes every activation
    assert torch.allclose(acts["out"].t.float().cpu(), got2, atol=2e-2)
    gpu.setParams(gpu.params().t * 0.5)                               # nothing is kept from one call to the next
    cpu.setParams(cpu.params().t * 0.5)
    want = cpu.output(x)[0].t
    assert (gpu.output(x.cuda())[0].t.cpu() - want).norm() <= 2 ** -8 * (2 * len(layers)) ** 0.5 * want.norm() * 2


@pytest.mark.parametrize("k,residual", [(1, True), (3, True), (1, False)])
def test_inputs_the_folded_kernels_do_not_read(k, residual):
    """Another channel count is refused as by the layers; a view off the 16-byte grid gives what its copy gives."""
    gpu, _ = _net(16, 9, 16, [(k, 1, 16), (1, 1, 16)], residual=residual)
    x = torch.randn(2, 16, 9, 12, device="cuda")
    want = gpu.output(x)[0].t
    for c in (8, 24, 64):
        with pytest.raises(Exception):
            gpu.output(torch.randn(2, c, 9, 12, device="cuda"))
    for cl in (False, True):
        xb = x.bfloat16().contiguous(memory_format=torch.channels_last if cl else torch.contiguous_format)
        off = torch.empty(xb.numel() + 1, dtype=xb.dtype, device="cuda")[1:].as_strided(xb.shape, xb.stride())
        off.copy_(xb)
        assert off.data_ptr() % 16
        assert torch.equal(gpu.output(off)[0].t, want)


@pytest.mark.parametrize("layers,opts", [
    ([(1, 1, 16), (1, 1, 16)], {}), ([(3, 1, 16), (3, 1, 16)], {}), ([(3, 1, 16), (3, 1, 16)], {"residual": False}),
    ([(7, 2, 16), (1, 2, 40), (5, 1, 8)], {"residual": False}), ([(3, 1, 16), (3, 1, 12), (1, 1, 16)], {}),
])
@pytest.mark.parametrize("cin", [3, 16])
def test_nan_reaches_the_output(layers, opts, cin):
    """A NaN in one image makes that image's probabilities NaN and no others, as the layers give it."""
    gpu, cpu = _net(cin, 9, 16, layers, **opts)
    x = torch.randn(3, cin, 9, 12)
    x[1, 0, 4, 4] = float("nan")
    got, want = gpu.output(x.cuda())[0].t.cpu(), cpu.output(x)[0].t
    assert torch.isnan(want[1]).all() and torch.isfinite(want[[0, 2]]).all()
    assert torch.equal(torch.isnan(got), torch.isnan(want))


def test_epilogue_relu_passes_nan_and_infinities():
    from deeplearning4j_b200.ops import native
    special = torch.tensor([float("nan"), float("inf"), float("-inf"), -0.0, 0.0, -1.0, 2.0, 3e-39], device="cuda")
    a = torch.zeros(40, 64, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    z = special.repeat(8)
    want = torch.relu(z).bfloat16()

    def same(y):
        assert torch.equal(torch.isnan(y), torch.isnan(want.expand_as(y))) and torch.equal(y.nan_to_num(7.0), want.expand_as(y).nan_to_num(7.0))
    same(native.gemm_raw(a, w, bias=z, act=1))
    same(native.gemm_raw(a, w, bias=z, act=1, out_dtype=torch.float32).bfloat16())
    same(native.gemm_raw(a[:, :24], w[:24], bias=z, act=1, block_n=128))
    x = torch.zeros(1, 64, 5, 8, device="cuda", dtype=torch.bfloat16).contiguous(memory_format=torch.channels_last)
    same(native.conv_infer_1x1(x, w, z, True).permute(0, 2, 3, 1).reshape(-1, 64))
    res = want.new_zeros(1, 64, 5, 8).contiguous(memory_format=torch.channels_last)
    same(native.conv_infer_1x1(x, w, z, True, res).permute(0, 2, 3, 1).reshape(-1, 64))
    for k in (3, 5):
        y = native.conv_infer_kxk(x, torch.zeros(64, k * k * 64, device="cuda", dtype=torch.bfloat16), z, k, k, (k // 2,) * 2, (1, 1), True)
        same(y.permute(0, 2, 3, 1).reshape(-1, 64))
    zz = z.bfloat16().reshape(1, 64, 1, 1).expand(1, 64, 5, 8).contiguous(memory_format=torch.channels_last)
    one, zero = torch.ones(64, device="cuda"), torch.zeros(64, device="cuda")
    same(native.bn_act_eval(zz, None, one, zero, True).permute(0, 2, 3, 1).reshape(-1, 64))
    same(native.bn_act_eval(zz, res, one, zero, True).permute(0, 2, 3, 1).reshape(-1, 64))
    same(native.add_relu(zz, res).permute(0, 2, 3, 1).reshape(-1, 64))


@pytest.mark.parametrize("act", ["IDENTITY", "TANH"])
@pytest.mark.parametrize("shape", [(1, 1), (9, 12)])
def test_residual_that_broadcasts(act, shape):
    """Add after a batch norm with a [N, C, 1, 1] input, in a folded (identity) and an unfolded convolution; output and gradients."""
    from deeplearning4j_b200 import DataType, nn
    from deeplearning4j_b200.nn.conf.base import InputType, PoolingType
    from deeplearning4j_b200.nn.conf.graphconf import ElementWiseVertex
    from deeplearning4j_b200.nn.graph import ComputationGraph
    from deeplearning4j_b200.nn.layers.conv import BatchNormalization, ConvolutionLayer, GlobalPoolingLayer
    from deeplearning4j_b200.nn.layers.core import ActivationLayer, OutputLayer

    def build(compute):
        b = nn.NeuralNetConfiguration.Builder().seed(3)
        gb = (b.computeDataType(DataType.BFLOAT16) if compute else b).graphBuilder()
        gb.addInputs("in", "in2").setInputTypes(InputType.convolutional(9, 12, 16), InputType.convolutional(*shape, 16))
        gb.addLayer("c", ConvolutionLayer([1, 1], [1, 1], nOut=16, activation=act), "in").addLayer("n", BatchNormalization(), "c")
        gb.addVertex("add", ElementWiseVertex("Add"), "n", "in2").addLayer("r", ActivationLayer("RELU"), "add")
        gb.addLayer("p", GlobalPoolingLayer(PoolingType.AVG), "r").addLayer("out", OutputLayer("MCXENT", nOut=5, activation="SOFTMAX"), "p")
        return ComputationGraph(gb.setOutputs("out").build())
    gpu, cpu = build(True), build(False)
    gpu.device = torch.device("cuda")
    gpu.init(), cpu.init()
    gpu.setParams(cpu.params().t)
    g = torch.Generator().manual_seed(2)
    x, s, y = torch.randn(3, 16, 9, 12, generator=g), torch.randn(3, 16, *shape, generator=g), torch.eye(5)[:3]
    want = cpu.output([x, s])[0].t
    assert (gpu.output([x.cuda(), s.cuda()])[0].t.cpu() - want).norm() <= 2e-2 * want.norm()
    off = torch.empty(s.numel() + 1, device="cuda", dtype=torch.bfloat16)[1:].view(s.shape)
    off.copy_(s)
    assert (gpu.output([x.cuda(), off])[0].t.cpu() - want).norm() <= 2e-2 * want.norm()
    _, sg = gpu.computeGradientAndScore([x.cuda(), s.cuda()], y.cuda())
    _, sc = cpu.computeGradientAndScore([x, s], y)
    assert abs(sg - sc) <= 2e-2 * abs(sc)
