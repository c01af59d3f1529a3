"""Performance cases of the framework: what its users have it compute, called through its public entry points.

Kinds of case (``"kind"``):

``mlp``        one ``fit`` of a small dense classifier (launch-bound; fp32, the default data type, or bf16 compute)
``attention``  scaled dot-product attention, op by op: forward (inference) or the gradient op (training), with the lengths, key
               masks and causal masks that batches of text have
``layer_norm`` gradient op of layer normalisation over rows of activations
``lm_head``    vocabulary projection + sparse softmax cross entropy, loss gradients through a SameDiff graph
``lstm``       truncated-BPTT ``fit`` of a stacked character LSTM
``rnn_step``   stateful generation, one character per call
``conv_block`` one ``fit`` step of a residual convolution block with batch norm
``resnet50``   ResNet-50 inference
``bert``       one ``fit`` step of a BERT-width masked-LM encoder, Adam, bf16 compute
``codec``      gradient compression: encode + decode, threshold or bitmap form

Inputs are drawn on the GPU from the seed alone.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from deeplearning4j_b200 import DataType, nn
from deeplearning4j_b200.models.bert import BertConfig, build_bert_mlm
from deeplearning4j_b200.models.zoo import ResNet50
from deeplearning4j_b200.nd.nd4j import Nd4j
from deeplearning4j_b200.nn.conf.base import BackpropType, ConvolutionMode, InputType, PoolingType
from deeplearning4j_b200.nn.conf.graphconf import ElementWiseVertex
from deeplearning4j_b200.nn.graph import ComputationGraph
from deeplearning4j_b200.nn.layers.conv import BatchNormalization, ConvolutionLayer, GlobalPoolingLayer
from deeplearning4j_b200.nn.layers.core import ActivationLayer, OutputLayer, RnnOutputLayer
from deeplearning4j_b200.nn.layers.recurrent import LSTM
from deeplearning4j_b200.samediff.core import SameDiff

DEV = "cuda"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def listed():
    return [
        # the smallest training step: an MNIST-shaped classifier at its usual minibatch, bound by launches and host work
        {"name": "mlp_fit_b128", "kind": "mlp", "batch": 128, "nIn": 784, "hidden": 512, "nOut": 10, "dtype": "float"},
        # one request served by a base-size encoder: attention of a single sequence
        {"name": "attention_b1_t128", "kind": "attention", "B": 1, "H": 12, "Tq": 128, "Tk": 128, "D": 64, "mask": False,
         "causal": False, "train": False},
        # pre-training batch of a base-size encoder
        {"name": "attention_grad_b32_t512", "kind": "attention", "B": 32, "H": 12, "Tq": 512, "Tk": 512, "D": 64, "mask": False,
         "causal": False, "train": True},
        # fine-tuning batch: sequences padded to the longest of the batch, padding masked
        {"name": "attention_grad_masked_t200", "kind": "attention", "B": 24, "H": 12, "Tq": 200, "Tk": 200, "D": 64, "mask": True,
         "causal": False, "train": True},
        # normalisation of one pre-training batch's activations (32 x 512 tokens)
        {"name": "layer_norm_grad_16384x768", "kind": "layer_norm", "rows": 16384, "C": 768, "dtype": "bfloat16"},
        # masked-LM head: 15 % of 32 x 512 tokens against a WordPiece vocabulary
        {"name": "lm_head_grad_2456x30522", "kind": "lm_head", "rows": 2456, "hidden": 768, "vocab": 30522},
        # character model training, two truncated-BPTT segments of 50
        {"name": "lstm_fit_1024", "kind": "lstm", "mb": 64, "hidden": 1024, "vocab": 98, "T": 100, "layers": 2},
        # character generation from the text-generation network at its default width
        {"name": "rnn_step_256", "kind": "rnn_step", "mb": 1, "hidden": 256, "vocab": 77, "layers": 2},
        # second stage of a residual network, training
        {"name": "conv_block_fit_n64_c64", "kind": "conv_block", "N": 64, "HW": 56, "width": 64, "classes": 1000},
        # image classification service
        {"name": "resnet50_output_b32", "kind": "resnet50", "N": 32, "HW": 224},
        # two layers of the pre-training workload, whole step with the updater
        {"name": "bert_fit_2layer_b32_t512", "kind": "bert", "B": 32, "T": 512, "layers": 2, "hidden": 768, "heads": 12, "vocab": 30522},
        # gradient sharing of a 25.6 M parameter network
        {"name": "threshold_codec_25m", "kind": "codec", "n": 25_600_000, "form": "threshold", "density": 0.01},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "attention", "attention", "attention", "layer_norm", "lm_head", "lstm", "rnn_step", "conv_block",
                       "resnet50", "bert", "codec"])
    if kind == "mlp":
        return {"kind": kind, "batch": _log(rng, 16, 1024), "nIn": _log(rng, 30, 1024), "hidden": _log(rng, 64, 1024),
                "nOut": rng.randint(2, 100), "dtype": rng.choice(["float", "float", "bfloat16"])}
    if kind == "attention":
        T = rng.choice([_log(rng, 16, 1024), _log(rng, 16, 1024) // 8 * 8 + 8, 128 * rng.randint(1, 8)])
        causal = rng.random() < 0.25
        Tk = T if causal or rng.random() < 0.8 else _log(rng, 16, 512)
        return {"kind": kind, "B": max(1, min(_log(rng, 1, 64), 16384 // max(T, Tk))), "H": rng.choice([4, 8, 12, 16]), "Tq": T, "Tk": Tk,
                "D": rng.choice([32, 64, 64, 64]), "mask": rng.random() < 0.5, "causal": causal, "train": rng.random() < 0.6}
    if kind == "layer_norm":
        C = rng.choice([128, 256, 384, 512, 768, 1024, 1536, 2048, 4096, rng.randint(8, 512) * 2 + 1])
        return {"kind": kind, "rows": _log(rng, 32, max(64, 16384 * 768 // C)), "C": C, "dtype": rng.choice(["bfloat16", "bfloat16", "float"])}
    if kind == "lm_head":
        return {"kind": kind, "rows": _log(rng, 64, 2456), "hidden": rng.choice([256, 512, 768]), "vocab": rng.randint(1000, 30522)}
    if kind == "lstm":
        return {"kind": kind, "mb": rng.choice([16, 32, 50, 64]), "hidden": rng.choice([128, 200, 256, 300, 512, 768, 1024]),
                "vocab": rng.randint(40, 128), "T": rng.choice([50, 75, 100]), "layers": rng.choice([1, 2])}
    if kind == "rnn_step":
        return {"kind": kind, "mb": _log(rng, 1, 64), "hidden": rng.choice([128, 200, 256, 512, 1024]), "vocab": rng.randint(40, 128),
                "layers": rng.choice([1, 2, 3])}
    if kind == "conv_block":
        w = rng.choice([32, 64, 128, 256])
        hw = rng.choice([7, 14, 19, 28, 56])
        return {"kind": kind, "N": max(1, min(_log(rng, 4, 256), 64 * 56 * 56 * 64 // (hw * hw * w))), "HW": hw, "width": w,
                "classes": rng.choice([10, 100, 1000])}
    if kind == "resnet50":
        return {"kind": kind, "N": _log(rng, 1, 32), "HW": rng.choice([192, 208, 224])}
    if kind == "bert":
        T = rng.choice([64, 128, 200, 256, 384, 512])
        hidden, heads = rng.choice([(256, 4), (512, 8), (768, 12)])
        return {"kind": kind, "B": max(1, min(_log(rng, 4, 32), 16384 // T)), "T": T, "layers": rng.choice([1, 2]), "hidden": hidden,
                "heads": heads, "vocab": rng.choice([1000, 8000, 30522])}
    return {"kind": kind, "n": _log(rng, 20_000, 25_600_000), "form": rng.choice(["threshold", "bitmap"]),
            "density": rng.choice([0.001, 0.01, 0.05])}


# ------------------------------------------------------------------------------------------------ inputs, shared with exact()
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, std=1.0, dtype=F32):
    return (torch.randn(shape, generator=g, device=DEV, dtype=F32) * std).to(dtype)


def _onehot(g, n, *shape):
    return F.one_hot(torch.randint(0, n, shape, generator=g, device=DEV), n).to(F32)


def _fmat(t):
    """A dense weight in the order in which a network's flat parameter vector holds it."""
    return t.t().reshape(-1)


def _mlp_in(c, seed):
    g = _gen(seed)
    sizes = [(c["nIn"], c["hidden"]), (c["hidden"], c["hidden"]), (c["hidden"], c["nOut"])]
    Ws = [_randn(g, i, o, std=(2.0 / (i + o)) ** 0.5) for i, o in sizes]
    bs = [_randn(g, o, std=0.01) for _, o in sizes]
    x = torch.rand((c["batch"], c["nIn"]), generator=g, device=DEV)
    return Ws, bs, x, _onehot(g, c["nOut"], c["batch"])


def _attention_in(c, seed):
    g = _gen(seed)
    B, H, Tq, Tk, D = (c[k] for k in ("B", "H", "Tq", "Tk", "D"))
    if Tq == Tk:           # views of one packed projection, as a multi-head layer has them
        qkv = _randn(g, B, Tq, 3, H, D, dtype=BF16)
        q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    else:
        q = _randn(g, B, Tq, H, D, dtype=BF16).permute(0, 2, 1, 3)
        kv = _randn(g, B, Tk, 2, H, D, dtype=BF16)
        k, v = (kv[:, :, i].permute(0, 2, 1, 3) for i in range(2))
    mask = None
    if c["mask"]:
        lens = torch.randint(max(1, Tk // 4), Tk + 1, (B,), generator=g, device=DEV)
        mask = (torch.arange(Tk, device=DEV)[None, :] < lens[:, None]).to(F32)
    dout = _randn(g, B, Tq, H, D, dtype=BF16).permute(0, 2, 1, 3)
    return q, k, v, mask, dout


def _layer_norm_in(c, seed):
    g = _gen(seed)
    dt = BF16 if c["dtype"] == "bfloat16" else F32
    return (_randn(g, c["rows"], c["C"], dtype=dt) + 0.25, 1 + _randn(g, c["C"], std=0.1), _randn(g, c["C"], std=0.1),
            _randn(g, c["rows"], c["C"], dtype=dt))


def _lm_head_in(c, seed):
    g = _gen(seed)
    return (_randn(g, c["rows"], c["hidden"], dtype=BF16), _randn(g, c["hidden"], c["vocab"], std=0.02, dtype=BF16),
            _randn(g, c["vocab"], std=0.02, dtype=BF16), torch.randint(0, c["vocab"], (c["rows"],), generator=g, device=DEV))


def _lstm_params(c, g):
    out, n_in, n = [], c["vocab"], c["hidden"]
    for _ in range(c["layers"]):
        b = _randn(g, 4 * n, std=0.02)
        b[n:2 * n] += 1.0
        out.append((_randn(g, n_in, 4 * n, std=(1.0 / n) ** 0.5), _randn(g, n, 4 * n, std=(1.0 / n) ** 0.5), b))
        n_in = n
    out.append((_randn(g, n, c["vocab"], std=(1.0 / n) ** 0.5), _randn(g, c["vocab"], std=0.02)))
    return out


def _lstm_in(c, seed):
    g = _gen(seed)
    ps = _lstm_params(c, g)
    if c["kind"] == "rnn_step":
        return ps, _onehot(g, c["vocab"], c["mb"]), None
    idx = torch.randint(0, c["vocab"], (c["mb"], c["T"] + 1), generator=g, device=DEV)
    oh = F.one_hot(idx, c["vocab"]).to(F32).permute(0, 2, 1)
    return ps, oh[:, :, :-1].contiguous(), oh[:, :, 1:].contiguous()


def _he(g, co, ci, k):
    return _randn(g, co, ci, k, k, std=(2.0 / (ci * k * k)) ** 0.5)


def _bn(g, n, scale=1.0):
    """gamma, beta, running mean, running log10 standard deviation."""
    return scale * (1 + _randn(g, n, std=0.1)), _randn(g, n, std=0.1), _randn(g, n, std=0.1), _randn(g, n, std=0.02)


def _conv_block_in(c, seed):
    g = _gen(seed)
    w = c["width"]
    convs = [(4 * w, 3, 3), (w, 4 * w, 1), (w, w, 3), (4 * w, w, 1)]          # stem, then a bottleneck
    ps = [((_randn(g, co, std=0.02), _he(g, co, ci, k)), _bn(g, co)) for co, ci, k in convs]
    out = (_randn(g, 4 * w, c["classes"], std=(1.0 / (4 * w)) ** 0.5), _randn(g, c["classes"], std=0.02))
    x = _randn(g, c["N"], 3, c["HW"], c["HW"])
    return ps, out, x, _onehot(g, c["classes"], c["N"])


def _resnet_blocks():
    """(filters, stride, has projection) of the zoo network's bottlenecks, in order."""
    out = []
    for f, n, s in (((64, 64, 256), 3, 2), ((128, 128, 512), 4, 2), ((256, 256, 1024), 6, 2), ((512, 512, 2048), 3, 2)):
        out += [(f, s if i == 0 else 1, i == 0) for i in range(n)]
    return out


def _resnet_names():
    return [s + b for s, bs in (("2", "abc"), ("3", "abcd"), ("4", "abcdef"), ("5", "abc")) for b in bs]


def _resnet_in(c, seed):
    """Parameters by vertex name, scaled so that activations stay at the size they have in a trained network."""
    g = _gen(seed)
    p = {"stem-cnn1": (_randn(g, 64, std=0.02), _he(g, 64, 3, 7)), "stem-batch1": _bn(g, 64, 0.5)}
    ci = 64
    for (f, _, proj), nm in zip(_resnet_blocks(), _resnet_names()):
        for part, co, k, i, sc in (("2a", f[0], 1, ci, 1.0), ("2b", f[1], 3, f[0], 1.0), ("2c", f[2], 1, f[1], 0.3)):
            p["res%s_branch%s" % (nm, part)] = (_randn(g, co, std=0.02), _he(g, co, i, k))
            p["bn%s_branch%s" % (nm, part)] = _bn(g, co, 0.7 * sc)
        if proj:
            p["res%s_branch1" % nm] = (_randn(g, f[2], std=0.02), _he(g, f[2], ci, 1))
            p["bn%s_branch1" % nm] = _bn(g, f[2], 0.7)
        ci = f[2]
    p["output"] = None                     # its width depends on the image size: filled in by the caller
    return p, _randn(g, c["N"], 3, c["HW"], c["HW"]), g


def _resnet_head(g, n_in):
    return _randn(g, n_in, 1000, std=0.5 * (1.0 / n_in) ** 0.5), _randn(g, 1000, std=0.02)


def _bert_in(c, seed):
    g = _gen(seed)
    n_tok = c["B"] * c["T"]
    n_masked = max(8, int(n_tok * 0.15) // 8 * 8)
    tok = torch.randint(0, c["vocab"], (c["B"], c["T"]), generator=g, device=DEV)
    pos = torch.randperm(n_tok, generator=g, device=DEV)[:n_masked].sort().values
    return g, tok, pos, tok.reshape(-1)[pos]


def _bert_params(c, g, shapes):
    """Variables by name, as in the middle of training: biases are not zero, gains not one."""
    out = {}
    for name, shape in shapes:
        t = _randn(g, *shape, std=0.02)
        if "gamma" in name:
            t = t + 1.0
        elif name == "mlm/decoder_W":
            t[:, c["vocab"]:] = 0.0
        elif name == "mlm/decoder_b":
            t[c["vocab"]:] = -30000.0
        out[name] = t
    return out


def _bert_shapes(c):
    H, ffn, V = c["hidden"], 4 * c["hidden"], (c["vocab"] + 7) // 8 * 8
    s = [("embeddings/word", (c["vocab"], H)), ("embeddings/position", (512, H)), ("embeddings/ln_gamma", (H,)), ("embeddings/ln_beta", (H,))]
    for l in range(c["layers"]):
        p = "layer%d/" % l
        s += [(p + "attn/Wqkv", (H, 3 * H)), (p + "attn/bqkv", (3 * H,)), (p + "attn/Wo", (H, H)), (p + "attn/bo", (H,)),
              (p + "ln1_gamma", (H,)), (p + "ln1_beta", (H,)), (p + "ffn/W1", (H, ffn)), (p + "ffn/b1", (ffn,)),
              (p + "ffn/W2", (ffn, H)), (p + "ffn/b2", (H,)), (p + "ln2_gamma", (H,)), (p + "ln2_beta", (H,))]
    return s + [("mlm/transform_W", (H, H)), ("mlm/transform_b", (H,)), ("mlm/ln_gamma", (H,)), ("mlm/ln_beta", (H,)),
                ("mlm/decoder_W", (H, V)), ("mlm/decoder_b", (V,))]


def _codec_in(c, seed):
    g = _gen(seed)
    grad = _randn(g, c["n"], std=1e-3)
    # two-sided tail of a normal distribution
    tau = 1e-3 * math.sqrt(2.0) * float(torch.erfinv(torch.tensor(1.0 - c["density"], dtype=F64)))
    return grad, _randn(g, c["n"], std=1e-3), float(torch.tensor(tau, dtype=F32))


# ------------------------------------------------------------------------------------------------ prepare / run
def _start(net):
    net.device = torch.device(DEV)
    return net.init()


def prepare(case, seed):
    c = case
    kind = c["kind"]
    st = {"case": c}
    if kind == "mlp":
        Ws, bs, x, y = _mlp_in(c, seed)
        b = nn.NeuralNetConfiguration.Builder().seed(123).updater(nn.Adam(1e-3))
        if c["dtype"] == "bfloat16":
            b = b.computeDataType(DataType.BFLOAT16)
        net = _start(nn.MultiLayerNetwork(
            b.list().layer(nn.DenseLayer(nIn=c["nIn"], nOut=c["hidden"], activation="relu"))
            .layer(nn.DenseLayer(nIn=c["hidden"], nOut=c["hidden"], activation="relu"))
            .layer(nn.OutputLayer("MCXENT", nIn=c["hidden"], nOut=c["nOut"], activation="softmax")).build()))
        net.setParams(torch.cat([t for W, bb in zip(Ws, bs) for t in (_fmat(W), bb)]))
        net.setCudaGraphs(True)
        st.update(net=net, x=x, y=y)
    elif kind == "attention":
        st["q"], st["k"], st["v"], st["mask"], st["dout"] = _attention_in(c, seed)
        st["scale"] = c["D"] ** -0.5
    elif kind == "layer_norm":
        st["x"], st["g"], st["b"], st["dy"] = _layer_norm_in(c, seed)
    elif kind == "lm_head":
        h, W, b, labels = _lm_head_in(c, seed)
        sd = SameDiff.create()
        hv = sd.placeHolder("hidden", DataType.BFLOAT16, -1, c["hidden"])
        lv = sd.placeHolder("labels", DataType.LONG, -1)
        logits = sd.nn.linear("logits", hv, sd.var("W", W), sd.var("b", b))
        sd.setLossVariables(sd.loss.sparseSoftmaxCrossEntropy("loss", logits, lv))
        sd.to(DEV)
        st.update(sd=sd, ph={"hidden": h, "labels": labels})
    elif kind in ("lstm", "rnn_step"):
        ps, x, y = _lstm_in(c, seed)
        lb = nn.NeuralNetConfiguration.Builder().seed(1).updater(nn.Adam(1e-3)).computeDataType(DataType.BFLOAT16).list()
        n_in = c["vocab"]
        for _ in range(c["layers"]):
            lb.layer(LSTM(nIn=n_in, nOut=c["hidden"], activation="TANH"))
            n_in = c["hidden"]
        lb.layer(RnnOutputLayer("MCXENT", nIn=n_in, nOut=c["vocab"], activation="SOFTMAX"))
        net = _start(nn.MultiLayerNetwork(lb.backpropType(BackpropType.TruncatedBPTT).tBPTTForwardLength(50).tBPTTBackwardLength(50).build()))
        net.setParams(torch.cat([t for p in ps for t in [_fmat(m) if m.dim() == 2 else m for m in p]]))
        if kind == "lstm":
            net.setCudaGraphs(True)
        st.update(net=net, x=x, y=y)
    elif kind == "conv_block":
        ps, out, x, y = _conv_block_in(c, seed)
        w = c["width"]
        gb = (nn.NeuralNetConfiguration.Builder().seed(1).updater(nn.Nesterovs(0.01, 0.9)).activation("IDENTITY")
              .convolutionMode(ConvolutionMode.Same).computeDataType(DataType.BFLOAT16).graphBuilder())
        gb.addInputs("input").setInputTypes(InputType.convolutional(c["HW"], c["HW"], 3))
        prev = "input"
        for i, (co, k) in enumerate(((4 * w, 3), (w, 1), (w, 3), (4 * w, 1))):
            gb.addLayer("conv%d" % i, ConvolutionLayer([k, k], nOut=co), prev)
            gb.addLayer("bn%d" % i, BatchNormalization(), "conv%d" % i)
            prev = "bn%d" % i
            if i < 3:
                gb.addLayer("act%d" % i, ActivationLayer("RELU"), prev)
                prev = "act%d" % i
        gb.addVertex("add", ElementWiseVertex("Add"), "bn3", "act0")
        gb.addLayer("act3", ActivationLayer("RELU"), "add")
        gb.addLayer("pool", GlobalPoolingLayer(PoolingType.AVG), "act3")
        gb.addLayer("output", OutputLayer("MCXENT", nOut=c["classes"], activation="SOFTMAX"), "pool")
        net = _start(ComputationGraph(gb.setOutputs("output").build()))
        parts = []
        for (b, W), bn in ps:
            parts += [b, W.reshape(-1)] + list(bn)
        net.setParams(torch.cat(parts + [_fmat(out[0]), out[1]]))
        net.setCudaGraphs(True)
        st.update(net=net, x=x, y=y)
    elif kind == "resnet50":
        p, x, g = _resnet_in(c, seed)
        net = _start(ComputationGraph(ResNet50(numClasses=1000, inputShape=[3, c["HW"], c["HW"]], updater=nn.Nesterovs(0.01, 0.9),
                                               computeDataType=DataType.BFLOAT16).conf()))
        table = net.paramTable()           # "<vertex>_<parameter>", in the order of the flat vector
        p["output"] = _resnet_head(g, table["output_W"].shape()[0])
        parts = []
        for key in table:
            vertex, name = key.rsplit("_", 1)
            k = {"b": 1 if vertex == "output" else 0, "W": 0 if vertex == "output" else 1, "gamma": 0, "beta": 1, "mean": 2, "log10stdev": 3}[name]
            t = p[vertex][k]
            parts.append(_fmat(t) if t.dim() == 2 else t.reshape(-1))
        net.setParams(torch.cat(parts))
        st.update(net=net, x=x)
    elif kind == "bert":
        g, tok, pos, lab = _bert_in(c, seed)
        cfg = BertConfig(vocabSize=c["vocab"], hidden=c["hidden"], layers=c["layers"], heads=c["heads"], ffn=4 * c["hidden"])
        sd = build_bert_mlm(cfg, c["B"], c["T"], nn.Adam(1e-4), DataType.BFLOAT16).to(DEV)
        for name, t in _bert_params(c, g, _bert_shapes(c)).items():
            sd.setArrayForVariable(name, t)
        sd.getTrainingConfig().cudaGraphs = True
        st.update(sd=sd, ph={"tokens": tok, "maskedPositions": pos, "maskedLabels": lab}, names=[n for n, _ in _bert_shapes(c)])
    elif kind == "codec":
        st["grad"], st["target"], st["tau"] = _codec_in(c, seed)
    else:
        raise ValueError(kind)
    return st


def run(state):
    st, c = state, state["case"]
    kind = c["kind"]
    if kind in ("mlp", "lstm", "conv_block"):
        net = st["net"]
        net.fit(st["x"], st["y"])
        return {"score": net.score(), "params": net.params().t}
    if kind == "attention":
        if c["train"]:
            dq, dv, dk = Nd4j.exec("dot_product_attention_v2_bp", st["q"], st["v"], st["k"], st["dout"], vMask=st["mask"],
                                   scale=st["scale"], useCausalMask=c["causal"])
            return {"dq": dq.t, "dk": dk.t, "dv": dv.t}
        return {"out": Nd4j.exec("dot_product_attention_v2", st["q"], st["v"], st["k"], None, None, st["mask"], scale=st["scale"],
                                 useCausalMask=c["causal"]).t}
    if kind == "layer_norm":
        dx, dg, db = Nd4j.exec("layer_norm_bp", st["x"], st["g"], st["b"], st["dy"])
        return {"dx": dx.t, "dgain": dg.t, "dbias": db.t}
    if kind == "lm_head":
        g = st["sd"].calculateGradients(st["ph"], "hidden", "W", "b")
        return {k: v.t for k, v in g.items()}
    if kind == "rnn_step":
        net = st["net"]
        out = {"probabilities": net.rnnTimeStep(st["x"]).t}
        for i in range(c["layers"]):
            out["h%d" % i], out["c%d" % i] = net.rnnGetPreviousState(i)
        return out
    if kind == "resnet50":
        return {"probabilities": st["net"].output(st["x"])[0].t}
    if kind == "bert":
        hist = st["sd"].fit(st["ph"], 1)
        return {"loss": hist.losses[-1][-1], "variables": {n: st["sd"].getVariable(n).getArr().t for n in st["names"]}}
    if c["form"] == "bitmap":
        residual, msg, count = Nd4j.exec("encode_bitmap", st["grad"], threshold=st["tau"])
        return {"residual": residual.t, "message": msg.t, "count": count.t,
                "decoded": Nd4j.exec("decode_bitmap", st["target"], msg).t}
    residual, msg = Nd4j.exec("encode_threshold", st["grad"], threshold=st["tau"])
    return {"residual": residual.t, "decoded": Nd4j.exec("decode_threshold", st["target"], msg).t}


# ------------------------------------------------------------------------------------------------ work
def _lstm_work(c, T, train):
    n, v, L, mb = c["hidden"], c["vocab"], c["layers"], c["mb"]
    weights = sum((v if i == 0 else n) * 4 * n + n * 4 * n for i in range(L)) + n * v
    flops = 2.0 * mb * T * weights * (3 if train else 1)
    act = mb * T * (2 * v * 4 + L * n * (2 + 4 + 8)) if train else mb * (2 * v * 4 + L * n * 12)
    segments = math.ceil(T / 50)
    return {"bytes": float(weights * 24 * segments + act if train else weights * 2 + act), "flops": flops}


def work(case):
    c = case
    kind = c["kind"]
    if kind == "mlp":
        n = c["nIn"] * c["hidden"] + c["hidden"] ** 2 + c["hidden"] * c["nOut"] + 2 * c["hidden"] + c["nOut"]
        return {"bytes": 24.0 * n + 4.0 * c["batch"] * (c["nIn"] + c["nOut"]), "flops": 6.0 * c["batch"] * n}
    if kind == "attention":
        B, H, Tq, Tk, D = (c[k] for k in ("B", "H", "Tq", "Tk", "D"))
        pairs = B * H * (Tq * Tk if not c["causal"] else Tq * (Tq + 1) / 2)
        q, kv = 2.0 * B * H * Tq * D, 2.0 * B * H * Tk * D
        # forward: S, PV; the gradient op computes the forward too: + dV, dP, dQ, dK
        return {"bytes": (3 * q + 4 * kv) if c["train"] else (2 * q + 2 * kv), "flops": (12.0 if c["train"] else 4.0) * pairs * D}
    if kind == "layer_norm":
        e = 2 if c["dtype"] == "bfloat16" else 4
        return {"bytes": 3.0 * e * c["rows"] * c["C"] + 16.0 * c["C"], "flops": 16.0 * c["rows"] * c["C"]}
    if kind == "lm_head":
        R, H, V = c["rows"], c["hidden"], c["vocab"]
        return {"bytes": 2.0 * (2 * R * H + 2 * H * V + 2 * V), "flops": 6.0 * R * H * V}
    if kind == "lstm":
        return _lstm_work(c, c["T"], True)
    if kind == "rnn_step":
        return _lstm_work(c, 1, False)
    if kind == "conv_block":               # activations: written forward, read and differentiated backward
        w, px = c["width"], c["N"] * c["HW"] ** 2
        macs = px * (27 * 4 * w + 4 * w * w + 9 * w * w + 4 * w * w)
        acts = px * w * (4 + 1 + 1 + 4)
        return {"bytes": 4.0 * 3 * px + 2.0 * 4 * acts, "flops": 6.0 * macs}
    if kind == "resnet50":
        macs, ci, hw = 0, 64, (c["HW"] + 6 - 7) // 2 + 1
        macs += hw * hw * 64 * 147
        acts = hw * hw * 64
        hw, nparam = (hw - 3) // 2 + 1, 64 * 147
        for f, s, proj in _resnet_blocks():
            hw = (hw - 1) // s + 1
            m = ci * f[0] + 9 * f[0] * f[1] + f[1] * f[2] + (ci * f[2] if proj else 0)
            macs += hw * hw * m
            nparam += m
            acts += hw * hw * (f[0] + f[1] + f[2])
            ci = f[2]
        return {"bytes": c["N"] * (12.0 * c["HW"] ** 2 + 4.0 * acts) + 2.0 * nparam, "flops": 2.0 * c["N"] * macs}
    if kind == "bert":
        n_tok, H, T = c["B"] * c["T"], c["hidden"], c["T"]
        n_masked = max(8, int(n_tok * 0.15) // 8 * 8)
        n_par = sum(math.prod(s) for _, s in _bert_shapes(c))
        flops = 6.0 * n_tok * c["layers"] * 12 * H * H + 12.0 * n_tok * T * H * c["layers"] + 6.0 * n_masked * (H * H + H * c["vocab"])
        return {"bytes": 24.0 * n_par + 2.0 * n_tok * H * (c["layers"] * 34 + 4), "flops": flops}
    n = c["n"]
    if c["form"] == "bitmap":
        return {"bytes": 4.0 * 4 * n + 2 * n / 4.0, "flops": 4.0 * n}
    return {"bytes": 4.0 * 4 * n + 8.0 * c["density"] * n, "flops": 4.0 * n}


# ------------------------------------------------------------------------------------------------ tolerance
def tolerance(case):
    """About four times the error against 64 bits (or between summation orders) that the data types give at these sizes."""
    c = case
    kind = c["kind"]
    if kind == "codec":
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "mlp":                         # weights after an Adam step: a gradient near zero may change its sign
        return {"rel": 1e-2, "max": 0.2} if c["dtype"] == "bfloat16" else {"rel": 2e-5, "max": 0.05}
    if kind == "layer_norm":
        return {"rel": 7e-3, "max": 0.1} if c["dtype"] == "bfloat16" else {"rel": 1e-5, "max": 1e-3}
    if kind == "attention":
        return {"rel": 1.5e-2, "max": 0.25}
    if kind == "lm_head":
        return {"rel": 1.2e-2, "max": 0.4}
    if kind == "lstm":
        return {"rel": 1e-2, "max": 0.4}
    if kind == "rnn_step":
        return {"rel": 1.4e-2, "max": 0.2}
    if kind == "conv_block":                  # weights after a Nesterov step, running statistics among them
        return {"rel": 5e-4, "max": 0.05}
    if kind == "resnet50":
        return {"rel": 1e-2, "max": 0.15}
    return {"rel": 3e-3, "max": 0.3}          # bert: weights after one step


# ------------------------------------------------------------------------------------------------ 64-bit values
def _adam(p, g, m, v, t, lr):
    m = 0.9 * m + 0.1 * g
    v = 0.999 * v + 0.001 * g * g
    e = lr * math.sqrt(1 - 0.999 ** t) / (1 - 0.9 ** t)
    return p - e * m / (v.sqrt() + 1e-8), m, v


def _leaf(t):
    return t.double().requires_grad_(True)


def _layer_norm64(x, g, b):
    m = x.mean(-1, keepdim=True)
    v = (x - m).square().mean(-1, keepdim=True)
    return (x - m) / (v + 1e-5).sqrt() * g + b


def _attend64(q, k, v, scale, mask=None, causal=False):
    s = q @ k.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    if mask is not None:
        s = s.masked_fill(mask[:, None, None, :] == 0, float("-inf"))
    return torch.softmax(s, -1) @ v


def _lstm64(ps, x, state):
    """[mb, vocab, T] -> logits [mb, vocab, T] and the carried state."""
    h_all, new = x.permute(2, 0, 1), []
    for (W, R, b), (h, c) in zip(ps[:-1], state):
        z_in, n, outs = h_all @ W + b, R.shape[0], []
        for t in range(h_all.shape[0]):
            z = z_in[t] + h @ R
            a, f, o, i = torch.tanh(z[:, :n]), torch.sigmoid(z[:, n:2 * n]), torch.sigmoid(z[:, 2 * n:3 * n]), torch.sigmoid(z[:, 3 * n:])
            c = f * c + i * a
            h = o * torch.tanh(c)
            outs.append(h)
        h_all = torch.stack(outs)
        new.append((h, c))
    W, b = ps[-1]
    return (h_all @ W + b).permute(1, 2, 0), new


def exact(case, seed):
    c = case
    kind = c["kind"]
    with torch.enable_grad():
        return {"mlp": _exact_mlp, "attention": _exact_attention, "layer_norm": _exact_layer_norm, "lm_head": _exact_lm_head,
                "lstm": _exact_lstm, "rnn_step": _exact_rnn_step, "conv_block": _exact_conv_block, "resnet50": _exact_resnet50,
                "bert": _exact_bert, "codec": _exact_codec}[kind](c, seed)


def _exact_mlp(c, seed):
    Ws, bs, x, y = _mlp_in(c, seed)
    Ws, bs = [_leaf(W) for W in Ws], [_leaf(b) for b in bs]
    h = x.double()
    for i, (W, b) in enumerate(zip(Ws, bs)):
        h = h @ W + b
        h = torch.relu(h) if i < 2 else h
    loss = -(y.double() * torch.log_softmax(h, 1)).sum() / c["batch"]
    loss.backward()
    out = []
    for W, b in zip(Ws, bs):
        for t in (W, b):
            p = _adam(t.detach(), t.grad, 0.0, 0.0, 1, 1e-3)[0]
            out.append(_fmat(p) if p.dim() == 2 else p)
    return {"score": float(loss.detach()), "params": torch.cat(out)}


def _exact_attention(c, seed):
    q, k, v, mask, dout = _attention_in(c, seed)
    scale, outs = c["D"] ** -0.5, []
    for b in range(c["B"]):                    # one sequence at a time: the score matrix in 64 bits is large
        qq, kk, vv = (_leaf(t[b:b + 1]) for t in (q, k, v))
        o = _attend64(qq, kk, vv, scale, None if mask is None else mask[b:b + 1], c["causal"])
        outs.append(torch.autograd.grad(o, (qq, kk, vv), dout[b:b + 1].double()) if c["train"] else (o.detach(),))
    outs = [torch.cat(t) for t in zip(*outs)]
    return dict(zip(("dq", "dk", "dv"), outs)) if c["train"] else {"out": outs[0]}


def _exact_layer_norm(c, seed):
    x, g, b, dy = _layer_norm_in(c, seed)
    x, g, b = _leaf(x), _leaf(g), _leaf(b)
    dx, dg, db = torch.autograd.grad(_layer_norm64(x, g, b), (x, g, b), dy.double())
    return {"dx": dx, "dgain": dg, "dbias": db}


def _exact_lm_head(c, seed):
    h, W, b, labels = _lm_head_in(c, seed)
    h, W, b = _leaf(h), _leaf(W), _leaf(b)
    g = torch.autograd.grad(F.cross_entropy(h @ W + b, labels), (h, W, b))
    return dict(zip(("hidden", "W", "b"), g))


def _zero_state(c):
    z = torch.zeros(c["mb"], c["hidden"], dtype=F64, device=DEV)
    return [(z, z) for _ in range(c["layers"])]


def _exact_lstm(c, seed):
    ps, x, y = _lstm_in(c, seed)
    ps = [[_leaf(t) for t in p] for p in ps]
    mv = [[(0.0, 0.0) for _ in p] for p in ps]
    state = _zero_state(c)
    for k, s in enumerate(range(0, c["T"], 50)):
        xs, ys = x[:, :, s:s + 50].double(), y[:, :, s:s + 50].double()
        logits, state = _lstm64(ps, xs, state)
        loss = -(ys * torch.log_softmax(logits, 1)).sum() / c["mb"]
        loss.backward()
        state = [(h.detach(), cc.detach()) for h, cc in state]
        for i, p in enumerate(ps):
            for j, t in enumerate(p):
                new, m, v = _adam(t.detach(), t.grad, *mv[i][j], k + 1, 1e-3)
                mv[i][j] = (m, v)
                p[j] = new.requires_grad_(True)
    return {"score": float(loss.detach()),
            "params": torch.cat([_fmat(t.detach()) if t.dim() == 2 else t.detach() for p in ps for t in p])}


def _exact_rnn_step(c, seed):
    ps, x, _ = _lstm_in(c, seed)
    logits, state = _lstm64([[t.double() for t in p] for p in ps], x.double()[:, :, None], _zero_state(c))
    out = {"probabilities": torch.softmax(logits, 1)[:, :, 0]}
    for i, (h, cc) in enumerate(state):
        out["h%d" % i], out["c%d" % i] = h, cc
    return out


def _exact_conv_block(c, seed):
    ps, out, x, y = _conv_block_in(c, seed)
    leaves, stats = [(_leaf(W), _leaf(bn[0]), _leaf(bn[1])) for (_, W), bn in ps], {}
    Wo, bo = _leaf(out[0]), _leaf(out[1])

    def conv_bn(i, h):
        W, g, b = leaves[i]
        z = F.conv2d(h, W, padding=W.shape[2] // 2)
        m = z.mean((0, 2, 3), keepdim=True)
        v = (z - m).square().mean((0, 2, 3), keepdim=True)
        (bias, _), (_, _, mean, ls) = ps[i]
        var = 0.9 * 10.0 ** (2 * ls.double()) + 0.1 * v.detach().flatten()
        stats[i] = [0.9 * mean.double() + 0.1 * (m.detach().flatten() + bias.double()), 0.5 * torch.log10(var)]
        return (z - m) / (v + 1e-5).sqrt() * g[None, :, None, None] + b[None, :, None, None]
    a0 = torch.relu(conv_bn(0, x.double()))
    a = torch.relu(conv_bn(2, torch.relu(conv_bn(1, a0))))
    a = torch.relu(conv_bn(3, a) + a0).mean((2, 3))
    loss = -(y.double() * torch.log_softmax(a @ Wo + bo, 1)).sum() / c["N"]
    loss.backward()
    step = lambda t: t.detach() - 1.9 * 0.01 * t.grad  # noqa: E731   (first Nesterov step, momentum 0.9)
    new = []
    for i, (W, g, b) in enumerate(leaves):     # a bias in front of a batch norm has no gradient
        new += [ps[i][0][0].double(), step(W).reshape(-1), step(g), step(b)] + stats[i]
    return {"score": float(loss.detach()), "params": torch.cat(new + [_fmat(step(Wo)), step(bo)])}


def _exact_resnet50(c, seed):
    p, x, g = _resnet_in(c, seed)

    def conv_bn(cn, bn, h, stride=1, pad=0):
        b, W = p[cn]
        gamma, beta, mean, ls = (t.double()[None, :, None, None] for t in p[bn])
        z = F.conv2d(h, W.double(), b.double(), stride, pad)
        return (z - mean) / (10.0 ** (2 * ls) + 1e-5).sqrt() * gamma + beta
    with torch.no_grad():
        h = torch.relu(conv_bn("stem-cnn1", "stem-batch1", x.double(), 2, 3))
        h = F.max_pool2d(h, 3, 2)
        for (_, s, proj), nm in zip(_resnet_blocks(), _resnet_names()):
            a = torch.relu(conv_bn("res%s_branch2a" % nm, "bn%s_branch2a" % nm, h, s))
            a = torch.relu(conv_bn("res%s_branch2b" % nm, "bn%s_branch2b" % nm, a, 1, 1))
            a = conv_bn("res%s_branch2c" % nm, "bn%s_branch2c" % nm, a)
            h = torch.relu(a + (conv_bn("res%s_branch1" % nm, "bn%s_branch1" % nm, h, s) if proj else h))
        h = F.max_pool2d(h, 3, 2).flatten(1)
        W, b = _resnet_head(g, h.shape[1])
        return {"probabilities": torch.softmax(h @ W.double() + b.double(), 1)}


def _exact_bert(c, seed):
    g, tok, pos, lab = _bert_in(c, seed)
    P = {k: _leaf(v) for k, v in _bert_params(c, g, _bert_shapes(c)).items()}
    B, T, H, nh = c["B"], c["T"], c["hidden"], c["heads"]
    gelu = lambda z: z * torch.sigmoid(1.702 * z)  # noqa: E731
    x = P["embeddings/word"][tok.reshape(-1)] + P["embeddings/position"][:T].repeat(B, 1)
    x = _layer_norm64(x, P["embeddings/ln_gamma"], P["embeddings/ln_beta"])
    for l in range(c["layers"]):
        w = {k[len("layer%d/" % l):]: v for k, v in P.items() if k.startswith("layer%d/" % l)}
        qkv = (x @ w["attn/Wqkv"] + w["attn/bqkv"]).reshape(B, T, 3, nh, H // nh)
        q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
        a = _attend64(q, k, v, (H // nh) ** -0.5).permute(0, 2, 1, 3).reshape(B * T, H)
        x = _layer_norm64(x + a @ w["attn/Wo"] + w["attn/bo"], w["ln1_gamma"], w["ln1_beta"])
        h = gelu(x @ w["ffn/W1"] + w["ffn/b1"]) @ w["ffn/W2"] + w["ffn/b2"]
        x = _layer_norm64(x + h, w["ln2_gamma"], w["ln2_beta"])
    hm = _layer_norm64(gelu(x[pos] @ P["mlm/transform_W"] + P["mlm/transform_b"]), P["mlm/ln_gamma"], P["mlm/ln_beta"])
    loss = F.cross_entropy(hm @ P["mlm/decoder_W"] + P["mlm/decoder_b"], lab)
    loss.backward()
    return {"loss": float(loss.detach()), "variables": {k: _adam(v.detach(), v.grad, 0.0, 0.0, 1, 1e-4)[0] for k, v in P.items()}}


def _exact_codec(c, seed):
    grad, target, tau = _codec_in(c, seed)
    x, t = grad.double(), target.double()
    big = x.abs() >= tau
    step = torch.where(big, torch.sign(x) * tau, torch.zeros_like(x))
    if c["form"] == "bitmap":
        step = torch.where(~big & (x < 0) & (x.abs() >= tau / 2), torch.full_like(x, -tau / 2), step)
        return {"residual": x - step, "message": None, "count": None, "decoded": t + step}
    return {"residual": x - step, "decoded": t + step}
