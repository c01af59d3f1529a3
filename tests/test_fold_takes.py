"""What the folded inference convolutions accept (host rule)."""
import torch


def test_only_what_the_kernels_read():
    from deeplearning4j_b200 import nn
    from deeplearning4j_b200.nn.conf.base import InputType
    from deeplearning4j_b200.nn.graph import ComputationGraph
    from deeplearning4j_b200.nn.layers.conv import BatchNormalization, ConvolutionLayer, GlobalPoolingLayer
    from deeplearning4j_b200.nn.layers.core import OutputLayer
    gb = nn.NeuralNetConfiguration.Builder().activation("IDENTITY").graphBuilder().addInputs("in").setInputTypes(InputType.convolutional(4, 4, 16))
    gb.addLayer("c", ConvolutionLayer([1, 1], [1, 1], nOut=8), "in").addLayer("n", BatchNormalization(), "c")
    gb.addLayer("p", GlobalPoolingLayer(), "n").addLayer("out", OutputLayer("MCXENT", nOut=3, activation="SOFTMAX"), "p")
    net = ComputationGraph(gb.setOutputs("out").build()).init()
    assert "c" in net._fold_specs()
    ok = torch.zeros(2, 16, 4, 4, dtype=torch.bfloat16, device=net.flat_params.device)
    assert net._fold_takes("c", ok)
    for bad in (ok[:, :8], torch.cat([ok, ok], 1), ok.float(), ok.half(), ok[0], ok[:0], ok.to("meta")):
        assert not net._fold_takes("c", bad)
