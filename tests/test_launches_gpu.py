"""Kernels that are launched behind one another, as other programs launch them: captured into a CUDA
graph, on several streams and from several threads. Each result is held to the same calls made one
after the other with a synchronization between them.
"""

import threading

import pytest
import torch

from mmh3_b200 import attention, gemm, synthetic
from mmh3_b200.gemm import ColumnMaxima, Output

pytestmark = pytest.mark.gpu

HEAD_DIM = 128
SCALE = synthetic.softmax_scale()


class Layer:
    """An attention layer: the qkv projection, then norm and RoPE and BF16 attention, or the fused
    input pass and INT8/FP8 attention over the maxima of |v| that the projection leaves."""

    def __init__(self, tokens, heads, hidden, quantized, seed):
        generator = torch.Generator(device="cuda").manual_seed(seed)
        inner = heads * HEAD_DIM
        self.shape = tokens, heads, hidden
        self.quantized = quantized
        self.activations = torch.empty((tokens, hidden), dtype=torch.int8, device="cuda")
        self.weights = torch.randint(-127, 128, (3 * inner, hidden), dtype=torch.int8, device="cuda",
                                     generator=generator)
        self.row_scales = torch.rand(tokens, device="cuda", generator=generator) + 0.5
        self.column_scales = (torch.rand(3 * inner, device="cuda", generator=generator) + 0.5) * 1e-5
        weight = torch.ones(HEAD_DIM, dtype=torch.bfloat16, device="cuda")
        angles = torch.rand((tokens, 64), device="cuda", generator=generator) * 6.0
        self.norm = attention.HeadNorm(weight, weight, angles, 64, 1e-6)
        self.qkv = torch.zeros((tokens, 3, heads, HEAD_DIM), dtype=torch.bfloat16, device="cuda")
        self.maxima = torch.zeros(heads, device="cuda")
        self.output = torch.zeros((tokens, heads, HEAD_DIM), dtype=torch.bfloat16, device="cuda")
        self.workspace = attention.QuantizedWorkspace(tokens, heads)

    def load(self, seed):
        generator = torch.Generator(device="cuda").manual_seed(seed)
        self.activations.copy_(torch.randint(-127, 128, self.activations.shape, device="cuda",
                                             generator=generator, dtype=torch.int8))

    def run(self, between=lambda: None):
        tokens, heads, hidden = self.shape
        self.maxima.zero_()
        between()
        gemm.int8(None, self.activations, self.weights, self.row_scales, self.column_scales,
                  Output(self.qkv.view(torch.int16),
                         column_maxima=ColumnMaxima(self.maxima, 2 * heads * HEAD_DIM)),
                  tokens, 3 * heads * HEAD_DIM, hidden)
        between()
        if self.quantized:
            attention.prepare_inputs(self.qkv, self.norm, tokens, heads, self.workspace,
                                     value_head_maxima=self.maxima)
            between()
            attention.dense_quantized(self.qkv, self.output, SCALE, self.workspace,
                                      inputs=attention.AttentionInputs.PREPARED_WITH_VALUES)
        else:
            attention.qk_norm_rope(self.qkv, self.norm, tokens, heads)
            between()
            attention.dense_bf16(self.qkv, self.output, tokens, heads, SCALE)
        between()

    def expected(self):
        self.run(torch.cuda.synchronize)
        result = self.output.clone()
        self.output.zero_()
        torch.cuda.synchronize()
        return result


@pytest.mark.parametrize("quantized", [False, True])
def test_a_captured_layer_gives_the_same_bits(quantized):
    """The layer twice in one graph, the second on a stream that forks from the first and joins it
    again, replayed over new inputs."""
    layers = [Layer(tokens, 8, 256, quantized, tokens) for tokens in (300, 1101)]
    for layer in layers:
        layer.load(1)
        layer.run()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layers[0].run()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            layers[1].run()
        layers[0].run()
        torch.cuda.current_stream().wait_stream(side)
        layers[0].run()
    for seed in (2, 3, 4):
        expected = []
        for layer in layers:
            layer.load(seed)
            expected.append(layer.expected())
        graph.replay()
        torch.cuda.synchronize()
        assert attention.take_status() == 0
        for layer, result in zip(layers, expected):
            assert torch.equal(layer.output.view(torch.int16), result.view(torch.int16))


def test_several_threads_give_the_same_bits():
    """Four threads, each on a stream of its own, every one with both kinds of layers."""
    layers = [[Layer(tokens, 4, 256, quantized, tokens) for quantized in (False, True)]
              for tokens in (200, 513, 700, 1300)]
    expected = []
    for index, pair in enumerate(layers):
        for layer in pair:
            layer.load(index)
        expected.append([layer.expected() for layer in pair])
    wrong = []

    def work(index):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    for layer, result in zip(layers[index], expected[index]):
                        layer.output.zero_()
                        layer.run()
                        if not torch.equal(layer.output.view(torch.int16),
                                           result.view(torch.int16)):
                            wrong.append((index, layer.quantized))
        except Exception as error:
            wrong.append(error)

    threads = [threading.Thread(target=work, args=(index,)) for index in range(len(layers))]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert attention.take_status() == 0
    assert not wrong
