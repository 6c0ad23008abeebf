"""Weight-only 8-bit layers above 8 tokens: the GEMM has to wait for the expansion of ITS weight, and the expansion for the GEMM that still reads
the memory before it.  Two different weights take turns back to back, so a GEMM that reads too early multiplies with the other one."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
TOL = 1e-2          # bf16 rows, weights and results: 2 ** -8 each


def _layer(wdtype, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return ref.quantize_per_channel(torch.randn(n, k, device="cuda", generator=g) * 0.05, wdtype)


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm()).item()


@pytest.mark.parametrize("wdtype", [torch.int8, torch.float8_e4m3fn])
@pytest.mark.parametrize("T", [9, 64, 256, 1024])       # weights as the M operand (9, 64), one-CTA tiles (256), CTA pairs (1024)
def test_two_weights_back_to_back(wdtype, T):
    n = k = 4096
    (qa, sa), (qb, sb) = _layer(wdtype, n, k, 1), _layer(wdtype, n, k, 2)
    x = torch.randn(T, k, device="cuda", dtype=torch.bfloat16)
    want_a, want_b = ref.linear(x.float(), qa, scale=sa), ref.linear(x.float(), qb, scale=sb)
    outs = [(ops.linear(x, qa, scale=sa), ops.linear(x, qb, scale=sb)) for _ in range(30)]
    for a, b in outs:
        assert _rel(a, want_a) < TOL and _rel(b, want_b) < TOL


def test_chained_layers_in_a_graph_and_on_two_streams():
    n = k = 2048
    layers = [_layer(torch.int8, n, k, s) for s in range(4)]
    x = torch.randn(40, k, device="cuda", dtype=torch.bfloat16)

    def chain(h, order):
        for i in order:
            h = ops.linear(h, layers[i][0], scale=layers[i][1])
        return h

    def want(order):
        h = x
        for i in order:
            h = ref.linear(h.float(), layers[i][0], scale=layers[i][1]).bfloat16()
        return h
    fwd, bwd = (0, 1, 2, 3), (3, 2, 1, 0)
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = []
    for _ in range(10):
        for s, order in zip(streams, (fwd, bwd)):
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                outs.append((order, chain(x, order)))
    torch.cuda.synchronize()
    for order, y in outs:
        assert _rel(y, want(order)) < 4 * TOL
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = chain(x, fwd)
    for _ in range(5):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert _rel(y, want(fwd)) < 4 * TOL
