"""The CTA-pair GEMM (csrc/gemm_pair.cu): rows and columns around its 256 x 256 tiles, short and long K, every epilogue.

Bound: results are rounded to bf16 once (2^-9 at most, 1.7e-3 rms for random values); sums are fp32."""
import math

import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def _rel(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / b.norm().clamp_min(1e-9)).item()


@pytest.mark.parametrize("M,N,K", [(513, 8, 64), (600, 264, 128), (768, 256, 64), (1023, 520, 4096), (1025, 6144, 192), (130, 10256, 320), (4097, 1000, 448)])
def test_plain(M, N, K):
    x = torch.randn(M, K, device=DEV, dtype=BF)
    w = (torch.randn(N, K, device=DEV) / math.sqrt(K)).to(BF)
    b, r = torch.randn(N, device=DEV, dtype=BF), torch.randn(M, N, device=DEV, dtype=BF)
    assert _rel(ops.linear(x, w), ref.linear(x.float(), w.float())) < 3e-3
    assert _rel(ops.linear(x, w, b, residual=r), ref.linear(x.float(), w.float(), b.float()) + r.float()) < 3e-3


@pytest.mark.parametrize("act", ["silu_mul", "gelu_tanh_mul", "gelu_mul"])
@pytest.mark.parametrize("M,I,K", [(513, 8, 64), (777, 200, 256), (129, 5128, 128), (1000, 1344, 2048), (2049, 72, 64)])
def test_gate_product(M, I, K, act):
    x = torch.randn(M, K, device=DEV, dtype=BF)
    w = (torch.randn(2 * I, K, device=DEV) / math.sqrt(K)).to(BF)
    b = torch.randn(2 * I, device=DEV, dtype=BF)
    assert _rel(ops.linear(x, w, b, act=act), ref.linear(x.float(), w.float(), b.float(), act=act)) < 3e-3
