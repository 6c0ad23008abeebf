"""1 .. 8 rows of more than 14336 columns: the streaming GEMV normalises and converts a row in rounds of 14336 columns (csrc/gemv2_body.cuh).

Bounds: products and sums are fp32.  8-bit weights: rows in f16 (2^-11), result in bf16 (1.7e-3 rms).  A norm: x gamma is rounded to bf16 too before the product."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16
TYPES = [BF, torch.int8, torch.float8_e4m3fn]


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-9)).item()


def _layer(T, N, K, wdtype):
    x, w, n = torch.randn(T, K, device=DEV, dtype=BF), torch.randn(N, K, device=DEV) / K ** 0.5, torch.randn(K, device=DEV, dtype=BF)
    x[:, -(K // 8):] *= 3                      # columns that are left out show
    q, s = (w.to(BF), None) if wdtype == BF else ref.quantize_per_channel(w, wdtype)
    return x, q, s, n, q.double() if s is None else q.double() * s.double().view(-1, 1)


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T,K", [(1, 14336), (2, 14464), (5, 14464), (1, 16384), (2, 16384), (3, 16384), (5, 16384), (4, 18432), (1, 28672), (2, 28672), (3, 28672), (1, 28800),
                                 (1, 43136), (1, 87040)])
@pytest.mark.parametrize("N", [64, 2064])
def test_every_column_counts(wdtype, T, K, N):
    x, q, s, n, w = _layer(T, N, K, wdtype)
    h = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * n.double()
    assert _rel(ops.linear(x, q, scale=s), x.double() @ w.t()) < 3e-3
    assert _rel(ops.linear(x, q, scale=s, act="silu_mul"), ref.linear(x.double(), w, act="silu_mul")) < 5e-3
    assert _rel(ops.linear(x, q, norm_weight=n, norm_eps=1e-5, scale=s), h @ w.t()) < 6e-3
    assert _rel(ops.linear(x, q, norm_weight=n, norm_eps=1e-5, scale=s, act="silu_mul"), ref.linear(h, w, act="silu_mul")) < 1e-2


@pytest.mark.parametrize("T,K", [(1, 87296), (2, 43776), (2, 54016), (3, 28928), (4, 22016), (4, 26880), (5, 17664), (5, 18432), (6, 16640), (6, 17920)])
@pytest.mark.parametrize("N", [64, 2064])
def test_norm_of_rows_wider_than_the_norm_kernel_takes(T, K, N):
    """Rows above 16384 columns that the streaming kernel has no shared memory for: the kernel that normalises them itself."""
    x, w, _, n, wd = _layer(T, N, K, BF)
    h = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * (n.double() + 1)
    r = torch.randn(T, N, device=DEV, dtype=BF)
    assert _rel(ops.linear(x, w, norm_weight=n, norm_eps=1e-5, norm_offset=1.0, residual=r), h @ wd.t() + r.double()) < 6e-3
    assert _rel(ops.linear(x, w, norm_weight=n, norm_eps=1e-5, norm_offset=1.0, act="silu_mul"), ref.linear(h, wd, act="silu_mul")) < 1e-2
