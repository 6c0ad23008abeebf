"""Grouped CTA-pair GEMMs of the routed experts (csrc/gemm_pair.cu, csrc/moe_grouped.cu) at the edges of their 256-row tiles.

Bound: the experts' intermediate rows and the results are rounded to bf16 (2^-9 each); sums are fp32."""
import math

import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def _experts(E, H, I):
    return ((torch.randn(E, 2 * I, H, device=DEV) / math.sqrt(H)).to(BF), (torch.randn(E, H, I, device=DEV) / math.sqrt(I)).to(BF))


def _check(x, wg, wd, w, i, offset=0):
    got = ops.moe_experts(x, wg, wd, w, i, "silu_mul", offset)
    want = ref.moe_experts(x.float(), wg.float(), wd.float(), w, i, "silu_mul", offset).float()
    assert ((got.float() - want).norm() / want.norm()).item() < 5e-3
    row = (got.float() - want).norm(dim=-1) / want.norm(dim=-1).clamp_min(want.norm() / math.sqrt(len(want)) * 0.1)
    assert row.max().item() < 2e-2                # no single row of another expert


@pytest.mark.parametrize("counts", [(1, 127, 128, 129, 255, 256, 257, 0), (0, 0, 511, 512, 513, 1, 0, 2), (129, 0, 0, 0, 0, 0, 0, 0), (0, 0, 0, 0, 0, 0, 0, 300)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_segment_sizes(counts, shuffled):
    E, H, I = len(counts), 256, 192
    wg, wd = _experts(E, H, I)
    i = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)]).to(DEV).view(-1, 1)
    if shuffled:
        i = i[torch.randperm(len(i), device=DEV)]
    x, w = torch.randn(len(i), H, device=DEV, dtype=BF), torch.rand(len(i), 1, device=DEV) + 0.5
    _check(x, wg, wd, w, i)
    if counts[0]:
        _check(x, wg[1:].contiguous(), wd[1:].contiguous(), w, i, 1) if sum(counts[1:]) else None


@pytest.mark.parametrize("N", [129, 300])
def test_a_token_may_name_an_expert_again(N):
    E, k, H, I = 6, 4, 256, 192
    wg, wd = _experts(E, H, I)
    x, w = torch.randn(N, H, device=DEV, dtype=BF), torch.rand(N, k, device=DEV)
    i = torch.randint(0, E, (N, k), device=DEV)
    i[:, 1] = i[:, 0] = 3
    _check(x, wg, wd, w, i)


def test_workspaces_follow_the_entries():
    E, k, N, H, I = 256, 8, 129, 1024, 64
    wg, wd = _experts(E, H, I)
    x, w = torch.randn(N, H, device=DEV, dtype=BF), torch.rand(N, k, device=DEV)
    i = torch.rand(N, E, device=DEV).topk(k, -1).indices
    _check(x, wg, wd, w, i)
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    ops.moe_experts(x, wg, wd, w, i, "silu_mul")
    rows = 2 * N * k * (2 * H + I) + 2 * N * H               # permuted rows, products, intermediate rows and the result in bf16
    assert torch.cuda.max_memory_allocated() - base < rows + (1 << 20)


@pytest.mark.parametrize("N", [2, 16, 200])            # a warp per weight row, weights as the M operand, CTA pairs
def test_ids_of_either_width(N):
    E, k, H, I = 8, 2, 256, 192
    wg, wd = _experts(E, H, I)
    x, w = torch.randn(N, H, device=DEV, dtype=BF), torch.rand(N, k, device=DEV)
    i = torch.rand(N, E + 4, device=DEV).topk(k, -1).indices          # some experts live elsewhere
    assert torch.equal(ops.moe_experts(x, wg, wd, w, i, "silu_mul", 2), ops.moe_experts(x, wg, wd, w, i.int(), "silu_mul", 2))
    _check(x, wg, wd, w, i.int(), 2)
