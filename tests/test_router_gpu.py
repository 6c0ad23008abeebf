"""fp32 router on tensor cores (csrc/router_tc.cu; choice: csrc/moe_plain.cu): logits against 64 bits at the edges of its blocks and column parts; choice and weights against the definition.

Bound: products of bf16 rows and split fp32 weights are exact in fp32, sums of at most 64 go through the tensor core (its adder drops bits below
2^-23 of the running sum: 64 * 2^-23 relative at worst, 1e-7 seen), the rest are fp32 additions; 1e-6 is asked for."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.modules.moe import RouterTopK
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 255, 256, 257, 1000, 4097])
@pytest.mark.parametrize("E,W", [(8, 512), (64, 64), (65, 128), (128, 2048), (300, 192), (512, 1088)])
def test_logits_and_choice(N, E, W):
    x = torch.randn(N, W, device="cuda", dtype=torch.bfloat16)
    w, b = torch.randn(E, W, device="cuda") * 0.05, torch.randn(E, device="cuda")
    k = min(8, E)
    for bias in (None, b):
        logits, weights, ids = ops.router_topk(x, w, k, bias=bias)
        exact = x.double() @ w.double().t() + (0 if bias is None else bias.double())
        assert ((logits.double() - exact).norm() / exact.norm()).item() < 1e-6
        want_w, want_i = ref.moe_route(logits, k)
        assert torch.equal(ids.long().sort(-1).values, want_i.sort(-1).values)
        assert torch.allclose(weights.sort(-1).values, want_w.sort(-1).values, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N", [1, 32, 33, 300, 4737])
@pytest.mark.parametrize("E,W", [(1, 4), (4, 516), (5, 4096), (8, 132), (9, 1028), (16, 6144), (8, 130)])
def test_few_experts_share_the_columns(N, E, W, dtype):
    """Up to 16 experts: the warps of a block share the columns.  fp32 sums of W terms in 32 lanes and up to 4 parts: at most W / 128 + 9 additions in a
    row, 57 * 2^-24 = 3.4e-6 at worst of the terms' size (4e-7 seen); 1e-6 of the result is asked for."""
    x = torch.randn(N, W, device="cuda", dtype=dtype)
    w = torch.randn(E, W, device="cuda") * 0.05
    logits, weights, ids = ops.router_topk(x, w, min(2, E))
    exact = x.double() @ w.double().t()
    assert ((logits.double() - exact).norm() / exact.norm()).item() < 1e-6
    want_w, want_i = ref.moe_route(logits, min(2, E))
    assert torch.equal(ids.long().sort(-1).values, want_i.sort(-1).values)
    assert torch.allclose(weights.sort(-1).values, want_w.sort(-1).values, rtol=1e-5, atol=1e-7)


def test_module_ids_keep_their_type():
    r = RouterTopK(16, 2, 256, device="cuda")
    r.linear_router.weight.data.normal_()
    x = torch.randn(5, 256, device="cuda", dtype=torch.bfloat16)
    assert r(x)[2].dtype == torch.int64 and ops.router_topk(x, r.linear_router.weight, 2)[2].dtype == torch.int64
    assert ops.router_topk(x, r.linear_router.weight, 2, "sigmoid")[2].dtype == torch.int32


@pytest.mark.parametrize("N", [1, 5, 32, 33, 100, 203, 204, 255, 256])
@pytest.mark.parametrize("E,W,k", [(5, 64, 2), (8, 4096, 2), (16, 516, 4), (17, 128, 4), (128, 2048, 8), (127, 260, 8), (512, 1024, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_split_columns(N, E, W, k, dtype):
    """Experts over the grid's second dimension, four and eight warps per four of them, ragged counts on both; rows that the kernel in front is still writing."""
    base = torch.randn(N, W, device="cuda", dtype=dtype)
    w = torch.randn(E, W, device="cuda") / W ** 0.5
    for i in range(3):
        x = base * (i + 1)                              # a kernel of the same stream
        logits, tw, ti = ops.router_topk(x, w, k)
        want = x.double() @ w.double().t()
        # fp32 sums of W products with independent rounding errors
        assert ((logits.double() - want).norm() / want.norm()).item() < 2e-6
        p = torch.softmax(logits.double(), -1)
        top = p.gather(1, ti.long())
        assert torch.allclose(top.sort(-1, descending=True).values, p.topk(k, -1).values, rtol=1e-5)
        assert torch.allclose(tw.double(), top / top.sum(-1, keepdim=True), rtol=1e-5)


@pytest.mark.parametrize("N,E,W", [(19, 512, 2048), (20, 512, 2048), (32, 512, 4096), (32, 384, 2052), (25, 400, 2880), (13, 512, 1024), (26, 512, 1024), (64, 206, 1024), (65, 206, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_split_columns_at_the_limits(N, E, W, dtype):
    """One or four tokens a block up to 32 tokens, and the last sizes before staged rows (tokens x experts up to 5000 + 8 W)."""
    test_split_columns(N, E, W, 8, dtype)
