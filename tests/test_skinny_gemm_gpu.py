"""The evenly split GEMM of a few tokens (csrc/skinny_gemm.cu): token counts around the instruction width, ragged feature tiles, tiles cut between
CTAs, and the routed experts of a small step.

Bound: results are rounded to bf16 once (2^-9 at most, 1.7e-3 rms); the experts' intermediate rows once more.  Sums are fp32."""
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


@pytest.mark.parametrize("T", [9, 15, 16, 17, 37, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(8, 64), (136, 128), (4104, 320), (1000, 4096), (256, 14336), (20000, 192)])
def test_plain(T, N, K):
    x = torch.randn(T, K, device=DEV, dtype=BF)
    w = (torch.randn(N, K, device=DEV) / math.sqrt(K)).to(BF)
    b, r = torch.randn(N, device=DEV, dtype=BF), torch.randn(T, N, device=DEV, dtype=BF)
    assert _rel(ops.linear(x, w), ref.linear(x.float(), w.float())) < 3e-3
    assert _rel(ops.linear(x, w, b, residual=r), ref.linear(x.float(), w.float(), b.float()) + r.float()) < 3e-3
    wide = torch.randn(T, K + 8, device=DEV, dtype=BF)[:, :K]             # rows of a wider tensor
    assert _rel(ops.linear(wide, w), ref.linear(wide.float(), w.float())) < 3e-3


@pytest.mark.parametrize("act", ["silu_mul", "gelu_tanh_mul", "gelu_mul"])
@pytest.mark.parametrize("T,I,K", [(9, 72, 64), (32, 1344, 512), (37, 14336, 4096), (64, 8640, 3904), (16, 200, 2048)])
def test_gate_product(T, I, K, act):
    x = torch.randn(T, K, device=DEV, dtype=BF)
    w = (torch.randn(2 * I, K, device=DEV) / math.sqrt(K)).to(BF)
    b = torch.randn(2 * I, device=DEV, dtype=BF)
    assert _rel(ops.linear(x, w, b, act=act), ref.linear(x.float(), w.float(), b.float(), act=act)) < 3e-3


@pytest.mark.parametrize("N", [1, 2, 3, 9, 16, 17, 100, 128])
@pytest.mark.parametrize("E,k,H,I,offset,local", [(8, 2, 256, 192, 0, 8), (128, 8, 512, 64, 32, 64), (300, 4, 128, 320, 0, 300), (4, 1, 1024, 2112, 0, 4)])
@pytest.mark.parametrize("form", ["plain", "bias", "scaled", "one expert"])
def test_experts(N, E, k, H, I, offset, local, form):
    x = torch.randn(N, H, device=DEV, dtype=BF)
    wg = (torch.randn(local, 2 * I, H, device=DEV) / math.sqrt(H)).to(BF)
    wd = (torch.randn(local, H, I, device=DEV) / math.sqrt(I)).to(BF)
    w, i = torch.topk(torch.softmax(torch.randn(N, E, device=DEV), -1), k, -1)
    if form == "one expert":
        i = torch.arange(k, device=DEV).expand(N, k) + offset
    kw, kf = {}, {}
    if form == "bias":
        bg, bd = torch.randn(local, 2 * I, device=DEV, dtype=BF), torch.randn(local, H, device=DEV, dtype=BF)
        kw, kf = dict(gate_up_bias=bg, down_bias=bd), dict(gate_up_bias=bg.float(), down_bias=bd.float())
    if form == "scaled":
        kw = kf = dict(scale_input=True)
    got = ops.moe_experts(x, wg, wd, w, i, "silu_mul", offset, **kw)
    want = ref.moe_experts(x.float(), wg.float(), wd.float(), w, i, "silu_mul", offset, **kf)
    assert got.shape == want.shape
    if want.abs().max() == 0:
        assert not got.any()
    else:
        assert _rel(got, want) < 5e-3


@pytest.mark.parametrize("N", [3, 16, 17, 33, 128])
@pytest.mark.parametrize("form", ["twice", "all slots", "shard"])
def test_a_token_may_name_an_expert_again(N, form):
    """An expert then owns up to N * k rows, more than one token tile of the GEMM holds."""
    E, k, H, I = 8, 4, 256, 192
    x = torch.randn(N, H, device=DEV, dtype=BF)
    wg = (torch.randn(E, 2 * I, H, device=DEV) / math.sqrt(H)).to(BF)
    wd = (torch.randn(E, H, I, device=DEV) / math.sqrt(I)).to(BF)
    w = torch.rand(N, k, device=DEV)
    i = torch.randint(0, E, (N, k), device=DEV)
    offset = 2 if form == "shard" else 0
    if form == "all slots":
        i[:] = 5
    else:
        i[:, 1] = i[:, 0] = 3
    wg, wd = wg[:E - offset].contiguous(), wd[:E - offset].contiguous()
    got = ops.moe_experts(x, wg, wd, w, i, "silu_mul", offset)
    want = ref.moe_experts(x.float(), wg.float(), wd.float(), w, i, "silu_mul", offset)
    assert _rel(got, want) < 5e-3


@pytest.mark.parametrize("T", [6, 7, 8, 24, 25, 41, 96])
@pytest.mark.parametrize("form", ["residual", "norm", "gate product"])
def test_groups_of_eight_tokens(T, form):
    """Rows of 6 .. 8 tokens that fill the streaming kernel's shared memory, and token counts around the epilogue's groups."""
    K = 16384 if form == "norm" else 14336
    x = torch.randn(T, K, device=DEV, dtype=BF)
    w = (torch.randn(1040, K, device=DEV) / math.sqrt(K)).to(BF)
    kw, kf = {}, {}
    if form == "residual":
        r, b = torch.randn(T, 1040, device=DEV, dtype=BF), torch.randn(1040, device=DEV, dtype=BF)
        kw, kf = dict(residual=r, bias=b), dict(residual=r.float(), bias=b.float())
    if form == "norm":
        n = torch.randn(K, device=DEV, dtype=BF)
        kw, kf = dict(norm_weight=n, norm_eps=1e-5), dict(norm_weight=n.float(), norm_eps=1e-5)
    if form == "gate product":
        kw = kf = dict(act="silu_mul")
    res = kf.get("residual")
    want = ref.linear(x.float(), w.float(), **{k: v for k, v in kf.items() if k != "residual"})
    # the normalised rows are rounded to bf16 too
    assert _rel(ops.linear(x, w, **kw), want if res is None else want + res) < (5e-3 if form == "norm" else 3e-3)


@pytest.mark.parametrize("N,form", [(129, "even"), (190, "even"), (190, "one expert"), (191, "half"), (130, "bias"), (190, "scaled")])
def test_large_experts_of_a_few_hundred_tokens(N, form):
    """Segments of up to 128 rows where an expert has more, boxes of 64 and 16 token rows; the same bits every time."""
    E, k, H, I = 8, 2, 1024, 512
    x = torch.randn(N, H, device=DEV, dtype=BF)
    wg = (torch.randn(E, 2 * I, H, device=DEV) / math.sqrt(H)).to(BF)
    wd = (torch.randn(E, H, I, device=DEV) / math.sqrt(I)).to(BF)
    w, i = torch.topk(torch.softmax(torch.randn(N, E, device=DEV), -1), k, -1)
    if form == "one expert":
        i[:, 0], i[:, 1] = 3, 5
    if form == "half":
        i[:N // 2, 0], i[:N // 2, 1] = 3, 6
    kw, kf = {}, {}
    if form == "bias":
        bg, bd = torch.randn(E, 2 * I, device=DEV, dtype=BF), torch.randn(E, H, device=DEV, dtype=BF)
        kw, kf = dict(gate_up_bias=bg, down_bias=bd), dict(gate_up_bias=bg.float(), down_bias=bd.float())
    if form == "scaled":
        kw = kf = dict(scale_input=True)
    before = ops.kernel_launches()["skinny_gemm"]
    got = ops.moe_experts(x, wg, wd, w, i, "silu_mul", 0, **kw)
    assert ops.kernel_launches()["skinny_gemm"] == before + 2
    assert _rel(got, ref.moe_experts(x.float(), wg.float(), wd.float(), w, i, "silu_mul", 0, **kf)) < 5e-3
    for _ in range(5):
        assert torch.equal(ops.moe_experts(x, wg, wd, w, i, "silu_mul", 0, **kw), got)
