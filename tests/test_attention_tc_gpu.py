"""The tcgen05 attention kernel (csrc/attention_tc.cu) at the edges of its tiles and over all forms of its mask, against the fp32 definition.

Bound: probabilities and results are rounded to bf16 (2^-9 relative each, at most); their rms is below 2^-9 / sqrt(3) * sqrt(2) = 1.6e-3, the fp32
sums are far below.  Random rows show 2.0e-3 .. 2.4e-3 because a result is a difference of many terms; 4e-3 is asked for."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / b.norm().clamp_min(1e-9)).item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv,window,causal,sinks", [
    (1, 1, 2, 1, 0, True, False), (2, 17, 4, 1, 0, True, True), (1, 128, 3, 1, 0, True, False), (3, 129, 4, 2, 0, True, False),
    (2, 255, 3, 3, 0, True, True), (1, 257, 8, 8, 100, True, False), (2, 640, 4, 1, 128, True, True), (1, 1000, 2, 2, 77, True, False),
    (2, 383, 6, 2, 0, False, True), (1, 1300, 4, 4, 0, False, False), (1, 2049, 2, 1, 1024, True, False)])
def test_contiguous(D, B, T, Hq, Hkv, window, causal, sinks):
    q, k, v = (torch.randn(B, T, h, D, device=DEV, dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv))
    sk = torch.randn(Hq, device=DEV) if sinks else None
    got = ops.attention_prefill(q, k, v, D ** -0.5, causal, window or None, sinks=sk)
    want = ref.attention_prefill(q.float(), k.float(), v.float(), D ** -0.5, causal, window or None, sinks=sk)
    assert _rel(got, want) < 4e-3


def _paged(B, T, Hq, G, D, page, ctx, n, std=1.0):
    blocks = -(-(max(c + m for c, m in zip(ctx, n))) // page)
    kc, vc = (torch.randn(B * blocks + 3, page, G, D, device=DEV, dtype=torch.bfloat16) * std for _ in range(2))
    table = torch.randperm(B * blocks + 3, device=DEV)[:B * blocks].view(B, blocks).int()
    used = torch.zeros(B * blocks + 3, page, dtype=torch.bool, device=DEV)
    for b in range(B):                   # rows that no request wrote hold garbage, as the rest of an allocation does
        slots = table[b].long().repeat_interleave(page) * page + torch.arange(page, device=DEV).repeat(blocks)
        used.view(-1)[slots[:ctx[b] + n[b]]] = True
    clean = (torch.where(used[..., None, None], t, torch.zeros_like(t)) for t in (kc, vc))
    dirty = (torch.where(used[..., None, None], t, torch.full_like(t, float("nan"))) for t in (kc, vc))
    q = torch.randn(B, T, Hq, D, device=DEV, dtype=torch.bfloat16) * std
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)          # noqa: E731
    return q, tuple(dirty), tuple(clean), table, i32(ctx), i32(n)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("page", [8, 16, 64, 128, 256])
@pytest.mark.parametrize("mask", [dict(), dict(window=100), dict(window=300, keep=4), dict(window=130, keep=200), dict(chunk=96)])
def test_paged(D, page, mask):
    ctx, n = (0, 517, 130, 64), (300, 16, 0, 129)
    q, dirty, clean, table, c, m = _paged(4, 300, 4, 2, D, page, ctx, n)
    args = (table, c, m, D ** -0.5, None, mask.get("window", 0), mask.get("keep", 0))
    got = ops.paged_window_attention(q, *dirty, *args, chunk=mask.get("chunk"))
    want = ref.paged_window_attention(q.float(), *(t.float() for t in clean), *args, chunk=mask.get("chunk"))
    assert _rel(got, want) < 4e-3
    for b, live in enumerate(n):
        assert not got[b, live:].any()


@pytest.mark.parametrize("std", [1.0, 6.0])          # scores inside and beyond the range of the polynomial for tanh (|score| <= cap)
@pytest.mark.parametrize("Hq,G", [(4, 2), (3, 3)])
@pytest.mark.parametrize("gate", [None, "channel", "odd", "head"])
def test_paged_cap_gate_sinks_temperature(std, Hq, G, gate):
    D, ctx, n = 128, (77, 0), (140, 65)
    q, dirty, clean, table, c, m = _paged(2, 140, Hq, G, D, 64, ctx, n, std)
    wide = torch.randn(2, 140, Hq * D + 3, device=DEV, dtype=torch.bfloat16)
    g = {None: None, "channel": wide[..., :Hq * D].contiguous(), "odd": wide[..., 3:], "head": wide[..., :Hq]}[gate]
    kw = dict(gate=g, sinks=torch.randn(Hq, device=DEV), gate_per_head=gate == "head",
              head_scale=torch.tensor([0.7, 1.3, -0.5, 2.0], device=DEV)[:Hq])
    for cap in (None, 20.0):
        got = ops.paged_window_attention(q, *dirty, table, c, m, D ** -0.5, cap, 0, 0, **kw)
        want = ref.paged_window_attention(q.float(), *(t.float() for t in clean), table, c, m, D ** -0.5, cap, 0, 0,
                                          **dict(kw, gate=None if g is None else g.float()))
        assert _rel(got, want) < 4e-3


@pytest.mark.parametrize("D", [64, 128])
def test_soft_cap_does_not_depend_on_unseen_keys(D):
    """Bits must not change with cache rows past the end, later keys or queries past the end, whatever those hold."""
    g = torch.Generator(device="cuda").manual_seed(3)
    B, T, Hq, G, page, pages = 2, 200, 8, 2, 64, 8
    k, v = (torch.randn(B * pages, page, G, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    q = torch.randn(B, T, Hq, D, device="cuda", generator=g).bfloat16()
    table = torch.arange(B * pages, device="cuda", dtype=torch.int32).view(B, pages)
    ctx, n = (torch.tensor(x, device="cuda", dtype=torch.int32) for x in ([100, 37], [T, 150]))
    want = None
    for fill in (0.0, 3.0, 400.0, -1e4):
        kk, qq = k.clone(), q.clone()
        for b in range(B):
            rows = kk[b * pages:(b + 1) * pages].view(-1, G, D)
            rows[int(ctx[b] + n[b]):] = fill
            qq[b, int(n[b]):] = fill
        torch.full((64 << 20,), fill, device="cuda").mul_(2)          # other kernels in between
        got = ops.paged_window_attention(qq, kk, v, table, ctx, n, D ** -0.5, 30.0, 0, 0)
        assert want is None or torch.equal(got, want)
        want = got


def _two_tiles():
    return ops.kernel_launches()["attention_prefill_tc_two_tiles"]


# rows of more than 1152 keys and at least 148 CTAs take two query tiles per CTA: one tile more or less than that, whole and odd lengths, heads in pairs
# and alone; the bound above
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv,window,causal,sinks,two", [
    (1, 1152, 34, 17, 0, True, False, 0), (1, 1153, 32, 8, 0, True, True, 1), (1, 1281, 30, 30, 0, True, False, 1), (2, 1290, 16, 4, 1025, True, True, 1),
    (2, 1290, 16, 4, 1024, True, False, 0), (1, 1217, 32, 16, 0, False, False, 1), (2, 1408, 15, 5, 0, False, True, 1)])
def test_two_tiles(D, B, T, Hq, Hkv, window, causal, sinks, two):
    before = _two_tiles()
    test_contiguous(D, B, T, Hq, Hkv, window, causal, sinks)
    assert _two_tiles() - before == two


@pytest.mark.parametrize("D,cap", [(64, 20.0), (128, 20.0), (64, None), (128, None)])
@pytest.mark.parametrize("Hq,G", [(32, 8), (17, 17)])
@pytest.mark.parametrize("mask,two", [(dict(), 1), (dict(window=1300, keep=70), 1), (dict(window=200, keep=4), 0), (dict(chunk=1200), 1)])
def test_two_tiles_paged(D, cap, Hq, G, mask, two):
    ctx, n = (0, 1517, 130, 64, 1000), (300, 16, 0, 257, 290)
    q, dirty, clean, table, c, m = _paged(5, 300, Hq, G, D, 64, ctx, n)
    args = (table, c, m, D ** -0.5, cap, mask.get("window", 0), mask.get("keep", 0))
    before = _two_tiles()
    got = ops.paged_window_attention(q, *dirty, *args, chunk=mask.get("chunk"))
    assert _two_tiles() - before == two
    want = ref.paged_window_attention(q.float(), *(t.float() for t in clean), *args, chunk=mask.get("chunk"))
    assert _rel(got, want) < 4e-3
    for b, live in enumerate(n):
        assert not got[b, live:].any()


@pytest.mark.parametrize("std", [1.0, 6.0])          # scores inside and beyond the range of the polynomial for tanh (|score| <= cap)
@pytest.mark.parametrize("Hq,G", [(32, 8), (17, 17)])
@pytest.mark.parametrize("gate", [None, "channel", "odd", "head"])
def test_two_tiles_cap_gate_sinks_temperature(std, Hq, G, gate):
    D, ctx, n = 128, (0, 1100, 130, 64, 1000), (300, 140, 0, 257, 290)
    q, dirty, clean, table, c, m = _paged(5, 300, Hq, G, D, 64, ctx, n, std)
    wide = torch.randn(5, 300, Hq * D + 3, device=DEV, dtype=torch.bfloat16)
    g = {None: None, "channel": wide[..., :Hq * D].contiguous(), "odd": wide[..., 3:], "head": wide[..., :Hq]}[gate]
    kw = dict(gate=g, sinks=torch.randn(Hq, device=DEV), gate_per_head=gate == "head", head_scale=torch.linspace(-0.8, 2.0, Hq, device=DEV))
    for cap in (None, 20.0):
        before = _two_tiles()
        got = ops.paged_window_attention(q, *dirty, table, c, m, D ** -0.5, cap, 0, 0, **kw)
        assert _two_tiles() - before == 1
        want = ref.paged_window_attention(q.float(), *(t.float() for t in clean), table, c, m, D ** -0.5, cap, 0, 0,
                                          **dict(kw, gate=None if g is None else g.float()))
        assert _rel(got, want) < 4e-3


def test_soft_cap_of_scores_below_the_range():
    """Scores that overflow to -inf are capped to -cap like all others, also where a row sees nothing else in its first tiles."""
    B, T, Hq, G, D, page = 1, 300, 4, 2, 128, 64
    q, dirty, _, table, c, m = _paged(B, T, Hq, G, D, page, (0,), (T,))
    k, v = (t.nan_to_num(0.0) for t in dirty)
    low = table[0].long().repeat_interleave(page)[:200] * page + torch.arange(page, device=DEV).repeat(5)[:200]
    q[..., 0] = 1e20
    k[..., 0] = 0.0
    k.view(-1, G, D)[low, :, 0] = -1e20
    for cap in (1.0, 4.0):
        got = ops.paged_window_attention(q, k, v, table, c, m, D ** -0.5, cap, 0, 0)
        want = ref.paged_window_attention(q.float(), k.float(), v.float(), table, c, m, D ** -0.5, cap, 0, 0)
        assert _rel(got, want) < 4e-3


@pytest.mark.parametrize("D,B,T,Hq,G", [(128, 1, 40, 4, 2), (128, 5, 300, 8, 2), (64, 3, 140, 8, 8)])
@pytest.mark.parametrize("at", [0, 8, 3])
def test_gate_rows_of_a_wider_tensor(D, B, T, Hq, G, at):
    """The gate comes as tiles where its rows lie on 16 bytes, else element by element; the ends of the sigmoid's range, infinities, and padding rows that hold NaN."""
    ctx, n = [0, 77, 130, 64, 1000][:B], [T, T - 30, 0, T // 2, 290][:B]
    q, dirty, clean, table, c, m = _paged(B, T, Hq, G, D, 64, ctx, n)
    wide = torch.randn(B, T, Hq * D + 8, device=DEV, dtype=torch.bfloat16) * 4
    wide[:, 5] = torch.tensor([100.0, -100.0, 3e38, -3e38, float("inf"), -float("inf"), 88.5, -88.5], device=DEV).bfloat16().repeat(Hq * D // 8 + 1)
    for b in range(B):
        wide[b, n[b]:] = float("nan")
    gate = wide[..., at:at + Hq * D]
    got = ops.paged_window_attention(q, *dirty, table, c, m, D ** -0.5, 0.0, 0, 0, gate)
    want = ref.paged_window_attention(q.float(), *(t.float() for t in clean), table, c, m, D ** -0.5, 0.0, 0, 0, gate.nan_to_num(0.0, float("inf"), -float("inf")).float())
    assert torch.isfinite(got).all() and _rel(got, want) < 4e-3
    for b in range(B):
        assert not got[b, n[b]:].any()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("std", [1.0, 4.0, 12.0, 1e20])
@pytest.mark.parametrize("mask", [dict(), dict(window=100, keep=4), dict(chunk=96)])
def test_cap_of_many_short_rows(D, std, mask):
    """More CTAs than SMs, few key tiles each: the small code, with scores below, around and beyond the cap."""
    ctx, n = (0, 517, 130, 64), (300, 16, 0, 129)
    q, dirty, clean, table, c, m = _paged(4, 300, 16, 4, D, 64, ctx, n)
    args = (table, c, m, D ** -0.5, 20.0, mask.get("window", 0), mask.get("keep", 0))
    q = q * std
    kw = dict(chunk=mask.get("chunk"), head_scale=torch.linspace(-0.8, 2.0, 16, device=DEV))
    got = ops.paged_window_attention(q, *dirty, *args, **kw)
    want = ref.paged_window_attention(q.double(), *(t.double() for t in clean), *args, **dict(kw, head_scale=kw["head_scale"].double()))
    assert torch.isfinite(got).all() and _rel(got, want) < 4e-3
    alone = ops.paged_window_attention(q[:1], *dirty, table[:1], c[:1], m[:1], *args[3:], **kw)      # fewer CTAs: the unrolled code, where the scores allow it
    assert torch.equal(got[:1], alone)
