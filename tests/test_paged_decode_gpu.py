"""Paged decode attention: pages of any size (2^k and not), rows of very different length, every number of parts the split rule can pick, against the
fp32 definition.  Bound: bf16 probabilities and results, 2^-9 at most each (2.0e-3 .. 2.4e-3 seen on random rows)."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv,page,longest,window,sinks", [
    (1, 1, 8, 2, 16, 1, 0, False), (2, 3, 8, 1, 24, 700, 0, True), (5, 1, 4, 4, 64, 4096, 0, False), (12, 1, 32, 8, 8, 4000, 100, True),
    (48, 1, 16, 8, 32, 3100, 0, False), (130, 2, 8, 8, 48, 300, 0, True), (1, 4, 64, 4, 256, 1030, 65, False)])
def test_rows(B, T, Hq, Hkv, page, longest, window, sinks, D):
    g = torch.Generator().manual_seed(3)
    blocks = -(-longest // page)
    last = torch.randint(T, max(longest, T + 1), (B,), generator=g)
    last[0] = max(longest, T)
    pos = (last.view(B, 1) - T + torch.arange(T)).int().cuda()
    kc, vc = (torch.randn(B * blocks, page, Hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.randperm(B * blocks, device="cuda").view(B, blocks).int()
    q = torch.randn(B, T, Hq, D, device="cuda", dtype=torch.bfloat16)
    sk = torch.randn(Hq, device="cuda") if sinks else None
    for _ in range(2):                   # the second call finds the tickets that the first one left
        got = ops.paged_attention_decode(q, kc, vc, table, pos, D ** -0.5, window or None, sk)
        want = ref.paged_attention_decode(q.float(), kc.float(), vc.float(), table, pos, D ** -0.5, window or None, sk)
        assert ((got.float() - want).norm() / want.norm()).item() < 4e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Hkv", [1, 8])
def test_few_requests_with_long_contexts(Hkv, D):
    """One request takes up to 64 parts: the rows of the parts and their factors have to fit the workspace and the shared memory of the combine."""
    Hq, page, ctx = 8 * Hkv if Hkv == 1 else 4 * Hkv, 64, 40001
    n = -(-ctx // page)
    k, v = (torch.randn(n, page, Hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.randperm(n, device="cuda").view(1, n).int()
    for T in (1, 64 // (Hq // Hkv)):
        q = torch.randn(1, T, Hq, D, device="cuda", dtype=torch.bfloat16)
        pos = torch.arange(ctx - T, ctx, device="cuda", dtype=torch.int32).view(1, T)
        got = ops.paged_attention_decode(q, k, v, table, pos, D ** -0.5)
        kk, vv = (t[table[0].long()].reshape(-1, Hkv, D)[:ctx].float().repeat_interleave(Hq // Hkv, 1) for t in (k, v))
        sc = torch.einsum("thd,nhd->thn", q[0].float(), kk) * D ** -0.5
        sc = sc.masked_fill(torch.arange(ctx, device="cuda") > pos[0].view(T, 1, 1), float("-inf"))
        want = torch.einsum("thn,nhd->thd", torch.softmax(sc, -1), vv)
        assert ((got[0].float() - want).norm() / want.norm()).item() < 4e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Hkv,window,most", [(1, 0, 4096), (2, 0, 2600), (1, 1500, 4096), (1, 0, 65536 + 64)])
def test_parts_of_one_size(Hkv, window, most, D):
    """From 96 (row, kv head) pairs on a row has as many parts as it needs: rows at the edges of the parts, the shortest and the longest that the table holds."""
    ctx = [most, 1] + [c + d for c in (1024, 2048, 3072) for d in (-1, 0, 1) if c + d <= most] * 9 + [63, 64, 65, 500, most - 1]
    B = 96 // Hkv + 3
    ctx = (ctx * 3)[:B]
    page, Hq = 64, 4 * Hkv
    n = -(-most // page)
    kc, vc = (torch.randn(n + 7, page, Hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.stack([torch.randperm(n + 7, device="cuda")[:n] for _ in range(B)]).int()          # rows share pages
    q, pos = torch.randn(B, 1, Hq, D, device="cuda", dtype=torch.bfloat16), torch.tensor(ctx, device="cuda", dtype=torch.int32).view(B, 1) - 1
    for _ in range(2):
        got = ops.paged_attention_decode(q, kc, vc, table, pos, D ** -0.5, window or None)
        for b in range(0, B, 1 if most <= 4096 else 17):
            want = ref.paged_attention_decode(q[b:b + 1].float(), kc.float(), vc.float(), table[b:b + 1], pos[b:b + 1], D ** -0.5, window or None, None)
            assert ((got[b:b + 1].float() - want).norm() / want.norm()).item() < 4e-3


@pytest.mark.parametrize("Hkv,B", [(8, 12), (8, 33), (1, 100)])
def test_parts_do_not_depend_on_the_width_of_the_table(Hkv, B):
    """A serving layer may pass its full table: rows of a few thousand keys are cut as under a table of their own length."""
    page, D, n, Hq = 32, 128, 4096 // 32, 4 * Hkv
    kc, vc = (torch.randn(B * n, page, Hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.randperm(B * n, device="cuda").view(B, n).int()
    ctx = [(4096, 1, 1025, 3000, 2049, 1024)[b % 6] for b in range(B)]
    q, pos = torch.randn(B, 1, Hq, D, device="cuda", dtype=torch.bfloat16), torch.tensor(ctx, device="cuda", dtype=torch.int32).view(B, 1) - 1
    want = ops.paged_attention_decode(q, kc, vc, table, pos, D ** -0.5)
    for slots in (32768, 131072):
        wide = torch.zeros(B, slots // page, device="cuda", dtype=torch.int32)
        wide[:, :n] = table
        assert torch.equal(ops.paged_attention_decode(q, kc, vc, wide, pos, D ** -0.5), want)


@pytest.mark.parametrize("B,T,Hkv,window", [(13, 1, 8, 0), (96, 1, 1, 0), (129, 2, 1, 100), (256, 1, 1, 0), (257, 1, 1, 0), (50, 3, 2, 700)])
def test_order_of_the_rows(B, T, Hkv, window):
    """The longest rows start first from 96 (row, kv head) pairs on: a row's bits do not depend on its place, equal lengths and empty rows among them."""
    page, D, longest, Hq = 64, 64, 3500, 4 * Hkv
    n = -(-longest // page)
    kc, vc = (torch.randn(3 * n, page, Hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.stack([torch.randperm(3 * n, device="cuda")[:n] for _ in range(B)]).int()
    ctx = [(longest, 1, 700, 1200, 700, 64, 2049)[b % 7] for b in range(B)]
    pos = torch.tensor(ctx, device="cuda", dtype=torch.int32).view(B, 1) - T + torch.arange(T, device="cuda", dtype=torch.int32)
    q = torch.randn(B, T, Hq, D, device="cuda", dtype=torch.bfloat16)
    got = ops.paged_attention_decode(q, kc, vc, table, pos, D ** -0.5, window or None)
    i = torch.randperm(B, device="cuda")
    again = ops.paged_attention_decode(q[i].contiguous(), kc, vc, table[i].contiguous(), pos[i].contiguous(), D ** -0.5, window or None)
    assert torch.equal(again, got[i])
    for b in range(0, B, 11):
        if ctx[b] >= T:
            want = ref.paged_attention_decode(q[b:b + 1].float(), kc.float(), vc.float(), table[b:b + 1], pos[b:b + 1], D ** -0.5, window or None, None)
            assert ((got[b:b + 1].float() - want).norm() / want.norm()).item() < 4e-3
