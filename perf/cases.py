"""The calls whose speed is followed: single layers and blocks of prefill and decode, and one whole decode step.

A case names a KIND of call and its sizes.  ``listed()`` holds the ones that are followed by name, ``draw(rng)`` gives more of the same
ranges.  Every kind calls the engine the way its own models do (``ops`` and ``modules``), ``llama_step`` goes through the application's
``forward`` (pinned host ids and positions in, CUDA-graph replay, logits out).

===========  =====================================================================================================================
mlp          gated MLP block with its input norm and the residual (``modules.mlp.GatedMLP``): prompts and batched decode steps
linear8      projection with 8-bit weights and per-channel scales (weight-only quantisation), decode and prompt sizes
flash        attention over fresh prompts (``ops.attention_prefill``): causal, windowed, with sinks, bidirectional; head sizes 64, 128
paged_step   one decode step of attention for a batch of requests on the paged KV cache (``ops.paged_attention_decode``)
portion      ragged prompt portions over a paged cache that holds earlier tokens (``ops.paged_window_attention``)
ssd          Mamba-2 recurrence over ragged rows with a carried state (``ops.ssd_scan``)
moe          mixture-of-experts block: norm, fp32 router, routed experts, residual (``modules.moe.MoE``)
sample       top-k / top-p / temperature sampling of a batch of vocabulary rows (``ops.sample``)
llama_step   a whole decode step of a four-layer Llama with the 8B layer sizes, logits returned
===========  =====================================================================================================================
"""
import math
import random

import torch

from neuronx_distributed_inference_b200 import ops

DEV = "cuda"
BF = torch.bfloat16

# (hidden, intermediate): Llama-3.1-8B, Llama-2-7b, open_llama_3b and the 2048-wide benchmark stack
MLP_SIZES = ((4096, 14336), (4096, 11008), (3200, 8640), (2048, 8192))
# (q heads, kv heads) of the same models
HEADS = ((32, 8), (16, 4), (32, 32), (8, 1))
# experts, chosen, hidden, intermediate: Qwen3-MoE, Mixtral, a DBRX shard of eight
MOE_SIZES = ((128, 8, 2048, 768), (8, 2, 4096, 14336), (16, 4, 6144, 1344))
# heads, head size, state, groups of the Mamba-2 mixers of the benchmark stacks
SSD_SIZES = ((64, 64, 128, 1), (128, 64, 128, 8))
VOCABS = (128256, 32000)
PAGE = 64


def listed():
    return [
        # a long prompt through the MLP of an 8B model: the largest share of prefill
        dict(name="mlp_prompt", kind="mlp", tokens=4096, size=0),
        # a serving batch's decode step through the same block: weights dominate, 37 requests are neither a tile nor a power of two
        dict(name="mlp_batch_step", kind="mlp", tokens=37, size=0),
        # a quantised 7B model decoding for three users: the down projection with fp8 weights
        dict(name="linear8_step", kind="linear8", tokens=3, n=4096, k=11008, fp8=True),
        # one long prompt, the attention of an 8B model
        dict(name="flash_long", kind="flash", rows=1, tokens=8192, heads=0, dim=128, window=0, sinks=False, causal=True),
        # short prompts of a GPT-OSS layer: head size 64, sliding window, sinks, a length that is no multiple of anything
        dict(name="flash_window", kind="flash", rows=3, tokens=1000, heads=0, dim=64, window=128, sinks=True, causal=True),
        # continuous batching: 48 requests at contexts up to 4096 take one token each
        dict(name="paged_step", kind="paged_step", rows=48, context=4096, heads=0, dim=128, page=32),
        # chunked prefill: portions of three requests, two of them with earlier context, soft cap, window and output gate
        dict(name="portion_mixed", kind="portion", rows=3, tokens=1024, context=3000, heads=0, dim=128, window=2048, keep=4, cap=30.0, gate=True),
        # four prompt portions through a Mamba-2 mixer
        dict(name="ssd_prompt", kind="ssd", rows=4, tokens=1024, size=0),
        # a long prompt through a block with many small experts
        dict(name="moe_prompt", kind="moe", tokens=4096, size=0),
        # a small batch's decode step through a block with few large experts
        dict(name="moe_step", kind="moe", tokens=6, size=1),
        # a batch of users who sample
        dict(name="sample_batch", kind="sample", rows=32, vocab=0, fp32=False),
        # the smallest whole call: two requests take one token (headline benchmark, four of its layers)
        dict(name="llama_step", kind="llama_step", rows=2, context=130),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(("mlp", "mlp", "linear8", "flash", "flash", "flash", "paged_step", "portion", "portion", "ssd", "moe", "moe", "sample", "llama_step"))
    if kind == "mlp":
        return dict(kind=kind, tokens=_log(rng, 1, 4096), size=rng.randrange(len(MLP_SIZES)))
    if kind == "linear8":
        n, k = rng.choice(((4096, 11008), (4096, 4096), (12288, 4096), (11008, 4096)))
        return dict(kind=kind, tokens=_log(rng, 1, 2048), n=n, k=k, fp8=rng.random() < 0.6)
    if kind == "flash":
        causal = rng.random() < 0.85
        rows = rng.randint(1, 4)
        return dict(kind=kind, rows=rows, tokens=_log(rng, 17, (8192, 4096, 3072, 2048)[rows - 1] if causal else 2048), heads=rng.randrange(len(HEADS)),
                    dim=rng.choice((128, 128, 64)), window=rng.choice((0, 0, 128, 1024, 77)) if causal else 0, sinks=rng.random() < 0.25, causal=causal)
    if kind == "paged_step":
        return dict(kind=kind, rows=_log(rng, 1, 48), context=_log(rng, 20, 4096), heads=rng.randrange(len(HEADS)) if rng.random() < 0.5 else 0,
                    dim=rng.choice((128, 128, 64)), page=rng.choice((16, 32, 64)))
    if kind == "portion":
        return dict(kind=kind, rows=rng.randint(1, 4), tokens=_log(rng, 16, 1024), context=rng.choice((0, _log(rng, 1, 3000))), heads=rng.randrange(2),
                    dim=rng.choice((128, 128, 64)), window=rng.choice((0, 500, 2048)), keep=rng.choice((0, 4)), cap=rng.choice((0.0, 30.0)), gate=rng.random() < 0.5)
    if kind == "ssd":
        return dict(kind=kind, rows=rng.randint(1, 4), tokens=_log(rng, 1, 1024), size=rng.randrange(len(SSD_SIZES)))
    if kind == "moe":
        size = rng.randrange(len(MOE_SIZES))
        return dict(kind=kind, tokens=_log(rng, 1, (4096, 1024, 2048)[size]), size=size)
    if kind == "sample":
        return dict(kind=kind, rows=_log(rng, 1, 64), vocab=rng.randrange(len(VOCABS)), fp32=rng.random() < 0.5)
    return dict(kind=kind, rows=rng.randint(1, 8), context=_log(rng, 20, 1000))


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, *shape, dtype=BF, std=1.0):
    return (torch.randn(shape, device=DEV, generator=g, dtype=torch.float32) * std).to(dtype)


def _weight(g, *shape):
    """bf16 weights of the usual initial size."""
    w = torch.empty(shape, device=DEV, dtype=BF)
    w.normal_(0.0, 0.02, generator=g)
    return w


# ---- mlp ----------------------------------------------------------------------------------------------------------------------------
def _mlp_prepare(c, seed):
    from neuronx_distributed_inference_b200.modules.mlp import GatedMLP
    g = _gen(seed)
    H, I = MLP_SIZES[c["size"]]
    m = GatedMLP(H, I, dtype=BF, device=DEV)
    m.gate_up_proj.weight.data.copy_(_weight(g, 2 * I, H))
    m.down_proj.weight.data.copy_(_weight(g, H, I))
    return dict(m=m, x=_randn(g, 1, c["tokens"], H), norm=_randn(g, H, std=0.1) + 1)


def _mlp_run(s):
    return s["m"](s["x"], norm_weight=s["norm"], norm_eps=1e-5, residual=s["x"])


def _rms64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _mlp_exact(c, s):
    x, I = s["x"].double(), MLP_SIZES[c["size"]][1]
    h = _rms64(x, s["norm"].double(), 1e-5)
    g, u = (h @ w.double().t() for w in s["m"].gate_up_proj.weight.data.split(I))
    return (_silu(g) * u) @ s["m"].down_proj.weight.data.double().t() + x


def _mlp_work(c):
    T, (H, I) = c["tokens"], MLP_SIZES[c["size"]]
    return dict(bytes=2 * (3 * H * I + H + 2 * T * H), flops=6 * T * H * I)


# ---- linear8 ------------------------------------------------------------------------------------------------------------------------
def _linear8_prepare(c, seed):
    g = _gen(seed)
    w = _randn(g, c["n"], c["k"], dtype=torch.float32, std=0.02)
    w, scale = ops.quantize_per_channel(w, torch.float8_e4m3fn if c["fp8"] else torch.int8)
    return dict(x=_randn(g, 1, c["tokens"], c["k"]), w=w.contiguous(), scale=scale.float().reshape(-1).contiguous())


def _linear8_run(s):
    return ops.linear(s["x"], s["w"], scale=s["scale"])


def _linear8_exact(c, s):
    return s["x"].double() @ (s["w"].double() * s["scale"].double().view(-1, 1)).t()


def _linear8_work(c):
    T, N, K = c["tokens"], c["n"], c["k"]
    return dict(bytes=N * K + 4 * N + 2 * T * (N + K), flops=2 * T * N * K)


# ---- flash --------------------------------------------------------------------------------------------------------------------------
def _flash_prepare(c, seed):
    g = _gen(seed)
    Hq, Hkv = HEADS[c["heads"]]
    B, T, D = c["rows"], c["tokens"], c["dim"]
    s = dict(q=_randn(g, B, T, Hq, D), k=_randn(g, B, T, Hkv, D), v=_randn(g, B, T, Hkv, D), scale=D ** -0.5,
             window=c["window"] or None, causal=c["causal"])
    s["sinks"] = _randn(g, Hq, dtype=torch.float32) if c["sinks"] else None
    return s


def _flash_run(s):
    return ops.attention_prefill(s["q"], s["k"], s["v"], s["scale"], s["causal"], s["window"], sinks=s["sinks"])


def _softmax_rows(sc, sinks):
    """Softmax over the last axis; ``sinks`` (broadcastable) joins the denominator only."""
    m = sc.amax(-1, keepdim=True)
    if sinks is not None:
        m = torch.maximum(m, sinks)
    e = torch.exp(sc - m)
    d = e.sum(-1, keepdim=True)
    return e / (d if sinks is None else d + torch.exp(sinks - m))


def _flash_exact(c, s):
    B, T, Hq, D = s["q"].shape
    rep = Hq // s["k"].shape[2]
    out = torch.empty(B, T, Hq, D, dtype=torch.float64, device=DEV)
    j = torch.arange(T, device=DEV)
    step = 2048
    for b in range(B):
        for h in range(Hq):
            k, v = s["k"][b, :, h // rep].double(), s["v"][b, :, h // rep].double()
            for t in range(0, T, step):
                i = j[t:t + step].view(-1, 1)
                sc = s["q"][b, t:t + step, h].double() @ k.t() * s["scale"]
                if s["causal"]:
                    see = j <= i
                    if s["window"]:
                        see = see & (i - j < s["window"])
                    sc = sc.masked_fill(~see, float("-inf"))
                out[b, t:t + step, h] = _softmax_rows(sc, None if s["sinks"] is None else s["sinks"][h].double()) @ v
    return out


def _pairs(T, causal, window):
    if not causal:
        return T * T
    w = min(window or T, T)
    return w * (w + 1) // 2 + (T - w) * w


def _flash_work(c):
    Hq, Hkv = HEADS[c["heads"]]
    B, T, D = c["rows"], c["tokens"], c["dim"]
    return dict(bytes=2 * B * T * D * 2 * (Hq + Hkv), flops=4 * B * Hq * D * _pairs(T, c["causal"], c["window"]))


# ---- paged_step ---------------------------------------------------------------------------------------------------------------------
def _contexts(rng, rows, most):
    """Context lengths of a batch in flight: one request at the limit, the others anywhere up to it."""
    return [most] + [rng.randint(1, most) for _ in range(rows - 1)]


def _paged_contexts(c, seed):
    return _contexts(random.Random(c["rows"] * 1000003 + c["context"]), c["rows"], c["context"])


def _paged_prepare(c, seed):
    g = _gen(seed)
    Hq, Hkv = HEADS[c["heads"]]
    D, page = c["dim"], c["page"]
    ctx = _paged_contexts(c, seed)
    per = -(-c["context"] // page)
    blocks = c["rows"] * per
    table = torch.randperm(blocks, device=DEV, generator=g).view(c["rows"], per).int()
    return dict(q=_randn(g, c["rows"], 1, Hq, D), k=_randn(g, blocks, page, Hkv, D), v=_randn(g, blocks, page, Hkv, D), table=table,
                pos=torch.tensor(ctx, device=DEV, dtype=torch.int32).view(-1, 1) - 1, scale=D ** -0.5)


def _paged_run(s):
    return ops.paged_attention_decode(s["q"], s["k"], s["v"], s["table"], s["pos"], s["scale"])


def _paged_exact(c, s):
    B, _, Hq, D = s["q"].shape
    G = s["k"].shape[2]
    out = torch.empty(B, 1, Hq, D, dtype=torch.float64, device=DEV)
    for b, n in enumerate(_paged_contexts(c, 0)):
        k, v = (t[s["table"][b].long()].reshape(-1, G, D)[:n].double().repeat_interleave(Hq // G, 1) for t in (s["k"], s["v"]))
        p = torch.softmax(torch.einsum("hd,nhd->hn", s["q"][b, 0].double(), k) * s["scale"], -1)
        out[b, 0] = torch.einsum("hn,nhd->hd", p, v)
    return out


def _paged_work(c):
    Hq, Hkv = HEADS[c["heads"]]
    n = sum(_paged_contexts(c, 0))
    return dict(bytes=4 * n * Hkv * c["dim"] + 4 * c["rows"] * Hq * c["dim"], flops=4 * n * Hq * c["dim"])


# ---- portion ------------------------------------------------------------------------------------------------------------------------
def _portion_rows(c):
    """(earlier context, new tokens) of every row: the first row brings the longest portion, one row starts a new request."""
    rng = random.Random(c["tokens"] * 7919 + c["context"])
    rows = []
    for b in range(c["rows"]):
        rows.append((c["context"] if b == 1 else rng.randint(0, c["context"]), c["tokens"] if b == 0 else rng.randint(max(1, c["tokens"] // 16), c["tokens"])))
    return rows


def _portion_prepare(c, seed):
    g = _gen(seed)
    Hq, Hkv = HEADS[c["heads"]]
    D, T = c["dim"], c["tokens"]
    rows = _portion_rows(c)
    per = -(-(c["context"] + T) // PAGE)
    blocks = c["rows"] * per
    s = dict(q=_randn(g, c["rows"], T, Hq, D), k=_randn(g, blocks, PAGE, Hkv, D), v=_randn(g, blocks, PAGE, Hkv, D),
             table=torch.randperm(blocks, device=DEV, generator=g).view(c["rows"], per).int(),
             ctx=torch.tensor([r[0] for r in rows], device=DEV, dtype=torch.int32), n=torch.tensor([r[1] for r in rows], device=DEV, dtype=torch.int32),
             scale=D ** -0.5, cap=c["cap"], window=c["window"], keep=c["keep"])
    s["gate"] = _randn(g, c["rows"], T, Hq * D) if c["gate"] else None
    return s


def _portion_run(s):
    return ops.paged_window_attention(s["q"], s["k"], s["v"], s["table"], s["ctx"], s["n"], s["scale"], s["cap"], s["window"], s["keep"], s["gate"])


def _portion_exact(c, s):
    B, T, Hq, D = s["q"].shape
    G = s["k"].shape[2]
    out = torch.zeros(B, T, Hq, D, dtype=torch.float64, device=DEV)
    for b, (ctx, n) in enumerate(_portion_rows(c)):
        k, v = (t[s["table"][b].long()].reshape(-1, G, D)[:ctx + n] for t in (s["k"], s["v"]))
        i, j = torch.arange(ctx, ctx + n, device=DEV).view(-1, 1), torch.arange(ctx + n, device=DEV).view(1, -1)
        see = j <= i
        if c["window"]:
            see = see & ((i - j < c["window"]) | (j < c["keep"]))
        for h in range(Hq):
            sc = s["q"][b, :n, h].double() @ k[:, h * G // Hq].double().t() * s["scale"]
            if c["cap"]:
                sc = c["cap"] * torch.tanh(sc / c["cap"])
            out[b, :n, h] = torch.softmax(sc.masked_fill(~see, float("-inf")), -1) @ v[:, h * G // Hq].double()
    out = out.reshape(B, T, Hq * D)
    return out if s["gate"] is None else out * torch.sigmoid(s["gate"].double())


def _portion_work(c):
    Hq, Hkv = HEADS[c["heads"]]
    D, pairs, keys, new = c["dim"], 0, 0, 0
    for ctx, n in _portion_rows(c):
        w = c["window"] or ctx + n
        for i in range(ctx, ctx + n):
            pairs += min(i + 1, w + (min(c["keep"], i + 1 - w) if i + 1 > w else 0))
        keys += min(ctx + n, n + w - 1 + c["keep"])
        new += n
    return dict(bytes=4 * keys * Hkv * D + 2 * new * Hq * D * (3 if c["gate"] else 2), flops=4 * pairs * Hq * D)


# ---- ssd ----------------------------------------------------------------------------------------------------------------------------
def _ssd_rows(c):
    """(has earlier context, new tokens) of every row."""
    rng = random.Random(c["tokens"] * 31 + c["rows"])
    return [(b % 2, c["tokens"] if b == 0 else rng.randint(max(1, c["tokens"] // 2), c["tokens"])) for b in range(c["rows"])]


def _ssd_prepare(c, seed):
    g = _gen(seed)
    nh, P, N, G = SSD_SIZES[c["size"]]
    B, T, inner = c["rows"], c["tokens"], nh * P
    xbc = _randn(g, B, T, inner + 2 * G * N, dtype=torch.float32)
    xbc = _silu(xbc)                                              # after convolution and SiLU
    rows = _ssd_rows(c)
    a0 = torch.rand(nh, device=DEV, generator=g) * 15 + 1          # the usual initial decays: A in 1 .. 16, steps 1e-3 .. 1e-1
    dt0 = torch.exp(torch.rand(nh, device=DEV, generator=g) * math.log(100.0) + math.log(1e-3))
    return dict(xbc=xbc, dt=_randn(g, B, T, nh, std=0.5), z=_randn(g, B, T, inner), a=torch.log(a0), bias=dt0 + torch.log(-torch.expm1(-dt0)),
                skip=torch.ones(nh, device=DEV) + _randn(g, nh, dtype=torch.float32, std=0.1),
                state=_randn(g, B + 1, nh, N, P, dtype=torch.float32, std=0.3), slots=torch.arange(B, device=DEV, dtype=torch.int32),
                ctx=torch.tensor([100 * r[0] for r in rows], device=DEV, dtype=torch.int32), n=torch.tensor([r[1] for r in rows], device=DEV, dtype=torch.int32),
                sizes=(nh, P, N, G))


def _ssd_run(s):
    y = ops.ssd_scan(s["xbc"], s["dt"], s["z"], s["a"], s["bias"], s["skip"], s["state"], s["slots"], s["ctx"], s["n"], *s["sizes"])
    return dict(y=y, state=s["state"])


def _ssd_exact(c, s):
    nh, P, N, G = s["sizes"]
    B, T, inner = c["rows"], c["tokens"], nh * P
    state = s["state"].double().clone()
    y = torch.zeros(B, T, inner, dtype=torch.float64, device=DEV)
    A, skip = -torch.exp(s["a"].double()), s["skip"].double()
    for b, (has, n) in enumerate(_ssd_rows(c)):
        xbc = s["xbc"][b, :n].double()
        x = xbc[:, :inner].view(n, nh, P)
        Bm, Cm = (xbc[:, inner + k * G * N:inner + (k + 1) * G * N].view(n, G, N) for k in (0, 1))
        dt = torch.log1p(torch.exp(s["dt"][b, :n].double() + s["bias"].double()))
        dA = torch.exp(A * dt)
        S = state[b] if has else torch.zeros_like(state[b])
        S = S.view(G, nh // G, N, P)
        dx = (dt.unsqueeze(-1) * x).view(n, G, nh // G, 1, P)
        for t in range(n):
            S = S * dA[t].view(G, nh // G, 1, 1) + Bm[t].view(G, 1, N, 1) * dx[t]
            y[b, t] = torch.einsum("ghnp,gn->ghp", S, Cm[t]).reshape(inner) + (x[t] * skip.view(nh, 1)).reshape(inner)
        state[b] = S.reshape(nh, N, P)
        y[b, :n] *= _silu(s["z"][b, :n].double())
    return dict(y=y, state=state)


def _ssd_work(c):
    nh, P, N, G = SSD_SIZES[c["size"]]
    n = sum(r[1] for r in _ssd_rows(c))
    inner, live = nh * P, sum(1 + r[0] for r in _ssd_rows(c))
    return dict(bytes=n * (4 * (2 * inner + 2 * G * N) + 2 * inner + 2 * nh) + live * 4 * nh * N * P, flops=n * nh * N * P * 5)


# ---- moe ----------------------------------------------------------------------------------------------------------------------------
def _moe_prepare(c, seed):
    from neuronx_distributed_inference_b200.modules.moe import ExpertMLPs, MoE, RouterTopK
    g = _gen(seed)
    E, k, H, I = MOE_SIZES[c["size"]]
    router = RouterTopK(E, k, H, device=DEV)
    router.linear_router.weight.data.copy_(_randn(g, E, H, dtype=torch.float32, std=0.02))
    experts = ExpertMLPs(E, H, I, dtype=BF, device=DEV)
    experts.gate_up_proj.data.copy_(_weight(g, E, 2 * I, H))
    experts.down_proj.data.copy_(_weight(g, E, H, I))
    return dict(m=MoE(router, experts), x=_randn(g, 1, c["tokens"], H), norm=_randn(g, H, std=0.1) + 1)


def _moe_run(s):
    return s["m"](s["x"], norm_weight=s["norm"], norm_eps=1e-5, residual=s["x"])


def _moe_route64(c, s):
    """Normalised rows, expert ids and weights of every token, from the bf16 rows that the router reads."""
    E, k, H, I = MOE_SIZES[c["size"]]
    h = _rms64(s["x"].double(), s["norm"].double(), 1e-5).view(-1, H)
    p = torch.softmax(h.to(BF).double() @ s["m"].router.linear_router.weight.data.double().t(), -1)
    w, i = torch.topk(p, k, -1)
    return h, w / w.sum(-1, keepdim=True), i


def _moe_exact(c, s):
    E, k, H, I = MOE_SIZES[c["size"]]
    h, w, i = _moe_route64(c, s)
    y = s["x"].double().view(-1, H).clone()
    for e in range(E):
        t, slot = torch.where(i == e)
        if t.numel():
            g, u = (h[t] @ s["m"].expert_mlps.gate_up_proj.data[e].double().t()).split(I, -1)
            y.index_add_(0, t, (_silu(g) * u) @ s["m"].expert_mlps.down_proj.data[e].double().t() * w[t, slot].unsqueeze(-1))
    return y.view(s["x"].shape)


def _moe_work(c):
    E, k, H, I = MOE_SIZES[c["size"]]
    T = c["tokens"]
    used = E * (1.0 - (1.0 - k / E) ** T)                       # expected experts that any token chose
    return dict(bytes=2 * used * 3 * H * I + 4 * E * H + 4 * T * H, flops=6 * T * k * H * I + 2 * T * E * H)


# ---- sample -------------------------------------------------------------------------------------------------------------------------
def _sample_prepare(c, seed):
    g = _gen(seed)
    B, V = c["rows"], VOCABS[c["vocab"]]
    rng = random.Random(seed)
    return dict(logits=_randn(g, B, V, dtype=torch.float32 if c["fp32"] else BF, std=2.5),
                k=torch.tensor([rng.choice((1, 10, 40, 50, 200)) for _ in range(B)], device=DEV, dtype=torch.int32),
                p=torch.tensor([rng.choice((0.8, 0.9, 0.95, 1.0)) for _ in range(B)], device=DEV),
                t=torch.tensor([rng.choice((0.0, 0.6, 0.7, 1.0, 1.3)) for _ in range(B)], device=DEV), r=torch.rand(B, device=DEV, generator=g))


def _sample_run(s):
    return ops.sample(s["logits"], s["k"], s["p"], s["t"], s["r"])


def _sample_work(c):
    B, V = c["rows"], VOCABS[c["vocab"]]
    return dict(bytes=B * V * (4 if c["fp32"] else 2) + 24 * B, flops=0)


# ---- llama_step ---------------------------------------------------------------------------------------------------------------------
LLAMA = dict(hidden_size=4096, intermediate_size=14336, num_hidden_layers=4, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
             vocab_size=128256, max_position_embeddings=131072, rms_norm_eps=1e-5, rope_theta=500000.0, tie_word_embeddings=False)


def _llama_prepare(c, seed):
    from neuronx_distributed_inference_b200.config import OnDeviceSamplingConfig
    from neuronx_distributed_inference_b200.utils.testing import build_random_llama
    B, n = c["rows"], c["context"]
    ctx = -(-n // 128) * 128
    app = build_random_llama(LLAMA, batch_size=B, seq_len=ctx + 128, max_context_length=ctx, device=DEV, dtype="bfloat16", seed=seed, skip_warmup=True,
                             enable_bucketing=True, output_logits=True, on_device_sampling_config=OnDeviceSamplingConfig(top_k=1))
    g = torch.Generator()
    g.manual_seed(seed)
    prompt = torch.randint(0, LLAMA["vocab_size"], (B, n), generator=g)
    app(prompt, attention_mask=torch.ones_like(prompt, dtype=torch.int32))
    ids = torch.randint(0, LLAMA["vocab_size"], (B, 1), generator=g).pin_memory()
    pos = torch.full((B, 1), n, dtype=torch.int32).pin_memory()
    app(ids, position_ids=pos)                                      # the step's graph: captured once, as serving warms up
    return dict(app=app, prompt=prompt, ids=ids, pos=pos)


def _llama_run(s):
    o = s["app"](s["ids"], position_ids=s["pos"])
    return o.logits


def _llama_exact(c, s):
    """Logits of the last token from the whole sequence in 64 bits, with the application's weights."""
    sd = {k: v for k, v in s["app"].model.named_parameters()}
    ids = torch.cat([s["prompt"], s["ids"]], 1).to(DEV)
    B, T = ids.shape
    Hq, G, D, eps = 32, 8, 128, 1e-5
    get = lambda name: next(v for k, v in sd.items() if name in k).data          # noqa: E731
    x = get("embed_tokens")[ids].double()
    ang = torch.arange(T, device=DEV).double().view(T, 1) * (500000.0 ** (-torch.arange(0, D, 2, device=DEV).double() / D))
    cos, sin = torch.cat([ang.cos()] * 2, -1).view(1, T, 1, D), torch.cat([ang.sin()] * 2, -1).view(1, T, 1, D)
    rot = lambda t: t * cos + torch.cat([-t[..., D // 2:], t[..., :D // 2]], -1) * sin          # noqa: E731
    see = torch.ones(T, T, device=DEV, dtype=torch.bool).tril()
    for i in range(LLAMA["num_hidden_layers"]):
        lay = lambda name: get("layers.%d.%s" % (i, name)).double()              # noqa: E731,B023
        h = _rms64(x, lay("input_layernorm"), eps)
        qkv = (h @ lay("self_attn.qkv_proj").t()).view(B, T, Hq + 2 * G, D)
        q, k, v = rot(qkv[:, :, :Hq]), rot(qkv[:, :, Hq:Hq + G]).repeat_interleave(Hq // G, 2), qkv[:, :, Hq + G:].repeat_interleave(Hq // G, 2)
        p = torch.softmax((torch.einsum("bthd,bshd->bhts", q, k) * D ** -0.5).masked_fill(~see, float("-inf")), -1)
        x = x + torch.einsum("bhts,bshd->bthd", p, v).reshape(B, T, Hq * D) @ lay("self_attn.o_proj").t()
        g, u = (_rms64(x, lay("post_attention_layernorm"), eps) @ lay("mlp.gate_up_proj").t()).chunk(2, -1)
        x = x + (_silu(g) * u) @ lay("mlp.down_proj").t()
    last = _rms64(x[:, -1], next(v for k, v in sd.items() if "norm" in k and "layers" not in k).data.double(), eps)
    return (last @ get("lm_head").double().t()).view(B, 1, -1)


def _llama_work(c):
    H, I, V, L, B, n = 4096, 14336, 128256, 4, c["rows"], c["context"] + 1
    weights = L * (H * (32 + 16) * 128 + H * H + 3 * H * I) + V * H
    return dict(bytes=2 * weights + L * B * n * 8 * 128 * 4 + 2 * B * (H + V), flops=2 * B * weights + 4 * L * B * n * 32 * 128)


_KINDS = {
    "mlp": (_mlp_prepare, _mlp_run, _mlp_work, _mlp_exact),
    "linear8": (_linear8_prepare, _linear8_run, _linear8_work, _linear8_exact),
    "flash": (_flash_prepare, _flash_run, _flash_work, _flash_exact),
    "paged_step": (_paged_prepare, _paged_run, _paged_work, _paged_exact),
    "portion": (_portion_prepare, _portion_run, _portion_work, _portion_exact),
    "ssd": (_ssd_prepare, _ssd_run, _ssd_work, _ssd_exact),
    "moe": (_moe_prepare, _moe_run, _moe_work, _moe_exact),
    "sample": (_sample_prepare, _sample_run, _sample_work, None),
    "llama_step": (_llama_prepare, _llama_run, _llama_work, _llama_exact),
}

# about four times what each kind shows against ``exact`` (bf16 rows and weights, fp32 sums; the scan is fp32 throughout)
_TOLERANCE = {
    "mlp": {"rel": 0.012}, "linear8": {"rel": 0.01}, "flash": {"rel": 0.01}, "paged_step": {"rel": 0.01}, "portion": {"rel": 0.012},
    "ssd": {"rel": 1e-5, "max": 1e-3}, "moe": {"rel": 0.014}, "sample": {"rel": 0.0, "differ": 0.01}, "llama_step": {"rel": 0.03},
}


def prepare(case, seed):
    with torch.no_grad():
        s = _KINDS[case["kind"]][0](case, seed)
    s["run"] = _KINDS[case["kind"]][1]
    return s


def run(state):
    with torch.no_grad():
        return state["run"](state)


def work(case):
    return _KINDS[case["kind"]][2](case)


def tolerance(case):
    return _TOLERANCE[case["kind"]]


def exact(case, seed):
    fn = _KINDS[case["kind"]][3]
    if fn is None:
        return None
    with torch.no_grad():
        return fn(case, prepare(case, seed))
