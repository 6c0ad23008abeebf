"""Mamba-2 scan in chunks on tensor cores (csrc/ssd_chunk.cu) at the edges of its chunks, against the definition in 64 bits.

Bound: all operands carry at least 24 bits (three bf16 parts), sums are fp32.  A term of an output passes about 8 roundings as in the step-by-step kernel, a
sum of 128 terms in the tensor core's fp32 accumulator adds 8 more that all go towards zero: 16 * 2^-24 = 1e-6 of the sizes of the terms.  The state does
not cancel: 1e-6 of its norm."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from tests.test_ssd_pair_gpu import _definition

pytestmark = pytest.mark.gpu


def _inputs(nh, G, T, lens, dtype):
    B, P, N = len(lens), 64, 128
    inner = nh * P
    xbc = torch.randn(B, T, inner + 2 * G * N, device="cuda")
    wide = torch.randn(B, T, inner + nh + 5, device="cuda", dtype=dtype)          # strided views of one projection
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")             # noqa: E731
    return dict(xBC=xbc, dt_raw=wide[..., inner:inner + nh], z=wide[..., :inner], A_log=torch.rand(nh, device="cuda") * 3, dt_bias=torch.randn(nh, device="cuda") - 1,
                D_skip=torch.randn(nh, device="cuda"), state=torch.randn(B + 2, nh, N, P, device="cuda"), slots=i32([3, 0, 1, 2][:B]), ctx_len=i32([5, 0, 7, 1][:B]),
                q_len=i32(lens)), (nh, P, N, G)


def _run(args, sizes):
    before = dict(ops.kernel_launches())["ssd_chunk"]
    y = ops.ssd_scan(*args.values(), *sizes)
    assert dict(ops.kernel_launches())["ssd_chunk"] == before + 1
    torch.cuda.synchronize()
    ops.check_waits()
    return y


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("nh,G", [(2, 1), (4, 2), (8, 1)])
@pytest.mark.parametrize("T,lens", [(48, (48, 1, 0)), (64, (64, 63)), (65, (65, 64, 2)), (300, (300, 129, 0, 191)), (1000, (1000, 128))])
def test_scan(nh, G, T, lens, dtype):
    args, sizes = _inputs(nh, G, T, lens, dtype)
    want_state = args["state"].clone()
    want, size = _definition(*(dict(args, state=want_state)).values(), *sizes)
    got = _run(args, sizes)
    for b, live in enumerate(lens):
        if live:
            assert ((got[b, :live].double() - want[b, :live]).norm() / size[b, :live].norm()).item() < 1e-6
        assert not got[b, live:].any()
    assert ((args["state"].double() - want_state.double()).norm() / want_state.double().norm()).item() < 1e-6


@pytest.mark.parametrize("where", ["x", "B", "C", "dt", "state"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_values_that_are_not_finite_reach_no_earlier_token_and_no_other_row(where, value):
    args, sizes = _inputs(4, 2, 200, (200, 200), torch.float32)
    want = _run({k: v.clone() for k, v in args.items()}, sizes)
    at, inner = 100, 4 * 64
    if where == "dt":
        args["dt_raw"][0, at, 1] = value
    elif where == "state":
        args["state"][3, 1, 5, 7], at = value, 0
    else:
        args["xBC"][0, at, {"x": 70, "B": inner + 3, "C": inner + 2 * 128 + 3}[where]] = value
    got = _run(args, sizes)
    assert torch.equal(got[1], want[1])
    rel = ((got[0, :at] - want[0, :at]).norm() / want[0, :at].norm().clamp_min(1e-9)).item()
    assert at == 0 or rel < 1e-6
    assert not torch.isfinite(got[0, at:]).all()
    assert torch.isfinite(got[0, :, 128:]).all()                                  # heads 2 and 3: another group


def test_gate_at_the_ends_of_its_range():
    """silu(z) from -inf to inf: the outputs are those of z = 30 (whose silu is 30 to 1e-13) times silu(z) / 30.  Bound: the error of a gate, 6 * 2^-24, on both sides;
    gates below 1e-37 carry the fewer bits of subnormal numbers."""
    args, sizes = _inputs(2, 1, 64, (64,), torch.float32)
    args["slots"].fill_(1)
    inf = float("inf")
    z = torch.tensor([0.0, -0.0, 1.0, -1.0, 20.0, -20.0, 80.0, -80.0, 86.9, -86.9, 87.1, -87.1, 88.0, -88.0, 100.0, -100.0, 1e4, -1e4, 3e35, -1e38, inf, -inf],
                     device="cuda")
    args["xBC"] *= 0.1
    args["state"].zero_()
    args["z"] = torch.full_like(args["z"], 30.0)
    core = _run({k: v.clone() for k, v in args.items()}, sizes).double() / 30.0
    args["z"] = z.repeat(64 * 128 // len(z) + 1)[:64 * 128].view(1, 64, 128).contiguous()
    got, zz = _run(args, sizes).double(), args["z"].double()
    want = core * zz * torch.sigmoid(zz)
    fin = torch.isfinite(zz)
    assert ((got - want).abs()[fin] <= 8e-7 * want.abs()[fin] + 1e-37 * core.abs()[fin]).all()
    assert torch.equal(got[zz == inf], (core * inf)[zz == inf]) and got[zz == -inf].isnan().all()


@pytest.mark.parametrize("what", ["products", "state", "steps"])
def test_operands_whose_products_leave_the_range(what):
    """Products that the recurrence does not form (C B^T before it is weighted with x, S^T C before S has decayed) may leave fp32's range where its own values do not.
    Bound: as above, and a decay e^-a carries an error of a * 2^-23 (a = A dt: 60 and more with the large state)."""
    args, sizes = _inputs(2, 1, 128, (128,), torch.float32)
    args["slots"].fill_(1)
    inner = 128
    args["A_log"].fill_(3.0)
    x, Bm, Cm = args["xBC"][..., :inner], args["xBC"][..., inner:inner + 128], args["xBC"][..., inner + 128:]
    if what == "products":                # C B^T near 1e39
        x *= 1e-8
        Bm *= 1e19
        Cm *= 1e19
    elif what == "state":                 # S^T C near 1e41; the state decays by e^-20 and more before the first token reads it
        args["dt_bias"].fill_(3.0)
        args["state"] *= 1e30
        Cm *= 1e10
    else:                                 # C B^T times the step size
        args["A_log"].fill_(-70.0)
        args["dt_bias"].fill_(600.0)
        x *= 1e-20
        Bm *= 1e18
        Cm *= 1e18
    want_state = args["state"].clone()
    want, size = _definition(*(dict(args, state=want_state)).values(), *sizes)
    got = _run(args, sizes)
    assert torch.isfinite(got).all()
    assert ((got[0].double() - want[0]).norm() / size[0].norm()).item() < (2e-5 if what == "state" else 1e-6)
    assert ((args["state"][1].double() - want_state[1].double()).norm() / want_state[1].double().norm()).item() < 1e-6


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("nh,G", [(2, 1), (8, 2)])
@pytest.mark.parametrize("T,lens", [(48, (1, 48, 23)), (130, (1, 130, 1, 22)), (64, (2, 5, 17, 40))])
def test_rows_of_few_tokens_run_step_by_step(nh, G, T, lens, dtype):
    """Decode rows beside a prompt portion in one padded call: the bits of the step-by-step kernel, which a call of the short rows alone takes."""
    args, sizes = _inputs(nh, G, T, lens, dtype)
    alone = {k: v.clone() for k, v in args.items()}
    got = _run(args, sizes)
    most = 23
    short = [b for b, n in enumerate(lens) if n <= most]
    for k in ("xBC", "dt_raw", "z"):
        alone[k] = alone[k][short, :most]
    for k in ("slots", "ctx_len", "q_len"):
        alone[k] = alone[k][short]
    before = dict(ops.kernel_launches())["ssd_chunk"]
    want = ops.ssd_scan(*alone.values(), *sizes)
    assert dict(ops.kernel_launches())["ssd_chunk"] == before
    for i, b in enumerate(short):
        assert torch.equal(got[b, :most], want[i]) and not got[b, most:].any()
        assert torch.equal(args["state"][alone["slots"][i]], alone["state"][alone["slots"][i]])


def test_workspace_is_bounded():
    """Long prompts run in windows of tokens, many rows in groups: the bits of one window after the other, and no more than 514 MB beside the output."""
    nh, G, P, N = 16, 8, 64, 128
    T, cut = 40000, 37440                 # 585 chunks of 8 groups fill a window
    args, sizes = _inputs(nh, G, T, (T,), torch.bfloat16)
    args["slots"].fill_(1)
    parts = {k: v.clone() for k, v in args.items()}
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    got = _run(args, sizes)
    assert torch.cuda.max_memory_allocated() - base - got.numel() * 4 < 514 << 20
    first = {k: (v[:, :cut].contiguous() if k == "xBC" else v[:, :cut] if k in ("dt_raw", "z") else v) for k, v in parts.items()}
    first["q_len"] = torch.full_like(parts["q_len"], cut)
    y0 = _run(first, sizes)
    rest = {k: (v[:, cut:].contiguous() if k == "xBC" else v[:, cut:] if k in ("dt_raw", "z") else v) for k, v in parts.items()}
    rest["q_len"], rest["ctx_len"] = torch.full_like(parts["q_len"], T - cut), torch.full_like(parts["q_len"], cut)
    y1 = _run(rest, sizes)
    assert torch.equal(got, torch.cat([y0, y1], 1)) and torch.equal(args["state"], parts["state"])


def test_rows_in_groups():
    """More rows than the workspace holds chunks of: a short row, padding and prompts in every group."""
    nh, G, T, B = 256, 128, 64, 40        # 36 rows of 128 groups fill the workspace
    lens = [(64, 1, 50, 0, 33)[b % 5] for b in range(B)]
    args, sizes = _inputs(nh, G, 1, (1,), torch.bfloat16)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")             # noqa: E731
    P, N, inner = 64, 128, nh * 64
    args.update(xBC=torch.randn(B, T, inner + 2 * G * N, device="cuda"), dt_raw=torch.randn(B, T, nh, device="cuda").bfloat16(),
                z=torch.randn(B, T, inner, device="cuda").bfloat16(), state=torch.randn(B, nh, N, P, device="cuda"),
                slots=i32(list(range(B))[::-1]), ctx_len=i32([b % 2 for b in range(B)]), q_len=i32(lens))
    alone = args["state"].clone()
    got = _run(args, sizes)
    for b in range(B):
        one = {k: (alone if k == "state" else v if k in ("A_log", "dt_bias", "D_skip") else v[b:b + 1]) for k, v in args.items()}
        assert torch.equal(_run(one, sizes)[0], got[b])
    assert torch.equal(alone, args["state"])
