"""Mamba-2 scan with two channels per thread (csrc/seqmix.cu) at the edges of its batches of steps, channel blocks and state lanes, against the
definition in 64 bits.

Bound: everything is fp32.  A term of an output (a state element times C, or the skip) carries about 8 roundings (step size, decay, product, update, product,
the tree of sums, the gate) = 8 * 2^-24 = 5e-7 of its own size; outputs may cancel, so the error is held against the sum of the terms' sizes.  The state does
not cancel: 1e-6 of its norm."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,lens", [(1, (1, 1, 0)), (8, (8, 3, 1)), (17, (17, 16, 9)), (40, (33, 40, 24))])
@pytest.mark.parametrize("nh,P,N,G", [(2, 64, 128, 1), (4, 20, 4, 2), (2, 36, 100, 2), (3, 33, 16, 1), (2, 16, 64, 1), (1, 128, 24, 1)])
def test_scan(nh, P, N, G, T, lens, dtype):
    B, inner = 3, nh * P
    xbc = torch.randn(B, T, inner + 2 * G * N, device="cuda")
    wide = torch.randn(B, T, inner + nh + 5, device="cuda", dtype=dtype)          # strided views of one projection
    z, dt = wide[..., :inner], wide[..., inner:inner + nh]
    a, bias, skip = torch.rand(nh, device="cuda") * 2, torch.randn(nh, device="cuda"), torch.randn(nh, device="cuda")
    state = torch.randn(B + 2, nh, N, P, device="cuda")
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")            # noqa: E731
    slots, ctx, n = i32(3, 0, 1), i32(5, 0, 7), i32(*lens)
    want_state = state.clone()
    want, size = _definition(xbc, dt, z, a, bias, skip, want_state, slots, ctx, n, nh, P, N, G)
    got = ops.ssd_scan(xbc, dt, z, a, bias, skip, state, slots, ctx, n, nh, P, N, G)
    for b, live in enumerate(lens):
        if live:
            assert ((got[b, :live].double() - want[b, :live]).norm() / size[b, :live].norm()).item() < 5e-7
    assert ((state.double() - want_state.double()).norm() / want_state.double().norm()).item() < 1e-6


def _definition(xbc, dt, z, a, bias, skip, state, slots, ctx, n, nh, P, N, G):
    """The recurrence of ops/reference.py::ssd_scan in 64 bits, and the sum of the sizes of every output's terms."""
    B, T, inner = xbc.shape[0], xbc.shape[1], nh * P
    out, size = (torch.zeros(B, T, inner, dtype=torch.float64, device="cuda") for _ in range(2))
    for b in range(B):
        S = state[slots[b]].double() if ctx[b] > 0 else torch.zeros(nh, N, P, dtype=torch.float64, device="cuda")
        for t in range(int(n[b])):
            r = xbc[b, t].double()
            x = r[:inner].view(nh, P)
            Bm, Cm = (r[inner + k * G * N:inner + (k + 1) * G * N].view(G, N).repeat_interleave(nh // G, 0) for k in (0, 1))
            step = torch.log1p(torch.exp(dt[b, t].double() + bias.double()))
            S = S * torch.exp(-torch.exp(a.double()) * step).view(nh, 1, 1) + (step.view(nh, 1) * Bm).unsqueeze(-1) * x.unsqueeze(1)
            y = (S * Cm.unsqueeze(-1)).sum(1) + skip.double().view(nh, 1) * x
            zz = z[b, t].double()
            out[b, t] = y.reshape(-1) * zz * torch.sigmoid(zz)
            size[b, t] = ((S.abs() * Cm.abs().unsqueeze(-1)).sum(1) + (skip.double().view(nh, 1) * x).abs()).reshape(-1) * (zz * torch.sigmoid(zz)).abs()
        if int(n[b]) > 0:
            state[slots[b]] = S.float()
    return out, size
