"""int8 / fp8 weights of 9 .. 512 tokens, and of fewer with rows too wide for the GEMV (csrc/skinny_gemm.cu): the bytes are expanded on their way to the tensor cores.

Bound: rows are bf16, products and sums fp32, the scale is applied to the sum: results are rounded to bf16 once (2^-9 at most, 1.7e-3 rms)."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16
TYPES = [torch.int8, torch.float8_e4m3fn]


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-9)).item()


def _want(x, q, s, bias=None, act=None):
    return ref.linear(x.double(), q.double() * s.double().view(-1, 1), None if bias is None else bias.double(), act=act)


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T", [9, 16, 17, 37, 64, 65, 100, 128, 129, 250, 257, 512])
@pytest.mark.parametrize("N,K", [(8, 128), (136, 256), (4104, 384), (1000, 4096), (256, 14336), (20000, 128)])
def test_plain(wdtype, T, N, K):
    q, s = ref.quantize_per_channel(torch.randn(N, K, device=DEV) * 0.02, wdtype)
    x = torch.randn(T, K, device=DEV, dtype=BF)
    b, r = torch.randn(N, device=DEV, dtype=BF), torch.randn(T, N, device=DEV, dtype=BF)
    assert _rel(ops.linear(x, q, scale=s), _want(x, q, s)) < 3e-3
    assert _rel(ops.linear(x, q, b, scale=s, residual=r), _want(x, q, s, b) + r.double()) < 3e-3
    assert _rel(ops.linear(x, q, scale=s.view(-1)[:1].contiguous()), _want(x, q, s.view(-1)[:1])) < 3e-3


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T,I,K", [(9, 72, 128), (32, 1344, 512), (37, 14336, 4096), (64, 8640, 3840), (65, 200, 2048)])
@pytest.mark.parametrize("act", ["silu_mul", "gelu_tanh_mul"])
def test_gate_product(wdtype, T, I, K, act):
    q, s = ref.quantize_per_channel(torch.randn(2 * I, K, device=DEV) / K ** 0.5, wdtype)
    x = torch.randn(T, K, device=DEV, dtype=BF)
    b, n = torch.randn(2 * I, device=DEV, dtype=BF), torch.randn(K, device=DEV, dtype=BF)
    # above 64 tokens the weight itself is rounded to bf16
    assert _rel(ops.linear(x, q, b, scale=s, act=act), _want(x, q, s, b, act)) < (3e-3 if T <= 64 else 6e-3)
    h = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * n.double()
    assert _rel(ops.linear(x, q, b, norm_weight=n, norm_eps=1e-5, scale=s, act=act), _want(h, q, s, b, act)) < 8e-3


@pytest.mark.parametrize("wdtype", TYPES)
def test_every_byte(wdtype):
    """All 256 values of a byte, in every position of a 16-byte piece: the expansion is exact (fp8: NaN stays NaN)."""
    K = 256
    q = torch.arange(256, device=DEV).view(256, 1).add(torch.arange(K, device=DEV)).remainder(256).to(torch.uint8).view(wdtype)
    x = torch.zeros(16, K, device=DEV, dtype=BF)
    for t in range(16):
        x[t, 17 * t % K] = 1.0
    got = ops.linear(x, q, scale=torch.ones(256, device=DEV))
    want = torch.stack([q[:, 17 * t % K].float() for t in range(16)])
    bad = torch.isnan(q.float()).any(-1)                       # 0 x NaN is NaN
    assert torch.equal(got[:, ~bad].float(), want[:, ~bad])
    assert torch.isnan(got[:, bad]).all()
    if not bad.all():
        return
    q = torch.where(torch.isnan(q.float()), torch.zeros_like(q.float()), q.float()).to(wdtype)
    assert torch.equal(ops.linear(x, q, scale=torch.ones(256, device=DEV)).float(), torch.stack([q[:, 17 * t % K].float() for t in range(16)]))


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T,N,K", [(8, 4096, 11008), (7, 256, 14336), (8, 1000, 10624), (3, 136, 32768), (1, 8, 110592), (8, 1001, 11008)])
def test_rows_too_wide_for_the_gemv(wdtype, T, N, K):
    """1 .. 8 rows that do not fit one SM's shared memory; 1001 weight rows and a norm stay with the warp-per-row kernel."""
    q, s = ref.quantize_per_channel(torch.randn(N, K, device=DEV) / K ** 0.5, wdtype)
    x, b = torch.randn(T, K, device=DEV, dtype=BF), torch.randn(N, device=DEV, dtype=BF)
    r, n = torch.randn(T, N, device=DEV, dtype=BF), torch.randn(K, device=DEV, dtype=BF)
    wide = torch.randn(T, K + 8, device=DEV, dtype=BF)
    assert _rel(ops.linear(x, q, scale=s), _want(x, q, s)) < 3e-3
    assert _rel(ops.linear(wide[:, 8:], q, scale=s), _want(wide[:, 8:], q, s)) < 3e-3
    assert _rel(ops.linear(x, q, b, scale=s, residual=r), _want(x, q, s, b) + r.double()) < 3e-3
    assert _rel(ops.linear(x, q, scale=s.view(-1)[:1].contiguous()), _want(x, q, s.view(-1)[:1])) < 3e-3
    if N % 16 == 0:
        assert _rel(ops.linear(x, q, b, scale=s, act="silu_mul"), _want(x, q, s, b, "silu_mul")) < 3e-3
    h = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * n.double()
    assert _rel(ops.linear(x, q, norm_weight=n, norm_eps=1e-5, scale=s), _want(h, q, s)) < 6e-3


@pytest.mark.parametrize("wdtype", [BF, *TYPES])
@pytest.mark.parametrize("K", [128, 2048, 4096, 4224])
@pytest.mark.parametrize("norm", [False, True])
def test_rows_of_a_step_do_not_depend_on_their_number(wdtype, K, norm):
    """1 .. 8 rows are normalised and converted in pairs and a rest: each row has the bits that it has alone."""
    x, w = torch.randn(8, K, device=DEV, dtype=BF), torch.randn(512, K, device=DEV) / K ** 0.5
    w, s = (w.to(BF), None) if wdtype == BF else ref.quantize_per_channel(w, wdtype)
    n = torch.randn(K, device=DEV, dtype=BF) if norm else None
    one = torch.cat([ops.linear(x[t:t + 1], w, norm_weight=n, scale=s) for t in range(8)])
    for T in range(1, 9):
        assert torch.equal(ops.linear(x[:T], w, norm_weight=n, scale=s), one[:T])


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T,N,K", [(65, 512, 512), (128, 4096, 1024), (129, 1000, 384), (200, 8192, 1024), (257, 2048, 2048), (300, 8200, 512), (512, 136, 256), (512, 16384, 1024)])
def test_expanded_weights_are_not_rounded(wdtype, T, N, K):
    """Sizes whose bytes are expanded in memory first (both tile kernels, cut tiles): the scale goes to the sum, so only the result is rounded (1.7e-3 rms; 2.4e-3
    with a rounded weight)."""
    q, s = ref.quantize_per_channel(torch.randn(N, K, device=DEV) / K ** 0.5, wdtype)
    x, b, r = torch.randn(T, K, device=DEV, dtype=BF), torch.randn(N, device=DEV, dtype=BF), torch.randn(T, N, device=DEV, dtype=BF)
    before = dict(ops.stats)
    assert _rel(ops.linear(x, q, scale=s), _want(x, q, s)) < 1.9e-3
    assert ops.stats["dequant_gemm"] == before["dequant_gemm"] + 1
    assert _rel(ops.linear(x, q, b, scale=s, residual=r), _want(x, q, s, b) + r.double()) < 3e-3
    assert _rel(ops.linear(x, q, scale=s.view(-1)[:1].contiguous()), _want(x, q, s.view(-1)[:1])) < 1.9e-3


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T,I,K", [(33, 72, 128), (64, 500 * 8, 256), (64, 1024, 1024)])
def test_expanded_weights_with_a_gate_product(wdtype, T, I, K):
    q, s = ref.quantize_per_channel(torch.randn(2 * I, K, device=DEV) / K ** 0.5, wdtype)
    x, b = torch.randn(T, K, device=DEV, dtype=BF), torch.randn(2 * I, device=DEV, dtype=BF)
    before = dict(ops.stats)
    for act in ("silu_mul", "gelu_mul"):
        assert _rel(ops.linear(x, q, b, scale=s, act=act), _want(x, q, s, b, act)) < 3e-3
        assert _rel(ops.linear(x, q, scale=s.view(-1)[:1].contiguous(), act=act), _want(x, q, s.view(-1)[:1], None, act)) < 3e-3
    assert ops.stats["dequant_gemm"] == before["dequant_gemm"] + 4
