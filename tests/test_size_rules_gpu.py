"""Sizes on both sides of the rules between kernel variants, against 64 bits.

Bounds: fp32 sums, results (and normalised rows) rounded to bf16: 1.7e-3 rms each."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-9)).item()


def _launched(call):
    before = ops.kernel_launches()
    call()
    return {k: n - before[k] for k, n in ops.kernel_launches().items() if n > before[k]}


@pytest.mark.parametrize("wdtype", [BF, torch.int8, torch.float8_e4m3fn])
@pytest.mark.parametrize("N,K", [(800, 512), (792, 512), (1184, 512), (1192, 1024), (1600, 1024), (2368, 2048), (2384, 2048), (2050, 512), (4096, 1536), (8192, 512), (16400, 512)])
def test_two_gemv_kernels_per_sm(wdtype, N, K):
    """A second tile for the busiest CTA, a CTA on every SM, one and two stages a tile; 4, 5 and 8 tokens change what fits.  Launched back to back, so that they overlap."""
    w = torch.randn(N, K, device=DEV) / K ** 0.5
    q, s = (w.to(BF), None) if wdtype == BF else ref.quantize_per_channel(w, wdtype)
    wd = q.double() if s is None else q.double() * s.double().view(-1, 1)
    n = torch.randn(K, device=DEV, dtype=BF)
    xs = [torch.randn(T, K, device=DEV, dtype=BF) for T in (1, 4, 5, 8)]
    plain = [ops.linear(x, q, scale=s) for x in xs for _ in range(3)][::3]
    normed = [ops.linear(x, q, norm_weight=n, norm_eps=1e-5, scale=s) for x in xs for _ in range(3)][::3]
    gated = [ops.linear(x, q, scale=s, act="silu_mul") for x in xs for _ in range(3)][::3] if N % 16 == 0 else []
    for i, x in enumerate(xs):
        h = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * n.double()
        assert _rel(plain[i], x.double() @ wd.t()) < 3e-3
        assert _rel(normed[i], h @ wd.t()) < 6e-3
        if gated:
            assert _rel(gated[i], ref.linear(x.double(), wd, act="silu_mul")) < 5e-3


@pytest.mark.parametrize("rows", [1, 296, 297, 444, 445, 592, 593, 888, 889, 1023])
@pytest.mark.parametrize("H", [8, 2048, 4104, 16384])
def test_norm_blocks_per_sm(rows, H):
    x, r, w = torch.randn(rows, H, device=DEV, dtype=BF), torch.randn(rows, H, device=DEV, dtype=BF), torch.randn(H, device=DEV, dtype=BF)
    want = lambda v: v.double() * torch.rsqrt(v.double().pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    assert _rel(ops.rmsnorm(x, w, 1e-5), want(x)) < 2.5e-3
    y, s = ops.rmsnorm(x, w, 1e-5, residual=r)
    assert torch.equal(s, x + r) and _rel(y, want(s)) < 2.5e-3


@pytest.mark.parametrize("T,N,K,act,kernel", [
    (65, 4096, 2048, None, "gemm_tcgen05"), (65, 2048, 4096, None, "skinny_gemm"), (80, 3200, 3200, None, "skinny_gemm"), (81, 3200, 3200, None, "gemm_tcgen05"),
    (80, 8320, 3072, None, "gemm_tcgen05"), (128, 512, 1024, None, "skinny_gemm"), (33, 2048, 4096, "silu_mul", "gemm_tcgen05"), (64, 4096, 4096, "silu_mul", "skinny_gemm"),
    (64, 512, 8192, "silu_mul", "skinny_gemm")])
def test_few_token_gemm(T, N, K, act, kernel):
    x, w = torch.randn(T, K, device=DEV, dtype=BF), torch.randn(N, K, device=DEV, dtype=BF) / K ** 0.5
    out = []
    assert _launched(lambda: out.append(ops.linear(x, w, act=act))) == {kernel: 1}
    assert _rel(out[0], ref.linear(x.double(), w.double(), act=act)) < 3e-3


@pytest.mark.parametrize("T,N,K,act,kernel", [
    (32, 512, 384, None, "skinny_gemm"), (33, 512, 384, None, "gemm_tcgen05"), (64, 512, 512, None, "skinny_gemm"), (65, 512, 512, None, "gemm_tcgen05"),
    (96, 2048, 1024, None, "skinny_gemm"), (97, 2048, 1024, None, "gemm_tcgen05"), (256, 8192, 512, None, "skinny_gemm"), (257, 8192, 512, None, "gemm_pair"),
    (192, 2048, 2048, None, "skinny_gemm"), (193, 2048, 2048, None, "gemm_tcgen05"), (512, 512, 2048, None, "skinny_gemm"), (512, 256, 4096, None, "skinny_gemm"),
    (32, 512, 128, "silu_mul", "skinny_gemm"), (33, 512, 512, "silu_mul", "gemm_tcgen05"), (48, 2048, 1024, "silu_mul", "skinny_gemm"), (49, 2048, 1024, "silu_mul", "gemm_tcgen05")])
def test_small_8_bit_weights(T, N, K, act, kernel):
    q, s = ref.quantize_per_channel(torch.randn(N, K, device=DEV) / K ** 0.5, torch.float8_e4m3fn)
    x = torch.randn(T, K, device=DEV, dtype=BF)
    out = []
    assert _launched(lambda: out.append(ops.linear(x, q, scale=s, act=act))) == {kernel: 1}
    assert _rel(out[0], ref.linear(x.double(), q.double() * s.double().view(-1, 1), act=act)) < 3e-3
