"""Which tensor-core kernel a call takes: the size rules of csrc/bindings.cpp and ops, read off the extension's launch counters."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def _launched(call):
    before = ops.kernel_launches()
    call()
    return {k: n - before[k] for k, n in ops.kernel_launches().items() if n > before[k]}


@pytest.mark.parametrize("T,N,K,act,kernel", [
    (9, 512, 512, None, "skinny_gemm"), (64, 512, 512, None, "skinny_gemm"), (65, 512, 512, None, "gemm_tcgen05"), (128, 256, 512, None, "skinny_gemm"),
    (129, 512, 512, None, "gemm_tcgen05"), (513, 512, 512, None, "gemm_pair"), (256, 10240, 512, None, "gemm_pair"), (256, 9984, 512, None, "gemm_tcgen05"),
    (32, 1024, 512, "silu_mul", "skinny_gemm"), (33, 1024, 512, "silu_mul", "gemm_tcgen05"), (64, 16384, 4096, "silu_mul", "skinny_gemm"),
    (256, 10240, 512, "silu_mul", "gemm_pair")])
def test_linear(T, N, K, act, kernel):
    x, w = torch.randn(T, K, device=DEV, dtype=BF), torch.randn(N, K, device=DEV, dtype=BF)
    assert _launched(lambda: ops.linear(x, w, act=act)) == {kernel: 1}


@pytest.mark.parametrize("N,kernel", [(3, "skinny_gemm"), (128, "skinny_gemm"), (129, "gemm_pair")])
def test_experts(N, kernel):
    E, k, H, I = 8, 2, 256, 192
    x, wg, wd = (torch.randn(*s, device=DEV, dtype=BF) for s in ((N, H), (E, 2 * I, H), (E, H, I)))
    i, w = torch.rand(N, E, device=DEV).topk(k, -1).indices, torch.rand(N, k, device=DEV)
    assert _launched(lambda: ops.moe_experts(x, wg, wd, w, i)) == {kernel: 2}


@pytest.mark.parametrize("D", [64, 128])
def test_attention(D):
    q, k = torch.randn(1, 40, 4, D, device=DEV, dtype=BF), torch.randn(1, 40, 2, D, device=DEV, dtype=BF)
    assert _launched(lambda: ops.attention_prefill(q, k, k, D ** -0.5)) == {"attention_prefill_tc": 1}
    cache, table = torch.randn(4, 16, 2, D, device=DEV, dtype=BF), torch.arange(4, device=DEV, dtype=torch.int32).view(1, 4)
    ctx, n = torch.tensor([9], device=DEV, dtype=torch.int32), torch.tensor([40], device=DEV, dtype=torch.int32)
    for cap in (0.0, 30.0):
        assert _launched(lambda: ops.paged_window_attention(q, cache, cache, table, ctx, n, D ** -0.5, cap, 0, 0)) == {"attention_prefill_tc": 1}
