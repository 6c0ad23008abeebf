"""Arguments of ops.linear that its kernels do not take as they are: the few-row kernels read norm weights and biases as dense bf16."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16
TYPES = [BF, torch.int8, torch.float8_e4m3fn]


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-9)).item()


def _layer(T, N, K, wdtype):
    x, w, n = torch.randn(T, K, device=DEV, dtype=BF), torch.randn(N, K, device=DEV) / K ** 0.5, torch.randn(K, device=DEV)
    q, s = (w.to(BF), None) if wdtype == BF else ref.quantize_per_channel(w, wdtype)
    h = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5)
    return x, q, s, n, h, q.double() if s is None else q.double() * s.double().view(-1, 1)


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T,K", [(1, 512), (8, 512), (9, 512), (8, 11008), (600, 512)])
def test_norm_weight_of_another_type(wdtype, T, K):
    """fp32 norm weights, as checkpoints keep them, at every number of rows (rows, x gamma and result are rounded to bf16; from 513 rows on 8-bit weights too)."""
    x, q, s, n, h, w = _layer(T, 136, K, wdtype)
    assert _rel(ops.linear(x, q, norm_weight=n, norm_eps=1e-5, scale=s), (h * n.double()) @ w.t()) < 8e-3


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T", [1, 8, 9])
def test_strided_norm_weight(wdtype, T):
    x, q, s, n, h, w = _layer(T, 136, 512, wdtype)
    n2 = torch.stack([n.to(BF), torch.zeros_like(n, dtype=BF)], -1)[:, 0]
    assert _rel(ops.linear(x, q, norm_weight=n2, norm_eps=1e-5, scale=s), (h * n2.double()) @ w.t()) < 8e-3


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T", [1, 8, 9, 600])
def test_norm_weight_of_another_length(wdtype, T):
    x, q, s, n, _, _ = _layer(T, 136, 512, wdtype)
    with pytest.raises(RuntimeError):
        ops.linear(x, q, norm_weight=n.to(BF)[:256].contiguous(), scale=s)


@pytest.mark.parametrize("wdtype", TYPES)
@pytest.mark.parametrize("T", [1, 8, 9, 600])
def test_bias(wdtype, T):
    """A strided bias counts as its dense copy; one of another type is refused, as F.linear refuses it, and so is one of another length."""
    x, q, s, _, _, w = _layer(T, 136, 512, wdtype)
    b = torch.randn(136, device=DEV)
    b2 = torch.stack([b.to(BF), torch.zeros_like(b, dtype=BF)], -1)[:, 0]
    assert _rel(ops.linear(x, q, b2, scale=s), x.double() @ w.t() + b2.double()) < 5e-3
    for bad in (b, b.to(BF)[:64].contiguous()):
        with pytest.raises(RuntimeError):
            ops.linear(x, q, bad, scale=s)


@pytest.mark.parametrize("wdtype", TYPES[1:])
@pytest.mark.parametrize("T", [1, 9, 600])
def test_scale_in_host_memory(wdtype, T):
    x, q, s, _, _, _ = _layer(T, 136, 512, wdtype)
    with pytest.raises(RuntimeError):
        ops.linear(x, q, scale=s.cpu())


def test_fp8_rows_and_weights(monkeypatch):
    """W8A8: strided norm weights and biases count as their dense copies, scales may be a slice; other types and lengths are refused."""
    monkeypatch.setattr(ops, "_ACT_QUANT", True)
    x, q, s, n, _, _ = _layer(20, 136, 512, torch.float8_e4m3fn)
    n2, b2 = torch.randn(512, 2, device=DEV).to(BF)[:, 0], torch.randn(136, 2, device=DEV).to(BF)[:, 0]
    want = ops.linear(x, q, b2.contiguous(), norm_weight=n2.contiguous(), scale=s)
    assert torch.equal(ops.linear(x, q, b2, norm_weight=n2, scale=s), want)
    assert torch.equal(ops.linear(x, q, b2, norm_weight=n2, scale=torch.cat([s[:1], s])[1:]), want)
    for kw in (dict(bias=b2.float()), dict(bias=b2[:64].contiguous()), dict(norm_weight=n2[:64].contiguous())):
        with pytest.raises(RuntimeError):
            ops.linear(x, q, scale=s, **kw)


@pytest.mark.parametrize("wdtype", TYPES[1:])
@pytest.mark.parametrize("T,N,K", [(20, 136, 512), (100, 512, 512), (300, 8192, 512), (200, 1024, 1024)])
def test_scales_of_a_slice(wdtype, T, N, K):
    """Scales that start off a 16-byte boundary, through every kernel that loads several at a time (the last size: a split K)."""
    x, q, s, _, _, w = _layer(T, N, K, wdtype)
    assert _rel(ops.linear(x, q, scale=torch.cat([s[:1], s])[1:]), x.double() @ w.t()) < 3e-3
