"""Top-k / top-p sampling over rows whose order or ties stress the group bound, row lengths around the slice size, unaligned rows, and the
exhaustive path, against the PyTorch definition (tokens are equal: ties go to the lowest index there and here)."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _rows(kind, B, V, dtype):
    if kind == "random":
        return (torch.randn(B, V) * 3).to(dtype)
    if kind == "sorted":                                  # the largest values side by side
        return torch.linspace(-9, 9, V).expand(B, V).to(dtype).contiguous()
    if kind == "block":                                   # one stretch far above the rest
        x = torch.randn(B, V)
        x[:, V // 3:V // 3 + 300] += 40
        return x.to(dtype)
    return torch.randint(0, 4, (B, V)).to(dtype)          # "ties": long runs of equal values


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [1, 7, 256, 1000, 8191, 8192, 8193, 32000, 50257, 128256, 262144, 300001])
@pytest.mark.parametrize("kind", ["random", "sorted", "block", "ties"])
def test_tokens(kind, V, dtype):
    B = 6
    logits = _rows(kind, B, V, dtype).cuda()
    # an exact order of equal values: the definition's top-k on the CPU keeps no order among them, so distinct values are compared by token,
    # rows with ties by the value drawn
    top_k = torch.tensor([1, 5, 50, 0, 256, 10], dtype=torch.int32)
    top_p = torch.tensor([1.0, 0.9, 0.5, 1.0, 0.95, 1.0])
    temp = torch.tensor([1.0, 0.7, 1.3, 1.0, 0.0, 2.0])
    rand = torch.tensor([0.11, 0.97, 0.42, 0.63, 0.5, 0.29])
    got = ops.sample(logits, top_k.cuda(), top_p.cuda(), temp.cuda(), rand.cuda(), 256)
    want = ref.sample(logits.float().cpu(), top_k, top_p, temp, rand, 256)
    rows = torch.arange(B)
    value = logits.float().cpu()
    assert torch.equal(value[rows, got.cpu()], value[rows, want])
    if kind != "ties" and dtype == torch.float32:
        assert torch.equal(got.cpu(), want)


def test_more_rows_than_a_grid_dimension():
    """66000 rows: more than the second dimension of a grid can count."""
    B, V = 66000, 40
    logits = torch.randn(B, V, device="cuda")
    one = torch.ones(B, device="cuda")
    got = ops.sample(logits, torch.ones(B, device="cuda", dtype=torch.int32), one, one, one * 0.5)
    assert torch.equal(got, logits.argmax(-1))


@pytest.mark.parametrize("near", [1, 40, 70, 400, 32000])
@pytest.mark.parametrize("k", [1, 50, 200])
def test_values_that_share_their_leading_bytes(k, near):
    """The bound's last bytes are looked at only where many groups share the leading ones."""
    B, V = 4, 32000
    logits = torch.randn(B, V)
    for b in range(B):
        at = torch.randperm(V)[:near]
        logits[b, at] = 8.0 + torch.randperm(near).float() * 1e-6       # one 16-bit prefix
    one = torch.ones(B)
    top_k, rand = torch.full((B,), k, dtype=torch.int32), torch.rand(B)
    got = ops.sample(logits.cuda(), top_k.cuda(), one.cuda(), one.cuda(), rand.cuda())
    assert torch.equal(got.cpu(), ref.sample(logits, top_k, one, one, rand))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_strided_parameters(dtype):
    """Columns of one parameter matrix, and of one matrix of draws, give what dense copies of them give."""
    B, V = 5, 4000
    logits = (torch.randn(B, V, device="cuda") * 3).to(dtype)
    params = torch.stack([torch.randint(1, 200, (B,), device="cuda").float(), torch.linspace(0.2, 1.0, B, device="cuda"), torch.linspace(1.5, 0.3, B, device="cuda")], -1)
    ks, rand = torch.stack([params[:, 0].int(), torch.ones(B, device="cuda", dtype=torch.int32)], -1), torch.rand(B, 7, device="cuda")
    got = ops.sample(logits, ks[:, 0], params[:, 1], params[:, 2], rand[:, 3], global_topk=256)
    dense = [t.clone(memory_format=torch.contiguous_format) for t in (ks[:, 0], params[:, 1], params[:, 2], rand[:, 3])]
    assert torch.equal(got, ops.sample(logits, *dense, global_topk=256))
    assert torch.equal(got, ops.sample(logits, params[:, 0], params[:, 1], params[:, 2], rand[:, 3], global_topk=256))
    assert torch.equal(ops.sample(logits, ks[:, 0], params[:, 1], params[:, 2], global_topk=256), ops.sample(logits, *dense[:3], global_topk=256))


@pytest.mark.parametrize("bad", range(4))
def test_parameters_of_another_length(bad):
    args = [torch.ones(3 if i == bad else 4, device="cuda") for i in range(4)]
    with pytest.raises(RuntimeError):
        ops.sample(torch.randn(4, 100, device="cuda"), *args)
