"""A wait inside a tensor-core kernel that runs out has to reach the caller as an error."""
import pytest
import torch

from neuronx_distributed_inference_b200 import ops
from neuronx_distributed_inference_b200.utils.testing import build_random_llama


def test_every_step_of_the_engine_asks(monkeypatch):
    app = build_random_llama(dict(hidden_size=64, intermediate_size=128, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2,
                                  vocab_size=128, head_dim=16), batch_size=1, seq_len=32, max_context_length=16, device="cpu", dtype="float32")
    ids = torch.randint(0, 128, (1, 8))
    app(ids, attention_mask=torch.ones_like(ids))

    def failed():
        raise RuntimeError("a wait inside the kernel ran out")
    monkeypatch.setattr(ops, "check_waits", failed)
    with pytest.raises(RuntimeError, match="ran out"):
        app(torch.tensor([[3]]), position_ids=torch.tensor([[8]], dtype=torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["asked", "next launch"])
def test_a_wait_that_runs_out_raises_once_and_leaves_the_context_usable(where):
    from neuronx_distributed_inference_b200.ops._ext import load_extension
    ext = load_extension()
    ops.check_waits()
    out = torch.full((1,), 7, device="cuda", dtype=torch.int32)
    ext.wait_probe(1000000, out)                 # half a millisecond on a barrier that nobody arrives on
    torch.cuda.synchronize()
    assert out.item() == 0
    x, w = torch.randn(16, 256, device="cuda", dtype=torch.bfloat16), torch.randn(256, 256, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="wait_probe_kernel.*ran out"):
        ops.check_waits() if where == "asked" else ops.linear(x, w)
    ops.check_waits()
    assert ((ops.linear(x, w).float() - x.float() @ w.float().t()).norm() / (x.float() @ w.float().t()).norm()).item() < 3e-3


@pytest.mark.gpu
def test_the_first_launch_of_a_process_may_be_captured():
    """The words that kernels report to are allocated by the first launch, which may be inside a stream capture."""
    import subprocess
    import sys
    code = """
import torch
from neuronx_distributed_inference_b200 import ops
x, w = torch.randn(16, 256, device="cuda").bfloat16(), torch.randn(256, 256, device="cuda").bfloat16()
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    y = ops.linear(x, w)
g.replay()
torch.cuda.synchronize()
ops.check_waits()
want = x.float() @ w.float().t()
assert ((y.float() - want).norm() / want.norm()).item() < 3e-3
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
