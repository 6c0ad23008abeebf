"""A router inside an MoE block is a module like any other: hooks see its result and may replace it, a subclass may override it."""
import torch

from neuronx_distributed_inference_b200.modules.moe import ExpertMLPs, MoE, RouterTopK


def _block(router_class=RouterTopK):
    torch.manual_seed(0)
    m = MoE(router_class(4, 2, 16), ExpertMLPs(4, 16, 8))
    m.router.linear_router.weight.data.normal_()
    for p in m.expert_mlps.parameters():
        p.data.normal_()
    return m, torch.randn(1, 3, 16)


def test_hooks_capture_and_replace_the_routing():
    m, x = _block()
    plain, seen = m(x), []
    handle = m.router.register_forward_hook(lambda mod, args, out: seen.append(out) or None)
    assert torch.equal(m(x), plain) and len(seen) == 1 and seen[0][2].dtype == torch.int64
    handle.remove()
    logits, w, idx = seen[0]
    m.router.register_forward_hook(lambda mod, args, out: (out[0], torch.zeros_like(out[1]), out[2]))
    assert not m(x).any()


def test_a_subclass_decides():
    class First(RouterTopK):
        def forward(self, x):
            logits, w, idx = super().forward(x)
            return logits, torch.ones_like(w) / 2, torch.zeros_like(idx)
    m, x = _block(First)
    one = m.expert_mlps(x.view(3, 16), torch.ones(3, 1), torch.zeros(3, 1, dtype=torch.long))
    assert torch.allclose(m(x).view(3, 16), one, atol=1e-5)
