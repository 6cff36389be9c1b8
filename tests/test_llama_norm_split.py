"""Norms of a Llama block: the residual path's gradient is added in the norm's backward, and whatever
looks at the module's calls sees them."""
import torch
import torch.nn as nn

from necklace_b200.models.llama import Llama, LlamaConfig
from necklace_b200.ops.norm import RMSNorm


def _net():
    cfg = LlamaConfig(n_layer=1, d_model=128, n_head=1, d_ff=64, max_seq=16)
    return Llama(cfg, layers=range(1), with_embed=False, with_head=False, seed=0)


def _pass(net):
    g = torch.Generator().manual_seed(1)
    x = torch.randn(2, 9, 128, generator=g).bfloat16().requires_grad_(True)
    y = net(x)
    y.backward(torch.randn(y.shape, generator=g).bfloat16())
    return y.detach(), x.grad, {n: p.grad for n, p in net.named_parameters()}


class _Plain(nn.Module):
    def __init__(self, norm):
        super().__init__()
        self.inner = norm

    def forward(self, x):
        return self.inner(x)


def test_gradients_are_those_of_a_norm_and_a_sum():
    y, dx, grads = _pass(_net())
    net = _net()
    blk = net.blocks[0] if isinstance(net.blocks, nn.ModuleList) else net.blocks["0"]
    blk.ln1, blk.ln2 = _Plain(blk.ln1), _Plain(blk.ln2)     # not split: autograd adds the two
    y2, dx2, grads2 = _pass(net)
    assert torch.equal(y, y2)
    # the sum is rounded to bf16 once instead of twice, in both norms
    assert (dx.float() - dx2.float()).norm() <= 2.0 ** -7 * dx2.float().norm()
    for n, g in grads2.items():
        h = grads[n.replace(".inner", "")]
        assert (h.float() - g.float()).norm() <= 2.0 ** -6 * g.float().norm() + 1e-6


def test_hooks_and_subclasses_are_called():
    seen = []
    net = _net()
    blk = net.blocks[0] if isinstance(net.blocks, nn.ModuleList) else net.blocks["0"]
    blk.ln1.register_forward_hook(lambda m, a, out: seen.append("hook"))

    class Twice(RMSNorm):
        def forward(self, x):
            seen.append("subclass")
            return super().forward(x)

    other = Twice(128)
    other.load_state_dict(blk.ln2.state_dict())
    blk.ln2 = other
    y, _, _ = _pass(net)
    assert seen == ["hook", "subclass"]
    assert torch.equal(y, _pass(_net())[0])
