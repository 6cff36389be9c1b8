"""The convolution at the head of a residual block is called as a module where that can be noticed,
and computes no gradient that nobody asked for."""
import torch
import torch.nn as nn

from necklace_b200.models.resnet import Bottleneck
from necklace_b200.ops.conv import Conv2d


def _x(**kw):
    return torch.randn(2, 5, 4, 32, generator=torch.Generator().manual_seed(0), **kw).bfloat16()


def test_another_module_in_its_place():
    block = Bottleneck(32, 8, 1, False)
    want = block(_x().requires_grad_(True))

    class Wrapper(nn.Module):
        def __init__(self, conv):
            super().__init__()
            self.conv = conv

        def forward(self, x):
            return self.conv(x)

    block.conv1 = Wrapper(block.conv1)
    assert torch.equal(want, block(_x().requires_grad_(True)))


def test_what_sees_calls_of_the_module():
    x = _x().requires_grad_(True)
    conv = Conv2d(32, 8, 1)
    assert conv.split(x)[0] is not x

    class Twice(Conv2d):
        def forward(self, t):
            return 2 * super().forward(t)

    sub = Twice(32, 8, 1)
    alias, y = sub.split(x)
    assert alias is x and torch.equal(y, sub(x))
    plain = conv(x).detach()
    conv.forward = lambda t: 3 * Conv2d.forward(conv, t)
    alias, y = conv.split(x)
    assert alias is x and torch.equal(y, 3 * plain)
    del conv.forward
    seen = []
    h = nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(m))
    try:
        assert conv.split(x)[0] is x and seen == [conv]
    finally:
        h.remove()
    assert conv.split(x)[0] is not x


def test_input_without_gradient_stays_without():
    """A frozen stem: the residual path must not start to compute a gradient for it."""
    conv = Conv2d(32, 8, 1)
    alias, y = conv.split(_x())
    assert not alias.requires_grad and y.requires_grad
    y.sum().backward()
    assert conv.weight.grad is not None
