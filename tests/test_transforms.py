"""Function transforms refuse the operators, whether gradients are on or off: an operator that ran
under one would see a batch or a wrapper as a tensor of its own."""
import pytest
import torch

from necklace_b200.ops import LayerNorm, attention_qkv, linear, mlp
from necklace_b200.ops.conv import conv2d

W = torch.randn(16, 8, generator=torch.Generator().manual_seed(0))
CALLS = {"linear": lambda t: linear(t, W), "mlp": lambda t: mlp(t, W, None, W.t(), None),
         "attention": lambda t: attention_qkv(t.repeat(1, 1, 3), 1),
         "norm": LayerNorm(8, dtype=torch.float32),
         "conv": lambda t: conv2d(t[None], W, 1, 1)}


@pytest.mark.parametrize("name", CALLS)
@pytest.mark.parametrize("grad", [False, True])
def test_transforms_are_refused(name, grad):
    f, x = CALLS[name], torch.randn(3, 2, 4, 8)
    with torch.set_grad_enabled(grad):
        f(x[0])
        with pytest.raises(RuntimeError, match="autograd.Function"):
            torch.func.vmap(f)(x)

    def inside(t):
        with torch.set_grad_enabled(grad):
            return f(t).sum() + t.sum()

    with pytest.raises(RuntimeError, match="autograd.Function"):
        torch.func.grad(inside)(x[0])
