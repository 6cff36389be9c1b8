"""The 1x1 convolution at the head of a residual block, whose data gradient also adds the gradient of
the residual path, against fp64; a module with hooks is called as such."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, mag, terms):
    # bf16 rounding of the result and fp32 sums of `terms` products (each a few roundings)
    bound = want.abs() * 2.0 ** -8 + mag * (terms + 16) * 2.0 ** -24 + 1e-30
    err = (got.double() - want).abs()
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("shape", [(1, 1, 1, 8), (3, 7, 5, 72), (2, 9, 9, 256)])
def test_residual_head_adds_the_other_gradient(shape):
    from necklace_b200.ops.conv import Conv2d
    g = torch.Generator(device="cuda").manual_seed(1)
    conv = Conv2d(shape[-1], 40, 1, device="cuda")
    x = torch.randn(shape, generator=g, device="cuda").bfloat16().requires_grad_(True)
    dy = torch.randn(*shape[:3], 40, generator=g, device="cuda").bfloat16()
    dr = torch.randn(shape, generator=g, device="cuda").bfloat16()
    alias, y = conv.split(x)
    assert torch.equal(y, conv(x)) and alias.data_ptr() == x.data_ptr()
    torch.autograd.backward([alias, y], [dr, dy])
    w = conv.weight.detach().double()
    want = dy.double() @ w + dr.double()
    _close(x.grad, want, dy.double().abs() @ w.abs() + dr.double().abs(), 40)
    x.grad = None
    alias, y = conv.split(x)
    (alias.sum() + y.sum()).backward()            # expanded gradients
    want = w.sum(0).expand(shape) + 1.0
    _close(x.grad, want, w.abs().sum(0).expand(shape) + 1.0, 40)
    calls = []
    conv.register_forward_hook(lambda *a: calls.append(1))
    alias, y = conv.split(x)                      # a hooked module is called
    assert calls and alias is x
