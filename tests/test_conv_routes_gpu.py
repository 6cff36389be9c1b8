"""Calls that the convolution kernels on the image must leave to the gathered form, or answer as it
does."""
import importlib

import pytest
import torch
import torch.nn.functional as F

from test_conv_image_gpu import SHAPES, test_image_kernels_match_torch

pytestmark = pytest.mark.gpu


def _rand(*s, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*s, generator=g, device="cuda").bfloat16()


def _close(got, want, mag, terms):
    # bf16 rounding of the result and fp32 sums of `terms` products (each a few roundings)
    bound = want.abs() * 2.0 ** -8 + mag * (terms + 16) * 2.0 ** -24 + 1e-30
    err = (got.double() - want).abs()
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("route", [0, 1, 2, 3])
@pytest.mark.parametrize("shape", SHAPES)
def test_every_route_at_every_shape(shape, route, monkeypatch):
    monkeypatch.setattr(importlib.import_module("necklace_b200.ops.conv"), "_route",
                        lambda *a: route)
    test_image_kernels_match_torch(shape)


@pytest.mark.parametrize("stride", [1, 2])
def test_negative_padding_cuts_the_border_off(stride):
    from necklace_b200.ops.conv import conv2d
    x, w = _rand(2, 9, 10, 16).requires_grad_(True), _rand(24, 9 * 16, seed=1).requires_grad_(True)
    y = conv2d(x, w, 3, 3, stride, -1)
    inner = x.detach()[:, 1:-1, 1:-1].contiguous().requires_grad_(True)
    w2 = w.detach().clone().requires_grad_(True)
    ref = conv2d(inner, w2, 3, 3, stride, 0)
    assert torch.allclose(y.float(), ref.float(), rtol=2.0 ** -7, atol=1e-2)
    dy = _rand(*y.shape, seed=2)
    y.backward(dy)
    ref.backward(dy)
    assert torch.allclose(w.grad.float(), w2.grad.float(), rtol=2.0 ** -7, atol=1e-2)
    # taps are rounded to bf16 each
    assert torch.allclose(x.grad[:, 1:-1, 1:-1].float(), inner.grad.float(), rtol=2.0 ** -6,
                          atol=0.1)
    border = x.grad.clone()
    border[:, 1:-1, 1:-1] = 0
    assert not border.any()


def test_saved_tensors_that_come_back_strided():
    """Saved-tensor hooks may give back the same values in another layout."""
    from necklace_b200.ops.conv import conv2d
    grads = []
    dy = _rand(2, 9, 10, 24, seed=2)
    for unpack in (lambda t: t, lambda t: t.transpose(0, -1).contiguous().transpose(0, -1)):
        x, w = _rand(2, 9, 10, 16).requires_grad_(True), _rand(24, 144, seed=1).requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            y = conv2d(x, w, 3, 3, 1, 1)
        y.backward(dy)
        grads.append((x.grad, w.grad))
    for a, b in zip(*grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_weight_gradient_into_a_buffer_of_another_kind(dtype):
    """A gradient buffer in fp32 gets the fp32 sums; one that is not aligned is rounded once."""
    from necklace_b200.ops.conv import conv2d
    x, w, dy = _rand(3, 9, 10, 16), _rand(24, 144, seed=1), _rand(3, 9, 10, 24, seed=2)
    w = torch.nn.Parameter(w)
    flat = torch.zeros(24 * 144 + 1, dtype=dtype, device="cuda")
    w._nkb_grad, w._nkb_grad_has = flat[1:].view(24, 144), False
    ref = []
    for d in (dy, _rand(3, 9, 10, 24, seed=3)):
        conv2d(x, w, 3, 3, 1, 1).backward(d)
        for v in (x.double(), x.double().abs()):
            wr = torch.zeros(24, 16, 3, 3, dtype=torch.float64, device="cuda", requires_grad=True)
            y = F.conv2d(v.permute(0, 3, 1, 2), wr, padding=1)
            y.backward((d.double() if v.min() < 0 else d.double().abs()).permute(0, 3, 1, 2))
            ref.append(wr.grad.permute(0, 2, 3, 1).reshape(24, 144))
    want, mag = ref[0] + ref[2], ref[1] + ref[3]
    # fp32 sums of 270 products twice; bf16: the first sum is rounded too
    bound = mag * 300 * 2.0 ** -24 * 4
    if dtype == torch.bfloat16:
        bound = bound + (ref[0].abs() + want.abs()) * 2.0 ** -8
    assert bool(((w._nkb_grad.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("k,pad", [(1, 0), (3, 0), (2, 0)])
def test_pixels_that_no_window_has(k, pad):
    """The last row and column of an image that the stride does not divide."""
    from necklace_b200.ops.conv import _conv_wgrad
    N, H, W, ci, co = 3, 8, 10, 16, 24
    if k == 2:
        H, W = 9, 11
    x, w = _rand(N, H, W, ci), _rand(co, k * k * ci, seed=1)
    Ho, Wo = (H - k) // 2 + 1, (W - k) // 2 + 1
    dy = _rand(N, Ho, Wo, co, seed=2)
    clean = _conv_wgrad(x, dy.reshape(-1, co), w, k, k, 2, pad, None, False)
    x[:, (Ho - 1) * 2 + k:] = float("inf")
    x[:, :, (Wo - 1) * 2 + k:] = float("nan")
    assert not x.isfinite().all()
    assert torch.equal(clean, _conv_wgrad(x, dy.reshape(-1, co), w, k, k, 2, pad, None, False))
