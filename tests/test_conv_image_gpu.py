"""The convolution kernels that read the image itself, against ``F.conv2d`` in fp64 on the same
bf16 values.  Shapes sit at the edges of the boxes of positions (a last box that is nearly empty,
fewer positions than a box, boxes over several images), of the 64-channel chunks and of the
column tiles, with every class of a strided data gradient and a window smaller than the stride."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

# N, H, W, Cin, Cout, kernel, stride, padding
SHAPES = [
    (1, 1, 1, 8, 8, 3, 1, 1), (1, 5, 7, 8, 16, 3, 1, 1), (3, 9, 11, 64, 64, 3, 1, 1),
    (2, 8, 16, 64, 72, 3, 1, 1), (5, 7, 7, 72, 136, 3, 1, 1), (129, 2, 1, 128, 64, 3, 1, 1),
    (2, 13, 17, 40, 264, 3, 2, 1), (4, 14, 14, 256, 512, 1, 2, 0), (3, 7, 9, 64, 128, 1, 2, 0),
    (2, 16, 16, 136, 64, 3, 2, 1), (2, 12, 10, 16, 24, 5, 1, 2), (2, 12, 10, 16, 24, 5, 2, 0),
    (1, 131, 3, 24, 40, 3, 1, 1), (2, 6, 200, 32, 32, 3, 2, 1), (2, 9, 9, 320, 8, 3, 1, 0),
    (2, 20, 20, 8, 16, 7, 2, 3), (2, 6, 6, 64, 64, 2, 1, 1), (33, 40, 53, 64, 128, 3, 1, 1),
]


def _close(got, want, scale, terms):
    # bf16 rounding of the result (2^-8 of the value) and fp32 sums of `terms` products, whose
    # error is at most terms * 2^-24 of the sum of magnitudes (`scale`)
    err = (got.double() - want).abs()
    bound = want.abs() * 2.0 ** -8 + scale * (terms * 2.0 ** -24) + 1e-30
    assert bool((err <= bound).all()), float((err / bound).max())


def _run(shape, seed=0):
    from necklace_b200.ops.conv import Conv2d, _image_kernels
    N, H, W, ci, co, k, s, p = shape
    g = torch.Generator(device="cuda").manual_seed(seed)
    conv = Conv2d(ci, co, k, s, p, device="cuda")
    x = torch.randn(N, H, W, ci, generator=g, device="cuda").bfloat16().requires_grad_(True)
    assert _image_kernels(x, conv.weight, k, k, s, p)
    y = conv(x)
    dy = torch.randn(y.shape, generator=g, device="cuda").bfloat16()
    y.backward(dy)
    return conv, x, y, dy


@pytest.mark.parametrize("shape", SHAPES)
def test_image_kernels_match_torch(shape):
    from necklace_b200.ops._common import check_status
    N, H, W, ci, co, k, s, p = shape
    conv, x, y, dy = _run(shape)
    check_status()
    xr = x.detach().double().permute(0, 3, 1, 2).requires_grad_(True)
    wr = conv.weight_oihw().detach().double().requires_grad_(True)
    ref = F.conv2d(xr, wr, stride=s, padding=p)
    ref.backward(dy.double().permute(0, 3, 1, 2))
    xa, wa = xr.detach().abs().requires_grad_(True), wr.detach().abs().requires_grad_(True)
    mag = F.conv2d(xa, wa, stride=s, padding=p)
    mag.backward(dy.double().abs().permute(0, 3, 1, 2))
    _close(y.detach(), ref.detach().permute(0, 2, 3, 1), mag.detach().permute(0, 2, 3, 1),
           k * k * ci)
    # every tap's product is rounded to bf16 before the taps are added: 2^-8 of the magnitudes
    _close(x.grad, xr.grad.permute(0, 2, 3, 1), xa.grad.permute(0, 2, 3, 1),
           k * k * co + (2 ** 16 if k > 1 else 0))
    gw = conv.weight.grad[:, :k * k * ci].view(co, k, k, ci).permute(0, 3, 1, 2)
    _close(gw, wr.grad, wa.grad, y.numel() // co)


def test_weight_gradient_accumulates_into_the_flat_buffer():
    from necklace_b200.parallel.flat import FlatParams
    from necklace_b200.ops.conv import Conv2d
    conv = Conv2d(24, 40, 3, 1, 1, device="cuda")
    flat = FlatParams(conv)
    x = torch.randn(2, 9, 9, 24, device="cuda").bfloat16()
    flat.begin_step()
    conv(x).sum().backward()
    once = flat.grad.clone()
    conv(x).sum().backward()
    assert torch.allclose(flat.grad.float(), 2 * once.float(), rtol=2 ** -7, atol=1e-3)


def test_other_layers_keep_the_gathered_form():
    from necklace_b200.ops.conv import Conv2d, _image_kernels
    for ci, co, k, s in ((3, 16, 7, 2), (16, 12, 3, 1), (16, 16, 3, 3)):
        conv = Conv2d(ci, co, k, s, k // 2, device="cuda")
        x = torch.randn(2, 12, 12, ci, device="cuda").bfloat16()
        assert not _image_kernels(x, conv.weight, k, k, s, k // 2)
        ref = F.conv2d(x.float().permute(0, 3, 1, 2), conv.weight_oihw().float(), stride=s,
                       padding=k // 2).permute(0, 2, 3, 1)
        assert torch.allclose(conv(x).float(), ref, rtol=2 ** -7, atol=2e-2)
