"""The gather of layers with odd channel counts, the max pooling gradient and evaluation-mode batch
norm against their CPU forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(2, 9, 11, 3, 7, 7, 2, 3), (1, 5, 200, 3, 3, 3, 1, 1),
                                  (3, 8, 8, 5, 2, 3, 1, 0), (2, 6, 7, 12, 3, 3, 2, 1),
                                  (1, 4, 130, 1, 1, 1, 1, 0), (1, 3, 3, 1001, 3, 3, 1, 1),
                                  (1, 2, 2, 4099, 3, 3, 1, 1)])
def test_gather_of_odd_channel_counts(case):
    from necklace_b200.ops.conv import im2col
    N, H, W, C, KH, KW, s, p = case
    x = torch.randn(N, H, W, C, generator=torch.Generator().manual_seed(C)).bfloat16()
    assert torch.equal(im2col(x, KH, KW, s, p), im2col(x.cuda(), KH, KW, s, p).cpu())


@pytest.mark.parametrize("shape", [(1, 1, 1, 8), (2, 3, 4, 16), (3, 7, 5, 64), (1, 16, 17, 8)])
def test_max_pool_gradient(shape):
    from necklace_b200.ops.conv import max_pool_3x3_s2
    n = int(torch.tensor(shape).prod())          # distinct values: one winner per window
    x = (torch.randperm(n, generator=torch.Generator().manual_seed(3)) % 251 - 125).view(shape)
    x = x.bfloat16()
    a, b = x.clone().requires_grad_(True), x.cuda().requires_grad_(True)
    ya, yb = max_pool_3x3_s2(a), max_pool_3x3_s2(b)
    g = torch.randn(ya.shape, generator=torch.Generator().manual_seed(4)).bfloat16()
    ya.backward(g)
    yb.backward(g.cuda())
    assert torch.equal(ya, yb.cpu())
    # up to four windows are added in fp32 and rounded once on both sides
    assert torch.allclose(a.grad.float(), b.grad.cpu().float(), rtol=2.0 ** -8, atol=1e-6)


@pytest.mark.parametrize("C,relu,res", [(8, False, False), (72, True, True), (2048, True, False)])
@pytest.mark.parametrize("half_stats", [False, True])
def test_evaluation_batch_norm(C, relu, res, half_stats):
    from necklace_b200.ops.conv import BatchNorm2d
    g = torch.Generator().manual_seed(C)
    x = torch.randn(3, 5, 7, C, generator=g).bfloat16()
    r = torch.randn(3, 5, 7, C, generator=g).bfloat16() if res else None
    bn = BatchNorm2d(C, relu=relu).eval()
    bn.running_mean.copy_(torch.randn(C, generator=g) * 0.1)
    bn.running_var.copy_(torch.rand(C, generator=g) + 0.5)
    if half_stats:                        # a model converted as a whole
        bn.running_mean, bn.running_var = bn.running_mean.bfloat16(), bn.running_var.bfloat16()
    m, v = bn.running_mean.double(), bn.running_var.double()
    want = (x.double() - m) * torch.rsqrt(v + bn.eps) + (r.double() if res else 0.0)
    want = torch.relu(want) if relu else want
    got = bn.cuda()(x.cuda(), r.cuda() if res else None).cpu().double()
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -19).all())


@pytest.mark.parametrize("eps", [1e-5, 0.0, 1e-3])
def test_evaluation_batch_norm_bits(eps):
    """Variance and eps in the kernel give the bits of (mean, torch.rsqrt(variance + eps)): the
    same layer with statistics of another kind of memory takes that way."""
    from necklace_b200.ops.conv import BatchNorm2d
    g = torch.Generator(device="cuda").manual_seed(1)
    C = 4096
    bn = BatchNorm2d(C, eps=eps, device="cuda").eval()
    with torch.no_grad():
        bn.weight.copy_(torch.randn(C, generator=g, device="cuda"))
        bn.bias.copy_(torch.randn(C, generator=g, device="cuda"))
    bn.running_mean.normal_(generator=g)
    bn.running_var.copy_(torch.rand(C, generator=g, device="cuda").add(1e-4) * 4)
    x = torch.randn(64, 1, 1, C, generator=g, device="cuda").bfloat16()
    one = bn(x)
    bn.running_mean = torch.stack([bn.running_mean, bn.running_mean], 1)[:, 0]   # strided
    assert not bn.running_mean.is_contiguous()
    assert torch.equal(one, bn(x))


@pytest.mark.parametrize("C", [24, 72, 136, 264, 520, 8192])
@pytest.mark.parametrize("M", [1, 13, 5003])
def test_batch_norm_strips(C, M):
    """Channel counts whose chunks of 8 do not fill a power of two, there and back against fp64."""
    from necklace_b200.ops.conv import BatchNorm2d
    g = torch.Generator(device="cuda").manual_seed(C + M)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    bn = BatchNorm2d(C, relu=True, device="cuda")
    with torch.no_grad():
        bn.weight.copy_(r(C) * 0.3 + 1), bn.bias.copy_(r(C))
    x = (r(M, 1, 1, C) + r(C)).bfloat16().requires_grad_(True)
    res = r(M, 1, 1, C).bfloat16().requires_grad_(True)
    dy = r(M, 1, 1, C).bfloat16()
    y = bn(x, res)
    y.backward(dy)
    xd = x.detach().double().view(M, C).requires_grad_(True)
    wd, bd = (t.detach().double().requires_grad_(True) for t in (bn.weight, bn.bias))
    var, mean = torch.var_mean(xd, 0, unbiased=False)
    rstd = torch.rsqrt(var + bn.eps)
    xhat = (xd - mean) * rstd
    out = xhat * wd + bd + res.detach().double().view(M, C)
    # fp32 statistics: a rounding of the mean or of a square moves xhat by about 2^-22 of the
    # channel's (largest value / spread)^2; one row has no spread but eps
    move = 2.0 ** -22 * (1 + (xd.detach().abs().amax(0) * rstd.detach()).square())
    err = (y.detach().double().view(M, C) - torch.relu(out)).abs()
    assert bool((err <= out.abs() * 2.0 ** -8 + move * wd.abs() * 4 + 1e-6).all())
    on = (y.detach().view(M, C) > 0).double()            # the signs of the stored output
    d = dy.double().view(M, C) * on
    assert torch.equal(res.grad.double().view(M, C), d)
    out.backward(d)
    h = xhat.detach().abs() + move
    for got, want, mag in ((bn.bias.grad, bd.grad, d.abs().sum(0)),
                           (bn.weight.grad, wd.grad, (d.abs() * h).sum(0))):
        slack = mag * ((M + 16) * 2.0 ** -24 + move * 4)
        assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-6).all())
    k = (wd.abs() * rstd).detach()
    mag = k * (d.abs() + d.abs().mean(0) + h * (d.abs() * h).mean(0))
    bound = xd.grad.abs() * 2.0 ** -8 + mag * ((M + 16) * 2.0 ** -24 + move * 8) + 1e-6
    assert bool(((x.grad.double().view(M, C) - xd.grad).abs() <= bound).all())
