"""The one-pass norm backward (dx, weight and bias gradient) against fp64 autograd on the same bf16
values: one row, fewer rows than a batch, more rows than one round of the grid; columns below a
warp, at and around the 512- and 1024-thread forms, at the largest size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, mag, terms):
    # bf16 rounding of the result and fp32 sums of `terms` products (each a few roundings)
    bound = want.abs() * 2.0 ** -8 + mag * (terms + 16) * 2.0 ** -24 + 1e-30
    err = (got.double() - want).abs()
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("rows,C", [(1, 8), (3, 64), (5, 256), (2500, 264), (700, 1024),
                                    (33, 2048), (9, 4096), (600, 4096), (7, 4104), (301, 8192)])
@pytest.mark.parametrize("rms,res", [(False, True), (True, False)])
def test_against_fp64(rows, C, rms, res):
    from necklace_b200.ops.norm import LayerNorm, RMSNorm
    from necklace_b200.parallel.flat import FlatParams
    g = torch.Generator(device="cuda").manual_seed(rows + C)
    mod = (RMSNorm(C, device="cuda") if rms else LayerNorm(C, device="cuda"))
    with torch.no_grad():
        for p in mod.parameters():
            p.copy_(torch.randn(C, generator=g, device="cuda"))
    x = (torch.randn(rows, C, generator=g, device="cuda") + 0.5).bfloat16().requires_grad_(True)
    dy = torch.randn(rows, C, generator=g, device="cuda").bfloat16()
    dr = torch.randn(rows, C, generator=g, device="cuda").bfloat16()
    flat = FlatParams(mod)
    flat.begin_step()

    def backward():
        alias, y = mod.split(x)
        torch.autograd.backward([alias, y] if res else [y], [dr, dy] if res else [dy])

    backward()
    xd = x.detach().double().requires_grad_(True)
    wd = mod.weight.detach().double().requires_grad_(True)
    bd = mod.bias.detach().double().requires_grad_(True) if not rms else None
    mean = 0.0 if rms else xd.mean(1, keepdim=True)
    rstd = torch.rsqrt(((xd - mean) ** 2).mean(1, keepdim=True) + mod.eps)
    xhat = (xd - mean) * rstd
    out = xhat * wd + (bd if bd is not None else 0.0)
    out.backward(dy.double())
    dx = xd.grad + (dr.double() if res else 0.0)
    a = (dy.double() * wd).abs()
    r, h = rstd.detach(), xhat.detach().abs()
    # the statistics are fp32, so xhat carries their rounding
    mag = r * (a + a.mean(1, keepdim=True) + h * (a * h).mean(1, keepdim=True))
    _close(x.grad, dx, mag * 8 + dr.abs().double() * res, 1)
    _close(mod.weight._nkb_grad, wd.grad, (dy.double().abs() * (h + r * xd.detach().abs())).sum(0),
           rows)
    if not rms:
        _close(mod.bias._nkb_grad, bd.grad, dy.double().abs().sum(0), rows)
    once = flat.grad.clone()
    backward()                                    # second micro-batch: adds to the first
    want = 2 * once.double()
    # the sum once more, its rows in any order, on top of the rounded first one: roundings of 2^-9
    # of each, and where a sum cancels the fp32 error of its terms
    slack = 2.0 ** -7 * want.abs() + 1e-30
    for p, m in ((mod.weight, (dy.double().abs() * (h + r * xd.detach().abs())).sum(0)),
                 (getattr(mod, "bias", None), dy.double().abs().sum(0))):
        if p is not None:
            o = (p._nkb_grad.data_ptr() - flat.grad.data_ptr()) // 2
            slack[o:o + C] += m * 2 * (rows + 16) * 2.0 ** -24
    assert bool(((flat.grad.double() - want).abs() <= slack).all())
