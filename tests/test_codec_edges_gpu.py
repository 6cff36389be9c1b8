"""The flat and matrix codec at word, half-word and vector edges: the same bits as the CPU form."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 15, 16, 17, 31, 33, 255, 4099, 1000003])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_flat(n, dt):
    from necklace_b200.ops import dequantize_flat, quantize_flat
    g = torch.Generator().manual_seed(n)
    a = (torch.randn(n, generator=g) * 1e-3).to(dt)
    a[::5] = float("nan") if n > 8 else 1e-3
    a[3:4] = float("inf")
    r = torch.randn(n, generator=g) * 3e-4
    thr = 1e-3
    rc, rg = r.clone(), r.cuda()
    cc, cg = quantize_flat(a, rc, thr), quantize_flat(a.cuda(), rg, thr)
    assert torch.equal(cc, cg.cpu())
    assert torch.equal(rc.view(torch.int32)[~rc.isnan()], rg.cpu().view(torch.int32)[~rc.isnan()])
    assert torch.equal(rc.isnan(), rg.cpu().isnan())
    for off in (0, 1):                       # off = 1: not 16-byte aligned
        for acc in (False, True):
            base = torch.randn(n + 1, generator=g).to(dt)
            oc, og = base[off:off + n].clone(), base.cuda()[off:off + n]
            dequantize_flat(cc, oc, thr, 0.5, acc)
            dequantize_flat(cg, og, thr, 0.5, acc)
            assert torch.equal(oc, og.cpu())


@pytest.mark.parametrize("n,ncol", [(1, 1), (15, 3), (16, 32), (17, 33), (32, 1), (47, 129)])
def test_matrix(n, ncol):
    from necklace_b200.ops import matrix_dequantize, matrix_quantize
    a = torch.randn(n, ncol, generator=torch.Generator().manual_seed(n)) * 1e-3
    cc, rc = matrix_quantize(a, 1e-3)
    cg, rg = matrix_quantize(a.cuda(), 1e-3)
    assert torch.equal(cc, cg.cpu()) and torch.equal(rc, rg.cpu())
    assert torch.equal(matrix_dequantize(cc, n, 1e-3), matrix_dequantize(cg, n, 1e-3).cpu())


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4099, 1000003])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_sum_of_squares(n, dt):
    from necklace_b200.ops.optim import sumsq
    base = torch.randn(n + 1, generator=torch.Generator().manual_seed(n)).to(dt).cuda()
    for off in (0, 1):
        out = torch.zeros(1, device="cuda")
        sumsq(base[off:off + n], out)
        want = base[off:off + n].double().square().sum()
        assert abs(float(out) - float(want)) <= float(want) * (n ** 0.5 + 8) * 2.0 ** -24
