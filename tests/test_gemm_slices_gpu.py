"""GEMMs with few output tiles and a long contraction, cut into many slices, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, mag, terms):
    # bf16 rounding of the result and fp32 sums of `terms` products (each a few roundings)
    bound = want.abs() * 2.0 ** -8 + mag * (terms + 16) * 2.0 ** -24 + 1e-30
    err = (got.double() - want).abs()
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("M,N,K", [(64, 64, 50000), (64, 256, 20011), (132, 68, 9000),
                                   (512, 512, 12544), (256, 64, 2048)])
def test_long_contractions_in_many_slices(M, N, K):
    from necklace_b200.ops.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(K)
    a = torch.randn(K, M, generator=g, device="cuda").bfloat16()
    b = torch.randn(K, N, generator=g, device="cuda").bfloat16()
    out = gemm(a, b, a_mn=True, b_mn=True)
    want = a.double().t() @ b.double()
    mag = a.double().abs().t() @ b.double().abs()
    _close(out, want, mag, K)
    acc = gemm(a, b, a_mn=True, b_mn=True, out=out.clone(), accumulate=True)
    assert bool(((acc.double() - 2 * want).abs() <= want.abs() * 2.0 ** -6 + mag * K * 2.0 ** -23).all())


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [
    (333, 776, 768, 0, 0), (333, 1024, 4104, 0, 1),          # 128 x 128, whole and split
    (771, 3080, 768, 0, 1), (2313, 1032, 2752, 0, 0),        # 128 x 256
    (4097, 3072, 1032, 0, 0), (1032, 1024, 8200, 1, 1),      # pairs, whole and split
    (129, 129, 64, 0, 0), (128, 264, 2048, 0, 0)])
def test_every_kind_of_tile_that_the_sizes_choose(M, N, K, a_mn, b_mn):
    from necklace_b200.ops.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(*((K, M) if a_mn else (M, K)), generator=g, device="cuda").bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), generator=g, device="cuda").bfloat16()
    A, B = (a.t() if a_mn else a).double(), (b.t() if b_mn else b).double()
    _close(gemm(a, b, a_mn=bool(a_mn), b_mn=bool(b_mn)), A @ B.t(), A.abs() @ B.abs().t(), K)


@pytest.mark.parametrize("M,N,K", [(64, 64, 2048), (64, 64, 4096), (64, 64, 4608), (132, 260, 4160),
                                   (1032, 1024, 8200)])
@pytest.mark.parametrize("fp32", [False, True])
def test_reduction_of_few_and_many_slices(M, N, K, fp32):
    """Up to eight slices are added by one thread per group of columns, more by four: both, at the
    line between them, written and added to, with rows apart."""
    from necklace_b200 import _lib
    from necklace_b200.ops.gemm import gemm
    assert _lib.value("nkb_gemm_slices", M, N, K, N + 8, 0) > 1
    g = torch.Generator(device="cuda").manual_seed(K)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    want, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    wide = torch.full((M, N + 8), 3.0, dtype=torch.float32 if fp32 else torch.bfloat16,
                      device="cuda")
    out, rel = wide[:, :N], 0.0 if fp32 else 2.0 ** -8
    gemm(a, b, out=out, alpha=0.5)
    assert bool(((out.double() - want / 2).abs() <= want.abs() * rel + mag * (K + 16) * 2.0 ** -24).all())
    gemm(a, b, out=out, accumulate=True, alpha_dev=torch.full((1,), 2.0, device="cuda"))
    bound = want.abs() * 4 * rel + mag * (K + 16) * 2.0 ** -21
    assert bool(((out.double() - 2.5 * want).abs() <= bound).all())
    assert bool((wide[:, N:] == 3).all())


@pytest.mark.parametrize("M,N,K", [(333, 1024, 4096), (64, 68, 2048), (129, 260, 4608)])
@pytest.mark.parametrize("bias,res,pitch,shift", [(True, False, 0, 0), (True, True, 0, 0),
                                                  (False, True, 4, 0), (True, True, 2, 0),
                                                  (True, True, 0, 1)])
def test_slices_with_bias_and_residual(M, N, K, bias, res, pitch, shift):
    """The kernel that adds the slices adds bias and residual; rows or bases that it cannot read four
    values at a time go through one slice."""
    from necklace_b200 import _lib
    from necklace_b200.ops.gemm import gemm
    assert _lib.value("nkb_gemm_slices", M, N, K, N, 0) > 1
    g = torch.Generator(device="cuda").manual_seed(K)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    # (a bias is contiguous in any case; rows of the residual may lie apart)
    bv = torch.randn(N + shift, generator=g, device="cuda").bfloat16()[shift:] if bias else None
    r = torch.randn(M, N + pitch, generator=g, device="cuda").bfloat16()[:, :N] if res else None
    want, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    if bias:
        want, mag = want + bv.double(), mag + bv.double().abs()
    if res:
        want, mag = want + r.double(), mag + r.double().abs()
    _close(gemm(a, b, bias=bv, res=r), want, mag, K)
    out32 = gemm(a, b, bias=bv, res=r, out_dtype=torch.float32)
    assert bool(((out32.double() - want).abs() <= mag * (K + 16) * 2.0 ** -24).all())
