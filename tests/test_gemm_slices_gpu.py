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
