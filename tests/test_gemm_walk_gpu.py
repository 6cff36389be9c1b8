"""The order in which a GEMM takes its tiles: every order covers every tile once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [128, 256, 512])
@pytest.mark.parametrize("M,N,K", [
    (4224, 520, 5632),     # rows in groups of eight blocks (what fits in L2 is fewer), a last group
    (520, 4224, 5632),     # the same with columns
    (2304, 2304, 72), (264, 2056, 64), (2056, 264, 64)])  # one group; one block on a side
def test_walk_covers_all_tiles(bn, M, N, K):
    from necklace_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    bias = torch.zeros(N, dtype=torch.bfloat16, device="cuda")   # (no split of K)
    got = gemm(a, b, bias=bias, out=torch.full((M, N), float("nan"), dtype=torch.bfloat16,
                                               device="cuda"), bn=bn).double()
    want, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + mag * (K + 16) * 2.0 ** -24).all())
