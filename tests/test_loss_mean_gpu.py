"""Mean loss and its gradient factor in one launch each: around the block size, with ignored targets,
with none left."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 31, 33, 1023, 1024, 1025, 8192])
@pytest.mark.parametrize("ignored", [0.0, 0.3, 1.0])
def test_against_fp64(T, ignored):
    from necklace_b200.ops.loss import _loss_corr, _mean_loss
    g = torch.Generator().manual_seed(T)
    losses = torch.rand(T, generator=g) * 10
    targets = torch.randint(0, 9, (T,), generator=g)
    drop = torch.rand(T, generator=g) < ignored
    targets[drop], losses[drop] = -100, 0.0
    loss, n = _mean_loss(losses.cuda(), targets.cuda())
    want_n = max(1, int((targets >= 0).sum()))
    want = losses.double().sum() / want_n
    assert int(n) == want_n and loss.shape == ()
    # at most T / 1024 + 10 additions in a chain, then a division
    assert abs(float(loss) - float(want)) <= float(want) * (T / 1024 + 12) * 2.0 ** -24
    d = torch.tensor(0.37, device="cuda")
    assert float(_loss_corr(d, n, T)) == pytest.approx(float(d) * T / want_n, rel=2.0 ** -22)
