"""The compressed all-reduce on one rank against the codec's arithmetic: word edges, both gradient
types, buffers that 16-byte accesses cannot take."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 4096, 4096 + 5, 100003])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 1])
def test_one_rank(n, dt, off):
    from necklace_b200.comm.symm import SymmetricHeap
    heap = SymmetricHeap(8 << 20)
    grp = heap.peer_group()
    gen = torch.Generator().manual_seed(n)
    base = (torch.randn(n + 1, generator=gen) * 1e-3).to(dt).cuda()
    res = (torch.randn(n, generator=gen) * 3e-4).cuda()
    g = base[off:off + n]
    words = (n + 15) // 16
    codes, counts = heap.alloc(words, torch.int32), heap.alloc(words * 16, torch.int8)
    a = g.float() + res
    thr, scale = torch.tensor(1e-3, device="cuda"), 0.5
    pos, neg = a >= thr, a <= -thr
    want_res = torch.where(pos, a - thr, torch.where(neg, a + thr, a))
    want = ((pos.float() - (neg & ~pos).float()) * (thr * scale)).to(dt)
    grp.dp_quant_allreduce(g, res, codes, counts, g, 1e-3, scale)
    torch.cuda.synchronize()
    assert torch.equal(res, want_res) and torch.equal(g, want)
