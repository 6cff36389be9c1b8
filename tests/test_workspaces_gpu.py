"""Scratch memory of kernels that go through it: work on several streams, in several threads and in
several captured graphs at the same time gives the bits of the same work one after the other."""
import threading

import pytest
import torch


def test_slices_of_a_gemm():
    from necklace_b200 import _lib
    if not _lib.available():
        pytest.skip("native library not built")
    n = lambda *a: _lib.value("nkb_gemm_slices", *a)  # noqa: E731
    assert n(64, 64, 50000, 64, 0) > 8
    assert n(64, 64, 2047, 64, 0) == 1          # K too short
    assert n(64, 66, 50000, 68, 0) == 1         # columns not in fours
    assert n(64, 64, 50000, 66, 0) == 1
    assert n(8192, 4096, 4096, 4096, 0) == 1    # fills the machine
    assert n(0, 64, 4096, 64, 0) == 1
    assert n(4096, 4096, 1 << 20, 4096, 0) * 4096 * 4096 <= 32 << 20


def _gemms(seed):
    """A few split GEMMs; called again it writes the same outputs."""
    from necklace_b200.ops.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(seed)
    ops = []
    for M, N, K in ((64, 64, 50000), (512, 512, 12544), (256, 1024, 8192)):
        a = torch.randn(K, M, generator=g, device="cuda").bfloat16()
        b = torch.randn(K, N, generator=g, device="cuda").bfloat16()
        ops.append((a, b, torch.empty(M, N, dtype=torch.bfloat16, device="cuda")))

    def run():
        for a, b, o in ops:
            gemm(a, b, a_mn=True, b_mn=True, out=o)
    return run, [o for _, _, o in ops]


def _same_side_by_side(make, how, same=torch.equal):
    from necklace_b200.ops._common import check_status
    runs, outs = zip(*(make(s) for s in range(2)))
    for r in runs:
        r()
    torch.cuda.synchronize()
    want = [[o.clone() for o in out] for out in outs]
    for out in outs:
        for o in out:
            o.zero_()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in runs]
    if how == "streams":
        for _ in range(20):
            for r, s in zip(runs, streams):
                with torch.cuda.stream(s):
                    r()
    elif how == "threads":                            # on one stream, launches in any order
        ts = [threading.Thread(target=lambda r=r: [r() for _ in range(20)]) for r in runs]
        [t.start() for t in ts]
        [t.join() for t in ts]
    else:                                             # captured one after the other, replayed at once
        graphs = []
        for r in runs:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                r()
            graphs.append(g)
        for _ in range(20):
            for g, s in zip(graphs, streams):
                with torch.cuda.stream(s):
                    g.replay()
    torch.cuda.synchronize()
    check_status()
    for out, w in zip(outs, want):
        for o, v in zip(out, w):
            assert same(o, v)


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["streams", "threads", "graphs"])
def test_split_gemms_side_by_side(how):
    _same_side_by_side(_gemms, how)


@pytest.mark.gpu
def test_output_that_a_split_cannot_write():
    """A base between 8-byte boundaries: the GEMM runs whole."""
    from necklace_b200.ops.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(0)
    a = torch.randn(4096, 64, generator=g, device="cuda").bfloat16()
    b = torch.randn(4096, 64, generator=g, device="cuda").bfloat16()
    for dt, rel in ((torch.bfloat16, 2.0 ** -8), (torch.float32, 0.0)):
        flat = torch.empty(64 * 64 + 1, dtype=dt, device="cuda")
        out = gemm(a, b, a_mn=True, b_mn=True, out=flat[1:].view(64, 64))
        want, mag = a.double().t() @ b.double(), a.double().abs().t() @ b.double().abs()
        bound = want.abs() * rel + mag * 4112 * 2.0 ** -24
        assert bool(((out.double() - want).abs() <= bound).all())


def _sums(seed):
    """Norms and column sums there and back; inputs of the two sets are far apart, so that a sum
    that gets a share of the other's shows."""
    from necklace_b200.ops import LayerNorm
    from necklace_b200.ops.conv import BatchNorm2d
    from necklace_b200.ops.gemm import colsum
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    ln, bn = LayerNorm(512, device="cuda"), BatchNorm2d(512, relu=True, device="cuda")
    x = (r(3000, 512) * (1 + 3 * seed) + 4 * seed).bfloat16()
    dy = (r(3000, 512) + 2 - 4 * seed).bfloat16()
    xs = [x.clone().requires_grad_(True) for _ in range(2)]
    outs = [torch.empty_like(t) for t in (ln.weight, ln.bias, xs[0], bn.weight, bn.bias, xs[1],
                                          ln.bias)]

    def run():
        got = torch.autograd.grad(ln(xs[0]), [ln.weight, ln.bias, xs[0]], dy)
        got += torch.autograd.grad(bn(xs[1].view(50, 60, 1, 512)).view(3000, 512),
                                   [bn.weight, bn.bias, xs[1]], dy)
        for o, v in zip(outs, got + (colsum(dy),)):
            o.copy_(v)
    return run, outs


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["streams", "threads", "graphs"])
def test_sums_side_by_side(how):
    # the sums are added in any order (fp32, rounded to bf16 once)
    _same_side_by_side(_sums, how, lambda o, v: bool(
        ((o.double() - v.double()).abs() <= v.double().abs() * 2.0 ** -6
         + v.double().square().mean().sqrt() * 2.0 ** -6).all()))


@pytest.mark.gpu
def test_first_use_inside_a_capture():
    """Scratch made while a graph is captured is cleared by the graph, not by the capture."""
    from necklace_b200.ops.gemm import colsum
    dy = torch.randn(700, 264, device="cuda").bfloat16()
    want = colsum(dy)
    s = torch.cuda.Stream()                           # nothing has run on it yet
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        out = colsum(dy)
    for _ in range(3):
        g.replay()
        torch.cuda.synchronize()
        assert torch.allclose(out.float(), want.float(), rtol=2.0 ** -7, atol=1e-2)
    with torch.cuda.stream(s):                        # the stream's own scratch afterwards
        again = colsum(dy)
    torch.cuda.synchronize()
    assert torch.allclose(again.float(), want.float(), rtol=2.0 ** -7, atol=1e-2)
