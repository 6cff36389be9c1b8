"""The compiled operators on tensors: what they leave to the general way, and on a GPU the same bits as
it over the forms that they accept."""
import os

import pytest
import torch

from necklace_b200 import _build, _lib

DEV = "cuda"


def test_a_failing_compiler_is_a_warning(tmp_path, monkeypatch):
    target = str(tmp_path / os.path.basename(_build.OPS))
    monkeypatch.setattr(_build, "OPS", target)
    open(target, "w").close()                    # what an earlier build left
    monkeypatch.setenv("CXX", "false")
    with pytest.warns(UserWarning, match="through Python"):
        assert not _build.build_ops(force=True)
    assert not os.listdir(tmp_path)


@pytest.mark.skipif(not os.path.exists(_build.OPS), reason="operators not built")
def test_other_arguments_are_left_to_the_general_way():
    ops = _lib.ops()
    x, w = torch.randn(4, 8).bfloat16(), torch.randn(8, 8).bfloat16()      # not on a GPU
    assert ops.linear(x, w, None, None, 0) is None
    assert ops.linear("x", w, None, None, 0) is None
    assert ops.gemm(x, w, 0, 0, None, 0, 0, 1.0, None, None, 0, None, 0, None, 0) is None
    assert ops.norm(x, w[0], None, "eps", 0) is None
    assert ops.attn(torch.randn(1, 4, 192).bfloat16(), 1.5, 1, 0) is None
    assert ops.bn_eval(x, None, None, 1e-5, w[0], w[0], None, 1) is None
    with pytest.raises(TypeError, match="wanted"):
        ops.linear(x, w)


def _both(monkeypatch, fn):
    """``fn()`` by the compiled operators and the general way."""
    got = fn()
    with monkeypatch.context() as m:
        m.setattr(_lib, "ops", lambda: None)
        want = fn()
    return got, want


def _same(got, want):
    assert len(got) == len(want)
    for a, b in zip(got, want):
        if a is None or b is None:
            assert a is None and b is None
            continue
        assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride()
        assert torch.equal(a, b)


def _rand(*shape, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV).bfloat16()


# leading dimensions, in, out; `gap`: the input is a part of wider rows; `flip`: of transposed storage
FORMS = [((5,), 8, 8, ""), ((2, 3), 72, 136, ""), ((3, 0), 8, 16, "skip"), ((4, 33), 2048, 64, ""),
         ((2, 7), 64, 24, "gap"), ((6, 5), 40, 12, ""), ((3, 4), 16, 16, "flip"), ((9,), 20, 10, "")]


@pytest.mark.gpu
@pytest.mark.parametrize("lead,K,N,form", [f for f in FORMS if f[3] != "skip"])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("res", [False, True])
def test_linear(monkeypatch, lead, K, N, form, bias, res):
    from necklace_b200.ops import linear

    def fn():
        x = _rand(*lead, K + (8 if form == "gap" else 0), seed=1)
        x = x[..., :K] if form == "gap" else x
        x = x.transpose(0, 1) if form == "flip" else x
        x = x.detach().requires_grad_(True)
        w, b = _rand(N, K, seed=2).requires_grad_(True), _rand(N, seed=3).requires_grad_(True)
        r = _rand(*x.shape[:-1], N, seed=4).requires_grad_(True) if res else None
        y = linear(x, w, b if bias else None, r)
        y.backward(_rand(*y.shape, seed=5))
        with torch.no_grad():
            z = linear(x, w, b if bias else None, r)
        return [y.detach(), z, x.grad.contiguous(), w.grad, b.grad, r.grad if res else None]

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("lead,K,F", [((7,), 8, 16), ((2, 5), 72, 264), ((3, 4), 20, 36)])
@pytest.mark.parametrize("frozen_x", [False, True])
def test_mlp_and_flat_gradients(monkeypatch, lead, K, F, frozen_x):
    from necklace_b200.ops import mlp
    from necklace_b200.parallel.flat import FlatParams

    def fn():
        torch.manual_seed(0)
        m = torch.nn.ParameterList([torch.nn.Parameter(_rand(*s, seed=i)) for i, s in
                                    enumerate([(F, K), (F,), (K, F), (K,)])])
        flat = FlatParams(m)
        x = _rand(*lead, K, seed=9).requires_grad_(not frozen_x)
        flat.begin_step()
        for _ in range(2):                       # the second pass adds to the first one's gradients
            y = mlp(x, m[0], m[1], m[2], m[3], residual=x)
            y.backward(_rand(*y.shape, seed=10))
        flat.finish_backward()
        with torch.no_grad():
            z = mlp(x, m[0], m[1], m[2], m[3])
        return [y.detach(), z, x.grad, flat.grad]

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(5, 8), (2, 3, 264), (4, 1, 1024)])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("flip", [False, True])
def test_norms(monkeypatch, shape, rms, split, flip):
    from necklace_b200.ops.norm import LayerNorm, RMSNorm

    def fn():
        n = (RMSNorm if rms else LayerNorm)(shape[-1], device=DEV)
        x = _rand(*shape, seed=1)
        x = (x.transpose(0, 1) if flip and x.dim() > 2 else x).detach().requires_grad_(True)
        a, y = n.split(x) if split else (x, n(x))
        out = y + a if split else y
        out.backward(_rand(*out.shape, seed=2))
        with torch.no_grad():
            z = n(x)
        return [y.detach().contiguous(), z.contiguous(), x.grad.contiguous(), n.weight.grad,
                None if rms else n.bias.grad]

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("S,H,D,causal", [(1, 1, 64, True), (130, 3, 64, False), (200, 2, 128, True)])
def test_attention(monkeypatch, S, H, D, causal):
    from necklace_b200.ops.attention import attention_qkv, attn_bwd, attn_fwd

    def fn():
        qkv = _rand(2, S, 3 * H * D, seed=1).requires_grad_(True)
        out = attention_qkv(qkv, H, causal)
        out.backward(_rand(*out.shape, seed=2))
        o, lse = attn_fwd(qkv.detach(), H, causal)
        assert (attn_bwd(qkv.detach(), o, lse, _rand(2, H * D, S, seed=2).transpose(1, 2), H,
                         causal)).shape == qkv.shape     # a gradient of other strides
        return [out.detach(), o, lse], qkv.grad

    (got, gd), (want, wd) = _both(monkeypatch, fn)
    _same(got, want)
    # dQ's fp32 sums over key blocks arrive in any order
    assert ((gd.float() - wd.float()).norm() / wd.float().norm()).item() < 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("C,Cout,k,stride", [(64, 64, 1, 1), (64, 128, 3, 1), (128, 64, 3, 2),
                                             (64, 128, 1, 2), (3, 64, 7, 2), (20, 24, 1, 1)])
@pytest.mark.parametrize("flip", [False, True])
def test_evaluated_convolutions_and_norms(monkeypatch, C, Cout, k, stride, flip):
    from necklace_b200.ops.conv import BatchNorm2d, Conv2d

    def fn():
        torch.manual_seed(1)
        conv = Conv2d(C, Cout, k, stride, k // 2, device=DEV)
        bn = BatchNorm2d(Cout, relu=True, device=DEV).eval()
        bn.running_mean.normal_()
        bn.running_var.uniform_(0.5, 1.5)
        x = _rand(3, 28, 24, C, seed=1)
        x = x.transpose(1, 2) if flip and k == stride == 1 and C % 8 == 0 else x
        with torch.no_grad():
            y = conv(x)
            z = bn(y, y) if Cout % 8 == 0 else y
            t = bn(y.transpose(1, 2)) if Cout % 8 == 0 else y
        return [y, z, t.contiguous()]

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
def test_wrong_arguments_fail_as_before():
    from necklace_b200.ops import gemm
    a, b = _rand(8, 16), _rand(8, 24)
    with pytest.raises(AssertionError, match="contraction"):
        gemm(a, b)
    with pytest.raises(AssertionError):
        gemm(a.float(), _rand(8, 16).float())
    with pytest.raises(AssertionError):
        gemm(a, _rand(8, 16), bias=_rand(9))
