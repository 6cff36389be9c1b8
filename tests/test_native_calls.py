"""The compiled call layer against ctypes, and operators without an autograd node (gradients off)
against the same operators with one: same values, and the node stays where something looks at it."""
import pytest
import torch


def _nkpy():
    from necklace_b200 import _lib
    if not _lib.available():
        pytest.skip("native library not built")
    if not _lib._fast:
        pytest.skip("extension not built")
    return _lib


def test_same_answers_as_ctypes():
    lib = _nkpy()
    ct = lib.load().nkb_conv_wgrad_split
    for geom in ((1, 1, 1, 8, 8, 3, 3, 1, 1), (256, 56, 56, 64, 64, 3, 3, 1, 1),
                 (33, 40, 53, 64, 128, 3, 3, 2, 1), (2, 9, 9, 12, 8, 3, 3, 1, 1)):
        assert lib.value("nkb_conv_wgrad_split", *geom) == ct(*geom)


def test_arguments_are_checked():
    lib = _nkpy()
    f = lib._fast["nkb_conv_wgrad_split"]
    with pytest.raises(TypeError):
        f(1, 2)
    with pytest.raises(TypeError):
        f(1, 1, 1, 8, 8, 3, 3, 1, "x")
    with pytest.raises(OverflowError):
        f(1, 1, 1, 8, 8, 3, 3, 1, 1 << 40)
    with pytest.raises(lib.NativeLibraryError, match="empty problem"):
        lib.call("nkb_gemm_bf16", None, 0, 0, None, 0, 0, None, 0, 0, 0, 0, 0, 0, 1.0, None, None,
                 0, 0, None, 0, None, None, 0, 0, 0, 0, None, None)


def _ops(device):
    from necklace_b200.ops import LayerNorm, RMSNorm, attention_qkv, linear, mlp
    from necklace_b200.ops.conv import BatchNorm2d, Conv2d
    from necklace_b200.ops.rotary import linear_rope
    g = torch.Generator().manual_seed(0)
    r = lambda *s: torch.randn(*s, generator=g).bfloat16().to(device)  # noqa: E731
    x, w1, b1, w2, b2, res = r(2, 9, 128), r(256, 128), r(256), r(128, 256), r(128), r(2, 9, 128)
    qkv, w3, img = r(2, 9, 384), r(384, 128), r(2, 7, 5, 16)
    ln, rn = LayerNorm(128, device=device), RMSNorm(128, device=device)
    convs = [Conv2d(16, 24, k, s, k // 2, device=device) for k, s in ((1, 1), (3, 1), (3, 2), (1, 2))]
    stem, bn = Conv2d(3, 8, 7, 2, 3, device=device), BatchNorm2d(16, relu=True, device=device).eval()
    bn.running_mean.normal_(generator=None), bn.running_var.uniform_(0.5, 2)
    return {"linear": lambda: linear(x, w1, b1), "linear_res": lambda: linear(x, w2.t().contiguous(), None, r(2, 9, 256) * 0),
            "mlp": lambda: mlp(x, w1, b1, w2, b2, res), "mlp_relu": lambda: mlp(x, w1, b1, w2, b2, None, "relu"),
            "ln": lambda: ln(x), "rms": lambda: rn(x), "ln_split": lambda: ln.split(x)[1],
            "rms_split": lambda: rn.split(x)[0], "attention": lambda: attention_qkv(qkv, 2, True),
            "rope": lambda: linear_rope(x, w3, 2), "stem": lambda: stem(r(1, 12, 12, 3) * 0 + 1),
            **{f"conv{i}": (lambda c=c: c(img)) for i, c in enumerate(convs)},
            "split": lambda: convs[0].split(img)[1], "bn": lambda: bn(img)}


def _same_without_a_node(device):
    for name, op in _ops(device).items():
        with torch.no_grad():
            a = op()
        assert not a.requires_grad and a.grad_fn is None
        assert torch.equal(a, op().detach()), name


def test_forward_by_itself_cpu():
    _same_without_a_node("cpu")


@pytest.mark.gpu
def test_forward_by_itself_gpu():
    from necklace_b200.ops._common import check_status
    _same_without_a_node("cuda")
    check_status()


def test_the_node_stays_where_something_looks():
    import torch.autograd.forward_ad as fwd_ad
    from necklace_b200.ops import linear
    from necklace_b200.ops._common import plain_call
    assert not plain_call()
    with torch.no_grad():
        assert plain_call()
        with fwd_ad.dual_level():
            assert not plain_call()
        seen = []
        torch.jit.trace(lambda t: (seen.append(plain_call()), t + 1)[1], torch.zeros(1),
                        check_trace=False)
        assert seen == [False]
    with torch.inference_mode():
        assert plain_call()
        assert linear(torch.ones(2, 8), torch.ones(4, 8)).shape == (2, 4)


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_forward_by_itself_adds_the_residual(device):
    from necklace_b200.ops import linear
    g = torch.Generator().manual_seed(5)
    x, w, res = (torch.randn(*s, generator=g).bfloat16().to(device)
                 for s in ((2, 9, 128), (256, 128), (2, 9, 256)))
    with torch.no_grad():
        y = linear(x, w, None, res)
        bare = linear(x, w)
    assert torch.equal(y, linear(x, w, None, res).detach())
    assert float((y.float() - bare.float() - res.float()).abs().max()) < 0.3
    assert float(res.float().abs().max()) > 2
