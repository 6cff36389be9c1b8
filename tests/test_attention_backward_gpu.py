"""Attention gradients against fp64 at the edges of the 128-row blocks, for one, two and more blocks
per key block (the pipeline's start, its steady state and its end), causal and full."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 2, 127, 128, 129, 255, 256, 257, 384, 511, 640, 1111, 2049])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("D", [64, 128])
def test_gradients(S, causal, D):
    from necklace_b200.ops import attention_qkv
    from necklace_b200.ops._common import check_status
    B, H = (2, 3) if S < 600 else (1, 2)
    g = torch.Generator(device="cuda").manual_seed(S)
    qkv = torch.randn(B, S, 3 * H * D, generator=g, device="cuda").bfloat16().requires_grad_(True)
    dout = torch.randn(B, S, H * D, generator=g, device="cuda").bfloat16()
    for _ in range(2):
        qkv.grad = None
        out = attention_qkv(qkv, H, causal)
        out.backward(dout)
    check_status()                       # no wait of the pipeline ran out
    x = qkv.detach().double().requires_grad_(True)
    q, k, v = x.view(B, S, 3, H, D).permute(2, 0, 3, 1, 4)
    s = q @ k.transpose(-1, -2) / D ** 0.5
    if causal:
        s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    prob = torch.softmax(s, -1)
    ref = (prob @ v).permute(0, 2, 1, 3).reshape(B, S, H * D)
    ref.backward(dout.double())
    # P, dS and the results are rounded to bf16 (2^-9 each): a few times 2^-9 in norm.  delta is
    # the product with an output rounded to 2^-9; in dS = P (dP - delta) that error, 2^-9 of
    # |dout| sqrt(D), meets a difference that may vanish (one key): it reaches dq and dk times P,
    # D^-1/2 and a key or query of length sqrt(D)
    spread = prob.detach().square().sum(-1).mean().sqrt()
    scale = dout.double().norm() * spread
    for i, name in enumerate(("dq", "dk", "dv")):
        a = qkv.grad.double().view(B, S, 3, H * D)[:, :, i]
        b = x.grad.view(B, S, 3, H * D)[:, :, i]
        err = (a - b).norm()
        assert float(err) <= 5 * 2.0 ** -9 * float(b.norm()) + 2.0 ** -8 * float(scale) * (i < 2), \
            (name, float(err / b.norm()))


@pytest.mark.parametrize("D", [64, 128])
def test_many_blocks_per_sm(D):
    """Two heads' worth of every SM: roles drift apart and waits meet every order of arrival."""
    from necklace_b200.ops.attention import attn_bwd, attn_fwd, set_bwd_impl
    from necklace_b200.ops._common import check_status
    B, H, S = 4, 16, 1024
    g = torch.Generator(device="cuda").manual_seed(1)
    qkv = torch.randn(B, S, 3 * H * D, generator=g, device="cuda").bfloat16()
    dout = torch.randn(B, S, H * D, generator=g, device="cuda").bfloat16()
    for causal in (True, False):
        out, lse = attn_fwd(qkv, H, causal)
        got = [attn_bwd(qkv, out, lse, dout, H, causal) for _ in range(20)][-1]
        check_status()
        set_bwd_impl(0)
        try:
            want = attn_bwd(qkv, out, lse, dout, H, causal).double()
        finally:
            set_bwd_impl(1)
        # both round P and dS to bf16 at the same places; fp32 sums in another order
        assert float((got.double() - want).norm()) <= 2.0 ** -8 * float(want.norm())
