"""Kernels that work on packed pairs and on words of two bf16, at the sizes and values where those can
go wrong: remainders of their strips and rows, masks of every byte, values that are not numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,C", [(1, 8), (3, 24), (255, 136), (1030, 264), (777, 64)])
@pytest.mark.parametrize("relu,with_res", [(True, False), (True, True), (False, False)])
def test_batch_norm_there_and_back(M, C, relu, with_res):
    from necklace_b200.ops.conv import BatchNorm2d
    g = torch.Generator(device=DEV).manual_seed(M)
    x = (torch.randn(M, 1, 1, C, generator=g, device=DEV) + 0.5).bfloat16().requires_grad_(True)
    r = torch.randn(M, 1, 1, C, generator=g, device=DEV).bfloat16().requires_grad_(True) \
        if with_res else None
    dy = torch.randn(M, 1, 1, C, generator=g, device=DEV).bfloat16()
    bn = BatchNorm2d(C, relu=relu, device=DEV)
    bn.weight.data.uniform_(0.5, 1.5, generator=g)
    bn.bias.data.normal_(generator=g)
    y = bn(x, r)
    y.backward(dy)
    X = x.detach().double().view(M, C)
    mean, var = X.mean(0), X.var(0, unbiased=False)
    rstd = (var + 1e-5).rsqrt()
    xh = (X - mean) * rstd
    w, b = bn.weight.double(), bn.bias.double()
    z = xh * w + b + (r.detach().double().view(M, C) if with_res else 0)
    want = z.relu() if relu else z
    # one bf16 rounding, and the fp32 statistics: sums of M terms of magnitude x^2 over the variance
    slack = 2.0 ** -8 * want.abs() + 2.0 ** -20 * (1 + w.abs() * rstd * (X.abs() + mean.abs() +
                                                   (X * X).mean(0) * rstd))
    assert bool(((y.detach().double().view(M, C) - want).abs() <= slack).all())
    # the backward takes the signs of the stored output
    keep = (y.detach().view(M, C) > 0).double() if relu else torch.ones(M, C, device=DEV).double()
    d = dy.double().view(M, C) * keep
    dx = w * rstd * (d - d.mean(0) - xh * (d * xh).mean(0))
    mag = w.abs() * rstd * (d.abs() + d.abs().mean(0) + xh.abs() * (d * xh).abs().mean(0))
    assert bool(((x.grad.double().view(M, C) - dx).abs() <= 2.0 ** -8 * dx.abs() + 2e-4 * mag).all())
    for got, ref, m in ((bn.weight.grad, (d * xh).sum(0), (d * xh).abs().sum(0)),
                        (bn.bias.grad, d.sum(0), d.abs().sum(0))):
        assert bool(((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-4 * m + 1e-30).all())
    if with_res:
        assert torch.equal(r.grad.double().view(M, C), d)


def test_batch_norm_mask_of_every_byte_and_odd_values():
    """All 256 masks of eight neighbouring channels; zeros, negative zeros, infinities and NaN."""
    from necklace_b200.ops.conv import BatchNorm2d
    M, C = 256, 8
    bn = BatchNorm2d(C, relu=True, device=DEV)
    signs = torch.tensor([[1.0 if m >> j & 1 else -1.0 for j in range(C)] for m in range(M)],
                         device=DEV)
    x = signs.view(M, 1, 1, C).bfloat16().requires_grad_(True)
    res = torch.zeros(M, 1, 1, C, device=DEV).bfloat16().requires_grad_(True)
    y = bn(x, res)
    dy = torch.full_like(y, 3.0)
    y.backward(dy)
    assert torch.equal(res.grad.view(M, C), (3.0 * (signs > 0)).bfloat16())
    ev = BatchNorm2d(C, relu=True, device=DEV).eval()
    odd = torch.tensor([float("nan"), float("inf"), -float("inf"), -0.0, 0.0, 1e-40, -1e-40, 2.0],
                       device=DEV).bfloat16().view(1, 1, 1, C)
    with torch.no_grad():
        out = ev(odd).view(C)
    s = (torch.ones((), device=DEV) + ev.eps).rsqrt()
    ref = torch.clamp((odd.float() * s).bfloat16().view(C).nan_to_num(nan=0.0, posinf=float("inf"),
                                                                     neginf=0.0), min=0.0)
    assert torch.equal(out, ref) and not bool(torch.signbit(out).any())


@pytest.mark.parametrize("n", [1, 7, 8, 17, 4096, 100003])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("offset", [0, 1])
def test_decoder_of_every_code(n, dtype, offset):
    from necklace_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(n)
    codes = torch.randint(-2 ** 31, 2 ** 31 - 1, ((n + 15) // 16,), generator=g, device=DEV,
                          dtype=torch.int64).to(torch.int32)
    c = torch.stack([(codes >> (2 * k)) & 3 for k in range(16)], 1).reshape(-1)[:n]
    val = torch.tensor([0.0, 0.37, -0.37, 0.0], device=DEV)[c.long()] * 0.5
    for accumulate in (0, 1):
        buf = torch.randn(n + 1, generator=g, device=DEV).to(dtype)
        out = buf[offset:offset + n]
        want = (out.float() + val if accumulate else val).to(dtype)
        _lib.call("nkb_dequant2_flat", codes.data_ptr(), out.data_ptr(),
                  int(dtype == torch.float32), n, 0.37, 0.5, accumulate, _lib.stream_ptr())
        assert torch.equal(out, want)


@pytest.mark.parametrize("rows", [1, 7, 63, 64, 65, 513, 4100])
@pytest.mark.parametrize("C,ld", [(2, 2), (8, 8), (254, 256), (264, 264), (1024, 1032)])
def test_column_sums(rows, C, ld):
    from necklace_b200.ops.gemm import colsum
    g = torch.Generator(device=DEV).manual_seed(rows)
    dy = torch.randn(rows, ld, generator=g, device=DEV).bfloat16()[:, :C]
    want, mag = dy.double().sum(0), dy.double().abs().sum(0)
    got = colsum(dy)
    slack = 2.0 ** -8 * want.abs() + mag * rows * 2.0 ** -24
    assert bool(((got.double() - want).abs() <= slack).all())
    again = colsum(dy, got.clone(), True)
    assert bool(((again.double() - got.double() - want).abs() <=
                 slack + 2.0 ** -8 * (got.double() + want).abs()).all())


@pytest.mark.parametrize("S", [1, 3, 5, 127, 130])
@pytest.mark.parametrize("B,H,D", [(1, 1, 64), (3, 5, 64), (2, 3, 128)])
def test_attention_backward_of_few_positions(S, B, H, D):
    """Groups of four positions of the row sums, and the pieces of the gradient that are left over."""
    from necklace_b200.ops.attention import attention_qkv
    g = torch.Generator(device=DEV).manual_seed(S)
    qkv = torch.randn(B, S, 3 * H * D, generator=g, device=DEV).bfloat16().requires_grad_(True)
    dout = torch.randn(B, S, H * D, generator=g, device=DEV).bfloat16()
    attention_qkv(qkv, H, True).backward(dout)
    q64 = qkv.detach().double().requires_grad_(True)
    q, k, v = q64.view(B, S, 3, H, D).permute(2, 0, 3, 1, 4)
    s = (q @ k.transpose(-1, -2)) * D ** -0.5
    s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=DEV).tril(), float("-inf"))
    (torch.softmax(s, -1) @ v).permute(0, 2, 1, 3).reshape(B, S, H * D).backward(dout.double())
    err = (qkv.grad.double() - q64.grad).norm() / q64.grad.norm()
    assert err.item() < 1e-2           # bf16 probabilities and score gradients: 0.3 % each
