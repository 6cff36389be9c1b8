"""Kernels that start before the one ahead of them has ended: every result is the one that the same
calls give with the device idle between them, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _chain(case, x, w, sync):
    """Calls that read, overwrite and reuse each other's buffers, long kernels next to tiny ones."""
    from necklace_b200.ops import gemm
    from necklace_b200.ops.gemm import colsum
    from necklace_b200.ops.norm import norm_fwd
    from necklace_b200.ops.quant import dequantize_flat, quantize_flat
    outs, step = [], (torch.cuda.synchronize if sync else lambda: None)
    C = x.shape[1]
    ones, zeros = torch.ones(C, dtype=x.dtype, device=DEV), torch.zeros(C, dtype=x.dtype, device=DEV)
    buf = torch.empty(x.shape[0], C, dtype=x.dtype, device=DEV)
    res = torch.zeros(x.numel(), dtype=torch.float32, device=DEV)
    for k in range(6):
        gemm(x, w, out=buf, bn=case)                       # read below, overwritten next time round
        step()
        y, _ = norm_fwd(buf, ones, zeros, 1e-5, False)
        step()
        outs.append(colsum(buf))
        step()
        gemm(y, w, out=buf, bn=case, b_mn=True)            # overwrites what the two above read
        step()
        codes = quantize_flat(buf.view(-1), res, 0.5)      # and the residual carries on
        step()
        dequantize_flat(codes, buf.view(-1), 0.5)          # overwrites what was just encoded
        step()
        outs.append(colsum(buf))
        step()
        x = y
        outs.append(x.clone())
    return outs + [res]


@pytest.mark.parametrize("case", [0, 128, 256, 512])
@pytest.mark.parametrize("rows,C", [(8, 128), (1000, 512), (8192, 1024)])
def test_overlapping_launches_give_the_bits_of_separate_ones(case, rows, C):
    g = torch.Generator(device=DEV).manual_seed(rows)
    x = torch.randn(rows, C, generator=g, device=DEV).bfloat16()
    w = (torch.randn(C, C, generator=g, device=DEV) * C ** -0.5).bfloat16()
    want = _chain(case, x, w, True)
    for _ in range(3):
        got = _chain(case, x, w, False)
        for a, b in zip(got, want):
            # column sums of many rows are added by atomics in any order: a bf16 rounding apart
            if a.dim() == 1 and a.dtype == torch.bfloat16:
                scale = 2.0 ** -7 * b.float().abs() + rows * 2.0 ** -22 * 8
                assert bool(((a.float() - b.float()).abs() <= scale).all())
            else:
                assert torch.equal(a, b)


@pytest.mark.parametrize("D,S", [(64, 200), (128, 333)])
def test_attention_there_and_back_with_and_without_gaps(D, S):
    from necklace_b200.ops.attention import attn_bwd, attn_fwd
    g = torch.Generator(device=DEV).manual_seed(S)
    H = 5
    qkv = torch.randn(2, S, 3 * H * D, generator=g, device=DEV).bfloat16()
    dout = torch.randn(2, S, H * D, generator=g, device=DEV).bfloat16()
    out, lse = attn_fwd(qkv, H)
    torch.cuda.synchronize()
    want = attn_bwd(qkv, out, lse, dout, H).float()
    torch.cuda.synchronize()
    for _ in range(8):
        o, l = attn_fwd(qkv, H)
        d = attn_bwd(qkv, o, l, dout, H).float()
        assert torch.equal(o, out) and torch.equal(l, lse)
        # dQ's fp32 sums over key blocks arrive in any order
        assert ((d - want).norm() / want.norm()).item() < 1e-3
