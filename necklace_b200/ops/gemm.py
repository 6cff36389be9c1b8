"""bf16 GEMM on tcgen05/TMEM and the linear-layer autograd functions built on it.

``gemm`` computes ``C[M,N] = epi(alpha * A[M,K] @ B[N,K]^T + bias) + res`` with either
operand allowed to be stored transposed (``a_mn`` / ``b_mn``), which is how forward,
data-gradient and weight-gradient of a linear layer all map to the same kernel
without transpose copies.  CPU tensors take a PyTorch fp32 reference path (used
by the CPU test-suite); CUDA tensors always take the native kernel.

Replaces the ``F.linear`` (cuBLAS) calls in the reference's tensor-parallel layers
(necklace/frmwrk/pytorch/mpnn/layers.py:239-249, :314-328).
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import _lib
from ._common import on_gpu, plain_call, status_ptr, stream_scratch

EPI_NONE, EPI_GELU_FWD, EPI_GELU_BWD, EPI_RELU = 0, 1, 2, 3


def _gelu_tanh_grad(z: torch.Tensor) -> torch.Tensor:
    k0, k1 = 0.7978845608028654, 0.044715
    u = k0 * (z + k1 * z ** 3)
    t = torch.tanh(u)
    return 0.5 * (1 + t) + 0.5 * z * (1 - t * t) * k0 * (1 + 3 * k1 * z * z)


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False,
         out: torch.Tensor | None = None, out_dtype: torch.dtype | None = None,
         accumulate: bool = False, alpha: float = 1.0, bias: torch.Tensor | None = None,
         res: torch.Tensor | None = None, epi: int = EPI_NONE, aux: torch.Tensor | None = None,
         ready_flags: torch.Tensor | None = None, rows_per_flag: int = 0, ready_target: int = 0,
         max_ctas: int = 0, bn: int = 0,
         alpha_dev: torch.Tensor | None = None) -> torch.Tensor:
    """``a`` is stored ``[M,K]`` (or ``[K,M]`` when ``a_mn``); ``b`` is stored ``[N,K]``
    (or ``[K,N]`` when ``b_mn``).  Both must be 2-D with unit inner stride."""
    if a.is_cuda and ready_flags is None and max_ctas == 0 \
            and (out_dtype is None or out_dtype is torch.bfloat16 or out_dtype is torch.float32):
        ops = _lib.ops()
        if ops is not None:
            y = ops.gemm(a, b, a_mn, b_mn, out, out_dtype is torch.float32, accumulate, alpha, bias,
                         res, epi, aux, bn, alpha_dev, status_ptr(a))
            if _lib.done(y, "nkb_gemm_bf16_ws"):
                return y
    sa, sb = a.shape, b.shape
    assert len(sa) == 2 and len(sb) == 2
    M, K = (sa[1], sa[0]) if a_mn else sa
    N, Kb = (sb[1], sb[0]) if b_mn else sb
    assert K == Kb, f"contraction mismatch {K} vs {Kb}"
    if out is None:
        assert not accumulate
        out = torch.empty((M, N), dtype=out_dtype or a.dtype, device=a.device)
    else:
        assert out.shape == (M, N) and out.stride(1) == 1

    if not on_gpu(a, b, out):
        A = a.float().t() if a_mn else a.float()
        B = b.float().t() if b_mn else b.float()
        y = alpha * (A @ B.t())
        if alpha_dev is not None:
            y = y * alpha_dev.float()
        if bias is not None:
            y = y + bias.float()
        if epi == EPI_GELU_FWD:
            aux.copy_(y.to(aux.dtype))
            y = F.gelu(y, approximate="tanh")
        elif epi == EPI_GELU_BWD:
            y = y * _gelu_tanh_grad(aux.float())
        elif epi == EPI_RELU:
            y = torch.relu(y)
        if res is not None:
            y = y + res.float()
        if accumulate:
            y = y + out.float()
        out.copy_(y.to(out.dtype))
        return out

    assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16
    (lda, ia), (ldb, ib) = a.stride(), b.stride()
    assert ia == 1 and ib == 1
    fp32 = out.dtype == torch.float32
    assert fp32 or out.dtype == torch.bfloat16
    if bias is not None:
        assert bias.dtype == torch.bfloat16 and bias.is_contiguous() and bias.numel() == N
    if res is not None:
        assert res.dtype == torch.bfloat16 and res.shape == (M, N) and res.stride(1) == 1
    if epi == EPI_GELU_FWD or epi == EPI_GELU_BWD:
        assert aux is not None and aux.dtype == torch.bfloat16 and aux.shape == (M, N)
        assert aux.stride(1) == 1
    pa, pb = a.data_ptr(), b.data_ptr()
    # TMA: 16-byte aligned base and row pitch; repack the rare operand that is not
    if lda % 8 or pa % 16:
        a = _repack(a)
        pa, lda = a.data_ptr(), a.stride(0)
    if ldb % 8 or pb % 16:
        b = _repack(b)
        pb, ldb = b.data_ptr(), b.stride(0)
    slices, ws = 1, None
    if K >= 2048 and epi == EPI_NONE and out.data_ptr() % (16 if fp32 else 8) == 0 \
            and (bias is None or bias.data_ptr() % 8 == 0) \
            and (res is None or (res.data_ptr() % 8 == 0 and res.stride(0) % 4 == 0)):
        slices = _lib.value("nkb_gemm_slices", M, N, K, out.stride(0), bn)
        if slices > 1:
            # the partial sums' memory belongs to this call: the allocator orders its reuse on
            # the stream (also while a graph is captured), and no other thread gets it meanwhile
            ws = torch.empty(slices * M * N, dtype=torch.float32, device=a.device)
    _lib.call("nkb_gemm_bf16_ws", pa, lda, a_mn, pb, ldb, b_mn, out.data_ptr(), out.stride(0),
              fp32, accumulate, M, N, K, alpha, None if bias is None else bias.data_ptr(),
              None if res is None else res.data_ptr(), 0 if res is None else res.stride(0), epi,
              None if aux is None else aux.data_ptr(), 0 if aux is None else aux.stride(0),
              status_ptr(a), None if ready_flags is None else ready_flags.data_ptr(),
              rows_per_flag, ready_target, max_ctas, bn,
              None if alpha_dev is None else alpha_dev.data_ptr(),
              None if ws is None else ws.data_ptr(), slices, _lib.stream_ptr())
    _lib.count_launch()
    return out


def set_splitk(enabled: bool) -> None:
    lib = _lib.load()
    lib.nkb_gemm_set_splitk.argtypes = [_lib.i32]
    lib.nkb_gemm_set_splitk.restype = None
    lib.nkb_gemm_set_splitk(int(enabled))


def _repack(t: torch.Tensor) -> torch.Tensor:
    """Copy into a buffer whose row pitch is a multiple of 8 elements (16 bytes)."""
    rows, cols = t.shape
    ld = (cols + 7) // 8 * 8
    buf = torch.zeros(rows, ld, dtype=t.dtype, device=t.device)
    buf[:, :cols].copy_(t)
    return buf[:, :cols]


def colsum(dy: torch.Tensor, out: torch.Tensor | None = None, accumulate: bool = False
           ) -> torch.Tensor:
    """Bias gradient: sum of ``dy[rows, C]`` over rows, bf16 out."""
    rows, Cn = dy.shape
    if out is None:
        out = torch.empty(Cn, dtype=dy.dtype, device=dy.device)
        accumulate = False
    if not on_gpu(dy):
        s = dy.float().sum(0)
        out.copy_(((out.float() + s) if accumulate else s).to(out.dtype))
        return out
    assert dy.dtype == torch.bfloat16 and dy.stride(1) == 1
    acc, tickets = colsum_scratch(Cn, dy.device)
    _lib.call("nkb_colsum_fused", dy.data_ptr(), acc.data_ptr(), tickets.data_ptr(),
              out.data_ptr(), int(accumulate), rows, Cn, dy.stride(0), _lib.stream_ptr())
    _lib.count_launch()
    return out


def colsum_scratch(Cn: int, device):
    """fp32 accumulator [2][C] and ticket counters of the kernels that sum columns (each leaves
    both at zero), shared by the calls on one stream."""
    assert Cn <= 65536
    return stream_scratch("colsum", device, lambda: (
        torch.zeros(2 * 65536, dtype=torch.float32, device=device),
        torch.zeros(256, dtype=torch.int32, device=device)))


# ---------------------------------------------------------------- autograd
def _deliver_grad(p: torch.Tensor, compute):
    """Weight/bias gradient delivery.

    When the parameter carries ``_nkb_grad`` (a view into a flat gradient buffer,
    set by the flat-parameter store) the gradient kernel writes or accumulates
    straight into it and autograd gets ``None``; otherwise the fresh gradient is
    returned for autograd to accumulate.  ``_nkb_grad_ready`` (if set) is called
    once the kernel is enqueued so data-parallel buckets can start reducing while
    backward continues.
    """
    buf = getattr(p, "_nkb_grad", None)
    if buf is None:
        return compute(None, False)
    compute(buf, bool(getattr(p, "_nkb_grad_has", False)))
    p._nkb_grad_has = True
    cb = getattr(p, "_nkb_grad_ready", None)
    if cb is not None:
        cb(p)
    return None


def _grad_target(p):
    """(tensor the kernel writes, accumulate?, what autograd gets) for parameter ``p``."""
    buf = getattr(p, "_nkb_grad", None)
    if buf is None:
        out = torch.empty_like(p)
        return out, False, out
    return buf, bool(getattr(p, "_nkb_grad_has", False)), None


def _grad_done(p):
    if getattr(p, "_nkb_grad", None) is None:
        return
    p._nkb_grad_has = True
    cb = getattr(p, "_nkb_grad_ready", None)
    if cb is not None:
        cb(p)


_NO_TARGET = (None, False, None)


def _deliver_nothing(p: torch.Tensor):
    """The gradient of a parameter whose output nobody used: zeros, delivered like any other."""
    return _deliver_grad(p, lambda out, acc: torch.zeros_like(p) if out is None
                         else (out if acc else out.zero_()))


class LinearFn(torch.autograd.Function):
    """``y = x @ w^T + b (+ residual)`` with ``w`` stored ``[out, in]``."""

    @staticmethod
    def forward(ctx, x, w, b, residual):
        x2 = x if x.is_contiguous() else x.reshape(-1, x.shape[-1])
        y = _linear(x2, w, b, residual)
        ctx.save_for_backward(x2, w)
        ctx.has_b = b is not None
        ctx.has_r = residual is not None
        ctx.b_ref = b
        return y if x2 is x else y.view(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        need = ctx.needs_input_grad
        dres = dy if ctx.has_r and need[3] else None
        if dy.is_cuda and (ops := _lib.ops()) is not None:
            b, bias = ctx.b_ref, ctx.has_b and need[2]
            tw, acc_w, dw = _grad_target(w) if need[1] else _NO_TARGET
            tb, acc_b, db = _grad_target(b) if bias else _NO_TARGET
            acc, tickets = colsum_scratch(w.shape[0], dy.device) if bias else (None, None)
            r = ops.linear_bwd(dy, x, w, need[0], tw, acc_w, tb, acc_b, acc, tickets,
                               status_ptr(dy))
            if _lib.done(r, "nkb_gemm_bf16_ws", need[0] + need[1] + bias):
                if need[1]:
                    _grad_done(w)
                if bias:
                    _grad_done(b)
                return r[0] if need[0] else None, dw, db, dres
        x2 = x.reshape(-1, x.shape[-1])
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = gemm(dy2, w, b_mn=True).view(*dy.shape[:-1], w.shape[1])
        if ctx.needs_input_grad[1]:
            dw = _deliver_grad(w, lambda out, acc: gemm(dy2, x2, a_mn=True, b_mn=True, out=out,
                                                        accumulate=acc))
        if ctx.has_b and ctx.needs_input_grad[2]:
            db = _deliver_grad(ctx.b_ref, lambda out, acc: colsum(dy2, out, acc))
        return dx, dw, db, dres


class MLPFn(torch.autograd.Function):
    """``y = act(x W1^T + b1) W2^T + b2 (+ residual)``, act = tanh-GELU or ReLU.

    The activation runs in the epilogue of the first GEMM (which also saves the
    pre-activation); its derivative runs in the epilogue of the data-gradient GEMM
    of the second layer, so no separate activation kernels exist in either direction.
    """

    @staticmethod
    def forward(ctx, x, w1, b1, w2, b2, residual, act):
        x2 = x if x.is_contiguous() else x.reshape(-1, x.shape[-1])
        y, h, z = _mlp(x2, w1, b1, w2, b2, residual, act)
        ctx.save_for_backward(x2, w1, w2, h, z)
        ctx.act = act
        ctx.refs = (b1, b2)
        ctx.has_r = residual is not None
        return y if x2 is x else y.view(*x.shape[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x, w1, w2, h, z = ctx.saved_tensors
        b1, b2 = ctx.refs
        need_x = ctx.needs_input_grad[0]
        if dy.is_cuda and ctx.act == "gelu" and w1 is not w2 and (b1 is None or b1 is not b2) \
                and (ops := _lib.ops()) is not None:
            t = [_grad_target(p) if p is not None else _NO_TARGET for p in (w1, b1, w2, b2)]
            acc, tickets = (None, None) if b1 is None and b2 is None else \
                colsum_scratch(max(w1.shape[0], w2.shape[0]), dy.device)
            r = ops.mlp_bwd(dy, x, w1, w2, h, z, need_x, t[0][0], t[0][1], t[1][0], t[1][1], t[2][0],
                            t[2][1], t[3][0], t[3][1], acc, tickets, status_ptr(dy))
            if _lib.done(r, "nkb_gemm_bf16_ws", 3 + need_x + (b1 is not None) + (b2 is not None)):
                for p in (w2, b2, w1, b1):
                    if p is not None:
                        _grad_done(p)
                return (r[0] if need_x else None, t[0][2], t[1][2], t[2][2], t[3][2],
                        dy if ctx.has_r else None, None)
        x2 = x.reshape(-1, x.shape[-1])
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        if ctx.act == "gelu":
            dz = gemm(dy2, w2, b_mn=True, epi=EPI_GELU_BWD, aux=z)
        else:
            dz = gemm(dy2, w2, b_mn=True)
            dz = dz * (h > 0).to(dz.dtype)
        dw2 = _deliver_grad(w2, lambda out, acc: gemm(dy2, h, a_mn=True, b_mn=True, out=out,
                                                      accumulate=acc))
        db2 = None
        if b2 is not None:
            db2 = _deliver_grad(b2, lambda out, acc: colsum(dy2, out, acc))
        dx = gemm(dz, w1, b_mn=True).view(*dy.shape[:-1], w1.shape[1]) \
            if need_x else None
        dw1 = _deliver_grad(w1, lambda out, acc: gemm(dz, x2, a_mn=True, b_mn=True, out=out,
                                                      accumulate=acc))
        db1 = None
        if b1 is not None:
            db1 = _deliver_grad(b1, lambda out, acc: colsum(dz, out, acc))
        dres = dy if ctx.has_r else None
        return dx, dw1, db1, dw2, db2, dres, None


def _linear(x, w, b, residual):
    """The forward pass by itself."""
    if x.is_cuda and (ops := _lib.ops()) is not None:
        y = ops.linear(x, w, b, residual, status_ptr(x))
        if _lib.done(y, "nkb_gemm_bf16_ws"):
            return y
    r2 = residual.reshape(-1, w.shape[0]) if residual is not None else None
    y = gemm(x.reshape(-1, x.shape[-1]), w, bias=b, res=r2)
    return y.view(*x.shape[:-1], w.shape[0])


def _mlp(x, w1, b1, w2, b2, residual, act):
    """(output, activation, pre-activation or None) of the forward pass by itself."""
    if act == "gelu" and x.is_cuda and (ops := _lib.ops()) is not None:
        r = ops.mlp(x, w1, b1, w2, b2, residual, status_ptr(x))
        if _lib.done(r, "nkb_gemm_bf16_ws", 2):
            return r
    x2 = x.reshape(-1, x.shape[-1])
    r2 = residual.reshape(-1, w2.shape[0]) if residual is not None else None
    z = None
    if act == "gelu":
        z = torch.empty(x2.shape[0], w1.shape[0], dtype=x2.dtype, device=x2.device)
        h = gemm(x2, w1, bias=b1, epi=EPI_GELU_FWD, aux=z)
    else:
        h = gemm(x2, w1, bias=b1, epi=EPI_RELU)
    return gemm(h, w2, bias=b2, res=r2).view(*x.shape[:-1], w2.shape[0]), h, z


def linear(x, w, b=None, residual=None):
    if plain_call():
        return _linear(x, w, b, residual)
    return LinearFn.apply(x, w, b, residual)


def mlp(x, w1, b1, w2, b2, residual=None, act="gelu"):
    if plain_call():
        return _mlp(x, w1, b1, w2, b2, residual, act)[0]
    return MLPFn.apply(x, w1, b1, w2, b2, residual, act)


class Linear(nn.Module):
    """Drop-in ``nn.Linear`` whose matmuls run on the tcgen05 GEMM."""

    def __init__(self, in_features: int, out_features: int, bias: bool = True,
                 dtype=torch.bfloat16, device=None, init_std: float | None = None):
        super().__init__()
        self.in_features, self.out_features = in_features, out_features
        self.weight = nn.Parameter(torch.empty(out_features, in_features, dtype=dtype,
                                               device=device))
        self.bias = nn.Parameter(torch.zeros(out_features, dtype=dtype, device=device)) \
            if bias else None
        if init_std is None:
            nn.init.kaiming_uniform_(self.weight, a=5 ** 0.5)
        else:
            nn.init.normal_(self.weight, std=init_std)

    def forward(self, x, residual=None):
        return linear(x, self.weight, self.bias, residual)
