"""Shared helpers for the operator wrappers."""
from __future__ import annotations

import threading

import torch
import torch.autograd.forward_ad as _fwd_ad

from .. import _lib

_grad_on = torch.is_grad_enabled
_trace = torch._C._get_tracing_state
_transform = torch._C._functorch.peek_interpreter_stack
_capturing = getattr(torch._C, "_cuda_isCurrentStreamCapturing", None)   # (CUDA builds)

_status: dict[int, torch.Tensor] = {}
_status_at: dict[int, int] = {}      # their addresses: the tensors live as long as the process
_scratch: dict[tuple, object] = {}   # (tag, device, stream, capture) -> what `make` gave
_scratch_lock = threading.Lock()
_SCRATCH_KEPT = 48                   # of 1/2 MB at most

STATUS_TEXT = {
    0: "ok", 1: "MMA warp timed out waiting for a TMA stage",
    2: "TMA producer timed out waiting for a free stage",
    3: "epilogue timed out waiting for an accumulator",
    4: "MMA warp timed out waiting for a free accumulator",
    5: "timed out waiting for a readiness/peer flag", 6: "index check failed",
}


def on_gpu(*ts) -> bool:
    """True when the native path must be used (any CUDA tensor)."""
    return any(t is not None and t.is_cuda for t in ts)


def status_word(device=None) -> torch.Tensor:
    """Device int32 the kernels write their first error code to."""
    dev = torch.cuda.current_device() if device is None else torch.device(device).index
    t = _status.get(dev)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=f"cuda:{dev}")
        _status[dev] = t
    return t


def status_ptr(t: torch.Tensor) -> int:
    """Address of the status word of ``t``'s device."""
    dev = t.get_device()
    p = _status_at.get(dev)
    if p is None:
        p = _status_at[dev] = status_word(t.device).data_ptr()
    return p


def plain_call() -> bool:
    """Whether an operator may run its forward pass without an autograd node: gradients are off,
    and neither forward-mode differentiation, a trace nor a function transform is looking (the
    last refuse these operators, with a message of their own)."""
    return not _grad_on() and _fwd_ad._current_level < 0 and _trace() is None \
        and _transform() is None


def check_status(reset: bool = True) -> None:
    """Synchronise and raise if any kernel since the last check reported an error."""
    for dev, t in _status.items():
        code = int(t.item())
        if code != 0:
            if reset:
                t.zero_()
            raise _lib.NativeLibraryError(
                f"device-side error {code} on cuda:{dev}: {STATUS_TEXT.get(code, 'unknown')}")


def stream_scratch(tag: str, device: torch.device, make):
    """Scratch that kernels find at zero and leave at zero (accumulators, ticket counters), made by
    ``make()`` once per device and stream: what runs on another stream may run at the same time.
    A graph being captured gets scratch of its own, cleared by the graph itself, because replays
    of two graphs may overlap wherever they were captured."""
    s = _lib.stream_ptr()
    capture = _lib.value("nkb_capture_id", s) if _capturing() else 0
    k = (tag, device.index, s, capture)
    t = _scratch.get(k)
    if t is None:
        t = make()
        with _scratch_lock:
            # what is dropped goes back to the allocator, which orders its reuse on its stream
            for old in [o for o in _scratch if not capture or o[3] != capture][:-_SCRATCH_KEPT]:
                del _scratch[old]
            _scratch[k] = t
    return t


def ptr(t) -> int | None:
    return None if t is None else t.data_ptr()


def set_wait_cycles(cycles: int) -> None:
    """Limit (in SM clock cycles) of every bounded device-side wait: on a barrier, on a peer
    flag, on a readiness flag.  The default is about two seconds; a wait that runs out makes
    its kernel record a status code and return (see ``check_status``)."""
    lib = _lib.load()
    for tu in ("gemm", "attn", "comm", "conv"):
        fn = getattr(lib, f"nkb_set_wait_cycles_{tu}")
        fn.argtypes = [_lib.i64]
        fn.restype = _lib.i32
        _lib.check(fn(int(cycles)), f"nkb_set_wait_cycles_{tu}")
