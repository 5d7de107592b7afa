"""Per-atom scalar readout ``e + (h[:, :C] * w).sum(-1)`` as one launch per direction (``fasteq_readout_*``)."""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from .. import _cabi
from ._needs import wanted

_ready = False


def _lib():
    global _ready
    lib = _cabi.core()
    if not _ready:
        lib.fasteq_readout_forward.argtypes = [C.c_int32] + [C.c_void_p] * 4 + [C.c_int64, C.c_int32, C.c_int64, C.c_void_p]
        lib.fasteq_readout_backward.argtypes = [C.c_int32] + [C.c_void_p] * 3 + [C.c_int64, C.c_int32, C.c_int64, C.c_void_p]
        _ready = True
    return lib


class _Readout(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h, w, e):
        ctx.save_for_backward(h, w)
        n, d = h.shape
        out = torch.empty(n, dtype=h.dtype, device=h.device)
        lib = _lib()
        with _cabi.on_device(h.device):
            _cabi.check(lib.fasteq_readout_forward(1 if h.dtype == torch.float64 else 0, h.data_ptr(), w.data_ptr(),
                                                   e.data_ptr() if e is not None else None, out.data_ptr(), n, w.numel(), d,
                                                   _cabi.stream(h.device)), lib, "fasteq_readout_forward")
        return out

    @staticmethod
    def backward(ctx, g):
        h, w = ctx.saved_tensors
        n, d = h.shape
        gh = gw = None
        if ctx.needs_input_grad[0]:
            if torch.is_grad_enabled():      # to be differentiated again: the same values as torch operations
                gh = torch.nn.functional.pad(g.unsqueeze(-1) * w, (0, d - w.numel()))
            else:
                gh, lib, gc = torch.empty_like(h), _lib(), g.contiguous()
                with _cabi.on_device(h.device):
                    _cabi.check(lib.fasteq_readout_backward(1 if h.dtype == torch.float64 else 0, gc.data_ptr(), w.data_ptr(), gh.data_ptr(),
                                                            n, w.numel(), d, _cabi.stream(h.device)), lib, "fasteq_readout_backward")
        if wanted(ctx, 1):
            gw = (g.unsqueeze(-1) * h[:, : w.numel()]).sum(dim=0)
        return gh, gw, (g if ctx.needs_input_grad[2] else None)


def _one_launch(h: torch.Tensor, w: torch.Tensor, e: Optional[torch.Tensor]) -> bool:
    """Whether the kernel's view of the operands is theirs: rows of one matrix, a weight per column, a running sum per row, all
    dense, of one type and on one device.  Everything else is left to the expression below, which broadcasts it or raises."""
    return (h.dim() == 2 and h.is_contiguous() and h.dtype in (torch.float32, torch.float64)
            and w.dim() == 1 and w.is_contiguous() and w.dtype == h.dtype and w.device == h.device and w.numel() <= h.shape[1]
            and (e is None or (e.shape == h.shape[:1] and e.is_contiguous() and e.dtype == h.dtype and e.device == h.device)))


def scalar_readout(h: torch.Tensor, w: torch.Tensor, e: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``e + (h[:, : len(w)] * w).sum(-1)`` (``e`` omitted: without it)."""
    if h.is_cuda and _one_launch(h, w, e):
        return _Readout.apply(h, w, e)
    s = (h[:, : w.numel()] * w).sum(dim=-1)
    return s if e is None else e + s
