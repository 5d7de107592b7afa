"""SiLU whose first and second backward are one kernel each (``fasteq_silu``), for the radial MLP of a training step."""
from __future__ import annotations

import ctypes as C

import torch

from .. import _cabi

_ready = False


def _run(order: int, z, g=None, h=None):
    global _ready
    lib = _cabi.core()
    if not _ready:
        lib.fasteq_silu.argtypes = [C.c_int32, C.c_int32] + [C.c_void_p] * 5 + [C.c_int64, C.c_void_p]
        _ready = True
    ptr = lambda t: t.data_ptr() if t is not None else None
    out0 = torch.empty_like(z)
    out1 = torch.empty_like(z) if order == 2 else None
    with _cabi.on_device(z.device):
        _cabi.check(lib.fasteq_silu(1 if z.dtype == torch.float64 else 0, order, z.data_ptr(), ptr(g), ptr(h), out0.data_ptr(), ptr(out1),
                                    z.numel(), _cabi.stream(z.device)), lib, "fasteq_silu")
    return out0, out1


class _SiLU(torch.autograd.Function):
    @staticmethod
    def forward(ctx, z):
        ctx.save_for_backward(z)
        return _run(0, z)[0]

    @staticmethod
    def backward(ctx, g):
        (z,) = ctx.saved_tensors
        return _SiLUBackward.apply(g.contiguous(), z)


class _SiLUBackward(torch.autograd.Function):
    @staticmethod
    def forward(ctx, g, z):
        ctx.save_for_backward(g, z)
        return _run(1, z, g)[0]

    @staticmethod
    def backward(ctx, h):
        g, z = ctx.saved_tensors
        if torch.is_grad_enabled():      # a third order is asked for: the same expressions as torch operations
            s = torch.sigmoid(z)
            return h * s * (1 + z * (1 - s)), h * g * s * (1 - s) * (2 + z * (1 - 2 * s))
        return _run(2, z, g, h.contiguous())


def silu(z: torch.Tensor) -> torch.Tensor:
    if z.is_cuda and z.dtype in (torch.float32, torch.float64) and z.is_contiguous():
        return _SiLU.apply(z)
    return torch.nn.functional.silu(z)
