"""Edge vectors and radial basis of a radius graph in one kernel, with the force-pass gradient in another
(``fasteq_edge_geometry_forward`` / ``_backward``): ``vec = pos[src] + shift - pos[dst]``,
``basis = bessel(|vec|) * polynomial_cutoff(|vec|)``.  First order only."""
from __future__ import annotations

import ctypes as C

import torch

from .. import _cabi, _front

_ready = False


def _lib():
    global _ready
    lib = _cabi.core()
    if not _ready:
        lib.fasteq_edge_geometry_device_status.argtypes = [C.POINTER(C.c_int32)]
        _ready = True
    return lib


def edge_geometry_usable(pos: torch.Tensor, n_basis: int) -> bool:
    return pos.is_cuda and pos.dtype in (torch.float32, torch.float64) and pos.dim() == 2 and pos.shape[1] == 3 and 1 <= n_basis <= 16


def edge_geometry(pos, edge_src, edge_dst, edge_shift, r_max: float, n_basis: int, envelope_p: int):
    """``(vec [E, 3], basis [E, n_basis])``; differentiable once with respect to ``pos``."""
    return _front.lib().edge_geometry(pos, edge_src, edge_dst, edge_shift, float(r_max), int(n_basis), int(envelope_p))


def edge_geometry_device_status() -> int:
    """Reads and clears the kernels' status word (synchronises): 0, or 2 after an edge index outside the position array
    (such an edge is skipped: zero features, no gradient)."""
    lib = _lib()
    v = C.c_int32(0)
    _cabi.check(lib.fasteq_edge_geometry_device_status(C.byref(v)), lib, "fasteq_edge_geometry_device_status")
    return int(v.value)
