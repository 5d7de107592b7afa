"""Loader of the native host path (``csrc/front``): a torch extension compiled in-tree like the kernels and handed the addresses of the
core library's functions."""
from __future__ import annotations

import ctypes as C
import importlib.machinery
import importlib.util
import threading

from . import _build, _cabi

_CORE = ("eqlinear_pack", "eqlinear_forward", "eqlinear_dgrad", "eqlinear_forward_packed", "eqlinear_dgrad_packed", "eqlinear_wgrad_scratch",
         "eqlinear_wgrad_with", "gemm_tf32x3_split", "gemm_tf32x3_presplit", "radial_chain_prepare", "radial_chain_forward",
         "radial_chain_backward", "edge_geometry_forward", "edge_geometry_backward", "silu", "neighbors_work_bytes", "neighbors_count",
         "neighbors_fill", "graph_partition", "graph_partition_edges", "last_cuda_error")
_lib = None
_lock = threading.Lock()


def addresses(lib, names) -> dict:
    """``{name: address}`` of functions of a library opened with ctypes."""
    return {n: C.cast(getattr(lib, n), C.c_void_p).value for n in names}


def lib():
    global _lib
    if _lib is None:
        core = _cabi.core()
        path = _build.build_front()
        with _lock:
            if _lib is None:
                loader = importlib.machinery.ExtensionFileLoader("fasteq_front", path)
                mod = importlib.util.module_from_spec(importlib.util.spec_from_file_location("fasteq_front", path, loader=loader))
                loader.exec_module(mod)
                mod.bind_core(addresses(core, [f"fasteq_{n}" for n in _CORE]), _cabi.FasteqError)
                _lib = mod
    return _lib
