"""``fast_equi_linear``: drop-in for fasteq/ops/eqlinear.py:44-65 (forward and grad_x of the
uniform ``uv,iu,iv`` SO3Linear).

``x`` is ``[B, I*U]`` (viewed ``[B, I, U]``, irrep-row major, channel minor), ``w`` holds ``P*U*V``
elements (viewed ``[P, U, V]``), the result is ``[B, J*V]``.  Precision routing as in the reference
(fasteq/ops/eqlinear.py:24-41): float64 -> FP64; float32 -> ``compute_precision`` ``None`` /
``"tf32"`` / ``"tf32x3"`` (error bound of 3xTF32) or ``"fp32"``; anything else raises ``ValueError``.
The reference returns no gradient for ``w`` (eqlinear_runtime.py:104); here ``w`` gets one when it
requires grad (``fasteq_eqlinear_wgrad``: FP32 on the tensor cores in three bf16 parts per operand, short batches and FP64 on FMA tiles),
so the mixing weights can be trained.
Unsupported descriptors raise; there is no fallback path.
"""
from __future__ import annotations

import ctypes as C
import operator
from typing import Dict, List, Tuple

import torch

from .. import _cabi, _front
from ..descriptors import LinearDescriptor
from . import _prepared

__all__ = ["fast_equi_linear", "eqlinear_clear_plan_cache", "eqlinear_set_plan_cache", "eqlinear_debug_info"]

_TF32, _FP32, _FP64 = 0, 1, 2


class _Problem(C.Structure):
    _fields_ = [("precision", C.c_int32), ("u", C.c_int32), ("v", C.c_int32), ("in_rows", C.c_int32),
                ("out_rows", C.c_int32), ("num_paths", C.c_int32), ("batch", C.c_int64),
                ("in_row", C.POINTER(C.c_int32)), ("out_row", C.POINTER(C.c_int32)), ("rows", C.POINTER(C.c_int32)),
                ("coeff", C.POINTER(C.c_double))]


def _resolve_precision(x, w, compute_precision) -> int:
    if x.dtype != w.dtype:
        raise ValueError(f"eqlinear: x and w must have the same dtype; got {x.dtype} and {w.dtype}")
    if x.dtype == torch.float64:
        return _FP64
    if x.dtype != torch.float32:
        raise ValueError(f"eqlinear: only float32 and float64 are supported; got {x.dtype}")
    if compute_precision is None:
        return _TF32
    value = compute_precision.lower() if isinstance(compute_precision, str) else compute_precision
    if value in ("tf32", "tf32x3"):
        return _TF32
    if value == "fp32":
        return _FP32
    raise ValueError(f"eqlinear: compute_precision must be None, 'tf32', or 'fp32'; got {compute_precision!r}")


def _segments(operand) -> Tuple[Tuple[int, ...], ...]:
    segs = getattr(operand, "segments", operand)
    return tuple(tuple(operator.index(v) for v in seg) for seg in segs)


def _single(descriptor, name: str) -> int:
    vals = {operator.index(v) for v in descriptor.get_dims(name)}
    if len(vals) != 1:
        raise ValueError(f"eqlinear: descriptor must have exactly one {name!r} dimension, got {sorted(vals)}")
    return vals.pop()


def _descriptor_problem(descriptor):
    """(mapping [(in_row, out_row, weight_path, rows)], coefficients, u, v, I, J).

    Accepts both descriptor flavours the reference accepts (eqlinear_descriptor.py:228-310): paths
    with ``indices`` (explicit segment mapping) and index-free paths over a dense run-length layout."""
    if len(descriptor.operands) != 3:
        raise ValueError("eqlinear requires exactly three operands: uv, iu, iv")
    paths = list(descriptor.paths)
    if not paths:
        raise ValueError("eqlinear descriptor must contain at least one path")
    in_seg, out_seg = _segments(descriptor.operands[1]), _segments(descriptor.operands[2])
    u, v = _single(descriptor, "u"), _single(descriptor, "v")
    coeff = []
    for p in paths:
        c = p.coefficients
        c = float(c.item() if hasattr(c, "item") else c)
        coeff.append(c)
    if all(hasattr(p, "indices") for p in paths):
        subs = getattr(descriptor, "operands_and_subscripts", None)
        if subs is not None and tuple(s for _, s in subs) != ("uv", "iu", "iv") or getattr(descriptor, "coefficient_subscripts", ""):
            raise NotImplementedError("eqlinear requires scalar coefficients and uv,iu,iv subscripts")
        w_seg = _segments(descriptor.operands[0])
        if len(w_seg) != len(paths):
            raise NotImplementedError("eqlinear requires one weight block per path")
        if (any(len(s) != 2 or s[1] != u for s in in_seg) or any(len(s) != 2 or s[1] != v for s in out_seg)
                or any(tuple(s) != (u, v) for s in w_seg)):
            raise ValueError("eqlinear: inconsistent uniform operand segment dimensions")
        in_off, out_off, I, J = [], [], 0, 0
        for s in in_seg:
            in_off.append(I); I += s[0]
        for s in out_seg:
            out_off.append(J); J += s[0]
        mapping = []
        for p in paths:
            wp, ip, op = (operator.index(i) for i in p.indices)
            if not (0 <= wp < len(w_seg) and 0 <= ip < len(in_seg) and 0 <= op < len(out_seg)):
                raise ValueError("eqlinear: invalid descriptor path index")
            i = in_seg[ip][0]
            if i <= 0 or i != out_seg[op][0]:
                raise ValueError("eqlinear: path i dimensions disagree")
            mapping.append((in_off[ip], out_off[op], wp, i))
        return mapping, coeff, u, v, I, J
    i_dims = tuple(s[0] for s in in_seg)
    if len(i_dims) != len(paths):
        raise ValueError(f"eqlinear: derived {len(i_dims)} i_dims for {len(paths)} paths")
    mapping, in_row, out_row, prev = [], 0, 0, None
    for q, i in enumerate(i_dims):
        if prev is not None and prev != i:
            out_row += prev
        mapping.append((in_row, out_row, q, i))
        in_row += i
        prev = i
    J = out_row + i_dims[-1]
    if J != sum(s[0] for s in out_seg):
        raise NotImplementedError(f"eqlinear: output segments imply {sum(s[0] for s in out_seg)} rows, kernel grouping implies {J}")
    return mapping, coeff, u, v, in_row, J


_core_ready = False


def _core():
    global _core_ready
    lib = _cabi.core()
    if not _core_ready:
        lib.fasteq_eqlinear_forward.argtypes = [C.POINTER(_Problem), C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
        lib.fasteq_eqlinear_dgrad.argtypes = [C.POINTER(_Problem), C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
        lib.fasteq_eqlinear_wgrad.argtypes = [C.POINTER(_Problem), C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
        lib.fasteq_eqlinear_wgrad_scratch.argtypes = [C.POINTER(_Problem), C.c_void_p, C.c_void_p, C.POINTER(C.c_int64)]
        lib.fasteq_eqlinear_wgrad_with.argtypes = [C.POINTER(_Problem), C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int64, C.c_void_p]
        _core_ready = True
    return lib


def _make_problem(mapping, coeff, u, v, I, J, batch, precision):
    P = len(mapping)
    arr = lambda vals: (C.c_int32 * P)(*vals)
    prob = _Problem(precision, u, v, I, J, P, batch, arr([m[0] for m in mapping]), arr([m[1] for m in mapping]),
                    arr([m[3] for m in mapping]), (C.c_double * P)(*coeff))
    return prob


def wgrad_into(prob, x, g, dw) -> None:
    """The weight gradient of a problem, its partial sums in memory of torch's allocator."""
    lib, need = _core(), C.c_int64(0)
    with _cabi.on_device(dw.device):
        stream = _cabi.stream(dw.device)
        _cabi.check(lib.fasteq_eqlinear_wgrad_scratch(C.byref(prob), x.data_ptr(), g.data_ptr(), C.byref(need)), lib,
                    "fasteq_eqlinear_wgrad_scratch")
        scratch = torch.empty(max(need.value, 16), dtype=torch.uint8, device=dw.device)
        _cabi.check(lib.fasteq_eqlinear_wgrad_with(C.byref(prob), x.data_ptr(), g.data_ptr(), dw.data_ptr(), scratch.data_ptr(),
                                                   scratch.numel(), stream), lib, "fasteq_eqlinear_wgrad_with")


class _Plan:
    """The weight gradient of one operator call: ``x`` is ``[batch, I * u]``, ``g`` ``[batch, J * v]``, the result shaped like the caller's
    weights."""

    def __init__(self, geom, precision, batch, w_shape):
        self.geom, self.precision, self.batch, self.w_shape = geom, precision, batch, tuple(w_shape)

    def wgrad(self, x, g):
        mapping, coeff, u, v, I, J = self.geom
        x3 = x.reshape(self.batch, I, u).contiguous()
        g3 = g.reshape(self.batch, J, v).contiguous()
        dw = torch.empty((len(mapping), u, v), dtype=g3.dtype, device=g3.device)
        table = [(m[0], m[1], q, m[3]) for q, m in enumerate(mapping)]
        wgrad_into(_make_problem(table, coeff, u, v, I, J, self.batch, self.precision), x3, g3, dw)
        wps = [m[2] for m in mapping]
        if wps != list(range(len(wps))):      # block q of the table is block wps[q] of the caller's tensor
            full = torch.empty_like(dw)
            full[torch.tensor(wps, device=dw.device)] = dw
            dw = full
        return dw.reshape(self.w_shape)


def _native(geom):
    """The native form of a geometry (``csrc/front/layers.cpp``): the operator, its gradient and its second order."""
    mapping, coeff, u, v, I, J = geom
    return _front.lib().Geometry([list(m) for m in mapping], list(coeff), u, v, I, J,
                                 lambda x, g, precision, batch, w_shape: _Plan(geom, precision, batch, w_shape).wgrad(x, g))


def _geometry(descriptor):
    """Native geometry of a descriptor.  One of this package keeps its own, with the tables it was made from: they can be changed."""
    if type(descriptor) is not LinearDescriptor:
        return _native(_descriptor_problem(descriptor))
    tables = (tuple(descriptor.paths), tuple(descriptor.operands), descriptor.operands_and_subscripts, descriptor.u, descriptor.v,
              descriptor.coefficient_subscripts)
    kept = descriptor.__dict__.get("_native")
    if kept is None or kept[0] != tables:
        kept = descriptor._native = (tables, _native(_descriptor_problem(descriptor)))
    return kept[1]


def fast_equi_linear(descriptor, w, x, *, compute_precision=None):
    """Forward, grad_x and grad_w for the uniform uv/iu/iv eqlinear operator."""
    precision = _resolve_precision(x, w, compute_precision)
    return _front.lib().eqlinear(_geometry(descriptor), w, x, precision)


def eqlinear_clear_plan_cache() -> None:
    """Drop the prepared weights (same name as the reference's call, fasteq/ops/eqlinear.py)."""
    _prepared.clear()


def eqlinear_set_plan_cache(max_bytes=None) -> None:
    """Byte budget of the prepared-weight cache; ``0`` disables it, ``None`` restores the default (256 MiB)."""
    _prepared.set_budget(max_bytes)


def eqlinear_debug_info(descriptor, w, x, *, compute_precision=None) -> dict:
    mapping, coeff, u, v, I, J = _descriptor_problem(descriptor)
    return {"precision": _resolve_precision(x, w, compute_precision), "forward_impl": 0, "a_view": 1, "j_rows": J}
