"""``fast_uniform1d_jit``: drop-in for fasteq/ops/uniform1d_jit.py:3328-3349.

Same call: ``fast_uniform1d_jit(w, x, y, input_indices, output_indices, meta)`` with
``input_indices = {1: src}`` (gather x), ``{2: src}`` (gather y), ``output_indices =
{0: dst}`` (scatter-sum the result), ``meta`` the reference's dict
(``i_list, j_list, k_list, v_list, coeff_list, w_seg_num, x_seg_num, y_seg_num,
out_seg_num, u_dim, size_list``).  Tensors are 2-D ``[rows, segments * u]`` in
ir_mul layout, CUDA, contiguous (a non-contiguous operand raises ``RuntimeError``
as in the reference; there is no CPU path).

Underneath, the path table is compiled into an sm_100a module (one per
signature, cached in-tree) and called through the C ABI of
include/fasteq_b200.h.  Scattered outputs use a receiver-sorted CSR plan that is
built once per index tensor and cached.
"""
from __future__ import annotations

import dataclasses
import threading
from collections import OrderedDict
from contextlib import contextmanager
from typing import Dict, List, Optional, Tuple

import numpy as np
import torch

from .. import _build, _cabi, _front
from .. import tuning as _tuning
from ..codegen import u1d as _emit
from ..codegen.u1d_common import U1DSpec, make_spec
from ._needs import asked

_EMITTER_VERSION = "u1d-v9"
_MODULES: Dict[Tuple, _cabi.U1DModule] = {}
_TUNING_OVERRIDE: Dict[str, _emit.Tuning] = {}
_lock = threading.Lock()


def _dtype_str(t: torch.Tensor) -> str:
    if t.dtype == torch.float32:
        return "f32"
    if t.dtype == torch.float64:
        return "f64"
    raise ValueError(f"fast_uniform1d_jit supports float32 and float64, got {t.dtype}")


def get_module(spec: U1DSpec, direction: str, needs=(False, False, False), tuning: Optional[_emit.Tuning] = None) -> _cabi.U1DModule:
    """Build (or load from the in-tree cache) the module of one signature."""
    tun = tuning or _TUNING_OVERRIDE.get(direction) or _tuning.lookup(spec, direction, needs) or _emit.untuned(spec, direction)
    key = (spec, direction, tuple(needs), tun)
    with _lock:
        mod = _MODULES.get(key)
    if mod is None:
        # compile outside the lock: different signatures build in parallel; the build itself is
        # atomic (temporary file + rename), so a duplicate build of one signature is harmless
        tag = spec.key(f"{_EMITTER_VERSION}|{direction}|{tuple(needs)}|{tun}")
        if direction == "fwd":
            source = _emit.emit_forward(spec, tun)
        else:
            source = _emit.emit_backward(spec, tun, *needs)
        so = _build.build_generated(f"u1d_{direction}_{tag}", source)
        with _lock:
            mod = _MODULES.get(key)
            if mod is None:
                mod = _cabi.U1DModule(so)
                _MODULES[key] = mod
    return mod


# ----------------------------------------------------------------------------- graph plan

class GraphPlan:
    """Receiver-sorted CSR view of a scatter index: sortedness, permutation, segment offsets, largest degree
    and per-grid partitions.  Built once per index tensor (one host sync) and cached.  Each build step
    leaves an event behind it; ``ready_on_current_stream`` makes a later user on another stream wait for them."""

    def __init__(self, dst: torch.Tensor, n_rows: int, seg_ptr: Optional[torch.Tensor] = None, max_degree: Optional[int] = None):
        if dst.dim() != 1:
            raise ValueError("scatter index must be 1-D")
        core = _cabi.core()
        self.n_rows = int(n_rows)
        self.n_edges = int(dst.numel())
        dev = dst.device
        self.device = dev
        if seg_ptr is not None:
            # the caller vouches for a receiver-sorted index and brings its CSR offsets (the GPU
            # neighbour-list builder does): nothing to check, nothing to build, no host sync
            if seg_ptr.numel() != self.n_rows + 1 or seg_ptr.dtype != torch.int32 or seg_ptr.device != dev:
                raise ValueError("seg_ptr must be an int32 tensor of n_rows + 1 offsets on the index's device")
            self.sorted, self.perm, self.seg_ptr = True, None, seg_ptr.contiguous()
            # where the caller does not know it: no receiver set has a smaller one, and to read it back would be the sync saved
            self.max_degree = int(max_degree) if max_degree is not None else -(-self.n_edges // max(self.n_rows, 1))
            self.native = self._native()
            return
        stream = _cabi.stream(dev)
        dst32 = dst.to(torch.int32).contiguous()
        survey = torch.empty(2 + self.n_rows, dtype=torch.int32, device=dev)
        with _cabi.on_device(dev):
            _cabi.check(core.fasteq_graph_survey(dst32.data_ptr(), self.n_edges, self.n_rows, survey.data_ptr(), stream), core,
                        "fasteq_graph_survey")
            unsorted, self.max_degree = survey[:2].tolist()
            self.sorted = not unsorted
            if self.sorted:
                self.perm = None
                sorted_dst = dst32
            else:
                sorted_dst64, perm = torch.sort(dst32.to(torch.int64), stable=True)
                self.perm = perm.to(torch.int32).contiguous()
                sorted_dst = sorted_dst64.to(torch.int32).contiguous()
            self.seg_ptr = torch.empty(self.n_rows + 1, dtype=torch.int32, device=dev)
            _cabi.check(core.fasteq_graph_build_csr(sorted_dst.data_ptr(), self.n_edges, self.n_rows,
                                                    self.seg_ptr.data_ptr(), stream), core, "fasteq_graph_build_csr")
        self.native = self._native()
        self.native.mark_built()

    def _native(self):
        """The offsets, partitions and events (``csrc/front/u1d.cpp``), which operator calls use without this object."""
        n_rows, n_edges, max_degree, device = self.n_rows, self.n_edges, self.max_degree, self.device
        return _front.lib().Plan(self.seg_ptr, self.perm, n_rows, n_edges, lambda mod: _shares(mod.desc, n_rows, n_edges, max_degree, device))

    @property
    def _parts(self) -> Dict[Tuple[int, bool], torch.Tensor]:
        return self.native.parts()

    def ready_on_current_stream(self) -> None:
        """Order the current stream behind the kernels that built this plan on other streams."""
        self.native.order_current_stream()

    def shares(self, desc: _cabi.U1DDesc) -> Tuple[torch.Tensor, int, bool]:
        """``(partition, its pipelines, whether it cuts receivers)`` for a module's launches."""
        n, split = _shares(desc, self.n_rows, self.n_edges, self.max_degree, self.device)
        return self.partition(n, split), n, split

    def record(self) -> None:
        """Enter the plan into the lists of ``record_plans``."""
        for rec in _RECORDERS:
            if not any(p is self for p in rec):
                rec.append(self)

    def partition(self, n_parts: int, split: bool = False) -> torch.Tensor:
        """First row of each share (``[1, n_parts + 1]``); with ``split`` shares are cut between edges and a second row holds
        their first edges."""
        return self.native.partition(n_parts, split)


def _shares(desc: _cabi.U1DDesc, n_rows: int, n_edges: int, max_degree: int, device) -> Tuple[int, bool]:
    """``(pipelines with a share, whether shares cut receivers)`` for a module's launches over a graph."""
    pipelines = _sm_count(device) * int(desc.ctas_per_sm)
    split = split_receivers(desc, n_rows, n_edges, max_degree, pipelines)
    return max(1, min(pipelines, max(n_rows, (n_edges + 3) // 4) if split else n_rows)), split


_PLANS: "OrderedDict[Tuple, GraphPlan]" = OrderedDict()   # least recently used first
_PLAN_LIMIT = 64
_OWNED: Dict[str, Tuple] = {}          # owner tag -> key of the plan that owner registered last
_RECORDERS: List[list] = []            # lists that collect every plan a call uses (see record_plans)


def _plan_key(dst: torch.Tensor, n_rows: int) -> Tuple:
    return (dst.data_ptr(), dst.numel(), dst._version, str(dst.device), dst.dtype, int(n_rows))


def _insert_plan(key: Tuple, plan: GraphPlan) -> None:
    while len(_PLANS) >= _PLAN_LIMIT:
        _PLANS.popitem(last=False)
    _PLANS[key] = plan


def graph_plan(dst: torch.Tensor, n_rows: int) -> GraphPlan:
    """Cached plan of a scatter index.  The key is the index tensor's storage address, length and torch
    version counter: an index rewritten in place OUTSIDE torch's version tracking (memory shared with an
    engine through DLPack / ``from_blob``, a write through ``.data``) keeps its key, so such callers must
    treat index tensors as immutable or call ``invalidate_plan`` after every rewrite."""
    key = _plan_key(dst, n_rows)
    plan = _PLANS.get(key)
    if plan is None:
        plan = GraphPlan(dst, n_rows)
        plan._keepalive = dst.detach()  # the key is the storage address: keep the storage from being recycled
        _insert_plan(key, plan)
    else:
        _PLANS.move_to_end(key)
    return plan


def register_sorted_plan(dst: torch.Tensor, n_rows: int, seg_ptr: torch.Tensor, owner: Optional[str] = None,
                         max_degree: Optional[int] = None) -> GraphPlan:
    """Install the plan of a receiver-sorted index whose CSR offsets (and largest degree, if the caller has it) are known.  ``owner``: a tag of
    the caller that rebuilds its graph over and over (a neighbour-list builder): its previous plan is dropped
    instead of filling the cache with dead index tensors."""
    key = _plan_key(dst, n_rows)
    if owner is not None:
        old = _OWNED.get(owner)
        if old is not None and old != key:
            _PLANS.pop(old, None)
        _OWNED[owner] = key
    _PLANS.pop(key, None)
    plan = GraphPlan(dst, n_rows, seg_ptr, max_degree)
    plan._keepalive = dst.detach()
    _insert_plan(key, plan)
    return plan


def invalidate_plan(dst: torch.Tensor) -> int:
    """Forget every cached plan of this index tensor's storage (after an in-place rewrite that torch's
    version counter does not see).  Returns the number of plans dropped."""
    hits = [k for k in _PLANS if k[0] == dst.data_ptr() and k[3] == str(dst.device)]
    for k in hits:
        del _PLANS[k]
    return len(hits)


@contextmanager
def record_plans():
    """Collect the plans used by the operator calls made inside the block.  A CUDA graph captured there
    bakes the plans' device pointers into its launches; whoever owns the graph must hold the collected
    plans for as long as the graph is replayed (the cache alone may evict them)."""
    got: list = []
    _RECORDERS.append(got)
    _front.lib().u1d_on_record(GraphPlan.record)
    _front.lib().u1d_recording(1)
    try:
        yield got
    finally:
        _front.lib().u1d_recording(-1)
        _RECORDERS.remove(got)


_SM_COUNT: Dict[int, int] = {}


def _sm_count(dev: torch.device) -> int:
    idx = dev.index if dev.index is not None else torch.cuda.current_device()
    if idx not in _SM_COUNT:
        _SM_COUNT[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    return _SM_COUNT[idx]


# ----------------------------------------------------------------------------- helpers

def _validate(w, x, y):
    for name, t in (("w", w), ("x", x), ("y", y)):
        if not isinstance(t, torch.Tensor):
            raise TypeError(f"{name} must be a tensor")
        if not t.is_cuda:
            raise RuntimeError(f"{name} must be a CUDA tensor: fasteq_b200 has no CPU path")
        if not t.is_contiguous():
            raise RuntimeError(f"{name} must be contiguous")
    if not (w.dtype == x.dtype == y.dtype):
        raise ValueError("w, x, y must share one dtype")


def _index32(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    if t is None:
        return None
    if t.dtype != torch.int32:
        t = t.to(torch.int32)
    return t.contiguous()


class _Call:
    """Resolved shapes / indices / plan of one operator call, shared by forward and backward."""

    def __init__(self, w, x, y, input_indices, output_indices, meta):
        input_indices = {} if input_indices is None else input_indices
        output_indices = {} if output_indices is None else output_indices
        self.u = int(meta["u_dim"])
        self.w_segs, self.x_segs = int(meta["w_seg_num"]), int(meta["x_seg_num"])
        self.y_segs, self.out_segs = int(meta["y_seg_num"]), int(meta["out_seg_num"])
        size_list = meta["size_list"]
        # extension of the reference's meta: "y_sh" = (degrees, normalize, normalization) says that the y
        # operand holds edge vectors [rows, 3] whose spherical harmonics the kernel evaluates itself
        self.y_sh = tuple(meta["y_sh"]) if meta.get("y_sh") else ()
        y_cols = int(size_list[2]) // self.y_segs
        if y_cols not in (1, self.u):
            raise ValueError("y must carry 1 or u_dim values per segment")
        self.y_vec = y_cols != 1
        y_row = 3 if self.y_sh else self.y_segs * y_cols
        if self.y_sh and (self.y_vec or y.shape[-1] != 3):
            raise ValueError("with in-kernel spherical harmonics y must be the edge vectors [rows, 3]")
        for name, t, cols in (("w", w, self.w_segs * self.u), ("x", x, self.x_segs * self.u), ("y", y, y_row)):
            if t.dim() < 2 or t.numel() % cols != 0:
                raise ValueError(f"{name} has {t.numel()} elements, not a multiple of {cols}")
        self.w_rows, self.x_rows, self.y_rows = w.numel() // (self.w_segs * self.u), x.numel() // (self.x_segs * self.u), y.numel() // y_row
        self.x_indexed, self.y_indexed = 1 in input_indices, 2 in input_indices
        self.scattered = 0 in output_indices
        src = input_indices.get(1, input_indices.get(2))
        self.src = _index32(src)
        dst = output_indices.get(0)
        # row count of the per-edge operands: dst, else src, else x (uniform1d_forward.py:163-168)
        if dst is not None:
            self.n_edges = int(dst.numel())
        elif src is not None:
            self.n_edges = int(src.numel())
        else:
            self.n_edges = self.x_rows
        self.w_shared = self.w_rows == 1 and self.n_edges != 1
        if not self.w_shared and self.w_rows != self.n_edges:
            raise ValueError(f"w has {self.w_rows} rows for {self.n_edges} edges")
        if not self.x_indexed and self.x_rows != self.n_edges:
            raise ValueError("x rows must equal the edge count when x is not gathered")
        if not self.y_indexed and self.y_rows != self.n_edges:
            raise ValueError("y rows must equal the edge count when y is not gathered")
        # scattered output has as many rows as x (uniform1d_forward.py:109)
        self.n_out_rows = self.x_rows if self.scattered else self.n_edges
        self.plan = graph_plan(dst, self.n_out_rows) if self.scattered else None
        self.dtype = _dtype_str(w)
        skey = tuple((id(meta[k]), getattr(meta[k], "_version", 0)) for k in ("i_list", "j_list", "k_list", "v_list", "coeff_list")) + (
            self.w_segs, self.x_segs, self.y_segs, self.out_segs, self.u, self.dtype, self.y_vec, self.w_shared,
            self.x_indexed, self.y_indexed, self.scattered, self.y_sh)
        hit = _SPEC_CACHE.get(skey)
        if hit is None:
            spec = make_spec(
                _np(meta["i_list"]), _np(meta["j_list"]), _np(meta["k_list"]), _np(meta["v_list"]), _np(meta["coeff_list"], True),
                w_segs=self.w_segs, x_segs=self.x_segs, y_segs=self.y_segs, out_segs=self.out_segs, u=self.u,
                dtype=self.dtype, y_vec=self.y_vec, w_shared=self.w_shared, x_indexed=self.x_indexed,
                y_indexed=self.y_indexed, scattered=self.scattered, y_sh=self.y_sh)
            if len(_SPEC_CACHE) > 256:
                _SPEC_CACHE.clear()
            # the entry holds the table objects so their ids stay unique while it exists
            hit = (spec, [meta[k] for k in ("i_list", "j_list", "k_list", "v_list", "coeff_list")])
            _SPEC_CACHE[skey] = hit
        self.spec = hit[0]

    def graph(self, mod: _cabi.U1DModule, dev) -> Tuple[_cabi.U1DGraph, Optional[int]]:
        """The launch's graph record and, when the shares of its pipelines split receivers, the address of their first edges."""
        g, part_edge = _cabi.U1DGraph(), None
        g.n_edges, g.n_out_rows, g.x_rows, g.y_rows = self.n_edges, self.n_out_rows, self.x_rows, self.y_rows
        g.x_index = self.src.data_ptr() if self.x_indexed else None
        g.y_index = self.src.data_ptr() if self.y_indexed else None
        if self.plan is not None:
            g.seg_ptr = self.plan.seg_ptr.data_ptr()
            g.perm = self.plan.perm.data_ptr() if self.plan.perm is not None else None
            part, g.n_parts, split = self.plan.shares(mod.desc)
            g.part_ptr, part_edge = part.data_ptr(), part[1].data_ptr() if split else None
            g.part = part               # under capture nobody else holds it
            self.plan.ready_on_current_stream()
            self.plan.record()
        return g, part_edge


# Below this many receivers per pipeline shares may be cut between edges, backward and forward.
SPLIT_ROWS_PER_PIPELINE = 32
SPLIT_ROWS_PER_PIPELINE_FORWARD = 14


def split_receivers(desc: _cabi.U1DDesc, n_rows: int, n_edges: int, max_degree: int, pipelines: int) -> bool:
    """Whether a launch's shares are cut between edges instead of between receivers.

    The longest share of whole receivers is the longest receiver where each has a pipeline, and about one receiver longer than the
    mean where pipelines take several.

    The backward pays only for receivers that two pipelines begin, and takes the cut throughout: 0.02 to 1.02 of the time on whole
    receivers over graphs of 1 to 15,000 receivers of 1 to 60 edges (once 1.08: 18.7 against 17.4 us, 512 equal rows of 33 channels).  The exception are FP64 rows in two thread groups, whose
    beginning costs as much as several edges: where equal receivers fill whole shares almost evenly they keep them (2,000 receivers of
    exactly 8 edges: 425 whole, 482 us cut; of 8 on average 516 and 489).

    The forward also pays for the carry rows and their launch, 2 to 18 us: what 24 to 30 edges of one pipeline take in FP32, half as
    many in the kernels with the slowest edges (rows that cannot travel as bulk copies; FP64 rows in two thread groups).  55 segments
    of 128 channels: 512 receivers of 8 edges 16.8 whole, 24.4 us cut; of 30 edges on average 48.3 and 42.6; of exactly 30 edges 30.1
    and 42.6; 4,000 receivers of 16 edges 97 and 102, of 30 edges 167 and 162; 55 segments of 64 channels, 2,000 of 30 edges 69.5
    and 60.9.  With these limits no forward of the sweep (529 graphs over seven signatures) is slower than on whole receivers by
    more than two runs of one differ.  With many receivers per pipeline the cut gains nothing and the forward loses by it: 52 edges
    on average, 55 segments of 128 channels, 4,000 receivers (7 per pipeline) 288 whole, 267 us cut; 6,000 (10) 411 and 393;
    9,000 (15) 594 and 607; 12,288 (21) 803 and 862; FP64, 55 segments of 64 channels, 10 per pipeline 462 and 445, 15 675 and 721."""
    if n_edges == 0 or n_rows >= SPLIT_ROWS_PER_PIPELINE * pipelines:
        return False
    wide = desc.dtype == 1 and desc.out_segs > 64
    if desc.direction == 1:
        even = 4 * max_degree * n_rows <= 5 * n_edges and n_rows > pipelines
        return not (wide and even and -(-n_rows // pipelines) * max_degree * pipelines - n_edges < 8 * pipelines)
    if n_rows >= SPLIT_ROWS_PER_PIPELINE_FORWARD * pipelines:
        return False
    slow = wide or desc.u * (8 if desc.dtype == 1 else 4) % 16 != 0
    if n_rows <= pipelines:
        return max_degree * pipelines - n_edges >= (16 if slow else 32) * pipelines
    return max_degree >= (24 if slow else 40)


_META_CACHE: Dict[Tuple, Tuple[torch.Tensor, np.ndarray]] = {}


def _np(t, is_float=False) -> np.ndarray:
    """Host copy of a meta tensor.  Cached by storage identity; the cache keeps the storage alive,
    so its address cannot be handed to another tensor while the entry exists."""
    if isinstance(t, torch.Tensor):
        key = (t.data_ptr(), t.numel(), t._version, t.dtype, str(t.device))
        hit = _META_CACHE.get(key)
        if hit is None:
            a = t.detach().cpu().numpy().astype(np.float64 if is_float else np.int64)
            if len(_META_CACHE) > 512:
                _META_CACHE.clear()
            _META_CACHE[key] = (t.detach(), a)
            return a
        return hit[1]
    return np.asarray(t, dtype=np.float64 if is_float else np.int64)


_SPEC_CACHE: Dict[Tuple, U1DSpec] = {}


def _tuning_for(spec: U1DSpec, direction: str, tensors, needs=(False, False, False)) -> Optional[_emit.Tuning]:
    """The launch configuration of this call: the measured winner of the signature when the tuning database has one,
    else the heuristic default.  Packed two-channel modules read and write 8-byte pairs; operands at an odd 4-byte
    offset (a contiguous view into a larger buffer) get the one-channel-per-thread module instead."""
    return _tuning_at(spec, direction, any(t is not None and t.data_ptr() % 8 for t in tensors), needs)


def _tuning_at(spec: U1DSpec, direction: str, odd: bool, needs) -> Optional[_emit.Tuning]:
    tun = _TUNING_OVERRIDE.get(direction) or _tuning.lookup(spec, direction, needs) or _emit.untuned(spec, direction)
    if odd and tun.vec == 2:
        return dataclasses.replace(tun, vec=1, pipes=1, groups=max(tun.groups, 1), min_blocks=min(tun.min_blocks + 1, 3))
    return tun


def _run_fwd(call: _Call, w, x, y) -> torch.Tensor:
    dev = x.device
    out = torch.empty((call.n_out_rows, call.out_segs * call.u), dtype=x.dtype, device=dev)
    mod = get_module(call.spec, "fwd", tuning=_tuning_for(call.spec, "fwd", (w, x, y, out)))
    with _cabi.on_device(dev):
        g, part_edge = call.graph(mod, dev)
        stream = _cabi.stream(dev)
        if part_edge is not None:
            carry = torch.empty((g.n_parts, call.out_segs * call.u), dtype=x.dtype, device=dev)
            mod.forward_split(g, part_edge, carry.data_ptr(), w.data_ptr(), x.data_ptr(), y.data_ptr(), out.data_ptr(), stream)
        else:
            mod.forward(g, w.data_ptr(), x.data_ptr(), y.data_ptr(), out.data_ptr(), stream)
    return out


def _run_bwd(call: _Call, grad_out, w, x, y, needs):
    dev = x.device
    gw = torch.empty_like(w) if needs[0] else None
    gx = torch.empty_like(x) if needs[1] else None
    gy = torch.empty_like(y) if needs[2] else None
    mod = get_module(call.spec, "bwd", needs, tuning=_tuning_for(call.spec, "bwd", (grad_out, w, x, y, gw, gx, gy), needs))
    ptr = lambda t: t.data_ptr() if t is not None else None
    with _cabi.on_device(dev):
        g, part_edge = call.graph(mod, dev)
        args = (grad_out.data_ptr(), w.data_ptr(), x.data_ptr(), y.data_ptr(), ptr(gw), ptr(gx), ptr(gy),
                _cabi.stream(dev))
        if part_edge is not None:
            mod.backward_split(g, part_edge, *args)
        else:
            mod.backward(g, *args)
    return gw, gx, gy


_DUAL_SPECS: Dict[Tuple[U1DSpec, Tuple[bool, bool, bool]], Optional[U1DSpec]] = {}


def _dual_spec(spec: U1DSpec, has: Tuple[bool, bool, bool]) -> Optional[U1DSpec]:
    """The second-order signature with tangents where ``has`` says so; ``None`` for the operand forms without such modules and for rows so
    wide that the modules would not fit an SM."""
    if not (spec.scattered and spec.x_indexed) or spec.w_shared or spec.y_vec or spec.y_indexed or spec.y_sh:
        return None
    if (spec, has) not in _DUAL_SPECS:
        if len(_DUAL_SPECS) > 256:
            _DUAL_SPECS.clear()
        dual = dataclasses.replace(spec, dual=has)
        _DUAL_SPECS[(spec, has)] = dual if _emit.second_order_fits(dual) else None
    return _DUAL_SPECS[(spec, has)]


def _second_order_composed(call: _Call, go, w, x, y, tangents, wants):
    """``(d_go, d_w, d_x, d_y)`` of ``<go, F(w', x, y) + F(w, x', y) + F(w, x, y')>``, ``tangents = (w', x', y')`` with ``None`` for those that
    are zero, from the first-order functions, so that autograd may go on differentiating.  The operator is trilinear in (w, x, y), so every term is a forward or a one-gradient backward of
    the same signature with an operand swapped for its tangent (the usual operand form has modules of its own for this, see
    ``csrc/front/u1d.cpp``):

        d_go = F(w', x, y) + F(w, x', y) + F(w, x, y')
        d_w  = Bw(go; x', y) + Bw(go; x, y')      (Bw = gradient with respect to the weight slot)
        d_x  = Bx(go; w', y) + Bx(go; w, y')
        d_y  = By(go; w', x) + By(go; w, x')
    """
    operands = (w, x, y)
    out = [None] * 4

    def swapped(i):
        return tuple(tangents[i] if k == i else t for k, t in enumerate(operands))

    for i, t in enumerate(tangents):
        if t is None:
            continue
        terms = [(0, FastUniform1dJITFunction.apply(*swapped(i), None, None, call))] if wants[0] else []
        terms += [(1 + k, FastUniform1dBackwardFunction.apply(go, *swapped(i), call, tuple(n == k for n in range(3)))[k])
                  for k in range(3) if k != i and wants[1 + k]]
        for k, v in terms:
            out[k] = v if out[k] is None else out[k] + v
    return tuple(out)


class FastUniform1dBackwardFunction(torch.autograd.Function):
    """First backward as a differentiable function (reference: fasteq/ops/uniform1d_jit.py:3098-3188),
    so that force losses can be trained."""

    @staticmethod
    def forward(ctx, grad_out, w, x, y, call, needs):
        gw, gx, gy = _run_bwd(call, grad_out, w, x, y, needs)
        ctx.call, ctx.needs = call, needs
        ctx.save_for_backward(grad_out, w, x, y)
        ctx.set_materialize_grads(False)
        outs = tuple(g if g is not None else t.new_empty((0,)) for g, t in ((gw, w), (gx, x), (gy, y)))
        return outs

    @staticmethod
    def backward(ctx, *tangents):
        go, w, x, y = ctx.saved_tensors
        tangents = tuple(t.contiguous() if (t is not None and n) else None for t, n in zip(tangents, ctx.needs))
        if all(t is None for t in tangents):
            return (None,) * 6
        wants = tuple(asked(ctx, i) for i in range(4))
        return _second_order_composed(ctx.call, go, w, x, y, tangents, wants) + (None, None)


class FastUniform1dJITFunction(torch.autograd.Function):
    """Autograd wrapper (reference: fasteq/ops/uniform1d_jit.py:3194-3326).  The backward produces
    exactly the gradients autograd asks for and is itself differentiable.  ``meta`` may be the resolved call."""

    @staticmethod
    def forward(ctx, w, x, y, input_indices, output_indices, meta):
        _validate(w, x, y)
        call = meta if isinstance(meta, _Call) else _Call(w, x, y, input_indices, output_indices, meta)
        ctx.call = call
        ctx.save_for_backward(w, x, y)
        return _run_fwd(call, w, x, y)

    @staticmethod
    def backward(ctx, grad_out):
        w, x, y = ctx.saved_tensors
        needs = tuple(asked(ctx, i) for i in range(3))
        if not any(needs):
            return None, None, None, None, None, None
        if ctx.call.y_sh:
            # not trilinear in the edge vector: the composed second backward does not apply
            if torch.is_grad_enabled() and any(t.requires_grad for t in (grad_out, w, x, y)):
                raise RuntimeError("fast_uniform1d_jit: no second-order gradient with in-kernel spherical harmonics; "
                                   "pass the harmonics as the y operand instead")
            gw, gx, gy = _run_bwd(ctx.call, grad_out.contiguous(), w, x, y, needs)
        else:
            gw, gx, gy = FastUniform1dBackwardFunction.apply(grad_out.contiguous(), w, x, y, ctx.call, needs)
        return (gw if needs[0] else None), (gx if needs[1] else None), (gy if needs[2] else None), None, None, None


_SIGNATURES: Dict[Tuple, Tuple] = {}
_TABLES = ("i_list", "j_list", "k_list", "v_list", "coeff_list")
_EXPORTS = tuple(f"fasteq_u1d_{n}" for n in ("forward", "forward_split", "backward", "backward_split", "tangent_forward", "tangent_backward")) + (
    "fasteq_last_cuda_error",)


def _signature(meta, dtype):
    """``(native signature, columns of x)`` of the usual operand form (per-edge weights, sender gather, receiver scatter, one y value per
    segment); ``None`` for the others."""
    y_sh = meta.get("y_sh")
    # whole numbers may come as tensors, which would be another key each time they are taken out of their list
    key = tuple((id(meta[k]), getattr(meta[k], "_version", 0)) for k in _TABLES) + (
        int(meta["w_seg_num"]), int(meta["x_seg_num"]), int(meta["y_seg_num"]), int(meta["out_seg_num"]), int(meta["u_dim"]),
        int(meta["size_list"][2]), dtype, tuple(y_sh) if y_sh else ())
    hit = _SIGNATURES.get(key)
    if hit is not None:
        return hit[0]
    made = None
    segs = [int(meta[k]) for k in ("w_seg_num", "x_seg_num", "y_seg_num", "out_seg_num")]
    u = int(meta["u_dim"])
    if dtype in (torch.float32, torch.float64) and int(meta["size_list"][2]) // segs[2] == 1:
        spec = make_spec(_np(meta["i_list"]), _np(meta["j_list"]), _np(meta["k_list"]), _np(meta["v_list"]), _np(meta["coeff_list"], True),
                         w_segs=segs[0], x_segs=segs[1], y_segs=segs[2], out_segs=segs[3], u=u, dtype="f32" if dtype == torch.float32 else "f64",
                         y_sh=tuple(y_sh) if y_sh else ())

        def load(direction, needs, tangents, odd):
            sp = spec if tangents is None else _dual_spec(spec, tuple(tangents))
            if sp is None:
                return None
            mod = get_module(sp, direction, tuple(needs), tuning=_tuning_at(sp, direction, odd, tuple(needs)))
            return mod, _front.addresses(mod.lib, _EXPORTS)
        made = (_front.lib().Signature(u, *segs, bool(y_sh), load), segs[1] * u)
    if len(_SIGNATURES) > 256:
        _SIGNATURES.clear()
    # the entry holds the table objects so their ids stay unique while it exists
    _SIGNATURES[key] = (made, [meta[k] for k in _TABLES])
    return made


def _native_call(w, x, y, input_indices, output_indices, meta) -> Optional[torch.Tensor]:
    """The call through the native host path, or ``None`` where its form is not the usual one (or something is wrong with it)."""
    if _TUNING_OVERRIDE or not input_indices or not output_indices or len(input_indices) != 1:
        return None
    src, dst = input_indices.get(1), output_indices.get(0)
    for t in (w, x, y, src, dst):
        if not isinstance(t, torch.Tensor) or not t.is_cuda:
            return None
    try:
        sig = _signature(meta, x.dtype)
    except TypeError:                    # a table key that cannot be hashed
        return None
    if sig is None or x.numel() % sig[1]:
        return None
    plan = graph_plan(dst, x.numel() // sig[1])
    return _front.lib().u1d(w, x, y, src, sig[0], plan.native, plan)


def fast_uniform1d_jit(w, x, y, input_indices, output_indices, meta, use_multiwarp_candidates: Optional[bool] = None):
    """See module docstring.  ``use_multiwarp_candidates`` is accepted and ignored, as in the reference."""
    out = _native_call(w, x, y, input_indices, output_indices, meta)
    return FastUniform1dJITFunction.apply(w, x, y, input_indices, output_indices, meta) if out is None else out
