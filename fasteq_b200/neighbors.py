"""Periodic radius graph built on the GPU (``fasteq_neighbors_*``): receiver-sorted edges in the
canonical (receiver, sender, image) order of ``fasteq_b200.graph.periodic_radius_graph`` plus the CSR
offsets, registered as a ready graph plan so that the tensor-product operator needs neither a
sortedness check nor a CSR build for the returned receiver index."""
from __future__ import annotations

from dataclasses import dataclass

import numpy as np
import torch

from . import _front

MAX_DEGREE = 1024


@dataclass
class RadiusGraph:
    edge_src: torch.Tensor     # [E] int32 sender
    edge_dst: torch.Tensor     # [E] int32 receiver, non-decreasing
    edge_shift: torch.Tensor   # [E, 3] float64 cartesian image offset of the sender
    seg_ptr: torch.Tensor      # [N + 1] int32 CSR offsets of edge_dst
    max_degree: int


def radius_graph(pos: torch.Tensor, atom_struct: torch.Tensor, box, cutoff: float, register_plan: bool = True) -> RadiusGraph:
    """``pos [N, 3]`` (CUDA, wrapped into the box; evaluated in float64), ``atom_struct [N]`` structure id of
    each atom, ``box [S, 3]`` (or ``[S]`` for cubes) host array of box lengths.  One host sync (the edge count)."""
    if not pos.is_cuda:
        raise RuntimeError("radius_graph: pos must be a CUDA tensor: fasteq_b200 has no CPU path (use fasteq_b200.graph on the host)")
    box = np.ascontiguousarray(np.asarray(box, dtype=np.float64))
    if box.ndim == 1:
        box = np.repeat(box[:, None], 3, axis=1).copy()
    src, dst, shift, seg_ptr, max_deg = _front.lib().radius_graph(pos, atom_struct, box, float(cutoff), MAX_DEGREE)
    if register_plan:
        from .ops.uniform1d_jit import register_sorted_plan
        register_sorted_plan(dst, int(pos.shape[0]), seg_ptr, owner=f"radius_graph:{pos.device}", max_degree=max_deg)
    return RadiusGraph(src, dst, shift, seg_ptr, max_deg)
