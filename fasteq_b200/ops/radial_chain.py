"""Fused hidden layers of the radial MLP: ``h_L = silu(W_L ... silu(W_1 basis))`` in one kernel, and
its gradient with respect to the basis in another (``fasteq_radial_chain_forward`` / ``_backward``).

Width 64, one to three hidden layers, at most 16 basis functions, FP32, no bias, weights that do not
require grad (inference and force evaluation); anything else returns ``None`` from
``radial_chain`` so that the caller takes the layered path.
"""
from __future__ import annotations

from typing import Optional, Sequence

import torch

from .. import _front

WIDTH = 64
MAX_BASIS = 16
MAX_HIDDEN = 3


def radial_chain_usable(basis: torch.Tensor, weights: Sequence[torch.Tensor]) -> bool:
    if not (basis.is_cuda and basis.dtype == torch.float32 and basis.dim() == 2 and basis.shape[0] > 0):
        return False
    if not (1 <= len(weights) <= MAX_HIDDEN and 1 <= basis.shape[1] <= MAX_BASIS):
        return False
    if tuple(weights[0].shape) != (WIDTH, basis.shape[1]):
        return False
    for w in weights:
        if w.dtype != torch.float32 or not w.is_cuda or (torch.is_grad_enabled() and w.requires_grad):
            return False
    return all(tuple(w.shape) == (WIDTH, WIDTH) for w in weights[1:])


def radial_chain(basis: torch.Tensor, weights: Sequence[torch.Tensor]) -> Optional[torch.Tensor]:
    """``silu(W_L ... silu(W_1 basis^T))^T`` for ``basis [E, n_basis]`` and ``torch.nn.Linear`` style weights
    (``[out, in]``), or ``None`` when the fused kernels do not take the arguments."""
    return _front.lib().radial_chain(basis, list(weights)) if basis.is_cuda else None
