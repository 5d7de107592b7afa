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


def radial_chain_usable(basis: torch.Tensor, weights: Sequence[torch.Tensor]) -> bool:
    """Whether the fused kernels take the arguments."""
    return _front.lib().radial_chain_takes(basis, list(weights))


def radial_chain(basis: torch.Tensor, weights: Sequence[torch.Tensor]) -> Optional[torch.Tensor]:
    """``silu(W_L ... silu(W_1 basis^T))^T`` for ``basis [E, n_basis]`` and ``torch.nn.Linear`` style weights
    (``[out, in]``), or ``None`` when the fused kernels do not take the arguments."""
    return _front.lib().radial_chain(basis, list(weights)) if basis.is_cuda else None
