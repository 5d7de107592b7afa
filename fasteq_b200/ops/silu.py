"""SiLU whose first and second backward are one kernel each (``fasteq_silu``), for the radial MLP of a training step."""
from __future__ import annotations

import torch

from .. import _front


def silu(z: torch.Tensor) -> torch.Tensor:
    if z.is_cuda and z.dtype in (torch.float32, torch.float64) and z.is_contiguous():
        return _front.lib().silu(z)
    return torch.nn.functional.silu(z)
