"""Cache of prepared (split / packed) weight forms for the tensor-core kernels, shared by the SO3Linear, dense and radial-chain
operators (``csrc/front/prepared.cpp``): keyed on the weights' storages and versions, ordered between streams, bounded.

Inside CUDA-graph capture a prepared form would be baked into the graph and go stale when the weights
change, so the cache is bypassed there unless the caller declares the weights frozen (``frozen_weights``)."""
from __future__ import annotations

from contextlib import contextmanager
from typing import Optional

from .. import _front


def set_budget(max_bytes: Optional[int]) -> None:
    _front.lib().prepared_set_budget(None if max_bytes is None else int(max_bytes))


def clear() -> None:
    _front.lib().prepared_clear()


@contextmanager
def frozen_weights():
    """Inside this block prepared weights may be used while a CUDA graph is being captured: the caller
    promises not to change the weights for as long as the graph is replayed."""
    lib = _front.lib()
    lib.prepared_freeze(1)
    try:
        yield
    finally:
        lib.prepared_freeze(-1)


def snapshot() -> list:
    """References to everything cached right now (hold them to keep graph-captured pointers valid)."""
    return _front.lib().prepared_snapshot()
