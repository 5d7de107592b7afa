"""Which gradients a backward has to produce.

``ctx.needs_input_grad`` says whether an input requires a gradient at all.  In the force pass of a training step
(``autograd.grad(energy, positions, create_graph=True)``) the layer weights do, yet nobody asks for their gradients there:
they are asked for when the loss is differentiated.  The engine knows which nodes the running pass will execute."""
from __future__ import annotations

import torch


def wanted(ctx, i: int) -> bool:
    """Whether the running backward asks for the gradient of the ``i``-th tensor input of ``ctx``'s function.  Only a pass that
    builds a graph is looked into; where the engine does not answer (it refuses leaves that are targets of the pass, and
    is not the one running under functional transforms) the gradient counts as wanted."""
    if not ctx.needs_input_grad[i]:
        return False
    return True if not torch.is_grad_enabled() else asked(ctx, i)


def asked(ctx, i: int) -> bool:
    """``wanted`` in every pass: the loss of a training step is differentiated with respect to the weights, and nobody asks for the
    gradients of the edge harmonics there."""
    if not ctx.needs_input_grad[i]:
        return False
    try:
        return bool(torch._C._will_engine_execute_node(ctx.next_functions[i][0]))
    except (RuntimeError, AttributeError, IndexError, TypeError):
        return True
