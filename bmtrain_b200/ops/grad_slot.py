"""Writing a parameter's gradient straight into the gradient buffer of the ZeRO block that owns it.

While the backward pass of a block runs, every parameter of the block has a slot in the block's flat gradient buffer
(``block_layer.py``).  The slots are open if the block is made of this package's own modules: other code may want the
gradient from autograd, in its own backward or on another stream.  A backward kernel that is about to produce the whole
gradient of such a parameter can write it there and return nothing to autograd: no zero-fill of the buffer, no gradient
tensor of its own, no add.  A table outside blocks whose gradient is attached already is added to in place (``attached``).
"""
from __future__ import annotations

from typing import Optional

import torch


def watched(param: torch.Tensor) -> bool:
    """Whether hooks expect the gradient of ``param`` to come from autograd."""
    return bool(param._backward_hooks or param._post_accumulate_grad_hooks)


def _nothing(*_):
    pass


def _node_watched(node) -> bool:
    """Whether hooks sit on the node that accumulates into a leaf; wrappers that reduce gradients register them there.  They are kept in a
    dictionary, to which only the handle of a hook leads (3 us)."""
    for register in (node.register_hook, node.register_prehook):
        handle = register(_nothing)
        hooks = handle.hooks_dict_ref()
        handle.remove()
        if hooks:
            return True
    return False


def attached(ctx, position: int, param: torch.Tensor) -> Optional[torch.Tensor]:
    """``param.grad`` if a backward that is running (``ctx``, whose input number ``position`` is the leaf ``param``) may add to it itself and
    return nothing to autograd, or None.  That is what autograd would do with a gradient that it got: the engine executes the leaf's
    accumulation in this very pass (a ``backward``, not a ``grad``, whose inputs if given contain the leaf), nothing watches the
    parameter or that node, no graph of the gradient is asked for, and the gradient is there, plain, of the parameter's type and on a 16-byte boundary.  Only on the default
    stream: elsewhere it is the engine that orders the accumulation with the leaf's own stream."""
    g = param.grad
    if (g is None or not g.is_cuda or g.dtype != param.dtype or g.shape != param.shape or not g.is_contiguous() or g.requires_grad
            or type(g) is not torch.Tensor or g.data_ptr() % 16 or torch.is_grad_enabled() or watched(param)
            or torch._C._cuda_getCurrentRawStream(g.device.index) != 0):
        return None
    node = ctx.next_functions[position][0]
    if getattr(node, "variable", None) is not param:
        return None
    try:
        if not torch._C._will_engine_execute_node(node) or _node_watched(node):
            return None
    except RuntimeError:        # torch.autograd.grad asks for this leaf
        return None
    torch.autograd.graph.increment_version(g)
    return g


def find(param: Optional[torch.Tensor]):
    """The slot a kernel may write the gradient of ``param`` to, or None: not a parameter of a block whose backward pass
    of known code is running (which includes that nothing watches its parameters), or not trained."""
    ref = getattr(param, "_bmt_grad_slot", None)
    slot = None if ref is None else ref()
    if slot is None or slot.param is not param or not slot.open or not param.requires_grad:
        return None
    return slot
