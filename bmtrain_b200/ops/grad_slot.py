"""Writing a parameter's gradient straight into the gradient buffer of the ZeRO block that owns it.

While a block's backward pass runs, every parameter of the block has a slot in the block's flat gradient buffer
(``block_layer.py``).  A backward kernel that is about to produce the whole gradient of such a parameter can write it
there and return nothing to autograd: no zero-fill of the buffer, no gradient tensor of its own, no add.
"""
from __future__ import annotations

from typing import Optional

import torch


def find(param: Optional[torch.Tensor]):
    """The slot a kernel may write the gradient of ``param`` to, or None: not a parameter of a block whose backward pass
    is running, not trained, or watched by hooks that expect the gradient to come from autograd."""
    slot = getattr(param, "_bmt_grad_slot", None)
    if slot is None or slot.param is not param or not slot.open or not param.requires_grad:
        return None
    if param._backward_hooks or getattr(param, "_post_accumulate_grad_hooks", None):
        return None
    return slot
