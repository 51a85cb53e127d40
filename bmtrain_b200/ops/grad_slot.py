"""Writing a parameter's gradient straight into the gradient buffer of the ZeRO block that owns it.

While the backward pass of a block runs, every parameter of the block has a slot in the block's flat gradient buffer
(``block_layer.py``).  The slots are open if the block is made of this package's own modules: other code may want the
gradient from autograd, in its own backward or on another stream.  A backward kernel that is about to produce the whole
gradient of such a parameter can write it there and return nothing to autograd: no zero-fill of the buffer, no gradient
tensor of its own, no add.
"""
from __future__ import annotations

from typing import Optional

import torch


def watched(param: torch.Tensor) -> bool:
    """Whether hooks expect the gradient of ``param`` to come from autograd."""
    return bool(param._backward_hooks or param._post_accumulate_grad_hooks)


def find(param: Optional[torch.Tensor]):
    """The slot a kernel may write the gradient of ``param`` to, or None: not a parameter of a block whose backward pass
    of known code is running (which includes that nothing watches its parameters), or not trained."""
    ref = getattr(param, "_bmt_grad_slot", None)
    slot = None if ref is None else ref()
    if slot is None or slot.param is not param or not slot.open or not param.requires_grad:
        return None
    return slot
