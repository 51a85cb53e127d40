"""Embedding gather / scatter-add kernels (the reference uses ``F.embedding``).

Index ``-1`` means "not in this shard": forward writes zeros, backward skips the row.  Backward orders the tokens by id
and writes every row of the table's gradient once, added in fp32 and rounded once.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch

from . import _native

_DT = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}


def embedding_forward(ids: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``out[..., :] = weight[ids[...]]`` (zeros where ``ids < 0``)."""
    d = weight.shape[1]
    if not weight.is_cuda:
        safe = ids.clamp(min=0)
        out = weight[safe.reshape(-1)].view(*ids.shape, d)
        return out * (ids >= 0).unsqueeze(-1).to(out.dtype)
    ids64 = ids.to(torch.int64).contiguous()
    out = torch.empty(*ids.shape, d, dtype=weight.dtype, device=weight.device)
    _native.check(_native.cuda_lib().bmt_embedding_fwd(
        ctypes.c_int64(ids64.numel()), ctypes.c_int64(d), _native.ptr(ids64), _native.ptr(weight.contiguous()),
        ctypes.c_int(_DT[weight.dtype]), _native.ptr(out), _native.stream_handle()), "embedding forward kernel")
    return out


def embedding_backward(ids: torch.Tensor, grad: torch.Tensor, rows: int, add_to: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``grad_weight[ids[t]] += grad[t]`` accumulated in fp32, returned in ``grad``'s dtype.  ``add_to`` (GPU): a gradient of the table,
    (rows, d) and contiguous, that the sums are added to; only its rows that occur in ``ids`` are touched."""
    d = grad.shape[-1]
    g2 = grad.reshape(-1, d)
    flat = ids.reshape(-1)
    if not grad.is_cuda:
        acc = torch.zeros(rows, d, dtype=torch.float32)
        keep = flat >= 0
        acc.index_add_(0, flat[keep], g2[keep].float())
        return acc.to(grad.dtype)
    if flat.numel() == 0:
        return torch.zeros(rows, d, dtype=grad.dtype, device=grad.device) if add_to is None else add_to
    lib = _native.cuda_lib()
    ids64, g2 = flat.to(torch.int64).contiguous(), g2.contiguous()
    out = torch.empty(rows, d, dtype=grad.dtype, device=grad.device) if add_to is None else add_to
    lib.bmt_embedding_bwd_scratch.restype = ctypes.c_int64
    words = lib.bmt_embedding_bwd_scratch(ctypes.c_int64(ids64.numel()), ctypes.c_int64(rows))
    scratch = torch.empty(words, dtype=torch.int32, device=grad.device)
    _native.check(_native.entry("bmt_embedding_bwd_ex", "qqqppipipp")(
        ids64.numel(), d, rows, ids64.data_ptr(), g2.data_ptr(), _DT[grad.dtype], out.data_ptr(), 0 if add_to is None else 1, scratch.data_ptr(),
        _native.stream()), "embedding backward kernels")
    return out


class EmbeddingFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, weight):
        ctx.save_for_backward(ids)
        ctx.rows = weight.shape[0]
        return embedding_forward(ids, weight)

    @staticmethod
    def backward(ctx, grad):
        (ids,) = ctx.saved_tensors
        return None, embedding_backward(ids, grad.contiguous(), ctx.rows)


def embedding(ids: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    return EmbeddingFunction.apply(ids, weight)
