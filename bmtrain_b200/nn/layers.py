"""Building-block modules on sharded parameters: embedding, LayerNorm, RMSNorm.

The reference keeps these in its example (``example/layers/embedding.py``,
``example/layers/layernorm.py``); they are part of the package here because
they sit on the framework's own kernels.
"""
from __future__ import annotations

from typing import Optional

import torch

from ..layer import DistributedModule, reads_parameters_only
from ..ops import embedding as _emb
from ..ops import gemm as _gemm
from ..ops import grad_slot as _grad_slot
from ..ops import norm as _norm
from ..parameter import DistributedParameter, ParameterInitializer, await_update, private_value, shard_is_value


class _ShardLookup(torch.autograd.Function):
    """Lookup in a table whose shard is the whole table: the kernel has read it before anything behind the call can write to
    it, backward does not need it, and its gradient is a fresh tensor.  So neither is copied; a gradient that is attached is added to."""

    @staticmethod
    def forward(ctx, ids, table):
        await_update(table)
        ctx.save_for_backward(ids)
        ctx.table = table
        return _emb.embedding_forward(ids, table.data.reshape(table._original_shape))

    @staticmethod
    def backward(ctx, grad):
        (ids,) = ctx.saved_tensors
        shape = ctx.table._original_shape
        held = _grad_slot.attached(ctx, 1, ctx.table) if grad.dtype == ctx.table.dtype else None
        if held is not None:
            _emb.embedding_backward(ids, grad.contiguous(), shape[0], add_to=held.view(shape))
            return None, None
        return None, _emb.embedding_backward(ids, grad.contiguous(), shape[0]).view(-1)


class _ShardProjection(torch.autograd.Function):
    """Multiplication by such a table: backward multiplies by the value of the forward pass, which is therefore a copy; the
    table's gradient is a fresh tensor and is not copied, or added to the one that is attached."""

    @staticmethod
    def forward(ctx, x, table):
        ctx.table = table
        return _gemm.LinearFunction.forward(ctx, x, private_value(table), None)

    @staticmethod
    def backward(ctx, grad):
        x, weight = ctx.saved_tensors
        held = _grad_slot.attached(ctx, 1, ctx.table) if ctx.needs_input_grad[1] and grad.dtype == weight.dtype else None
        if held is None:
            grad_x, grad_w, _ = _gemm.LinearFunction.backward(ctx, grad)
            return grad_x, None if grad_w is None else grad_w.view(-1)
        g2 = grad.reshape(-1, grad.shape[-1])
        grad_x = _gemm.gemm_nn(g2, weight).view(x.shape) if ctx.needs_input_grad[0] else None
        _gemm.gemm_tn(g2, x.reshape(-1, x.shape[-1]), out=held.view(weight.shape), accumulate=True)
        return grad_x, None


@reads_parameters_only
class Embedding(DistributedModule):
    """Token embedding; ``forward(x, projection=True)`` multiplies by the transposed table (tied LM head)."""

    def __init__(self, num_embeddings: int, embedding_dim: int, dtype=None, init_mean: float = 0.0, init_std: float = 1.0):
        super().__init__()
        self.num_embeddings = num_embeddings
        self.embedding_dim = embedding_dim
        self.weight = DistributedParameter(
            torch.empty(num_embeddings, embedding_dim, dtype=dtype, device="meta"),
            init_method=ParameterInitializer(torch.nn.init.normal_, mean=init_mean, std=init_std))

    def forward(self, input: torch.Tensor, projection: bool = False) -> torch.Tensor:
        table = self._parameters.get("weight")
        if type(self) is Embedding and isinstance(table, DistributedParameter) and shard_is_value(table):
            if not projection:
                return _ShardLookup.apply(input, table)
            if input.is_cuda or input.dtype != torch.float32:
                return _ShardProjection.apply(input, table)
        if projection:
            return _gemm.linear(input, self.weight)
        return _emb.embedding(input, self.weight)

    def extra_repr(self) -> str:
        return f"{self.num_embeddings}, {self.embedding_dim}"


@reads_parameters_only
class LayerNorm(DistributedModule):
    """LayerNorm over the last dimension."""

    def __init__(self, normalized_shape: int, eps: float = 1e-5, elementwise_affine: bool = True, dtype=None):
        super().__init__()
        if not isinstance(normalized_shape, int):
            (normalized_shape,) = tuple(normalized_shape)
        self.normalized_shape = (normalized_shape,)
        self.eps = eps
        self.elementwise_affine = elementwise_affine
        assert elementwise_affine, "LayerNorm without affine parameters is not provided"
        self.weight = DistributedParameter(torch.empty(normalized_shape, dtype=dtype, device="meta"),
                                           init_method=torch.nn.init.ones_)
        self.bias = DistributedParameter(torch.empty(normalized_shape, dtype=dtype, device="meta"),
                                         init_method=torch.nn.init.zeros_)

    def forward(self, input: torch.Tensor) -> torch.Tensor:
        return _norm.layer_norm(input, self.weight, self.bias, self.eps)

    def extra_repr(self) -> str:
        return f"{self.normalized_shape}, eps={self.eps}"


Layernorm = LayerNorm


@reads_parameters_only
class RMSNorm(DistributedModule):
    """Root-mean-square norm over the last dimension (Llama style)."""

    def __init__(self, dim: int, eps: float = 1e-6, dtype=None):
        super().__init__()
        self.dim = dim
        self.eps = eps
        self.weight = DistributedParameter(torch.empty(dim, dtype=dtype, device="meta"), init_method=torch.nn.init.ones_)

    def forward(self, input: torch.Tensor) -> torch.Tensor:
        return _norm.rms_norm(input, self.weight, self.eps)

    def extra_repr(self) -> str:
        return f"{self.dim}, eps={self.eps}"
