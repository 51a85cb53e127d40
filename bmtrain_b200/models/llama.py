"""Llama-shaped decoder: RMSNorm, rotary position embedding, SwiGLU FFN, grouped-query attention.

The reference ships no such model; it is here because the 13B / 70B shaped
configurations need one.  Built from the same sharded-parameter modules as
:mod:`bmtrain_b200.models.gpt`.
"""
from __future__ import annotations

import math
import os
from typing import Optional

import torch

from ..block_layer import Block, TransformerBlockList
from ..global_var import config
from ..layer import DistributedModule, reads_parameters_only
from ..nn import ColumnParallelLinear, Embedding, Linear, RMSNorm, RowParallelLinear, VPEmbedding
from ..ops import attention as _attn
from ..ops import elementwise as _ew
from ..ops import llama_block as _llama_block


_FUSED_BLOCK = os.environ.get("BMT_FUSED_BLOCK", "1") != "0"


@reads_parameters_only
class LlamaAttention(DistributedModule):
    def __init__(self, dim_model: int, num_heads: int, num_kv_heads: int, dim_head: int, dtype=None, rope_theta: float = 10000.0):
        super().__init__()
        tp = config["tp_size"]
        assert num_heads % tp == 0 and num_kv_heads % tp == 0 and num_heads % num_kv_heads == 0
        self.h, self.hk, self.dh = num_heads // tp, num_kv_heads // tp, dim_head
        out_qkv = (num_heads + 2 * num_kv_heads) * dim_head
        if tp > 1:
            self.project_qkv = ColumnParallelLinear(dim_model, out_qkv, bias=False, dtype=dtype)
            self.project_out = RowParallelLinear(num_heads * dim_head, dim_model, bias=False, dtype=dtype)
        else:
            self.project_qkv = Linear(dim_model, out_qkv, bias=False, dtype=dtype)
            self.project_out = Linear(num_heads * dim_head, dim_model, bias=False, dtype=dtype)
        self.rope_theta = rope_theta

    def forward(self, hidden: torch.Tensor) -> torch.Tensor:
        tp = config["tp_size"]
        qkv = self.project_qkv(hidden)
        if tp > 1:
            s, b = qkv.shape[0], qkv.shape[1]
            qkv = qkv.view(s, b, self.hk, self.h // self.hk + 2, self.dh).permute(1, 0, 2, 3, 4)
        else:
            b, s = qkv.shape[0], qkv.shape[1]
            qkv = qkv.view(b, s, self.hk, self.h // self.hk + 2, self.dh)
        q, k, v = _ew.rope_qkv(qkv, self.h // self.hk, self.rope_theta)
        out = _attn.attention(q, k, v, 1.0 / math.sqrt(self.dh), causal=True)
        if tp > 1:
            out = out.permute(1, 0, 2, 3).reshape(s, b, self.h * self.dh)
        else:
            out = out.reshape(b, s, self.h * self.dh)
        return self.project_out(out)


@reads_parameters_only
class LlamaMLP(DistributedModule):
    """``w_out(silu(gate) * up)`` with gate and up projections fused into one GEMM (interleaved per TP rank)."""

    def __init__(self, dim_model: int, dim_ff: int, dtype=None):
        super().__init__()
        if config["tp_size"] > 1:
            self.w_gate_up = ColumnParallelLinear(dim_model, 2 * dim_ff, bias=False, dtype=dtype)
            self.w_out = RowParallelLinear(dim_ff, dim_model, bias=False, dtype=dtype)
        else:
            self.w_gate_up = Linear(dim_model, 2 * dim_ff, bias=False, dtype=dtype)
            self.w_out = Linear(dim_ff, dim_model, bias=False, dtype=dtype)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return self.w_out(_ew.swiglu(self.w_gate_up(x)))


@reads_parameters_only
class LlamaBlock(DistributedModule):
    def __init__(self, dim_model, num_heads, num_kv_heads, dim_head, dim_ff, dtype=None, eps=1e-5):
        super().__init__()
        self.ln_attn = RMSNorm(dim_model, eps=eps, dtype=dtype)
        self.attn = LlamaAttention(dim_model, num_heads, num_kv_heads, dim_head, dtype=dtype)
        self.ln_ff = RMSNorm(dim_model, eps=eps, dtype=dtype)
        self.ff = LlamaMLP(dim_model, dim_ff, dtype=dtype)

    # A ``Block`` whose module is this one, as it stands, has it computed by the native executor (see ``Block._native_module``).
    def _bmt_native_takes(self, hidden):
        """The parameters in the executor's order if it takes these arguments, else None."""
        if not (torch.is_tensor(hidden) and hidden.is_cuda and hidden.dim() == 3 and hidden.numel() > 0 and config["tp_size"] == 1
                and hidden.is_contiguous()       # the result of the modules has the strides of what they are given
                and hidden.dtype in (torch.float16, torch.bfloat16) and _FUSED_BLOCK and os.environ.get("BMT_FLASH_ATTN", "1") != "0"):
            return None
        m = self._modules
        if type(m["ln_attn"]) is not RMSNorm or type(m["attn"]) is not LlamaAttention or type(m["ln_ff"]) is not RMSNorm or type(m["ff"]) is not LlamaMLP:
            return None                                  # other submodules
        a = m["attn"]
        attn, ff, d = a._modules, m["ff"]._modules, hidden.shape[-1]
        linears = (attn["project_qkv"], attn["project_out"], ff["w_gate_up"], ff["w_out"])
        if any(type(mod) is not Linear or mod._parameters["bias"] is not None for mod in linears):
            return None
        params = [mod._parameters["weight"] for mod in (m["ln_attn"], *linears[:2], m["ln_ff"], *linears[2:])]
        shapes = [tuple(p._original_shape) for p in params]
        f = shapes[5][1]
        if shapes != [(d,), ((a.h + 2 * a.hk) * a.dh, d), (d, a.h * a.dh), (d,), (2 * f, d), (d, f)]:
            return None
        # what the kernels take: head dims of the fused attention, rows of the norms, whole 16-byte vectors
        return params if a.dh % 16 == 0 and a.dh <= 128 and d % 8 == 0 and d <= 16384 and f % 8 == 0 else None

    def _bmt_native_pass(self, addresses, hidden):
        m = self._modules
        attn = m["attn"]
        return _llama_block.Pass(hidden.contiguous(), addresses, attn.h, attn.hk, attn.dh,
                                 m["ff"]._modules["w_out"]._parameters["weight"]._original_shape[1], m["ln_attn"].eps, m["ln_ff"].eps,
                                 attn.rope_theta)

    def forward(self, hidden: torch.Tensor) -> torch.Tensor:
        hidden = hidden + self.attn(self.ln_attn(hidden))
        return hidden + self.ff(self.ln_ff(hidden))


class Llama(DistributedModule):
    """``forward(input_ids (b, s)) -> logits`` ((b, s, vocab), or (s, b, vocab/tp) under tensor parallelism)."""

    def __init__(self, num_layers: int, vocab_size: int, dim_model: int, num_heads: int, dim_ff: int,
                 num_kv_heads: Optional[int] = None, dim_head: Optional[int] = None, dtype=None,
                 zero_level: int = 3, use_checkpoint: bool = True, init_std: float = 0.02):
        super().__init__()
        num_kv_heads = num_kv_heads or num_heads
        dim_head = dim_head or dim_model // num_heads
        tp = config["tp_size"]
        emb = VPEmbedding if tp > 1 else Embedding
        self.word_emb = emb(vocab_size, dim_model, dtype=dtype, init_std=init_std)
        self.lm_head = emb(vocab_size, dim_model, dtype=dtype, init_std=init_std)
        blocks = [Block(LlamaBlock(dim_model, num_heads, num_kv_heads, dim_head, dim_ff, dtype=dtype),
                        use_checkpoint=use_checkpoint, zero_level=zero_level,
                        mode="PIPE" if config["pipe_size"] > 1 else "BLOCK") for _ in range(num_layers)]
        if config["pipe_size"] > 1:
            from ..pipe_layer import PipelineTransformerBlockList

            self.transformers = PipelineTransformerBlockList(blocks)
        else:
            self.transformers = TransformerBlockList(blocks)
        self.layernorm = RMSNorm(dim_model, dtype=dtype)

    def forward(self, input: torch.Tensor) -> torch.Tensor:
        tp = config["tp_size"]
        if tp > 1:
            input = input.chunk(tp, dim=1)[config["tp_rank"]].t().contiguous()
        out = self.word_emb(input)
        out = self.transformers(out)
        out = self.layernorm(out)
        return self.lm_head(out, projection=True)
