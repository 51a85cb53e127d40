"""Whole Llama-shaped block (RMSNorm, rotary embedding, grouped-query attention, SwiGLU) on the native block executor
(``csrc/block_exec.cu``): each direction is one C++ call that issues all of the block's launches; what a pass keeps for backward, and
what backward scratches, is one allocation each.  Used by ``Block`` for ``models/llama.py`` as it stands; anything else runs the modules.
"""
from __future__ import annotations

import ctypes
import functools
import struct

import torch

from . import _native
from . import elementwise as _ew
from . import gemm as _gemm
from .gpt_block import _carve

# BmtLlamaBlock and BmtLlamaBlockGrad of csrc/api.h as they lie in memory
_BLOCK = struct.Struct("@7qiffi6Q3Q13QQq")
_GRAD = struct.Struct("@8Q13Qq")
_SAVED = ("ln1", "stats1", "q", "k", "v", "ctx", "lse", "h1", "ln2", "stats2", "gate_up", "ff", "packed")
_WORK = ("d_ff", "d_gate_up", "d_ln", "d_h1", "d_ctx", "dq", "dk", "dv", "d_packed", "norm_partial", "dq_acc", "delta", "dkv_part")
PARAM_NAMES = ("ln1_w", "qkv_w", "out_w", "ln2_w", "gate_up_w", "w_out")


@functools.lru_cache(maxsize=256)
def _saved_plan(b, s, d, h, hk, dh, dff):
    T = b * s
    return _carve([("ln1", 2 * T * d), ("stats1", 8 * T), ("q", 2 * T * h * dh), ("k", 2 * T * hk * dh), ("v", 2 * T * hk * dh),
                   ("ctx", 2 * T * h * dh), ("lse", 4 * T * h), ("h1", 2 * T * d), ("ln2", 2 * T * d), ("stats2", 8 * T),
                   ("gate_up", 4 * T * dff), ("ff", 2 * T * dff), ("packed", 2 * T * (h + 2 * hk) * dh)])


@functools.lru_cache(maxsize=256)
def _work_plan(b, s, d, h, hk, dh, dff, nblk):
    T, lib = b * s, _native.cuda_lib()
    lib.bmt_flash_attn_bwd_parts.restype = ctypes.c_int64
    i64, c_int = ctypes.c_int64, ctypes.c_int
    parts = lib.bmt_flash_attn_bwd_parts(i64(b), i64(s), c_int(h), c_int(hk), c_int(dh)) if hk != h else 0
    sizes = [("d_ff", 2 * T * dff), ("d_gate_up", 4 * T * dff), ("d_ln", 2 * T * d), ("d_h1", 2 * T * d), ("d_ctx", 2 * T * h * dh),
             ("dq", 2 * T * h * dh), ("dk", 2 * T * hk * dh), ("dv", 2 * T * hk * dh), ("d_packed", 2 * T * (h + 2 * hk) * dh),
             ("norm_partial", 16 * nblk * d), ("dq_acc", 4 * T * h * dh), ("delta", 4 * T * h)]
    return _carve(sizes + [("dkv_part", 4 * parts)] if parts else sizes)


class Pass:
    """One forward (or recomputation) of a block and what backward needs of it; ``addresses``: of the parameters, in the order of
    ``PARAM_NAMES``."""

    def __init__(self, x, addresses, h, hk, dh, dff, eps1, eps2, theta):
        b, s, d = self.shape = x.shape
        self.x, self.cfg = x, (h, hk, dh, dff)
        plan, total = _saved_plan(b, s, d, h, hk, dh, dff)
        self.saved = torch.empty(total, dtype=torch.uint8, device=x.device)
        base = self.saved.data_ptr()
        self.table = _ew._rope_table(s, dh, theta, x.device)
        self.head = (b, s, d, h, hk, dh, dff, 0 if x.dtype == torch.float16 else 1, eps1, eps2, 0, *addresses)
        self.tail = (self.table.data_ptr(), *[base + plan[n] for n in _SAVED])

    def _describe(self, y, scratch):
        return _BLOCK.pack(*self.head, self.x.data_ptr(), y, *self.tail, *scratch.gemm)

    def forward(self) -> torch.Tensor:
        y = torch.empty_like(self.x)
        scratch = _gemm.scratch()
        _native.check(_native.entry("bmt_llama_block_forward", "bip")(self._describe(y.data_ptr(), scratch), 9, scratch.stream), "Llama block forward")
        return y

    def recompute(self) -> None:
        """Forward again for ``backward``: without the last GEMM, whose result nothing reads."""
        scratch = _gemm.scratch()
        _native.check(_native.entry("bmt_llama_block_forward", "bip")(self._describe(0, scratch), 8, scratch.stream), "Llama block forward")

    def backward(self, dy: torch.Tensor, grads) -> torch.Tensor:
        """``grads``: addresses for the gradients of the parameters, in their order."""
        b, s, d = self.shape
        nblk = min(b * s, 296)
        plan, total = _work_plan(b, s, d, *self.cfg, nblk)
        work = torch.empty(total, dtype=torch.uint8, device=dy.device)
        base = work.data_ptr()
        dx = torch.empty_like(self.x)
        scratch = _gemm.scratch()
        g = _GRAD.pack(dy.data_ptr(), dx.data_ptr(), *grads, *[base + plan[n] if n in plan else 0 for n in _WORK], nblk)
        _native.check(_native.entry("bmt_llama_block_backward", "bbp")(self._describe(0, scratch), g, scratch.stream), "Llama block backward")
        return dx
