"""Whole pre-LN GPT block as one autograd node on the native block executor (``csrc/block_exec.cu``).

Each direction is one C++ call that issues all of the block's launches; what a pass keeps for backward, and what backward
scratches, is one allocation each, divided by a plan of the sizes.  All contractions run on the tcgen05 GEMM with fused
epilogues (bias, ReLU, residual add, ReLU-mask on dgrad) or in the fused attention kernels.  The big weight gradients are
written straight into the parameter's slot of the ZeRO block's gradient buffer, or into ``param.grad`` when a gradient of the
right dtype is already attached, which removes the separate accumulate pass.
"""
from __future__ import annotations

import ctypes
import functools
import os
import struct
from typing import Optional

import torch

from . import _native
from . import attention as _attn
from . import gemm as _gemm
from . import grad_slot as _grad_slot


_c_void_p, _i64, _int, _f32 = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int, ctypes.c_float


class _Block(ctypes.Structure):
    _fields_ = [
        ("batch", _i64), ("seq", _i64), ("d_model", _i64), ("n_heads", _i64), ("d_head", _i64), ("d_ff", _i64),
        ("dtype", _int), ("act", _int), ("eps", _f32), ("causal", _int), ("mask", _c_void_p),
        ("ln1_w", _c_void_p), ("ln1_b", _c_void_p), ("qkv_w", _c_void_p), ("qkv_b", _c_void_p), ("out_w", _c_void_p),
        ("out_b", _c_void_p), ("ln2_w", _c_void_p), ("ln2_b", _c_void_p), ("fc1_w", _c_void_p), ("fc1_b", _c_void_p),
        ("fc2_w", _c_void_p), ("fc2_b", _c_void_p),
        ("x", _c_void_p), ("y", _c_void_p),
        ("ln1", _c_void_p), ("stats1", _c_void_p), ("qkv", _c_void_p), ("probs", _c_void_p), ("probs_ld", _i64),
        ("ctx", _c_void_p), ("h1", _c_void_p), ("ln2", _c_void_p), ("stats2", _c_void_p), ("ff", _c_void_p), ("pre", _c_void_p),
        ("lse", _c_void_p), ("mask_packed", _c_void_p),
        ("colsum_scratch", _c_void_p), ("colsum_scratch_bytes", _i64), ("gemm_scratch", _c_void_p), ("gemm_scratch_bytes", _i64),
    ]


class _Grad(ctypes.Structure):
    _fields_ = [
        ("dy", _c_void_p), ("dx", _c_void_p),
        ("d_ln1_w", _c_void_p), ("d_ln1_b", _c_void_p), ("d_qkv_w", _c_void_p), ("d_qkv_b", _c_void_p),
        ("d_out_w", _c_void_p), ("d_out_b", _c_void_p), ("d_ln2_w", _c_void_p), ("d_ln2_b", _c_void_p),
        ("d_fc1_w", _c_void_p), ("d_fc1_b", _c_void_p), ("d_fc2_w", _c_void_p), ("d_fc2_b", _c_void_p),
        ("acc_w", _int),
        ("d_ff", _c_void_p), ("d_ln2", _c_void_p), ("d_h1", _c_void_p), ("d_ctx", _c_void_p), ("d_probs", _c_void_p),
        ("d_qkv", _c_void_p), ("norm_partial", _c_void_p), ("nblk", _int),
        ("dq_acc", _c_void_p), ("delta", _c_void_p),
        ("acc_small", _int), ("norm_partial2", _c_void_p),
    ]


# The same in one go: packing the block costs the host 2 us, filling the structure field by field 12.
_BLOCK = struct.Struct("@6q2ifi15Q4Qq8QQqQq")
_GRAD = struct.Struct("@14Qi4x7Qi4x2Qi4xQ")
assert _BLOCK.size == ctypes.sizeof(_Block) and _GRAD.size == ctypes.sizeof(_Grad)
_WORK = ("d_ff", "d_ln2", "d_h1", "d_ctx", "d_probs", "d_qkv", "norm_partial")


_PARAM_NAMES = ("ln1_w", "ln1_b", "qkv_w", "qkv_b", "out_w", "out_b", "ln2_w", "ln2_b", "fc1_w", "fc1_b", "fc2_w", "fc2_b")
_WEIGHTS = ("qkv_w", "out_w", "fc1_w", "fc2_w")
_SMALL = tuple(n for n in _PARAM_NAMES if n not in _WEIGHTS)


def _as_bytes(mask: torch.Tensor) -> torch.Tensor:
    """A boolean mask as bytes without a conversion pass (bool tensors are stored as one 0/1 byte per element)."""
    if mask.dtype == torch.bool:
        return mask.contiguous().view(torch.uint8)
    return mask.to(torch.uint8).contiguous()


def _carve(sizes):
    """Offsets of buffers of the given byte sizes inside one allocation (256-byte aligned), and its size.  One allocation per
    pass: at 1024 tokens the host is what bounds a block, and twenty tensors cost it 40 us a block."""
    offsets, at = {}, 0
    for name, n in sizes:
        offsets[name] = at
        at += (n + 255) // 256 * 256
    return offsets, at


@functools.lru_cache(maxsize=256)
def _saved_plan(b, s, d, n_heads, d_head, dff, gelu, fused_attn, masked):
    """What forward keeps for backward (16-bit activations, fp32 statistics)."""
    T, hd = b * s, n_heads * d_head
    sizes = [("ln1", 2 * T * d), ("stats1", 8 * T), ("qkv", 6 * T * hd), ("ctx", 2 * T * hd), ("h1", 2 * T * d), ("ln2", 2 * T * d),
             ("stats2", 8 * T), ("ff", 2 * T * dff)]
    if fused_attn:
        sizes.append(("lse", 4 * b * n_heads * s))
        if masked:
            sizes.append(("mask_packed", _attn.packed_mask_bytes(b, s, s)))
    else:
        sizes.append(("probs", 2 * b * n_heads * s * ((s + 7) // 8 * 8)))
    if gelu:
        sizes.append(("pre", 2 * T * dff))
    return _carve(sizes)


@functools.lru_cache(maxsize=256)
def _work_plan(b, s, d, n_heads, d_head, dff, fused_attn, nblk):
    """Scratch of a backward pass."""
    T, hd = b * s, n_heads * d_head
    sizes = [("d_ff", 2 * T * dff), ("d_ln2", 2 * T * d), ("d_h1", 2 * T * d), ("d_ctx", 2 * T * hd), ("d_qkv", 6 * T * hd),
             ("norm_partial", 8 * nblk * d), ("norm_partial2", 8 * nblk * d)]
    if fused_attn:
        sizes += [("dq_acc", 4 * T * hd), ("delta", 4 * b * n_heads * s)]
    else:
        sizes.append(("d_probs", 2 * b * n_heads * s * ((s + 7) // 8 * 8)))
    return _carve(sizes)


class Pass:
    """One forward (or recomputation) of a block by the native executor and what backward needs of it.  ``addresses``: of the parameters,
    in the order of ``_PARAM_NAMES``."""

    def __init__(self, x, mask, addresses, n_heads, d_head, d_ff, act, eps, causal):
        b, s, d = self.shape = x.shape
        self.x = x
        self.mask8 = None if mask is None else _as_bytes(mask)
        self.fused_attn = d_head % 16 == 0 and d_head <= 128 and os.environ.get("BMT_FLASH_ATTN", "1") != "0"
        self.cfg = (n_heads, d_head, d_ff)
        self.plan, total = _saved_plan(b, s, d, n_heads, d_head, d_ff, act == "gelu", self.fused_attn, self.mask8 is not None)
        self.saved = torch.empty(total, dtype=torch.uint8, device=x.device)
        base = self.saved.data_ptr()
        at = {name: base + offset for name, offset in self.plan.items()}
        self.scratch = _gemm.scratch()
        self.addresses = addresses
        self.head = (b, s, d, n_heads, d_head, d_ff, 0 if x.dtype == torch.float16 else 1, 1 if act == "relu" else 2, eps, 1 if causal else 0,
                     0 if self.mask8 is None else self.mask8.data_ptr())
        get = at.get
        # fused attention: scores and probabilities never reach memory, one log-sum-exp per row is kept instead
        self.tail = (at["ln1"], at["stats1"], at["qkv"], get("probs", 0), (s + 7) // 8 * 8 if "probs" in at else 0, at["ctx"], at["h1"], at["ln2"],
                     at["stats2"], at["ff"], get("pre", 0), get("lse", 0), get("mask_packed", 0),
                     0, 0, *self.scratch.gemm)         # forward adds no columns

    def forward(self) -> torch.Tensor:
        y = torch.empty_like(self.x)
        self.run(1, 9, y)
        return y

    def recompute(self) -> None:
        """Forward again for ``backward``: without the last GEMM, whose result nothing reads."""
        self.run(1, 8)

    def describe(self, y: int = 0) -> bytes:
        return _BLOCK.pack(*self.head, *self.addresses, self.x.data_ptr(), y, *self.tail)

    def run(self, first: int, last: int, y: Optional[torch.Tensor] = None) -> None:
        """Steps of the forward (``bmt_gpt_block_forward_steps``); the last one, 9, is what computes ``y``."""
        _native.check(_native.entry("bmt_gpt_block_forward_steps", "biip")(self.describe(0 if y is None else y.data_ptr()), first, last,
                                                                           self.scratch.stream), "GPT block forward")

    def backward(self, dy: torch.Tensor, grads, acc_weights: bool = False, acc_small: bool = False) -> torch.Tensor:
        """``grads``: addresses for the gradients of the parameters, in their order; ``acc_*``: added to what is there."""
        b, s, d = self.shape
        nblk = min(b * s, 296)
        plan, total = _work_plan(b, s, d, *self.cfg, self.fused_attn, nblk)
        work = torch.empty(total, dtype=torch.uint8, device=dy.device)
        base = work.data_ptr()
        at = lambda name: base + plan[name] if name in plan else 0  # noqa: E731
        dx = torch.empty_like(self.x)
        g = _GRAD.pack(dy.data_ptr(), dx.data_ptr(), *grads, 1 if acc_weights else 0, *[at(n) for n in _WORK], nblk, at("dq_acc"), at("delta"),
                       1 if acc_small else 0, at("norm_partial2"))
        scratch = _gemm.scratch()               # the forward may have been on another stream
        self.tail = self.tail[:-4] + (*scratch.colsum, *scratch.gemm)
        _native.check(_native.entry("bmt_gpt_block_backward", "bbp")(self.describe(), g, scratch.stream), "GPT block backward")
        return dx




class GPTBlockFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, mask, n_heads, d_head, act, eps, causal, deferred, *params):
        x = x.contiguous()
        b, s, d = x.shape
        run = Pass(x, mask, [p.data_ptr() for p in params], n_heads, d_head, params[8].shape[0], act, eps, causal)
        y = torch.empty_like(x)
        if deferred is None:
            run.run(1, 9, y)
        else:
            # the block's parameters are still on their way: norms and biases first; the QKV weight is gathered by the GEMM
            # that consumes it; the other big weights travel on the peer stream and have the attention core's duration to
            # arrive before the output projection.  They start together with the GEMM ("before") or when it is done
            # ("after", so that the QKV weight has the links to itself): BMT_REST_PUSH, default by group size.
            from ..parallel import fused_ops

            T, hd = b * s, n_heads * d_head
            plan, saved = run.plan, run.saved
            ln1 = saved[plan["ln1"]:plan["ln1"] + 2 * T * d].view(x.dtype).view(T, d)
            qkv = saved[plan["qkv"]:plan["qkv"] + 6 * T * hd].view(x.dtype).view(T, 3 * hd)

            cur = torch.cuda.current_stream()
            cur.wait_event(deferred["ev_small"])
            run.run(1, 1, y)
            when = os.environ.get("BMT_REST_PUSH") or ("before" if deferred["bucket"].comm.size <= 2 else "after")
            if when == "before":
                ev_rest = deferred["push_rest"]()
                fused_ops.zero_gather_gemm(ln1, qkv, params[3], deferred)
            else:
                fused_ops.zero_gather_gemm(ln1, qkv, params[3], deferred)
                ev_gemm = torch.cuda.Event()
                ev_gemm.record(cur)
                ev_rest = deferred["push_rest"](ev_gemm)
            run.run(3, 5, y)
            cur.wait_event(ev_rest)
            run.run(6, 9, y)
        ctx.run, ctx.params = run, params
        return y

    @staticmethod
    def backward(ctx, dy):
        run, params = ctx.run, ctx.params
        dt = run.x.dtype
        dy = dy.contiguous()
        run.addresses = [p.data_ptr() for p in params]

        # gradients of the parameters go straight into the owning block's gradient buffer, or accumulate in place when the
        # owner attached same-dtype gradient buffers (no tensor goes back to autograd for them then)
        def attached(p):
            return (p.is_leaf and p.requires_grad and p.grad is not None and p.grad.dtype == dt and p.grad.is_contiguous()
                    and not _grad_slot.watched(p))

        grads, where, acc = {}, {}, {}
        for names in (_WEIGHTS, _SMALL):
            mine = [(name, p) for name, p in zip(_PARAM_NAMES, params) if name in names]
            slots = [_grad_slot.find(p) if p.dtype == dt else None for _, p in mine]
            if all(s is not None for s in slots) and len({s.written for s in slots}) == 1:
                # the owning ZeRO block's gradient buffer: written on first use, added to afterwards
                acc[names] = slots[0].written
                for (name, _), slot in zip(mine, slots):
                    where[name] = slot.grad_ptr()
                    slot.written = True
                continue
            acc[names] = all(attached(p) for _, p in mine)
            for name, p in mine:
                if not acc[names]:
                    grads[name] = torch.empty_like(p)
                where[name] = (p.grad if acc[names] else grads[name]).data_ptr()
        dx = run.backward(dy, [where[n] for n in _PARAM_NAMES], acc[_WEIGHTS], acc[_SMALL])
        ctx.run = None
        out = [grads.get(name) if p.requires_grad else None for name, p in zip(_PARAM_NAMES, params)]
        return (dx, None, None, None, None, None, None, None) + tuple(out)


def gpt_block(x: torch.Tensor, mask: Optional[torch.Tensor], n_heads: int, d_head: int, act: str, eps: float, causal: bool,
              ln1_w, ln1_b, qkv_w, qkv_b, out_w, out_b, ln2_w, ln2_b, fc1_w, fc1_b, fc2_w, fc2_b, deferred=None) -> torch.Tensor:
    """``x`` (batch, seq, d_model) -> same shape.  ``mask``: optional bool (batch, seq, seq), True = attend.
    ``deferred``: gather-in-progress description from the owning ZeRO block (see ``Block._try_deferred_gather``)."""
    return GPTBlockFunction.apply(x, mask, n_heads, d_head, act, eps, causal, deferred, ln1_w, ln1_b, qkv_w, qkv_b, out_w, out_b,
                                  ln2_w, ln2_b, fc1_w, fc1_b, fc2_w, fc2_b)
