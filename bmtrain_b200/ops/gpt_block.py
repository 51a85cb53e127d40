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
        ("acc_small", _int),
    ]


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
             ("norm_partial", 8 * nblk * d)]
    if fused_attn:
        sizes += [("dq_acc", 4 * T * hd), ("delta", 4 * b * n_heads * s)]
    else:
        sizes.append(("d_probs", 2 * b * n_heads * s * ((s + 7) // 8 * 8)))
    return _carve(sizes)


def _describe(x, y, mask, params, saved, plan, n_heads, d_head, act, eps, causal):
    """The block as the native executor takes it; ``saved``: address of the buffer that ``plan`` divides."""
    b, s, d = x.shape
    work = _gemm.scratch()
    at = lambda name: saved + plan[name] if name in plan else None  # noqa: E731
    # fused attention: scores and probabilities never reach memory, one log-sum-exp per row is kept instead
    return _Block(b, s, d, n_heads, d_head, params[8].shape[0], 0 if x.dtype == torch.float16 else 1, 1 if act == "relu" else 2, eps,
                  1 if causal else 0, None if mask is None else mask.data_ptr(), *[p.data_ptr() for p in params], x.data_ptr(),
                  y.data_ptr(), at("ln1"), at("stats1"), at("qkv"), at("probs"), (s + 7) // 8 * 8 if "probs" in plan else 0,
                  at("ctx"), at("h1"), at("ln2"), at("stats2"), at("ff"), at("pre"), at("lse"), at("mask_packed"),
                  *work.colsum, *work.gemm)


class GPTBlockFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, mask, n_heads, d_head, act, eps, causal, deferred, *params):
        lib = _native.cuda_lib()
        x = x.contiguous()
        b, s, d = x.shape
        dff = params[8].shape[0]
        mask8 = None if mask is None else _as_bytes(mask)
        fused_attn = d_head % 16 == 0 and d_head <= 128 and os.environ.get("BMT_FLASH_ATTN", "1") != "0"
        plan, total = _saved_plan(b, s, d, n_heads, d_head, dff, act == "gelu", fused_attn, mask8 is not None)
        saved = torch.empty(total, dtype=torch.uint8, device=x.device)
        y = torch.empty_like(x)
        blk = _describe(x, y, mask8, params, saved.data_ptr(), plan, n_heads, d_head, act, eps, causal)
        if deferred is None:
            _native.check(lib.bmt_gpt_block_forward(ctypes.byref(blk), _native.stream_handle()), "GPT block forward")
        else:
            # the block's parameters are still on their way: norms and biases first; the QKV weight is gathered by the GEMM
            # that consumes it; the other big weights travel on the peer stream and have the attention core's duration to
            # arrive before the output projection.  They start together with the GEMM ("before") or when it is done
            # ("after", so that the QKV weight has the links to itself): BMT_REST_PUSH, default by group size.
            from ..parallel import fused_ops

            T, hd = b * s, n_heads * d_head
            ln1 = saved[plan["ln1"]:plan["ln1"] + 2 * T * d].view(x.dtype).view(T, d)
            qkv = saved[plan["qkv"]:plan["qkv"] + 6 * T * hd].view(x.dtype).view(T, 3 * hd)

            cur = torch.cuda.current_stream()
            cur.wait_event(deferred["ev_small"])
            _native.check(lib.bmt_gpt_block_forward_steps(ctypes.byref(blk), 1, 1, _native.stream_handle()), "GPT block forward")
            when = os.environ.get("BMT_REST_PUSH") or ("before" if deferred["bucket"].comm.size <= 2 else "after")
            if when == "before":
                ev_rest = deferred["push_rest"]()
                fused_ops.zero_gather_gemm(ln1, qkv, params[3], deferred)
            else:
                fused_ops.zero_gather_gemm(ln1, qkv, params[3], deferred)
                ev_gemm = torch.cuda.Event()
                ev_gemm.record(cur)
                ev_rest = deferred["push_rest"](ev_gemm)
            _native.check(lib.bmt_gpt_block_forward_steps(ctypes.byref(blk), 3, 5, _native.stream_handle()), "GPT block forward")
            cur.wait_event(ev_rest)
            _native.check(lib.bmt_gpt_block_forward_steps(ctypes.byref(blk), 6, 9, _native.stream_handle()), "GPT block forward")
        ctx.saved, ctx.plan, ctx.x, ctx.mask8, ctx.params = saved, plan, x, mask8, params
        ctx.cfg = (n_heads, d_head, act, eps, causal, fused_attn)
        return y

    @staticmethod
    def backward(ctx, dy):
        lib = _native.cuda_lib()
        x, saved, params = ctx.x, ctx.saved, ctx.params
        n_heads, d_head, act, eps, causal, fused_attn = ctx.cfg
        b, s, d = x.shape
        dev, dt = x.device, x.dtype
        dy = dy.contiguous()
        # (the forward output's pointer is not read by backward)
        blk = _describe(x, dy, ctx.mask8, params, saved.data_ptr(), ctx.plan, n_heads, d_head, act, eps, causal)
        g = _Grad()
        dx = torch.empty_like(x)
        g.dy, g.dx = dy.data_ptr(), dx.data_ptr()
        # gradients of the parameters go straight into the owning block's gradient buffer, or accumulate in place when the
        # owner attached same-dtype gradient buffers (no tensor goes back to autograd for them then)
        def attached(p):
            return (p.is_leaf and p.requires_grad and p.grad is not None and p.grad.dtype == dt and p.grad.is_contiguous()
                    and not _grad_slot.watched(p))

        grads = {}
        for names, flag in ((_WEIGHTS, "acc_w"), (_SMALL, "acc_small")):
            mine = [(name, p) for name, p in zip(_PARAM_NAMES, params) if name in names]
            slots = [_grad_slot.find(p) if p.dtype == dt else None for _, p in mine]
            if all(s is not None for s in slots) and len({s.written for s in slots}) == 1:
                # the owning ZeRO block's gradient buffer: written on first use, added to afterwards
                setattr(g, flag, 1 if slots[0].written else 0)
                for (name, _), slot in zip(mine, slots):
                    setattr(g, "d_" + name, slot.grad_ptr())
                    slot.written = True
                continue
            acc = all(attached(p) for _, p in mine)
            setattr(g, flag, 1 if acc else 0)
            for name, p in mine:
                if not acc:
                    grads[name] = torch.empty_like(p)
                setattr(g, "d_" + name, (p.grad if acc else grads[name]).data_ptr())
        nblk = min(b * s, 296)
        plan, total = _work_plan(b, s, d, n_heads, d_head, params[8].shape[0], fused_attn, nblk)
        work = torch.empty(total, dtype=torch.uint8, device=dev)
        base = work.data_ptr()
        for name, at in plan.items():
            setattr(g, name, base + at)
        g.nblk = nblk
        _native.check(lib.bmt_gpt_block_backward(ctypes.byref(blk), ctypes.byref(g), _native.stream_handle()), "GPT block backward")
        ctx.saved = None
        out = [grads.get(name) if p.requires_grad else None for name, p in zip(_PARAM_NAMES, params)]
        return (dx, None, None, None, None, None, None, None) + tuple(out)


def gpt_block(x: torch.Tensor, mask: Optional[torch.Tensor], n_heads: int, d_head: int, act: str, eps: float, causal: bool,
              ln1_w, ln1_b, qkv_w, qkv_b, out_w, out_b, ln2_w, ln2_b, fc1_w, fc1_b, fc2_w, fc2_b, deferred=None) -> torch.Tensor:
    """``x`` (batch, seq, d_model) -> same shape.  ``mask``: optional bool (batch, seq, seq), True = attend.
    ``deferred``: gather-in-progress description from the owning ZeRO block (see ``Block._try_deferred_gather``)."""
    return GPTBlockFunction.apply(x, mask, n_heads, d_head, act, eps, causal, deferred, ln1_w, ln1_b, qkv_w, qkv_b, out_w, out_b,
                                  ln2_w, ln2_b, fc1_w, fc1_b, fc2_w, fc2_b)
