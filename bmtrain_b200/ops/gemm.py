"""Dense GEMMs of the transformer blocks.

Three operand layouts cover a linear layer (reference does all of them through
cuBLAS: ``bmtrain/nn/linear.py:10-24``):

* ``gemm_nt(a[M,K], b[N,K])``  -> ``a @ b.T``   forward  (x, W)
* ``gemm_nn(a[M,K], b[K,N])``  -> ``a @ b``     dgrad    (grad_out, W)
* ``gemm_tn(a[K,M], b[K,N])``  -> ``a.T @ b``   wgrad    (grad_out, x)

On a B200 all three run the hand-written tcgen05 kernel (``csrc/gemm_sm100.cu``:
TMA-fed shared-memory pipeline, accumulators in tensor memory, persistent tile
scheduler) with optional fused epilogues (bias add, GELU/ReLU, accumulate into
an existing tensor).  CPU tensors take the PyTorch definition.
"""
from __future__ import annotations

import ctypes
import os
import threading
from typing import Optional

import torch

from . import _native
from . import grad_slot as _grad_slot

ACT_NONE, ACT_RELU, ACT_GELU = 0, 1, 2
_ACT = {None: ACT_NONE, "none": ACT_NONE, "relu": ACT_RELU, "gelu": ACT_GELU}
_DT = {torch.float16: 0, torch.bfloat16: 1}

# operand major-ness as seen by the kernel: 0 = reduction dim contiguous, 1 = output dim contiguous
_K_MAJOR, _MN_MAJOR = 0, 1


def _apply_act(x: torch.Tensor, act) -> torch.Tensor:
    if act in (None, "none"):
        return x
    if act == "relu":
        return torch.relu(x)
    if act == "gelu":
        return torch.nn.functional.gelu(x)
    raise ValueError(act)


_OUT_DT = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}


def _launch(a, b, out, m, n, k, a_major, b_major, bias, act, accumulate, lda, ldb):
    dt = a.dtype
    assert dt == b.dtype and dt in _DT, "tensor-core GEMM takes fp16 or bf16 operands"
    work = scratch()
    status = _native.entry("bmt_gemm", "qqqpqipqipqipiiipqp")(
        m, n, k, a.data_ptr(), lda, a_major, b.data_ptr(), ldb, b_major, out.data_ptr(), out.stride(0), _OUT_DT[out.dtype],
        0 if bias is None else bias.data_ptr(), _ACT[act], 1 if accumulate else 0, _DT[dt], work.gemm[0], work.gemm[1], work.stream)
    if status != 0:
        _native.check(status, f"tcgen05 GEMM (m={m}, n={n}, k={k})")


def _use_torch(t: torch.Tensor) -> bool:
    return (not t.is_cuda) or os.environ.get("BMT_GEMM_DEBUG_TORCH", "0") == "1"


def _rowmajor(t: torch.Tensor) -> torch.Tensor:
    """A view TMA can read: unit inner stride, 16-byte aligned base and row pitch (pads a copy when needed)."""
    (rows, cols), (pitch, step) = t.shape, t.stride()
    if step == 1 and pitch >= cols and pitch % 8 == 0 and t.data_ptr() % 16 == 0:
        return t
    if cols % 8 == 0:
        return t.contiguous()
    padded = torch.zeros(rows, (cols + 7) // 8 * 8, dtype=t.dtype, device=t.device)
    padded[:, :cols].copy_(t)
    return padded[:, :cols]


def gemm_nt(a: torch.Tensor, b: torch.Tensor, bias: Optional[torch.Tensor] = None, act=None,
            out: Optional[torch.Tensor] = None, accumulate: bool = False, out_dtype=None) -> torch.Tensor:
    """``act(a @ b.T + bias)``; ``a`` (M, K), ``b`` (N, K), both with contiguous K."""
    m, k = a.shape
    n = b.shape[0]
    assert b.shape[1] == k
    if _use_torch(a):
        r = torch.matmul(a.float(), b.float().t()) if a.dtype != torch.float32 else torch.matmul(a, b.t())
        if bias is not None:
            r = r + bias.float()
        r = _apply_act(r, act)
        if out is not None:
            out.copy_(out.float() + r if accumulate else r)
            return out
        return r.to(out_dtype or a.dtype)
    a, b = _rowmajor(a), _rowmajor(b)
    if out is None:
        assert not accumulate
        out = torch.empty(m, n, dtype=out_dtype or a.dtype, device=a.device)
    _launch(a, b, out, m, n, k, _K_MAJOR, _K_MAJOR, bias, act, accumulate, a.stride(0), b.stride(0))
    return out


def gemm_nn(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None, accumulate: bool = False,
            out_dtype=None) -> torch.Tensor:
    """``a @ b``; ``a`` (M, K) with contiguous K, ``b`` (K, N) with contiguous N."""
    m, k = a.shape
    n = b.shape[1]
    assert b.shape[0] == k
    if _use_torch(a):
        r = torch.matmul(a.float(), b.float()) if a.dtype != torch.float32 else torch.matmul(a, b)
        if out is not None:
            out.copy_(out.float() + r if accumulate else r)
            return out
        return r.to(out_dtype or a.dtype)
    a, b = _rowmajor(a), _rowmajor(b)
    if out is None:
        assert not accumulate
        out = torch.empty(m, n, dtype=out_dtype or a.dtype, device=a.device)
    _launch(a, b, out, m, n, k, _K_MAJOR, _MN_MAJOR, None, None, accumulate, a.stride(0), b.stride(0))
    return out


def gemm_tn(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None, accumulate: bool = False,
            out_dtype=None) -> torch.Tensor:
    """``a.T @ b``; ``a`` (K, M) with contiguous M, ``b`` (K, N) with contiguous N."""
    k, m = a.shape
    n = b.shape[1]
    assert b.shape[0] == k
    if _use_torch(a):
        r = torch.matmul(a.float().t(), b.float()) if a.dtype != torch.float32 else torch.matmul(a.t(), b)
        if out is not None:
            out.copy_(out.float() + r if accumulate else r)
            return out
        return r.to(out_dtype or a.dtype)
    a, b = _rowmajor(a), _rowmajor(b)
    if out is None:
        assert not accumulate
        out = torch.empty(m, n, dtype=out_dtype or a.dtype, device=a.device)
    _launch(a, b, out, m, n, k, _MN_MAJOR, _MN_MAJOR, None, None, accumulate, a.stride(0), b.stride(0))
    return out


_COLSUM_BYTES = 4 * (1024 + 2 * 1024 * 1024)
_MOST_SCRATCH = 16
_scratch = {}                   # by device and stream, the one that was used last at the end
_scratch_order = threading.Lock()
_latest = (None, None)


class _Scratch:
    """Work space of the kernels that add partial sums, one per device and stream, zeroed once: the kernels leave counters and flags
    at zero, and launches that share it take turns on their stream.  The first part belongs to the column sums (4 KB of ticket
    counters and the sums), the second to the GEMMs that divide tiles over several CTAs: (address, bytes) each."""

    __slots__ = ("buf", "colsum", "gemm", "stream")

    def __init__(self, index, stream):
        lib = _native.cuda_lib()
        lib.bmt_gemm_scratch_bytes.restype = ctypes.c_int64
        size = lib.bmt_gemm_scratch_bytes()
        self.buf = torch.zeros(_COLSUM_BYTES + size, dtype=torch.uint8, device=torch.device("cuda", index))
        base = self.buf.data_ptr()
        self.colsum = (base, _COLSUM_BYTES)
        self.gemm = (base + _COLSUM_BYTES, size)
        self.stream = stream


class _CapturedScratch:
    """The same for one captured call: a graph may be replayed next to anything else, on any stream, so what its launches use belongs to it
    (to its memory pool), and they set the counters to zero themselves.  GEMMs do not divide tiles there."""

    __slots__ = ("buf", "index", "stream")
    gemm = (0, 0)

    def __init__(self, index, stream):
        self.buf, self.index, self.stream = None, index, stream

    @property
    def colsum(self):
        if self.buf is None:
            self.buf = torch.empty(_COLSUM_BYTES, dtype=torch.uint8, device=torch.device("cuda", self.index))
            self.buf[:4096].zero_()
        return self.buf.data_ptr(), _COLSUM_BYTES


def scratch():
    """The current stream's, or the captured call's own.  Streams beyond the last ``_MOST_SCRATCH`` that used one give theirs back: to the
    allocator, which hands it out again in the order of the same stream."""
    global _latest
    index = torch._C._cuda_getDevice()
    stream = torch._C._cuda_getCurrentRawStream(index)
    if torch._C._cuda_isCurrentStreamCapturing():
        return _CapturedScratch(index, stream)
    key, (last, got) = (index, stream), _latest
    if last == key:
        return got
    with _scratch_order:
        got = _scratch.pop(key, None)
        if got is None:
            if len(_scratch) >= _MOST_SCRATCH:
                del _scratch[next(iter(_scratch))]
            got = _Scratch(index, stream)
        _scratch[key] = got
        _latest = (key, got)
    return got


def bias_grad(grad_out: torch.Tensor) -> torch.Tensor:
    """Column sums of ``grad_out`` (M, N), accumulated in fp32, returned in the input dtype."""
    if not grad_out.is_cuda:
        return grad_out.float().sum(0).to(grad_out.dtype)
    g = grad_out.contiguous()
    m, n = g.shape
    out = torch.empty(n, dtype=g.dtype, device=g.device)
    work = scratch()
    _native.check(_native.entry("bmt_colsum_ex", "qqpipipqp")(m, n, g.data_ptr(), _OUT_DT[g.dtype], out.data_ptr(), 0, *work.colsum, work.stream),
                  "column-sum kernel")
    return out


class LinearFunction(torch.autograd.Function):
    """``y = act(x W^T + b)`` with explicit dgrad / wgrad / bgrad GEMMs (activation only when no grad through it is needed: ``act`` must be None for training)."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        ctx.save_for_backward(x, weight)
        ctx.has_bias = bias is not None
        if x.dim() == 2:
            return gemm_nt(x, weight, bias)
        y = gemm_nt(x.reshape(-1, x.shape[-1]), weight, bias)
        return y.view(*x.shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, grad_output):
        x, weight = ctx.saved_tensors
        g2 = grad_output if grad_output.dim() == 2 else grad_output.reshape(-1, grad_output.shape[-1])
        x2 = x if x.dim() == 2 else x.reshape(-1, x.shape[-1])
        grad_x = grad_w = grad_b = None
        if ctx.needs_input_grad[0]:
            grad_x = gemm_nn(g2, weight).view(x.shape)
        if ctx.needs_input_grad[1]:
            slot = _grad_slot.find(weight) if weight.dtype == g2.dtype else None
            if slot is None:
                grad_w = gemm_tn(g2, x2)
            else:
                gemm_tn(g2, x2, out=slot.grad_view(), accumulate=slot.written)
                slot.written = True
        if ctx.has_bias and ctx.needs_input_grad[2]:
            grad_b = bias_grad(g2)
        return grad_x, grad_w, grad_b


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Differentiable ``x @ weight.T + bias`` on the framework's GEMM kernels."""
    if x.dtype == torch.float32 and not x.is_cuda:
        return torch.nn.functional.linear(x, weight, bias)
    return LinearFunction.apply(x, weight, bias)
