"""GELU and its derivative in 32 bits, for every 16-bit argument, against 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _arguments():
    """All fp16 values of magnitude 2^-10 to 5, eight to a row."""
    x = torch.arange(-2 ** 15, 2 ** 15, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.float16)
    x = x[(x.abs() >= 2.0 ** -10) & (x.abs() <= 5)]
    return x[:x.numel() // 8 * 8].view(-1, 8)


def test_gelu_in_32_bits(bmt_gpu):
    from bmtrain_b200.ops import gemm

    x = _arguments()
    got = gemm.gemm_nt(x, torch.eye(8, dtype=x.dtype, device="cuda"), act="gelu", out_dtype=torch.float32).double()
    d = x.double()
    phi = 0.5 * torch.special.erfc(-d * 0.5 ** 0.5)
    # |x| < 1.3: Phi is 1/2 + x P.  P (< 1/2) is good to one rounding of 2^-26 and two of its small terms of 2^-28, and the sum is rounded: 2^-25
    # above 1/2, 2^-26 below; then the product, 2^-24.  Beyond: the exponential's unit 2^-22 and q's error, the exponent's roundings, which grow
    # with u^2, and 1 - Phi
    absolute = d.abs() * 2.0 ** -25 + torch.where(d > 0, 2.0 ** -25, 2.0 ** -26)
    near = absolute / phi + 2.0 ** -24 + 1e-8
    far = torch.where(d > 0, 2.0 ** -23, 6e-7 + 2.0 ** -23 * d * d)
    bound = torch.where(d.abs() < 1.3, near, far)
    error = (got / (d * phi) - 1).abs()
    assert error.le(bound).all(), float((error - bound).max())


def test_gelu_gradient_in_32_bits(bmt_gpu):
    from bmtrain_b200.ops import _native
    from bmtrain_b200.parallel.fused_ops import _GemmDesc

    x = _arguments()
    ones = torch.ones_like(x)
    ones[:, 1:] = 0
    b = ones[:8].contiguous()
    out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
    g = _GemmDesc()
    g.m, g.n, g.k = x.shape[0], 8, 8
    g.a, g.lda, g.b, g.ldb = ones.data_ptr(), 8, b.data_ptr(), 8
    g.c, g.ldc, g.c_dtype, g.ab_dtype, g.alpha = out.data_ptr(), 8, 2, 0, 1.0
    g.batch_inner = g.batch_outer = g.b_inner_div = 1
    g.aux, g.ld_aux, g.aux_mode = x.data_ptr(), 8, 2
    _native.check(_native.cuda_lib().bmt_gemm_ex(ctypes.byref(g), _native.stream_handle()), "gemm")
    d = x.double()
    density = 0.3989422804014327 * torch.exp(-0.5 * d * d)
    ref = 0.5 * torch.special.erfc(-d * 0.5 ** 0.5) + d * density
    # Phi as above; x phi(x): an exponential of unit 2^-22 and three roundings, of a value below 0.25; the sum, below 1.13
    bound = d.abs().clamp(max=1.3) * 2.0 ** -25 + 2.0 ** -25 + (d * density).abs() * (2.0 ** -22 + 3 * 2.0 ** -24) + ref.abs() * 2.0 ** -24
    error = (out.double() - ref).abs()
    assert error.le(bound).all(), float((error - bound).max())
