"""Norm forward at the edges of its teams: every number of warps a row and of vectors a lane, ragged rows, row counts that leave a block
with idle teams, a constant row, against float64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

_UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("dtype", list(_UNIT))
@pytest.mark.parametrize("rms,bias", [(True, False), (True, True), (False, True), (False, False)])
@pytest.mark.parametrize("rows,d", [(1, 8), (5, 256), (7, 264), (4, 520), (3, 1032), (9, 1280), (2, 1288), (3, 2048), (3, 2560), (2, 2568), (5, 4104), (3, 5120),
                                    (2, 5128), (3, 8200), (2, 11008), (2, 13000), (2, 16384)])
def test_norm_forward(bmt_gpu, dtype, rms, bias, rows, d):
    from bmtrain_b200.ops import _native

    gen = torch.Generator(device="cuda").manual_seed(rows * d)
    x = (2 * torch.randn(rows, d, generator=gen, device="cuda") + 0.5).to(dtype)
    x[0] = 3.0
    w, b = ((torch.randn(d, generator=gen, device="cuda") + 1).to(dtype) for _ in range(2))
    y, stats = torch.full((rows + 1, d), 9.0, dtype=dtype, device="cuda"), torch.empty(2, rows, device="cuda")
    i64, c = ctypes.c_int64, ctypes.c_int
    _native.check(_native.cuda_lib().bmt_norm_fwd(i64(rows), i64(d), _native.ptr(x), _native.ptr(w), _native.ptr(b) if bias else ctypes.c_void_p(0),
                                                  ctypes.c_float(1e-5), c(rms), c(0 if dtype == torch.float16 else 1), _native.ptr(y),
                                                  _native.ptr(stats), _native.stream_handle()), "norm")
    xd = x.double()
    mean = torch.zeros(rows, 1, device="cuda", dtype=torch.double) if rms else xd.mean(1, keepdim=True)
    rstd = ((xd - mean).square().mean(1, keepdim=True) + 1e-5).rsqrt()
    want = (xd - mean) * rstd * w.double() + (b.double() if bias else 0)
    # one rounding of the result; fp32 inside: the mean to 2^-22 of the row's size, which the constant row multiplies by 316
    slack = 1e-6 * ((xd - mean).abs() + xd.abs().amax(1, keepdim=True)) * rstd * w.double().abs() + 1e-6 * want.abs() + 1e-7
    assert ((y[:rows].double() - want).abs() <= _UNIT[dtype] * (want.abs() + slack) + slack).all()
    assert (y[rows] == 9).all()
    assert ((stats[0].double() - mean[:, 0]).abs() <= 1e-6 * xd.abs().amax(1)).all()
    assert ((stats[1].double() / rstd[:, 0] - 1).abs()[1:] <= 1e-5).all()
