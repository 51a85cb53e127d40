"""Maximum, sum and target logit of the rows of a cross entropy: every number of vectors a thread holds, full and ragged trips, rows that
start off a 16-byte boundary, classes that are hidden, against float64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

_DT = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}


@pytest.mark.parametrize("dtype", list(_DT))
@pytest.mark.parametrize("n", [1, 7, 8, 33, 1024, 2048, 2056, 4095, 6144, 8192, 8200, 10240, 10247, 16384, 20481, 30001])
def test_row_statistics(bmt_gpu, dtype, n):
    from bmtrain_b200.ops import _native

    m, start = 5, 3
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = (4 * torch.randn(m, n, generator=gen, device="cuda") + 9).to(dtype)
    x[1, 1::2] = torch.finfo(dtype).min
    x[2, : n // 2] = -float("inf")
    x[3] = -float("inf")
    target = torch.randint(0, n, (m,), generator=gen, device="cuda") + start
    target[4] = n + start                                # another rank's class
    out = torch.full((3, m), 7.0, device="cuda")
    i64 = ctypes.c_int64
    _native.check(_native.cuda_lib().bmt_ce_row_stats(i64(m), i64(n), _native.ptr(x), ctypes.c_int(_DT[dtype]), _native.ptr(target), i64(start),
                                                      _native.ptr(out), _native.stream_handle()), "row statistics")
    xd = x.double()
    most = xd.amax(1)
    total = torch.where(most[:, None] == -float("inf"), torch.zeros_like(xd), torch.exp(xd - most[:, None])).sum(1)
    assert (out[0].double() == most).all()
    # an FMA's rounding of an exponent below 2^8 (2^-16 of the sum in the worst row, relative to terms that large exponents make small),
    # ex2 to 2^-22, and the additions
    assert ((out[1].double() - total).abs() <= 1e-5 * total + 1e-30).all()
    assert out[1, 3] == 0
    want = x.float().gather(1, (target - start).clamp(max=n - 1)[:, None])[:, 0]
    want[4] = 0
    assert (out[2] == want).all()


def test_a_nan_is_not_lost(bmt_gpu):
    from bmtrain_b200.ops import _native

    i64 = ctypes.c_int64
    for n, at in ((10240, 0), (10240, 9999), (10007, 10006), (33, 32)):
        x = torch.zeros(2, n, device="cuda", dtype=torch.bfloat16)
        x[1, at] = float("nan")
        out = torch.zeros(3, 2, device="cuda")
        _native.check(_native.cuda_lib().bmt_ce_row_stats(i64(2), i64(n), _native.ptr(x), ctypes.c_int(1), _native.ptr(torch.zeros(2, dtype=torch.int64, device="cuda")),
                                                          i64(0), _native.ptr(out), _native.stream_handle()), "row statistics")
        assert out[1, 0] == n and out[1, 1].isnan()
