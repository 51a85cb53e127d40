"""Column sums of several matrices in one launch, at the edges of its 32 columns and 64 (fp32: 32) row lanes, on both sides of the
line beyond which a matrix goes to the kernel that splits the rows, against float64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

_UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


class _Item(ctypes.Structure):
    _fields_ = [("x", ctypes.c_void_p), ("m", ctypes.c_int64), ("n", ctypes.c_int64), ("out", ctypes.c_void_p), ("f32", ctypes.c_int),
                ("first", ctypes.c_int)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("shapes", [[(1, 8)], [(0, 24), (63, 40), (65, 32)], [(512, 8), (513, 72), (296, 264, "f"), (1, 8, "f"), (33, 40, "f")],
                                    [(2048, 264), (2049, 264), (300, 64, "f"), (2047, 1000)]])
def test_column_sums(bmt_gpu, dtype, add, shapes):
    from bmtrain_b200.ops import _native, gemm

    gen = torch.Generator(device="cuda").manual_seed(7)
    xs = [torch.randn(s[0], s[1], generator=gen, device="cuda").to(torch.float32 if len(s) > 2 else dtype) for s in shapes]
    outs = [torch.randn(s[1], generator=gen, device="cuda").to(dtype) for s in shapes]
    had = [o.double() if add else torch.zeros_like(o, dtype=torch.double) for o in outs]
    items = (_Item * len(xs))(*[_Item(x.data_ptr(), x.shape[0], x.shape[1], o.data_ptr(), int(x.dtype == torch.float32), 0)
                                for x, o in zip(xs, outs)])
    work = gemm.scratch()
    _native.check(_native.cuda_lib().bmt_colsum_multi(items, ctypes.c_int(len(xs)), ctypes.c_int(0 if dtype == torch.float16 else 1),
                                                      ctypes.c_int(add), ctypes.c_void_p(work.colsum[0]), ctypes.c_int64(work.colsum[1]),
                                                      _native.stream_handle()), "column sums")
    for x, o, h in zip(xs, outs, had):
        want = x.double().sum(0) + h
        # at most ~100 additions in fp32 follow one another, then one rounding
        assert ((o.double() - want).abs() <= _UNIT[dtype] * want.abs() + 100 * 2.0 ** -24 * (x.double().abs().sum(0) + h.abs()) + 1e-7).all()


def test_items_that_are_refused(bmt_gpu):
    from bmtrain_b200.ops import _native

    call = _native.cuda_lib().bmt_colsum_multi
    one = (_Item * 1)(_Item(0, 4, 12, 0, 0, 0))         # 12 columns: not a multiple of 8
    rest = (ctypes.c_int(0), ctypes.c_void_p(0), ctypes.c_int64(0), _native.stream_handle())
    assert call(one, ctypes.c_int(1), ctypes.c_int(1), *rest) == -3
    assert call(one, ctypes.c_int(1), ctypes.c_int(2), *rest) == -3
    assert call(one, ctypes.c_int(13), ctypes.c_int(1), *rest) == -3
