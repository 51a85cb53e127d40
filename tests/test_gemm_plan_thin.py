"""Products of a few rows with an operand that L2 does not hold: whole tiles where they keep nearly all SMs reading, divided ones elsewhere."""
import ctypes

import pytest


@pytest.mark.parametrize("m,n,k,b_major,divided", [
    (88, 17944, 24864, 1, False), (24, 17752, 16256, 1, False), (96, 17944, 24864, 1, False),     # the rule
    (88, 17944, 24864, 0, True), (104, 17944, 24864, 1, True), (128, 17456, 16536, 1, True),      # the other layout, more rows
    (88, 8184, 19408, 1, True), (64, 17944, 3000, 1, False), (64, 3216, 20616, 1, True)])         # few tiles, an operand that fits, both
def test_thin_products(m, n, k, b_major, divided):
    from bmtrain_b200.ops import _native

    i64, plan, items = ctypes.c_int64, (ctypes.c_int64 * 6)(), (ctypes.c_int * (5 * 4096))()
    assert _native.cuda_lib().bmt_gemm_plan(i64(m), i64(n), i64(k), b_major, 0, plan, items, 4096) >= 0
    assert (plan[3] > 0) == divided, list(plan)
