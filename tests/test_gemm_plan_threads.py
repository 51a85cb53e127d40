"""Planning a GEMM changes nothing that launches of other threads read."""
import ctypes
import threading

import pytest
import torch


@pytest.mark.skipif(torch.cuda.is_available(), reason="looks at what is remembered of a device where there is none")
def test_planning_in_several_threads():
    from bmtrain_b200.ops import _native

    lib = _native.cuda_lib()
    i64 = ctypes.c_int64

    def plans():
        out, items = (ctypes.c_int64 * 6)(), (ctypes.c_int * (5 * 4096))()
        for n in range(300):
            assert lib.bmt_gemm_plan(i64(1024 + n), i64(2560), i64(8192), 0, 0, out, items, 4096) >= 0

    for _ in range(10):
        threads = [threading.Thread(target=plans) for _ in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    # the number of CTAs of a launch is not known without a device, and planning has not made it known
    assert lib.bmt_gemm_rs_grid(i64(1024), i64(2560), i64(2560), 0) == -1
