"""What the C entry points refuse and the sizes they ask for; nothing here launches a kernel."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    from bmtrain_b200.ops import _native

    return _native.cuda_lib()


def test_block_refuses_half_a_mask(lib):
    from bmtrain_b200.ops.gpt_block import _Block, _Grad

    for with_mask in (True, False):
        blk, grad = _Block(), _Grad()
        blk.batch, blk.seq, blk.d_model, blk.n_heads, blk.d_head, blk.d_ff = 1, 8, 16, 1, 16, 16
        blk.lse = 256                                            # selects the fused attention; never read
        setattr(blk, "mask" if with_mask else "mask_packed", 256)
        for first, last in ((1, 9), (3, 3)):
            assert lib.bmt_gpt_block_forward_steps(ctypes.byref(blk), first, last, None) == -40
        assert lib.bmt_gpt_block_backward(ctypes.byref(blk), ctypes.byref(grad), None) == -40
