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


@pytest.mark.parametrize("b,sq,sk", [(1, 1, 1), (2, 127, 129), (3, 437, 437), (1, 2048, 300)])
def test_mask_layout(lib, b, sq, sk):
    """The Python side asks the library; the parts hold a bit per query and padded key, per key and padded query, and a byte per
    tile, and start on 16-byte boundaries where they are read as vectors."""
    from bmtrain_b200.ops import attention as A

    size, by_key, classes = A.packed_mask_layout(b, sq, sk)
    qt, kt = -(-sq // 128), -(-sk // 128)
    assert (by_key, classes, size) == (b * sq * kt * 16, b * 16 * (sq * kt + sk * qt), b * (16 * (sq * kt + sk * qt) + qt * kt))
    assert A.packed_mask_bytes(b, sq, sk) == size and by_key % 16 == 0


def test_embedding_scratch(lib):
    """total and number of hot rows, count and start per row, the hot rows (above 64 tokens each), rank and order per token."""
    lib.bmt_embedding_bwd_scratch.restype = ctypes.c_int64
    for tokens, rows in ((1, 1), (63, 5), (64, 5), (6400, 50304)):
        need = 2 + 2 * rows + tokens // 65 + 2 * tokens
        assert need <= lib.bmt_embedding_bwd_scratch(ctypes.c_int64(tokens), ctypes.c_int64(rows)) <= need + tokens // 64 + 1
