"""Packing of dense attention masks at the edges of the 128 x 128 tiles and 32 x 32 bit blocks, for rows of 16-byte pieces and others,
against the same packing by numpy."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _words(m, tiles):
    """(rows, columns) of 0/1 -> (rows, tiles * 4) words of 32 columns, the lowest bit first."""
    full = np.zeros((m.shape[0], tiles * 128), np.uint8)
    full[:, :m.shape[1]] = m
    return np.packbits(full, axis=1, bitorder="little").view("<u4")


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("b,sq,sk", [(1, 1, 1), (2, 31, 33), (1, 128, 128), (2, 129, 144), (1, 127, 256), (3, 200, 131), (1, 1, 400), (1, 300, 16)])
def test_packing(bmt_gpu, b, sq, sk, shift):
    from bmtrain_b200.ops import _native, attention

    gen = torch.Generator().manual_seed(sq * 1000 + sk)
    m = (torch.rand(b, sq, sk, generator=gen) < 0.5).to(torch.uint8) * torch.randint(1, 256, (b, sq, sk), generator=gen).to(torch.uint8)
    m[0, :128] = 1                                       # a tile that is full as far as it goes
    m[-1, 128:, :128] = 0                                # and one that is empty
    held = torch.zeros(m.numel() + 16, dtype=torch.uint8, device="cuda")
    held[shift:shift + m.numel()] = m.flatten().cuda()
    size = attention.packed_mask_bytes(b, sq, sk)
    packed = torch.full((size + 16,), 0xa5, dtype=torch.uint8, device="cuda")
    i64 = ctypes.c_int64
    _native.check(_native.cuda_lib().bmt_attn_mask_pack(i64(b), i64(sq), i64(sk), ctypes.c_void_p(held.data_ptr() + shift), _native.ptr(packed),
                                                        _native.stream_handle()), "mask packing")
    got, qt, kt = packed.cpu().numpy(), -(-sq // 128), -(-sk // 128)
    on = (m != 0).numpy()
    want = np.concatenate([_words(x, kt).ravel() for x in on] + [_words(x.T, qt).ravel() for x in on]).view(np.uint8)
    cls = [0 if not t.any() else 2 if t.all() else 1 for x in on for i in range(qt) for t in
           [x[i * 128:(i + 1) * 128, j * 128:(j + 1) * 128] for j in range(kt)]]
    assert (got[:len(want)] == want).all()
    assert (got[len(want):len(want) + len(cls)] == np.array(cls, np.uint8)).all()
    assert (got[size:] == 0xa5).all()
