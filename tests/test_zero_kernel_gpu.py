"""Zeroing a list of gradients: slices off the 16-byte boundary, the edges of a chunk (1024 vectors), empty tensors, more than one launch,
what the kernel does not take, and the version counters that autograd checks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32, torch.float64])
def test_zeros_and_nothing_else(bmt_gpu, dtype):
    from bmtrain_b200.ops import infnan

    sizes = [1, 7, 8, 9, 0, 8191, 8192, 8193, 40001] * 4
    held = [torch.ones(n + 24, device="cuda", dtype=dtype) for n in sizes]
    starts = [(5 * i) % 12 for i in range(len(sizes))]
    views = [h[s:s + n] for h, s, n in zip(held, starts, sizes)]
    infnan.multi_zero(views)
    for h, s, n in zip(held, starts, sizes):
        assert not h[s:s + n].any() and bool((h[:s] == 1).all()) and bool((h[s + n:] == 1).all())
    odd = torch.ones(6, 4, device="cuda", dtype=dtype)
    infnan.multi_zero([odd[:, ::2]])
    assert odd.sum() == 12


def test_versions(bmt_gpu):
    from bmtrain_b200.ops import infnan

    x = torch.ones(64, device="cuda", requires_grad=True)
    saved = torch.full((64,), 2.0, device="cuda")
    y = (x * saved).sum()
    infnan.multi_zero([saved])
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()
