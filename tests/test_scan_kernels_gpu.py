"""Overflow scan, sum of squares and scaling over lists of tensors: edges of the 16-byte vectors, of the chunks of 1024 and 2048 vectors and
of the list, slices that begin between two 16-byte boundaries."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 7, 8, 9, 4095, 4096, 4097, 8191, 8192, 8193, 16383, 16385, 50001]


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda", 0)


def _slices(dev, dtype, offset):
    g = torch.Generator(device="cuda").manual_seed(offset)
    bases = [torch.randn(n + offset, generator=g, device=dev).to(dtype) for n in SIZES]
    return [b[offset:] for b in bases], bases


@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_scans_and_scaling(dev, dtype, offset):
    from bmtrain_b200.ops import infnan

    ts, bases = _slices(dev, dtype, offset)
    before = [t.clone() for t in ts]
    heads = [b[:offset].clone() for b in bases]
    total = torch.zeros(1, device=dev)
    infnan.multi_sq_norm(ts, total)
    ref = sum(float(t.double().square().sum()) for t in ts)
    assert abs(float(total) - ref) <= 1e-5 * ref          # sums of positive fp32 terms, at most a few hundred deep
    coef = torch.tensor([0.37], device=dev)
    infnan.multi_scale(ts, coef)
    for t, b, h, base in zip(ts, before, heads, bases):
        assert torch.equal(t, (b.float() * coef).to(dtype))
        assert torch.equal(base[:offset], h)
    flag = torch.zeros(1, dtype=torch.uint8, device=dev)
    infnan.multi_has_inf_nan(ts, flag)
    assert int(flag) == 0
    for t in ts:
        for at, value in ((0, float("nan")), (t.numel() // 2, float("-inf")), (t.numel() - 1, float("inf"))):
            old = t[at].clone()
            t[at] = value
            flag.zero_()
            infnan.multi_has_inf_nan(ts, flag)
            assert int(flag) == 1, (t.numel(), at)
            t[at] = old


def test_more_tensors_than_a_table_and_empty_ones(dev):
    from bmtrain_b200.ops import infnan

    ts = [torch.full((i % 5,), float(i), dtype=torch.float16, device=dev) for i in range(61)]
    total = torch.zeros(1, device=dev)
    infnan.multi_sq_norm(ts, total)
    assert float(total) == float(sum((i % 5) * i * i for i in range(61)))
    infnan.multi_scale(ts, torch.tensor([0.5], device=dev))
    assert all(torch.equal(t, torch.full_like(t, i * 0.5)) for i, t in enumerate(ts))


def test_sum_of_squares_of_many_values_is_not_biased(bmt_gpu):
    """Some two thousand values of a thread: summed one by one the roundings of fp16 squares went one way."""
    from bmtrain_b200.ops import infnan

    off = []
    for seed in range(4):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        x = (3 * torch.randn(1 << 28, generator=gen, device="cuda", dtype=torch.float16))
        out = torch.zeros(1, device="cuda")
        infnan.multi_sq_norm([x], out)
        want = torch.stack([part.double().square().sum() for part in x.split(1 << 24)]).sum()
        off.append(float((out.double() - want) / want))
    # a block's sum is off by a few 2^-24, the 600 that are added to one another by half a unit each, at random: 12 * 2^-24
    assert abs(sum(off) / 4) <= 6e-7 and max(map(abs, off)) <= 1.5e-6
