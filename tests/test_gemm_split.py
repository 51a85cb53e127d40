"""GEMMs whose tiles are divided along K over several CTAs: the division covers everything once (host arithmetic, no GPU), and
results against float64 at ragged sizes, in every operand layout and epilogue form, on several streams."""
import ctypes
import random

import pytest
import torch


def _plan(lib, m, n, k, b_major, worker):
    plan, items = (ctypes.c_int64 * 6)(), (ctypes.c_int * (5 * 4096))()
    i64 = ctypes.c_int64
    count = lib.bmt_gemm_plan(i64(m), i64(n), i64(k), ctypes.c_int(b_major), ctypes.c_int(worker), plan, items, ctypes.c_int(4096))
    assert count >= 0
    return list(plan), [tuple(items[5 * i:5 * i + 5]) for i in range(count)]


def test_division_covers_every_tile_once():
    from bmtrain_b200.ops import _native

    lib = _native.cuda_lib()
    rng, split = random.Random(3), 0
    sizes = [(1024, 2560, 8192), (1024, 2560, 2560), (777, 7680, 2560), (256, 256, 10240), (130, 64, 100000), (4096, 12288, 4096)]
    sizes += [tuple(int(2 ** rng.uniform(3, 14)) for _ in range(3)) for _ in range(60)]
    for m, n, k in sizes:
        for b_major in (0, 1):
            plan, _ = _plan(lib, m, n, k, b_major, 0)
            _, _, tiles, sk_tiles, sk_workers, grid = plan
            k_blocks = -(-k // 64)
            split += sk_tiles > 0
            assert sk_workers <= grid <= 148
            parts = {}
            for worker in range(grid):
                items = _plan(lib, m, n, k, b_major, worker)[1]
                assert sum(i[3] == 1 for i in items) <= 1 and sum(i[3] == 2 for i in items) <= 1      # one slot, one wait
                assert [i[3] for i in items] == sorted(i[3] for i in items)          # the storage of the pipeline is free at the end
                for tile, kb0, kb1, kind, first in items:
                    assert 0 <= tile < tiles and 0 <= kb0 < kb1 <= k_blocks
                    parts.setdefault(tile, []).append((worker, kb0, kb1, kind, first))
            assert sorted(parts) == list(range(tiles))
            for pieces in parts.values():
                pieces.sort(key=lambda x: x[1])
                assert pieces[0][1] == 0 and pieces[-1][2] == k_blocks
                assert all(a[2] == b[1] for a, b in zip(pieces, pieces[1:]))
                if len(pieces) == 1:
                    assert pieces[0][3] == 0
                else:       # the last one finishes the tile and waits for exactly the others, all of lower index
                    assert [x[3] for x in pieces] == [1] * (len(pieces) - 1) + [2]
                    assert [x[0] for x in pieces[:-1]] == list(range(pieces[-1][4], pieces[-1][0]))
    assert split > 20


SHAPES = [(1024, 2560, 2560), (777, 2560, 1288), (130, 520, 4096), (256, 256, 10240), (1311, 1000, 2560), (33, 72, 2048), (2100, 3000, 640)]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_against_float64(bmt_gpu, dtype, m, n, k):
    from bmtrain_b200.ops import _native
    from bmtrain_b200.ops import gemm as G

    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)  # noqa: E731
    a, b, bias = rand(m, k), rand(n, k), rand(n)
    exact = a.double() @ b.double().t()
    unit = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    # one rounding of the result and fp32 sums of k products
    bound = unit * (exact.abs() + bias.double().abs()) + 4 * 2.0 ** -24 * k ** 0.5 * (a.double().abs() @ b.double().abs().t()) + 1e-6
    y = G.gemm_nt(a, b, bias)
    assert ((y.double() - exact - bias.double()).abs() <= bound).all()
    assert torch.equal(G.gemm_nt(a, b, bias), y)                      # the sums are added in a fixed order
    if n % 8 == 0:
        assert ((G.gemm_nn(a, b.t().contiguous()).double() - exact).abs() <= bound).all()
    if n % 8 == 0 and m % 8 == 0:
        out = rand(m, n)
        old = out.double()
        G.gemm_tn(a.t().contiguous(), b.t().contiguous(), out=out, accumulate=True)
        assert ((out.double() - exact - old).abs() <= bound + unit * old.abs()).all()
    assert _native.cuda_lib().bmt_gemm_status() == 0


@pytest.mark.gpu
def test_streams_and_repeats(bmt_gpu):
    """Launches that share a stream's scratch, and launches of several streams at the same time."""
    from bmtrain_b200.ops import _native
    from bmtrain_b200.ops import gemm as G

    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").half()  # noqa: E731
    work = [(rand(m, k), rand(n, k)) for m, n, k in SHAPES]
    want = [G.gemm_nt(a, b) for a, b in work]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    got = []
    for i in range(30):
        for s in streams:
            with torch.cuda.stream(s):
                got.append((i % len(work), G.gemm_nt(*work[i % len(work)])))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i]) for i, y in got)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = G.gemm_nt(*work[0])
    graph.replay()
    torch.cuda.synchronize()
    assert (y.double() - want[0].double()).norm() <= 2.0 ** -11 * want[0].double().norm()
    assert _native.cuda_lib().bmt_gemm_status() == 0
