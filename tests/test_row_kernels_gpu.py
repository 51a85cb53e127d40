"""Row kernels at the edges of their work splits, against float64: norm backward (every team width, ragged lanes, fewer rows
than CTAs), the reduced cross-entropy, the embedding gradient (ids that repeat up to and beyond the hot-row limit)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

_UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,d", [(1, 8), (3, 256), (37, 264), (700, 512), (5, 520), (33, 768), (9, 776), (64, 1536), (300, 1544),
                                    (17, 2048), (1000, 2560), (2, 3072), (11, 4104), (600, 5120), (7, 6152), (149, 8192), (5, 8200),
                                    (3, 12288), (150, 12296), (4, 16384)])
def test_norm_backward(bmt_gpu, dtype, rms, rows, d):
    from bmtrain_b200.ops import _native
    from bmtrain_b200.ops import norm as N

    gen = torch.Generator(device="cuda").manual_seed(rows + d)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    x, dy = (2 * rand(rows, d) + 0.5).to(dtype), rand(rows, d).to(dtype)
    w, b = (1 + 0.2 * rand(d)).to(dtype), (0.2 * rand(d)).to(dtype)
    leaves = [t.clone().requires_grad_() for t in ((x, w) if rms else (x, w, b))]
    y = N.rms_norm(*leaves, 1e-5) if rms else N.layer_norm(*leaves, 1e-5)
    got = torch.autograd.grad(y, leaves, dy)
    assert _native.cuda_lib().bmt_norm_status() == 0
    exact = [t.double().requires_grad_() for t in ((x, w) if rms else (x, w, b))]
    if rms:
        ref = exact[0] * torch.rsqrt(exact[0].square().mean(-1, keepdim=True) + 1e-5) * exact[1]
    else:
        ref = torch.nn.functional.layer_norm(exact[0], (d,), exact[1], exact[2], 1e-5)
    want = torch.autograd.grad(ref, exact, dy.double())
    for name, a, e in zip(("dx", "dw", "db"), got, want):
        # one rounding of the result; fp32 inside (sums over a row or a column: relative 1e-5 of the norm)
        assert (a.double() - e).norm() <= (_UNIT[dtype] + 2e-5) * e.norm() + 1e-6, (name, float((a.double() - e).norm() / e.norm()))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,classes", [(1, 8), (3, 1000), (1023, 33), (1025, 2048), (130, 32003), (2049, 4096), (8192, 16), (8193, 16),
                                          (9217, 9), (151553, 8), (200000, 24)])       # from 8193 rows on several blocks
@pytest.mark.parametrize("reduction", ["mean", "sum"])
def test_reduced_cross_entropy(bmt_gpu, dtype, rows, classes, reduction):
    gen = torch.Generator(device="cuda").manual_seed(rows + classes)
    x = (2 * torch.randn(rows, classes, generator=gen, device="cuda")).to(dtype).requires_grad_()
    t = torch.randint(0, classes, (rows,), generator=gen, device="cuda")
    t[1::5] = -100
    loss = bmt_gpu.loss.FusedCrossEntropy(ignore_index=-100, reduction=reduction)(x, t)
    assert loss.dtype == torch.float32 and loss.dim() == 0
    (gx,) = torch.autograd.grad(loss * 64.0, (x,))
    xe = x.detach().double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(xe, t, ignore_index=-100, reduction=reduction)
    (ge,) = torch.autograd.grad(ref * 64.0, (xe,))
    assert abs(float(loss) - float(ref)) <= 3e-6 * abs(float(ref)) + 1e-6
    # half types: one rounding, gradients below the smallest normal fp16 number lose bits
    bound = 1.5 * _UNIT[dtype] * ge.norm() + (3e-8 * ge.numel() ** 0.5 if dtype == torch.float16 else 0) + 3e-6 * ge.norm()
    assert (gx.double() - ge).norm() <= bound


def test_reduced_cross_entropy_without_rows(bmt_gpu):
    x = torch.randn(4, 64, device="cuda", dtype=torch.float16, requires_grad=True)
    t = torch.full((4,), -100, device="cuda")
    loss = bmt_gpu.loss.FusedCrossEntropy()(x, t)
    assert torch.isnan(loss)
    (g,) = torch.autograd.grad(loss, (x,))
    assert not g.any()
    assert float(bmt_gpu.loss.FusedCrossEntropy(reduction="sum")(x, t)) == 0.0
    empty = torch.empty(0, 64, device="cuda", dtype=torch.float16)
    assert torch.isnan(bmt_gpu.loss.FusedCrossEntropy()(empty, t[:0]))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,rows,d", [(1, 1, 8), (65, 3, 8), (64, 1, 264), (700, 5, 2056), (2000, 4099, 512), (129, 70000, 64), (5000, 300, 96)])
def test_embedding_gradient(bmt_gpu, dtype, tokens, rows, d):
    from bmtrain_b200.ops import embedding as E

    gen = torch.Generator(device="cuda").manual_seed(tokens + rows)
    ids = torch.randint(0, rows, (tokens,), generator=gen, device="cuda")
    ids[torch.rand(tokens, generator=gen, device="cuda") < 0.1] = -1        # not in this shard
    if tokens > 1000:
        ids[:tokens // 3] = rows - 1                                        # one row far above the hot-row limit
    g = torch.randn(tokens, d, generator=gen, device="cuda").to(dtype)
    got = E.embedding_backward(ids, g, rows)
    keep = ids >= 0
    want = torch.zeros(rows, d, dtype=torch.float64, device="cuda").index_add_(0, ids[keep], g[keep].double())
    size = torch.zeros(rows, d, dtype=torch.float64, device="cuda").index_add_(0, ids[keep], g[keep].double().abs())
    assert got.dtype == dtype
    assert (got.double() - want).abs().le(_UNIT[dtype] * want.abs() + tokens * 2.0 ** -24 * size + 1e-7).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("classes", [33, 1000, 2047, 4096, 12289, 12296])       # odd and even, scalar, vector and streaming rows
@pytest.mark.parametrize("hide", ["inf", "lowest"])
def test_cross_entropy_of_hidden_classes(bmt_gpu, dtype, classes, hide):
    """Classes hidden with -inf or with the lowest number of the type: the first ones, the last ones, all but one, a thread's whole first trip, everything a thread
    sees; and rows with a NaN, which must not come out finite."""
    gen = torch.Generator(device="cuda").manual_seed(classes)
    x = torch.randn(8, classes, generator=gen, device="cuda").to(dtype)
    inf = float("inf") if hide == "inf" else torch.finfo(dtype).max
    x[0, :9] = -inf
    x[1, -9:] = -inf
    x[2, :] = -inf
    x[2, classes // 2] = 1.0
    x[3, : min(classes - 1, 8 * 256 * 4 + 5)] = -inf
    x[4, (torch.arange(classes, device="cuda") // 8) % 3 != 1] = -inf
    x[5, classes - 1] = float("nan")
    x[6, 0] = float("nan")
    t = torch.full((8,), classes - 1, device="cuda")
    t[1], t[2], t[4] = classes // 2, classes // 2, 9
    x = x.requires_grad_()
    loss = bmt_gpu.loss.FusedCrossEntropy(reduction="none")(x, t)
    (gx,) = torch.autograd.grad(loss, (x,), torch.ones_like(loss))
    xe = x.detach().double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(xe, t, reduction="none")
    (ge,) = torch.autograd.grad(ref, (xe,), torch.ones_like(ref))
    good = [0, 1, 2, 3, 4, 7]
    assert torch.isnan(loss[[5, 6]]).all()
    assert (loss[good].double() - ref[good]).abs().le(3e-6 * ref[good].abs() + 2e-6).all()
    assert (gx[good].double() - ge[good]).abs().le(1.5 * _UNIT[dtype] * ge[good].abs() + 2e-6 + (6e-8 if dtype == torch.float16 else 0)).all()
    assert torch.isnan(gx[[5, 6]]).any(1).all()


@pytest.mark.parametrize("classes", [33, 1024, 5001])
@pytest.mark.parametrize("level", [0.0, 14.0, 65.0, 700.0])
def test_cross_entropy_is_exact_near_the_target(bmt_gpu, classes, level):
    """fp32 logits around ``level``, one class far above the others.  The exponent is x - lse up to one rounding of that
    difference and the 1.3e-8 that the fp32 log2(e) is off; each 2^x is good to 2 ulp (4 units), each product to one unit."""
    from bmtrain_b200.ops import cross_entropy as C

    gen = torch.Generator(device="cuda").manual_seed(classes)
    x = torch.randn(64, classes, generator=gen, device="cuda") * 3 + level
    t = torch.randint(0, classes, (64,), generator=gen, device="cuda")
    x[torch.arange(32), t[:32]] = level + 30.0
    lse = torch.logsumexp(x.double(), 1).float()
    g = torch.rand(64, generator=gen, device="cuda") + 0.5
    got = C.ce_backward(x, t, lse, g, ignore_index=-100)
    gap = x.double() - lse.double()[:, None]
    p = gap.exp()
    want = (p - torch.nn.functional.one_hot(t, classes)) * g.double()[:, None]
    unit = 2.0 ** -24
    bound = g[:, None] * p * (10 * unit + 2 * unit * gap.abs()) + unit * want.abs() + 1e-37
    assert (got.double() - want).abs().le(bound).all(), float(((got.double() - want).abs() - bound).max())
    mx, se, _ = C.row_stats(x, t)
    top = x.double().max(1).values
    exact = (x.double() - top[:, None]).exp().sum(1)
    assert torch.equal(mx.double(), top)
    assert (se.double() - exact).abs().le((16 + classes / 256 + 8) * unit * exact).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("classes", [7, 100, 1001, 4096])
@pytest.mark.parametrize("reduction", ["mean", "none"])
def test_ignored_rows_get_no_gradient(bmt_gpu, dtype, classes, reduction):
    """... whatever their logits are."""
    x = torch.randn(5, classes, device="cuda").to(dtype)
    x[1, 3], x[2, classes - 1], x[3] = float("nan"), float("inf"), float("-inf")
    t = torch.tensor([0, -100, -100, -100, classes - 1], device="cuda")
    x = x.requires_grad_()
    loss = bmt_gpu.loss.FusedCrossEntropy(ignore_index=-100, reduction=reduction)(x, t)
    (g,) = torch.autograd.grad(loss, (x,), torch.ones_like(loss))
    assert torch.equal(g[1:4], torch.zeros_like(g[1:4]))
    assert torch.isfinite(g).all() and g[0].any() and g[4].any()
