"""GEMMs at sizes whose tiles are divided along K, in every epilogue form and operand layout: pairs of CTAs and single ones, with and without
whole tiles before the divided ones, ragged edges, CTAs that both leave sums and add others'.  Against float64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

_DT = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}
_UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}


def _plan(m, n, k, b_major):
    """(CTAs per tile, tiles, divided tiles, whether a CTA both leaves sums and adds others')"""
    from bmtrain_b200.ops import _native

    lib, i64 = _native.cuda_lib(), ctypes.c_int64
    plan, items, both = (ctypes.c_int64 * 6)(), (ctypes.c_int * (5 * 4096))(), False
    ask = lambda worker: lib.bmt_gemm_plan(i64(m), i64(n), i64(k), b_major, worker, plan, items, 4096)  # noqa: E731
    assert ask(0) >= 0
    for worker in range(plan[5]):
        kinds = [items[5 * i + 3] for i in range(ask(worker))]
        both |= 1 in kinds and 2 in kinds
    return plan[1], plan[2], plan[3], both


# m, n, k, layout of B, CTAs per tile, whole tiles before the divided ones, CTAs with both kinds
SIZES = [(1024, 2560, 8192, 1, 2, False, True), (4096, 4096, 16384, 0, 2, True, True), (2100, 4200, 4104, 1, 2, True, True),
         (256, 256, 10240, 0, 1, False, False), (56, 720, 9144, 0, 1, False, True), (300, 520, 8200, 1, 1, False, True),
         (129, 1000, 12000, 0, 2, False, True), (33, 72, 20000, 1, 1, False, False), (777, 2504, 9000, 1, 2, False, True)]
FORMS = ["plain", "bias", "bias_relu", "bias_gelu", "residual", "residual_rounded", "relu_mask", "gelu_mask", "accumulate", "float_out",
         "residual_accumulate", "odd_pitch"]


def _gelu_grad(x):
    return 0.5 * torch.special.erfc(-x * 0.5 ** 0.5) + x * torch.exp(-0.5 * x * x) * 0.3989422804014327


def test_sizes_are_divided(bmt_gpu):
    for m, n, k, b_major, ctas, behind, both in SIZES:
        plan = _plan(m, n, k, b_major)
        assert plan[0] == ctas and plan[2] > 0 and (plan[1] > plan[2]) == behind and plan[3] == both, (m, n, k, b_major, plan)


_operands = {}


def _inputs(m, n, k, dtype):
    """Kept from one form to the next: (A, B, their product in 64 bits, the product of their magnitudes)."""
    key = (m, n, k, dtype)
    if key not in _operands:
        _operands.clear()
        gen = torch.Generator(device="cuda").manual_seed(m + 3 * n + k)
        a, b = (torch.randn(rows, k, generator=gen, device="cuda").to(dtype) for rows in (m, n))
        _operands[key] = a, b, a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    return _operands[key]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s[:4])))
def test_forms(bmt_gpu, size, dtype):
    from bmtrain_b200.ops import _native
    from bmtrain_b200.ops import gemm as G
    from bmtrain_b200.parallel.fused_ops import _GemmDesc

    m, n, k, b_major = size[:4]
    lib = _native.cuda_lib()
    a, b, product, magnitude = _inputs(m, n, k, dtype)
    gen = torch.Generator(device="cuda").manual_seed(k)
    rand = lambda *s, dt=dtype: torch.randn(*s, generator=gen, device="cuda").to(dt)  # noqa: E731
    stored = b if b_major == 0 else b.t().contiguous()
    for form in FORMS:
        out_dt = torch.float32 if form == "float_out" else dtype
        ldc = n + 3 if form == "odd_pitch" else n
        store = rand(m, ldc, dt=out_dt)
        before = store.clone()
        bias, extra = rand(n), rand(m, n)
        g = _GemmDesc()
        g.m, g.n, g.k = m, n, k
        g.a, g.lda, g.b, g.ldb, g.b_major = a.data_ptr(), k, stored.data_ptr(), stored.stride(0), b_major
        alpha = 2.0 ** -6                     # results of magnitude about 1
        g.c, g.ldc, g.c_dtype, g.ab_dtype, g.alpha = store.data_ptr(), ldc, _DT[out_dt], _DT[dtype], alpha
        g.batch_inner = g.batch_outer = g.b_inner_div = 1
        g.scratch, g.scratch_bytes = G.scratch().gemm
        ref, old, e = alpha * product, before[:, :n].double(), extra.double()
        if form.startswith("bias"):
            g.bias, g.act = bias.data_ptr(), {"bias": 0, "bias_relu": 1, "bias_gelu": 2}[form]
            ref = ref + bias.double()
            ref = ref.relu() if form == "bias_relu" else torch.nn.functional.gelu(ref) if form == "bias_gelu" else ref
        grow = 1.0
        if "mask" in form:
            g.aux, g.ld_aux, g.aux_mode = extra.data_ptr(), n, 1 if form == "relu_mask" else 2
            ref = ref * ((e > 0) if form == "relu_mask" else _gelu_grad(e))
            grow = 1.13                       # largest derivative
        inner = ref.abs()
        if form.startswith("residual"):
            g.residual, g.ldr, g.round_first = extra.data_ptr(), n, 1 if form == "residual_rounded" else 0
            ref = ref + e
        if form.endswith("accumulate"):
            g.accumulate = 1
            ref = ref + old
        _native.check(lib.bmt_gemm_ex(ctypes.byref(g), _native.stream_handle()), "gemm")
        # one rounding to the output type (two where the product is rounded by itself), and fp32 sums of k products
        bound = _UNIT[out_dt] * (ref.abs() + (inner if form == "residual_rounded" else 0)) + 1e-6
        bound += 4 * 2.0 ** -24 * grow * (alpha * k ** 0.5 * magnitude + e.abs() + old.abs() + 1.0)
        error = (store[:, :n].double() - ref).abs()
        assert error.le(bound).all(), (form, float((error - bound).max()))
        assert torch.equal(store[:, n:], before[:, n:])
        again = before.clone()
        g.c = again.data_ptr()
        _native.check(lib.bmt_gemm_ex(ctypes.byref(g), _native.stream_handle()), "gemm")
        assert torch.equal(again, store), form                       # the sums are added in a fixed order
    assert lib.bmt_gemm_status() == 0


def test_back_to_back_on_several_streams(bmt_gpu):
    """Launches of different tile widths that share a stream's flags and slots, on several streams at the same time."""
    from bmtrain_b200.ops import _native
    from bmtrain_b200.ops import gemm as G

    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").half()  # noqa: E731
    sizes = [s[:4] for s in SIZES if s[0] < 2000]
    work = [(rand(m, k), rand(n, k) if b_major == 0 else rand(k, n), b_major) for m, n, k, b_major in sizes]
    call = lambda w: (G.gemm_nn if w[2] else G.gemm_nt)(*w[:2])  # noqa: E731
    want = [call(w) for w in work]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    got = []
    for i in range(6 * len(work)):
        for j, s in enumerate(streams):
            with torch.cuda.stream(s):
                at = (i + 2 * j) % len(work)
                got.append((at, call(work[at])))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i]) for i, y in got)
    assert _native.cuda_lib().bmt_gemm_status() == 0
