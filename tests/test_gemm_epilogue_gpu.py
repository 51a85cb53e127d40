"""Epilogue forms of the tcgen05 GEMM (bias, activation, residual, gradient mask, accumulation, output type) at tile edges,
odd widths and unaligned pitches, against float64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

_DT = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}


def _gelu_grad(x):
    cdf = 0.5 * (1.0 + torch.erf(x * 0.5 ** 0.5))
    return cdf + x * torch.exp(-0.5 * x * x) * 0.3989422804014327


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 8, 64, 8), (127, 136, 72, 136), (129, 40, 64, 48), (257, 520, 200, 520), (300, 97, 64, 104),
                                   (130, 264, 64, 267), (777, 1000, 64, 1000)])
@pytest.mark.parametrize("form", ["plain", "bias_relu", "bias_gelu", "residual", "relu_mask", "gelu_mask", "accumulate", "float_out",
                                  "residual_accumulate"])
def test_epilogue_forms(bmt_gpu, dtype, shape, form):
    from bmtrain_b200.ops import _native
    from bmtrain_b200.parallel.fused_ops import _GemmDesc

    m, n, k, ldc = shape                       # ldc > n: the output is a view with a pitch; 267: no 16-byte rows
    gen = torch.Generator(device="cuda").manual_seed(m * 31 + n)
    rand = lambda *s, dt=dtype: torch.randn(*s, generator=gen, device="cuda").to(dt)  # noqa: E731
    a, b = rand(m, k), rand(n, k)
    out_dt = torch.float32 if form == "float_out" else dtype
    store = rand(m, ldc, dt=out_dt)
    before = store.clone()
    bias, extra = rand(n), rand(m, n)
    g = _GemmDesc()
    g.m, g.n, g.k = m, n, k
    g.a, g.lda, g.b, g.ldb = a.data_ptr(), k, b.data_ptr(), k
    g.c, g.ldc, g.c_dtype, g.ab_dtype, g.alpha = store.data_ptr(), ldc, _DT[out_dt], _DT[dtype], 0.5
    g.batch_inner = g.batch_outer = g.b_inner_div = 1
    ref = 0.5 * (a.double() @ b.double().t())
    old, e = before[:, :n].double(), extra.double()
    if form.startswith("bias"):
        g.bias, g.act = bias.data_ptr(), 1 if form == "bias_relu" else 2
        ref = ref + bias.double()
        ref = ref.relu() if form == "bias_relu" else torch.nn.functional.gelu(ref)
    if "mask" in form:
        g.aux, g.ld_aux, g.aux_mode = extra.data_ptr(), n, 1 if form == "relu_mask" else 2
        ref = ref * ((e > 0) if form == "relu_mask" else _gelu_grad(e))
    if form.startswith("residual"):
        g.residual, g.ldr = extra.data_ptr(), n
        ref = ref + e
    if form.endswith("accumulate"):
        g.accumulate = 1
        ref = ref + old
    lib = _native.cuda_lib()
    _native.check(lib.bmt_gemm_ex(ctypes.byref(g), _native.stream_handle()), "gemm")
    got = store[:, :n].double()
    # one rounding to the output type, plus fp32 sums of k products of magnitude ~1 and the fp32 erf / exp of the epilogue
    unit = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}[out_dt]
    bound = unit * ref.abs() + (k + 8) * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t() + e.abs() + 1.0) + 1e-7
    assert (got - ref).abs().le(bound).all(), float(((got - ref).abs() - bound).max())
    assert torch.equal(store[:, n:], before[:, n:])      # columns behind the matrix are left alone
    assert lib.bmt_gemm_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,ldc", [(264, 264), (267, 272)])      # the compiled forms and the general one
@pytest.mark.parametrize("form", ["plain", "bias", "bias_relu", "bias_gelu", "residual", "relu_mask", "gelu_mask", "accumulate", "float_out"])
def test_epilogue_keeps_nan_and_inf(bmt_gpu, dtype, n, ldc, form):
    """A product that is not a number, or infinite, arrives as such in every form (a ReLU maps NaN to zero, as fmaxf does)."""
    from bmtrain_b200.ops import _native
    from bmtrain_b200.parallel.fused_ops import _GemmDesc

    m, k = 130, 64
    a, b = torch.ones(m, k, device="cuda", dtype=dtype), torch.ones(n, k, device="cuda", dtype=dtype)
    bad = {3: float("nan"), 64: float("inf"), 129: float("-inf")}
    for row, value in bad.items():
        a[row, 5] = value
    out_dt = torch.float32 if form == "float_out" else dtype
    store = torch.ones(m, ldc, device="cuda", dtype=out_dt)
    ones, bias = torch.ones(m, n, device="cuda", dtype=dtype), torch.ones(n, device="cuda", dtype=dtype)
    g = _GemmDesc()
    g.m, g.n, g.k = m, n, k
    g.a, g.lda, g.b, g.ldb = a.data_ptr(), k, b.data_ptr(), k
    g.c, g.ldc, g.c_dtype, g.ab_dtype, g.alpha = store.data_ptr(), ldc, _DT[out_dt], _DT[dtype], 1.0
    g.batch_inner = g.batch_outer = g.b_inner_div = 1
    if form.startswith("bias"):
        g.bias, g.act = bias.data_ptr(), {"bias": 0, "bias_relu": 1, "bias_gelu": 2}[form]
    if "mask" in form:
        g.aux, g.ld_aux, g.aux_mode = ones.data_ptr(), n, 1 if form == "relu_mask" else 2
    if form == "residual":
        g.residual, g.ldr = ones.data_ptr(), n
    if form == "accumulate":
        g.accumulate = 1
    lib = _native.cuda_lib()
    _native.check(lib.bmt_gemm_ex(ctypes.byref(g), _native.stream_handle()), "gemm")
    got = store[:, :n].float()
    finite = torch.ones(m, dtype=torch.bool, device="cuda")
    finite[list(bad)] = False
    assert torch.isfinite(got[finite]).all()
    if form == "bias_relu":
        assert not got[3].any() and not got[129].any()
    else:
        assert torch.isnan(got[3]).all()
        if form == "bias_gelu":
            assert not torch.isposinf(got[129]).any()        # -inf * 0 or -0, as the formula gives it
        else:
            assert torch.isneginf(got[129]).all()
    assert torch.isposinf(got[64]).all()
    assert lib.bmt_gemm_status() == 0
