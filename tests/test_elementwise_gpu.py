"""Gated activation, GELU and rotary embedding at the edges of their pieces (512 positions of 8 elements) and with odd row widths, against
float64; extreme arguments of the activations."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

_UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}
_DT = {torch.float16: 0, torch.bfloat16: 1}


def _gelu(x):
    from bmtrain_b200.ops import _native

    out = torch.empty_like(x)
    _native.check(_native.cuda_lib().bmt_gelu_fwd(ctypes.c_int64(x.numel()), _native.ptr(x), ctypes.c_int(_DT[x.dtype]), _native.ptr(out),
                                                  _native.stream_handle()), "gelu")
    return out


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,f", [(1, 8), (3, 16), (511, 8), (513, 8), (5, 4088), (2, 4104), (77, 328), (1, 70000)])
def test_swiglu(bmt_gpu, dtype, rows, f):
    from bmtrain_b200.ops import elementwise as E

    gen = torch.Generator(device="cuda").manual_seed(rows + f)
    x = (3 * torch.randn(rows, 2 * f, generator=gen, device="cuda")).to(dtype).requires_grad_()
    g = torch.randn(rows, f, generator=gen, device="cuda").to(dtype)
    y = E.swiglu(x)
    (dx,) = torch.autograd.grad(y, x, g)
    xd = x.detach().double().requires_grad_()
    yd = torch.nn.functional.silu(xd[:, :f]) * xd[:, f:]
    (dd,) = torch.autograd.grad(yd, xd, g.double())
    # one rounding, fp32 inside (a few 2^-22 of each factor; the gradient adds terms that may cancel)
    assert ((y.double() - yd).abs() <= _UNIT[dtype] * yd.abs() + 1e-6 * (1 + yd.abs())).all()
    assert ((dx.double() - dd).abs() <= _UNIT[dtype] * dd.abs() + 2e-6 * (1 + xd.abs().amax() * g.abs().amax())).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n", [8, 4088, 4096, 4104, 100008])
def test_gelu(bmt_gpu, dtype, n):
    x = torch.linspace(-12, 12, n, device="cuda").to(dtype)
    exact = 0.5 * x.double() * torch.special.erfc(x.double() * -0.5 ** 0.5)       # 1 + erf cancels on the negative side, in 64 bits too
    small = 2.0 ** -25 if dtype == torch.float16 else 1e-30          # half the smallest fp16 step
    assert ((_gelu(x).double() - exact).abs() <= (_UNIT[dtype] + 1e-5) * exact.abs() + small).all()


def test_extremes(bmt_gpu):
    from bmtrain_b200.ops import elementwise as E

    v = torch.tensor([0.0, -0.0, 60000.0, -60000.0, float("inf"), float("nan"), 3.4e38, -3.4e38], device="cuda")
    for dtype in (torch.float16, torch.bfloat16):
        x = v.to(dtype)
        got, want = _gelu(x).double(), torch.nn.functional.gelu(x.double())
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(0), want.to(dtype).double().nan_to_num(0))
        gate = torch.cat([x, torch.ones_like(x)])[None]
        got, want = E.swiglu(gate)[0].double(), torch.nn.functional.silu(x.double())
        assert torch.equal(got.isnan(), want.isnan())
        assert torch.allclose(got.nan_to_num(0), want.to(dtype).double().nan_to_num(0), rtol=2 * _UNIT[dtype], atol=1e-30)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,s,hk,g,d", [(1, 1, 1, 1, 16), (3, 1, 1, 1, 32), (2, 77, 3, 1, 80), (1, 200, 2, 4, 128), (40, 3, 1, 2, 64), (2, 129, 4, 1, 96)])
def test_rope(bmt_gpu, dtype, b, s, hk, g, d):
    from bmtrain_b200.ops import elementwise as E

    gen = torch.Generator(device="cuda").manual_seed(s + d)
    p = torch.randn(b, s, hk, g + 2, d, generator=gen, device="cuda").to(dtype).requires_grad_()
    q, k, v = E.rope_qkv(p, g)
    gr = [torch.randn(t.shape, generator=gen, device="cuda").to(dtype) for t in (q, k, v)]
    (dp,) = torch.autograd.grad([q, k, v], p, gr)
    cos, sin = (t.double() for t in E._rope_tables(s, d, 10000.0, p.device))

    def turn(x, sign):
        a, c = x[..., : d // 2], x[..., d // 2:]
        cc, ss = cos[None, :, None], sign * sin[None, :, None]
        return torch.cat([a * cc - c * ss, a * ss + c * cc], -1)

    pd = p.detach().double()
    for got, want in ((q, turn(pd[:, :, :, :g].reshape(b, s, hk * g, d), 1)), (k, turn(pd[:, :, :, g], 1)), (v, pd[:, :, :, g + 1])):
        assert ((got.double() - want).abs() <= _UNIT[dtype] * want.abs() + 1e-5).all()
    dq = turn(gr[0].double(), -1).view(b, s, hk, g, d)
    want = torch.cat([dq, turn(gr[1].double(), -1)[:, :, :, None], gr[2].double()[:, :, :, None]], 3)
    assert ((dp.double() - want).abs() <= _UNIT[dtype] * want.abs() + 1e-5).all()
