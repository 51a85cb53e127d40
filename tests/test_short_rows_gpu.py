"""Norms and lookups of short rows on both sides of the number of blocks from which they are launched normally."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,d", [(32768, 64), (32769, 64), (40003, 256), (32772, 8)])
@pytest.mark.parametrize("rms", [True, False])
def test_norm_rows(bmt_gpu, dtype, rows, d, rms):
    from bmtrain_b200.ops import norm

    gen = torch.Generator(device="cuda").manual_seed(rows + d)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)  # noqa: E731
    x, w, b = rand(rows, d), rand(d), rand(d)
    y = norm.rms_norm(x, w, 1e-5) if rms else norm.layer_norm(x, w, b, 1e-5)
    f = x.double()
    f = f if rms else f - f.mean(1, keepdim=True)
    exact = f * (f.square().mean(1, keepdim=True) + 1e-5).rsqrt() * w.double() + (0 if rms else b.double())
    unit = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    # one rounding of the result; fp32 statistics and three operations before it
    bound = unit * exact.abs() + 16 * 2.0 ** -24 * (f.abs().amax(1, keepdim=True) + 1) * (w.double().abs() + b.double().abs() + 1) * d ** 0.5 + 1e-6
    assert ((y.double() - exact).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,d", [(4096, 64), (4097, 64), (5000, 512), (5000, 1024), (5000, 1032)])
def test_lookups(bmt_gpu, dtype, tokens, d):
    from bmtrain_b200.ops import embedding

    gen = torch.Generator(device="cuda").manual_seed(tokens + d)
    table = torch.randn(301, d, generator=gen, device="cuda").to(dtype)
    ids = torch.randint(0, 301, (tokens,), generator=gen, device="cuda")
    for _ in range(3):       # each next to the kernel that writes its table
        table = table * 1
        assert torch.equal(embedding.embedding_forward(ids, table), table[ids])
