"""Fused attention at the edges of its 128 x 128 tiles, with one and with two query tiles per CTA, every padded head dim, and
the packed form of dense masks (empty, full and mixed tiles), against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(q, k, v, scale, keep):
    g = q.shape[2] // k.shape[2]
    k, v = k.repeat_interleave(g, 2), v.repeat_interleave(g, 2)
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) * scale
    p = torch.nan_to_num(torch.softmax(s.masked_fill(~keep, float("-inf")), -1))
    return torch.einsum("bhqk,bkhd->bqhd", p, v)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("cfg", [
    # b, sq, sk, h, hk, d, masking; more than 148 (head, query tile) pairs take two tiles per CTA
    (1, 1, 1, 1, 1, 16, None), (1, 127, 129, 3, 1, 32, None), (2, 129, 257, 2, 2, 48, "lens"), (1, 255, 255, 80, 10, 64, "causal"),
    (2, 385, 385, 40, 40, 80, "blocks"), (1, 384, 640, 60, 12, 96, "causal"), (1, 300, 300, 4, 4, 112, "blocks"),
    (2, 257, 257, 64, 8, 128, "random"), (3, 130, 300, 40, 40, 128, "lens"), (1, 513, 200, 40, 8, 128, "causal")])
def test_tiles(bmt_gpu, dtype, cfg):
    from bmtrain_b200.ops import _native
    from bmtrain_b200.ops import attention as AT

    b, sq, sk, h, hk, d, masking = cfg
    gen = torch.Generator(device="cuda").manual_seed(sq + sk + d)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)  # noqa: E731
    q, k, v, do = rand(b, sq, h, d), rand(b, sk, hk, d), rand(b, sk, hk, d), rand(b, sq, h, d)
    keep = torch.ones(b, 1, sq, sk, dtype=torch.bool, device="cuda")
    mask = lens = None
    causal = masking == "causal"
    if causal:
        keep = keep & torch.ones(sq, sk, dtype=torch.bool, device="cuda").tril(sk - sq)
    elif masking == "lens":
        lens = torch.tensor([max(0, sk - 150 * i) for i in range(b)], device="cuda")
        keep = keep & (torch.arange(sk, device="cuda") < lens.view(b, 1, 1, 1))
    elif masking == "blocks":          # whole tiles hidden, whole tiles visible, the rest mixed, one row that sees nothing
        keep = keep & torch.ones(sq, sk, dtype=torch.bool, device="cuda").tril()
        keep[:, :, :, 128:256] &= (torch.arange(sq, device="cuda") >= 256).view(1, 1, sq, 1)
        keep[0, :, 5] = False
    elif masking == "random":
        keep = torch.rand(b, 1, sq, sk, generator=gen, device="cuda") > 0.4
        keep[:, :, 200:] = False
    if masking in ("blocks", "random"):
        mask = keep[:, 0]
        packed = AT.pack_mask(mask.to(torch.uint8), b, sq, sk)
        kt, qt = (sk + 127) // 128, (sq + 127) // 128
        words = packed[: b * sq * kt * 16].view(b, sq, kt * 16)
        bits = ((words[..., None] >> torch.arange(8, device="cuda", dtype=torch.uint8)) & 1).reshape(b, sq, kt * 128)
        assert torch.equal(bits[:, :, :sk].bool(), mask) and not bits[:, :, sk:].any()
        by_key = packed[b * sq * kt * 16: b * 16 * (sq * kt + sk * qt)].view(b, sk, qt * 16)
        bits_t = ((by_key[..., None] >> torch.arange(8, device="cuda", dtype=torch.uint8)) & 1).reshape(b, sk, qt * 128)
        assert torch.equal(bits_t[:, :, :sq].bool(), mask.transpose(1, 2)) and not bits_t[:, :, sq:].any()
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    o = AT.attention(*leaves, causal=causal, mask=mask, kv_lens=lens)
    got = [o, *torch.autograd.grad(o, leaves, do)]
    torch.cuda.synchronize()
    assert _native.cuda_lib().bmt_attn_status() == 0
    exact = [t.double().requires_grad_() for t in (q, k, v)]
    ref = _oracle(*exact, 1.0 / math.sqrt(d), keep)
    want = [ref, *torch.autograd.grad(ref, exact, do.double())]
    # probabilities, dS and results are rounded once each; 0.6 units of the type were seen
    tol = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    for name, a, w in zip(("o", "dq", "dk", "dv"), got, want):
        assert torch.isfinite(a).all(), name
        assert (a.double() - w).norm() <= tol * w.norm() + 1e-6, (name, float((a.double() - w).norm() / w.norm()))


@pytest.mark.parametrize("hk,masking", [(8, None), (2, None), (8, "mask"), (8, "lens")])
def test_forward_and_backward_under_capture(bmt_gpu, hk, masking):
    """Both directions are captured into a graph on addresses that they have not seen, and replay on new inputs."""
    from bmtrain_b200.ops import attention as AT

    gen = torch.Generator(device="cuda").manual_seed(hk)
    fresh = lambda h: torch.randn(2, 200, h, 64, generator=gen, device="cuda").half()  # noqa: E731
    q, k, v, do = (fresh(h) for h in (8, hk, hk, 8))
    mask = torch.rand(2, 200, 200, generator=gen, device="cuda") > 0.3 if masking == "mask" else None
    lens = torch.tensor([77, 200], device="cuda") if masking == "lens" else None
    for t in (q, k, v):
        t.requires_grad_()

    def run():
        o = AT.attention(q, k, v, mask=mask, kv_lens=lens)
        return [o.detach(), *torch.autograd.grad(o, (q, k, v), do)]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = run()
    with torch.no_grad():
        for t in (q, k, v, do):
            t.copy_(fresh(t.shape[2]))
    graph.replay()
    torch.cuda.synchronize()
    got = [t.clone() for t in got]
    for a, b in zip(got, run()):
        # dQ is added up in another order
        assert (a - b).float().norm() <= 1e-3 * b.float().norm()
