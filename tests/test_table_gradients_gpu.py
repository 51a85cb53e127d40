"""Gradients of stand-alone tables that are attached: added to in place by a backward pass, left to autograd wherever something could
see the difference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _table(bmt, rows=300, d=64, dtype=torch.float16):
    emb = bmt.nn.Embedding(rows, d, dtype=dtype)
    with torch.no_grad():
        emb.weight.normal_() if emb._parameters["weight"].dim() == 2 else emb._parameters["weight"].data.normal_()
    return emb, emb._parameters["weight"]


def _loss(emb, ids, x):
    return emb(ids).float().square().sum() * 1e-2 + emb(x, projection=True).float().sum() * 1e-2


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_added_in_place_and_to_what_is_there(bmt_gpu, dtype):
    emb, p = _table(bmt_gpu, dtype=dtype)
    gen = torch.Generator(device="cuda").manual_seed(1)
    ids = torch.randint(0, 300, (7, 31), generator=gen, device="cuda")
    ids[0, :] = 5                                       # one row with many tokens
    ids[1:4, :] = 9                                     # ... beyond the limit of the per-row teams
    x = torch.randn(40, 64, generator=gen, device="cuda").to(dtype)
    _loss(emb, ids, x).backward()                       # nothing attached: autograd's
    first = p.grad.clone()
    w, g = p.detach().view(300, 64).double(), torch.zeros(300, 64, dtype=torch.float64, device="cuda")
    look = (2e-2 * w[ids.view(-1)].float()).to(dtype).double()
    g.index_add_(0, ids.view(-1), look)
    exact = (g + 1e-2 * x.double().sum(0)).view(-1)
    unit = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    # roundings of the loss gradient and of the two contributions, and of their sum
    bound = lambda k: 8 * k * unit * exact.norm()  # noqa: E731
    assert (first.double() - exact).norm() <= bound(1)
    held = p.grad
    held.zero_()
    _loss(emb, ids, x).backward()
    assert p.grad is held and (held.double() - exact).norm() <= bound(1)
    _loss(emb, ids, x).backward()
    assert p.grad is held and (held.double() - 2 * exact).norm() <= bound(2)
    untouched = torch.ones(300, dtype=torch.bool, device="cuda")
    untouched[ids.view(-1)] = False
    held.zero_()
    emb(ids).float().sum().backward()
    assert (held.view(300, 64)[untouched] == 0).all() and (held.view(300, 64)[~untouched] != 0).all()


def test_left_to_autograd(bmt_gpu):
    emb, p = _table(bmt_gpu)
    ids, x = torch.randint(0, 300, (50,), device="cuda"), torch.randn(8, 64, device="cuda").half()
    _loss(emb, ids, x).backward()
    want = p.grad.clone()
    held = p.grad
    held.zero_()
    (g,) = torch.autograd.grad(_loss(emb, ids, x), [p])                # asks for the gradient: nothing may be added to .grad
    assert torch.equal(g, want) and (held == 0).all()
    other = torch.zeros(64, device="cuda", dtype=torch.float16, requires_grad=True)
    (_loss(emb, ids, x) + (emb(ids) * other).sum()).backward(inputs=[other])
    assert (held == 0).all() and other.grad is not None
    seen = []
    handle = p.register_hook(lambda t: seen.append(t.clone()))
    _loss(emb, ids, x).backward()
    handle.remove()
    assert len(seen) == 1 and torch.equal(seen[0], want) and torch.equal(held, want)
    held.zero_()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _loss(emb, ids, x).backward()
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(held, want)
    held.zero_()
    _loss(emb, ids, x).backward(retain_graph=False)
    assert (held.double() - want.double()).norm() <= 2.0 ** -9 * want.double().norm()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_same_bits_with_and_without_zeros_attached(bmt_gpu, dtype):
    """A tied table: the first pass, which leaves the gradient to autograd, and passes that add to zeros in place."""
    emb, p = _table(bmt_gpu, dtype=dtype)
    gen = torch.Generator(device="cuda").manual_seed(3)
    perm = lambda: torch.randperm(300, generator=gen, device="cuda")  # noqa: E731
    ids = torch.cat([perm(), perm()[:107]])             # one or two tokens a row: their order does not matter
    x = torch.randn(40, 64, generator=gen, device="cuda").to(dtype)
    _loss(emb, ids, x).backward()
    first, held = p.grad.clone(), p.grad
    for _ in range(2):
        held.zero_()
        _loss(emb, ids, x).backward()
        assert p.grad is held and torch.equal(held, first)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_sums_are_rounded_before_they_are_added(bmt_gpu, dtype):
    from bmtrain_b200.ops import embedding as E

    gen = torch.Generator(device="cuda").manual_seed(4)
    ids = torch.randint(0, 300, (500,), generator=gen, device="cuda")
    ids[:40], ids[40:140] = 17, 33                      # rows of many tokens, one beyond the limit of the per-row teams
    g = (torch.randint(-128, 128, (500, 64), generator=gen, device="cuda") / 64).to(dtype)      # sums exact in any order
    held = torch.randn(300, 64, generator=gen, device="cuda").to(dtype)
    want = (held.float() + E.embedding_backward(ids, g, 300).float()).to(dtype)
    assert torch.equal(E.embedding_backward(ids, g, 300, add_to=held), want)


@pytest.mark.parametrize("kind", ["register_hook", "register_prehook"])
def test_hooks_on_the_accumulation(bmt_gpu, kind):
    """Hooks on the node that accumulates a table's gradient are given the gradient."""
    emb, p = _table(bmt_gpu)
    ids, x = torch.randint(0, 300, (50,), device="cuda"), torch.randn(8, 64, device="cuda").half()
    _loss(emb, ids, x).backward()
    want, held = p.grad.clone(), p.grad
    node = p.expand_as(p).grad_fn.next_functions[0][0]
    seen = []
    handle = getattr(node, kind)(lambda *grads: seen.append(grads[-1][0]))
    held.zero_()
    _loss(emb, ids, x).backward()
    handle.remove()
    assert len(seen) == 1 and torch.equal(seen[0], want) and torch.equal(held, want)
    held.zero_()
    _loss(emb, ids, x).backward()               # nobody watches any more
    assert len(seen) == 1 and p.grad is held and torch.equal(held, want)


def test_in_place_additions_are_counted(bmt_gpu):
    emb, p = _table(bmt_gpu)
    ids, x = torch.randint(0, 300, (50,), device="cuda"), torch.randn(8, 64, device="cuda").half()
    _loss(emb, ids, x).backward()
    weight = torch.ones(1, device="cuda", dtype=torch.float16, requires_grad=True)
    product = (p.grad * weight).sum()           # keeps p.grad for its own backward
    _loss(emb, ids, x).backward()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        product.backward()


def test_gradients_off_the_16_byte_boundary(bmt_gpu):
    """A gradient that is a slice of a larger buffer, as programs that keep all gradients in one have it, is left to autograd."""
    emb, p = _table(bmt_gpu)
    ids, x = torch.randint(0, 300, (50,), device="cuda"), torch.randn(8, 64, device="cuda").half()
    _loss(emb, ids, x).backward()
    want = p.grad.clone()
    for start in (1, 4, 7, 8):
        buffer = torch.zeros(p.numel() + 32, device="cuda", dtype=p.dtype)
        p.grad = buffer[start:start + p.numel()]
        _loss(emb, ids, x).backward()
        torch.cuda.synchronize()
        assert torch.equal(p.grad, want) and not buffer[:start].any() and not buffer[start + p.numel():].any()
