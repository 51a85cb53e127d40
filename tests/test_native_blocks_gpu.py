"""Blocks computed by the native executors against the same blocks run through their modules: outputs, gradients of the input and of
every parameter, with recomputation; what makes a block go through its modules again."""
import pytest
import torch

pytestmark = pytest.mark.gpu

_UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _llama(bmt, dtype, dim, heads, kv, dh, ff):
    from bmtrain_b200.models.llama import LlamaBlock

    return LlamaBlock(dim, heads, kv, dh, ff, dtype=dtype)


def _gpt(bmt, dtype, dim, heads, dh, ff, act, causal):
    from bmtrain_b200.models.gpt import TransformerEncoder

    return TransformerEncoder(dim, dh, heads, ff, True, dtype, act, causal=causal)


def _step(block, args, gy):
    x = args[0].detach().clone().requires_grad_()
    y = block(x, *args[1:])
    y.backward(gy)
    grads = {n: p.grad.clone() for n, p in block.named_parameters()}
    for b in block._buckets.values():
        b.storage.grad = None
    for p in block.parameters():
        p.grad = None
    return y.detach(), x.grad, grads


CASES = [("llama", dict(dim=256, heads=4, kv=4, dh=64, ff=704), (2, 128)), ("llama", dict(dim=264, heads=3, kv=1, dh=80, ff=328), (1, 77)),
         ("llama", dict(dim=512, heads=8, kv=2, dh=128, ff=1024), (3, 200)),
         ("gpt", dict(dim=256, heads=4, dh=64, ff=1024, act="relu", causal=True), (2, 128)),
         ("gpt", dict(dim=240, heads=3, dh=80, ff=520, act="gelu", causal=False), (2, 77)),
         ("gpt", dict(dim=256, heads=2, dh=8, ff=256, act="relu", causal=True), (1, 40))]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind,cfg,tokens", CASES)
def test_native_block(bmt_gpu, dtype, kind, cfg, tokens, monkeypatch):
    bmt = bmt_gpu
    gen = torch.Generator(device="cuda").manual_seed(3)
    block = bmt.Block((_llama if kind == "llama" else _gpt)(bmt, dtype, **cfg))
    with torch.no_grad():
        for name, p in block._module.named_parameters():
            shape = p._original_shape
            value = torch.randn(*shape, generator=gen, device="cuda") * (0.1 if len(shape) == 1 else shape[-1] ** -0.5) + (
                1.0 if len(shape) == 1 and name.endswith("weight") else 0.0)
            block._load_param(p, value.to(dtype))
    b, s = tokens
    x = torch.randn(b, s, cfg["dim"], generator=gen, device="cuda").to(dtype)
    gy = torch.randn(b, s, cfg["dim"], generator=gen, device="cuda").to(dtype)
    args = [x]
    if kind == "gpt" and not cfg["causal"]:
        mask = torch.rand(b, s, s, generator=gen, device="cuda") < 0.6
        mask[:, :, 0] = True
        args.append(mask)
    calls = []
    real = type(block)._native_backward
    monkeypatch.setattr(type(block), "_native_backward", lambda *a: calls.append(1) or real(*a))
    native = _step(block, args, gy)
    assert len(calls) == 1
    again = _step(block, args, gy)
    assert torch.equal(native[0], again[0])
    with torch.no_grad():
        assert torch.equal(block(*args), native[0])
    monkeypatch.setattr(type(block), "_native_module", lambda *a, **k: None)
    modules = _step(block, args, gy)
    assert len(calls) == 2
    assert torch.equal(native[0], modules[0])              # the same roundings forward
    # each is a few roundings of 16-bit intermediates away from the exact block; a chain of a dozen of them on either side
    for a, e in [(native[0], modules[0]), (native[1], modules[1])] + [(native[2][n], modules[2][n]) for n in modules[2]]:
        assert (a.double() - e.double()).norm() <= 12 * _UNIT[dtype] * e.double().norm() + 1e-6
    assert set(native[2]) == set(modules[2])


def test_hooks_and_partial_training_go_through_the_modules(bmt_gpu):
    bmt = bmt_gpu
    block = bmt.Block(_llama(bmt, torch.bfloat16, 256, 4, 4, 64, 512))
    bmt.init_parameters(block)
    x = torch.randn(1, 64, 256, device="cuda", dtype=torch.bfloat16)
    args = [x]
    assert block._native_module(args, True) is not None
    seen = []
    handle = block._module.ff.register_forward_hook(lambda m, i, o: seen.append(o))
    block(x.requires_grad_()).sum().backward()
    assert len(seen) == 2                                  # forward and recomputation
    handle.remove()
    block(x).sum().backward()
    assert len(seen) == 2
    p = block._module.attn.project_out.weight
    p.requires_grad_(False)
    from bmtrain_b200.layer import only_reads_parameters

    assert block._native_module(args, only_reads_parameters(block._module), training=True) is None
    assert block._native_module([x.float()], True) is None


@pytest.mark.parametrize("tokens,d,d_ff", [(370, 2560, 10240), (2272, 2496, 7936), (128, 256, 4096)])
def test_products_below_a_relu_are_not_divided(bmt_gpu, tokens, d, d_ff):
    """The block gives the bits that products of whole tiles give (the first two sizes are planned as divided ones elsewhere)."""
    from bmtrain_b200.ops import gpt_block

    gen = torch.Generator(device="cuda").manual_seed(d)
    dims = {"qkv": (3 * d, d), "out": (d, d), "fc1": (d_ff, d), "fc2": (d, d_ff)}
    rnd = lambda *s: (0.02 * torch.randn(*s, generator=gen, device="cuda")).bfloat16()  # noqa: E731
    params = {n + "_w": rnd(*s) for n, s in dims.items()} | {n + "_b": rnd(s[0]) for n, s in dims.items()}
    for n in ("ln1", "ln2"):
        params[n + "_w"], params[n + "_b"] = 1 + rnd(d), rnd(d)
    order = ("ln1_w", "ln1_b", "qkv_w", "qkv_b", "out_w", "out_b", "ln2_w", "ln2_b", "fc1_w", "fc1_b", "fc2_w", "fc2_b")
    x = torch.randn(1, tokens, d, generator=gen, device="cuda").bfloat16()

    def ran(without):
        run = gpt_block.Pass(x, None, [params[n].data_ptr() for n in order], d // 64, 64, d_ff, "relu", 1e-5, True)
        if without:
            run.tail = run.tail[:-2] + (0, 0)
        return run.forward()

    assert torch.equal(ran(False), ran(True))


class _Wrapped(torch.nn.Module):
    """A projection whose parameters are not its own."""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    weight = property(lambda self: self.inner.weight)
    bias = property(lambda self: self.inner.bias)

    def forward(self, x):
        return self.inner(x)


def test_block_with_a_wrapped_projection(bmt_gpu):
    bmt = bmt_gpu
    enc = _gpt(bmt, torch.float16, 256, 4, 64, 512, "relu", True)
    bmt.init_parameters(enc)
    x = torch.randn(1, 40, 256, device="cuda").half()
    want = enc(x)
    enc.attn.project_qkv = _Wrapped(enc.attn.project_qkv)
    assert torch.equal(enc(x), want)


def test_block_with_other_submodules(bmt_gpu):
    """A Llama block with another feed-forward layer of this package runs its modules."""
    from bmtrain_b200.models.gpt import Feedforward

    bmt = bmt_gpu
    inner = _llama(bmt, torch.bfloat16, 256, 4, 4, 64, 512)
    inner.ff = Feedforward(256, 512, bias=False, dtype=torch.bfloat16)
    block = bmt.Block(inner)
    bmt.init_parameters(block)
    x = torch.randn(1, 64, 256, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        assert torch.equal(block(x), block(x))
    y, dx, grads = _step(block, [x], torch.ones_like(x))
    assert torch.isfinite(dx).all() and len(grads) == 6


def test_parameters_show_the_partition_after_a_pass(bmt_gpu):
    """Whatever was assigned to a parameter's ``data``: a pass computes with the partition, and afterwards the parameters are its views again."""
    bmt = bmt_gpu
    block = bmt.Block(_llama(bmt, torch.bfloat16, 256, 4, 4, 64, 512))
    bmt.init_parameters(block)
    x = torch.randn(1, 64, 256, device="cuda", dtype=torch.bfloat16)
    _step(block, [x], torch.ones_like(x))
    want = [p.data_ptr() for p in block.parameters()]
    values = [p.detach().clone() for p in block.parameters()]
    for training in (True, False):
        for p in block.parameters():
            p.data = p.data.clone().zero_()
        if training:
            _step(block, [x], torch.ones_like(x))
        else:
            with torch.no_grad():
                block(x)
        assert [p.data_ptr() for p in block.parameters()] == want
        assert all(torch.equal(p.detach(), v) for p, v in zip(block.parameters(), values))


def _launches(call):
    import ctypes

    from bmtrain_b200.ops import _native

    lib = _native.cuda_lib()
    lib.bmt_launch_count.restype = ctypes.c_int64
    before = lib.bmt_launch_count()
    call()
    return lib.bmt_launch_count() - before


@pytest.mark.parametrize("tokens,act,masked,forward,backward", [(300, "relu", False, 7, 14), (300, "gelu", True, 9, 14), (2056, "relu", False, 7, 18)])
def test_launches_of_a_gpt_block(bmt_gpu, tokens, act, masked, forward, backward):
    from bmtrain_b200.ops import gpt_block

    d, f = 256, 512
    shapes = [(d,), (d,), (3 * d, d), (3 * d,), (d, d), (d,), (d,), (d,), (f, d), (f,), (d, f), (d,)]
    params = [torch.randn(*s, device="cuda").mul_(0.05).half() for s in shapes]
    grads = [torch.empty_like(p) for p in params]
    x = torch.randn(1, tokens, d, device="cuda").half()
    mask = torch.ones(1, tokens, tokens, dtype=torch.bool, device="cuda") if masked else None
    run = gpt_block.Pass(x, mask, [p.data_ptr() for p in params], 4, 64, f, act, 1e-5, True)
    assert _launches(run.forward) == forward
    assert _launches(lambda: run.backward(x, [g.data_ptr() for g in grads])) == backward


@pytest.mark.parametrize("kv,backward", [(4, 16), (1, 17)])
def test_launches_of_a_llama_block(bmt_gpu, kv, backward):
    from bmtrain_b200.ops import llama_block

    d, f, h, dh = 256, 512, 4, 64
    shapes = [(d,), ((h + 2 * kv) * dh, d), (d, h * dh), (d,), (2 * f, d), (d, f)]
    params = [torch.randn(*s, device="cuda").mul_(0.05).half() for s in shapes]
    grads = [torch.empty_like(p) for p in params]
    x = torch.randn(1, 300, d, device="cuda").half()
    run = llama_block.Pass(x, [p.data_ptr() for p in params], h, kv, dh, f, 1e-5, 1e-5, 10000.0)
    assert _launches(run.forward) == 9
    assert _launches(lambda: run.backward(x, [g.data_ptr() for g in grads])) == backward


def test_executor_and_operators_at_a_size_that_is_divided(bmt_gpu, monkeypatch):
    """Below a ReLU the executor's products are whole and the operators' are divided: equal but for the rounding of sums."""
    from bmtrain_b200.models import gpt

    bmt, dtype = bmt_gpu, torch.bfloat16
    gen = torch.Generator(device="cuda").manual_seed(9)
    enc = _gpt(bmt, dtype, 2560, 40, 64, 10240, "relu", True)
    bmt.init_parameters(enc)
    x = torch.randn(1, 370, 2560, generator=gen, device="cuda").to(dtype)
    with torch.no_grad():
        executor = enc(x)
        monkeypatch.setattr(gpt, "_FUSED_BLOCK", False)
        operators = enc(x)
    # a chain of a dozen 16-bit intermediates
    assert (executor.double() - operators.double()).norm() <= 12 * _UNIT[dtype] * operators.double().norm()


def test_strides_of_the_result(bmt_gpu, monkeypatch):
    """A sequence-first hidden state seen as batch-first: the result lies in memory as that of the modules does."""
    bmt = bmt_gpu
    block = bmt.Block(_llama(bmt, torch.float16, 256, 4, 2, 64, 512))
    bmt.init_parameters(block)
    x = torch.randn(40, 3, 256, device="cuda").half().transpose(0, 1)
    with torch.no_grad():
        got, contiguous = block(x), block(x.contiguous())
        assert block._native_module([x.contiguous()], True) is not None
        monkeypatch.setattr(type(block), "_native_module", lambda *a, **k: None)
        want = block(x)
    assert got.stride() == want.stride() and contiguous.is_contiguous()
    assert torch.equal(got, want) and torch.equal(contiguous, want)
    got.transpose(0, 1).view(120, 256)
