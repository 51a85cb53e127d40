"""Gradients of a block's parameters: written into the block's buffer by kernels, left in ``.grad`` by autograd, or
missing; parameters used in place on one rank."""
import pytest
import torch

from dist_utils import run_distributed


def _make(bmt, dtype):
    class Net(bmt.DistributedModule):
        def __init__(self):
            super().__init__()
            self.a = bmt.nn.Linear(24, 40, dtype=dtype)          # sizes that leave gaps between the slots
            self.twice = bmt.nn.Linear(40, 40, bias=False, dtype=dtype)
            self.norm = bmt.nn.RMSNorm(40, dtype=dtype) if dtype != torch.float32 else None
            self.unused = bmt.nn.Linear(8, 8, dtype=dtype)
            self.scale = bmt.DistributedParameter(torch.ones(40, dtype=dtype))
            self.out = bmt.nn.Linear(40, 24, dtype=dtype)

        def forward(self, x):
            h = self.twice(torch.tanh(self.a(x)))
            h = self.twice(torch.tanh(h)) * self.scale           # one weight, two gradients
            if self.norm is not None:
                h = self.norm(h)
            return self.out(h)

    return Net()


def _reference(state, x, grad, norm):
    p = {k: v.double().requires_grad_() for k, v in state.items()}
    x = x.double()
    h = torch.tanh(x @ p["a.weight"].t() + p["a.bias"]) @ p["twice.weight"].t()
    h = (torch.tanh(h) @ p["twice.weight"].t()) * p["scale"]
    if norm:
        h = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * p["norm.weight"]
    y = h @ p["out.weight"].t() + p["out.bias"]
    g = torch.autograd.grad(y, list(p.values()), grad.double(), allow_unused=True)
    return y, {k: torch.zeros_like(v) if gi is None else gi for (k, v), gi in zip(p.items(), g)}


def _check(bmt, dev, dtype, ckpt, hook, tol):
    torch.manual_seed(11)
    net = _make(bmt, dtype)
    state = {k: (torch.randn(v.shape) * 0.3).to(dtype) for k, v in net.state_dict().items()}
    seen = []
    blk = bmt.Block(net, use_checkpoint=ckpt)
    if hook:
        dict(blk.named_parameters())["out.weight"].register_hook(lambda g: seen.append(g.shape))
    blk.load_state_dict({k: v.to(dev) for k, v in state.items()})
    x, grad = torch.randn(6, 24).to(dtype), torch.randn(6, 24).to(dtype)
    y_ref, want = _reference(state, x, grad, "norm.weight" in state)
    for passes in (1, 2):                                        # the second pass accumulates
        y = blk(x.to(dev).requires_grad_())
        y.backward(grad.to(dev))
        bmt.synchronize()
        assert (y.double().cpu() - y_ref).norm() <= tol * y_ref.norm()
        got = {n: p.grad for n, p in blk.named_parameters()}
        assert set(got) == set(want)
        for n, g in want.items():
            err = (got[n].double().cpu().reshape(-1) - passes * g.reshape(-1)).norm()
            assert err <= tol * passes * g.norm() + 1e-12, (n, passes, float(err))
        whole = passes * torch.cat([g.reshape(-1) for g in want.values()]).norm()
        for b in blk._buckets.values():                          # the gaps between the slots hold zeros
            assert torch.isfinite(b.storage.grad).all()
            assert b.storage.grad.double().norm().cpu() <= (1 + tol) * whole
    assert len(seen) == (2 if hook else 0)
    for k, v in blk.state_dict().items():                        # parameters used in place are left as they were
        assert torch.equal(v.cpu(), state[k]), k


@pytest.mark.parametrize("ckpt", [True, False])
@pytest.mark.parametrize("hook", [False, True])
def test_block_gradients_cpu(bmt_cpu, ckpt, hook):
    _check(bmt_cpu, "cpu", torch.float32, ckpt, hook, 1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("ckpt", [True, False])
@pytest.mark.parametrize("hook", [False, True])
def test_block_gradients_gpu(bmt_gpu, dtype, ckpt, hook):
    # activations and gradients pass about ten roundings to 16 bits
    _check(bmt_gpu, "cuda", dtype, ckpt, hook, 10 * (2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7))


class _AddsToGrad(torch.autograd.Function):
    """The usual fused weight gradient: added to ``weight.grad`` in place, nothing returned to autograd."""

    @staticmethod
    def forward(ctx, x, weight):
        ctx.weight = weight
        ctx.save_for_backward(x)
        return x @ weight.t()

    @staticmethod
    def backward(ctx, g):
        (x,) = ctx.saved_tensors
        ctx.weight.grad.add_(g.t() @ x)
        return g @ ctx.weight, None


class _Nested(torch.autograd.Function):
    """Asks autograd for the gradient of a weight inside its own backward."""

    @staticmethod
    def forward(ctx, x, weight, linear):
        ctx.linear = linear
        ctx.save_for_backward(x, weight)
        with torch.no_grad():
            return linear(x)

    @staticmethod
    def backward(ctx, g):
        x, weight = ctx.saved_tensors
        x = x.detach().requires_grad_()
        with torch.enable_grad():
            y = ctx.linear(x)
        gx, gw = torch.autograd.grad(y, (x, weight), g)
        return gx, gw, None


def _check_foreign(bmt, dev, dtype, tol):
    class Net(bmt.DistributedModule):
        def __init__(self):
            super().__init__()
            self.a, self.b = (bmt.nn.Linear(24, 24, bias=False, dtype=dtype) for _ in range(2))

        def forward(self, x):
            x = _AddsToGrad.apply(x, self.a.weight)
            return _Nested.apply(x, self.b.weight, self.b)

    torch.manual_seed(5)
    blk = bmt.Block(Net())
    blk.load_state_dict({k: (torch.randn(24, 24) * 0.3).to(dtype).to(dev) for k in ("a.weight", "b.weight")})
    x, g = torch.randn(6, 24).to(dtype).to(dev).requires_grad_(), torch.randn(6, 24).to(dtype).to(dev)
    wa, wb = (v.double().to(dev).requires_grad_() for v in blk.state_dict().values())
    want = torch.autograd.grad((x.double() @ wa.t()) @ wb.t(), (wa, wb), g.double())
    for passes in (1, 2):
        blk(x).backward(g)
        bmt.synchronize()
        for (n, p), w in zip(blk.named_parameters(), want):
            assert (p.grad.double() - passes * w.reshape(-1)).norm() <= tol * passes * w.norm(), (n, passes)


def test_foreign_functions_cpu(bmt_cpu):
    _check_foreign(bmt_cpu, "cpu", torch.float32, 1e-5)


@pytest.mark.gpu
def test_foreign_functions_gpu(bmt_gpu):
    _check_foreign(bmt_gpu, "cuda", torch.float16, 6 * 2.0 ** -10)


def _check_known(bmt, dev, dtype, kind, tol):
    """Blocks of the package's own modules: no buffer is cleared for them, and a hook brings the general path back."""
    from bmtrain_b200.models.gpt import TransformerEncoder
    from bmtrain_b200.models.llama import LlamaBlock
    from oracle import OracleBlock

    torch.manual_seed(7)
    make = lambda: TransformerEncoder(64, 16, 4, 96, dtype=dtype, causal=True) if kind == "gpt" else LlamaBlock(64, 4, 2, 16, 96, dtype=dtype)  # noqa: E731
    blocks, seen = [bmt.Block(make()) for _ in range(2)], []
    state = {k: (torch.randn(v.shape) * 0.2).to(dtype) for k, v in blocks[0].state_dict().items()}
    for blk in blocks:
        blk.load_state_dict({k: v.to(dev) for k, v in state.items()})
    list(blocks[1].parameters())[0].register_hook(lambda g: seen.append(g.shape))
    x, g = torch.randn(2, 24, 64).to(dtype).to(dev), torch.randn(2, 24, 64).to(dtype).to(dev)
    with torch.no_grad():
        assert torch.equal(blocks[0](x), blocks[1](x))
    grads = []
    for blk in blocks:
        for _ in range(2):                                       # the second pass accumulates
            blk(x.clone().requires_grad_()).backward(g)
        bmt.synchronize()
        grads.append({n: p.grad.double().clone() for n, p in blk.named_parameters()})
    alone = bmt.world_size() == 1
    assert blocks[0]._may_run_in_place() == alone and not blocks[1]._may_run_in_place() and len(seen) == 2
    for n, a in grads[0].items():
        assert (a - grads[1][n]).norm() <= tol * grads[1][n].norm() + 1e-12, n
    if kind == "gpt" and alone:
        ref = OracleBlock(64, 16, 4, 96).double()
        ref.load_state_dict({k: v.double() for k, v in state.items()})
        ref(x.double().cpu(), torch.ones(24, 24).tril().bool().expand(2, 24, 24)).backward(g.double().cpu())
        for n, p in ref.named_parameters():
            assert (grads[0][n].cpu() - 2 * p.grad.reshape(-1)).norm() <= 4 * tol * p.grad.norm() + 1e-12, n


@pytest.mark.parametrize("kind", ["gpt", "llama"])
def test_known_blocks_cpu(bmt_cpu, kind):
    _check_known(bmt_cpu, "cpu", torch.float32, kind, 1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["gpt", "llama"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_known_blocks_gpu(bmt_gpu, kind, dtype):
    # the two paths add the second pass in 16 bits and in fp32; activations and gradients pass about ten roundings to 16 bits
    _check_known(bmt_gpu, "cuda", dtype, kind, 10 * (2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7))


def known_on_ranks(kind):
    import bmtrain_b200 as bmt
    from bmtrain_b200.ops import grad_slot

    found = []
    plain = grad_slot.find
    grad_slot.find = lambda p: found.append(plain(p)) or found[-1]
    _check_known(bmt, "cpu", torch.bfloat16, kind, 10 * 2.0 ** -7)
    assert any(s is not None for s in found)                     # the linear layers of the first block wrote into their slots


@pytest.mark.parametrize("world", [2, 3])
@pytest.mark.parametrize("kind", ["gpt", "llama"])
def test_known_blocks_on_ranks_cpu(kind, world):
    run_distributed("test_grad_slots", "known_on_ranks", world, kind=kind)


def test_gradient_buffers_are_attached_later(bmt_cpu):
    """Two backward passes into one buffer (micro-batches of a pipeline), the first without and the second with views."""
    from bmtrain_b200.models.llama import LlamaBlock

    blk = bmt_cpu.Block(LlamaBlock(16, 2, 2, 8, 24, dtype=torch.float32))
    bmt_cpu.init_parameters(blk)
    first, second = [s.param for s in blk._slots][:2]
    blk._enter_backward(attach=False)
    assert first.grad is None
    first.grad = torch.ones_like(first)
    blk._enter_backward()
    for s in blk._slots:
        assert s.param.grad.data_ptr() == s.grad_ptr()
    first.grad.add_(1)
    second.grad.add_(3)
    blk._exit_backward()
    bmt_cpu.synchronize()
    for i, p in enumerate(blk.parameters()):
        assert torch.equal(p.grad, torch.full_like(p.grad, [2.0, 3.0][i] if i < 2 else 0.0)), i
