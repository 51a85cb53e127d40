"""Gradients of a block's parameters: written into the block's buffer by kernels, left in ``.grad`` by autograd, or
missing; parameters used in place on one rank."""
import pytest
import torch


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
