"""One rank in the group: what a user's program may do with gathered parameters and gradients is what it may do on several
ranks, although there is nothing to gather or to reduce."""
import pytest
import torch


@pytest.fixture
def bmt(bmt_cpu):
    return bmt_cpu


def _two(bmt):
    class Two(bmt.DistributedModule):
        def __init__(self):
            super().__init__()
            self.a = bmt.DistributedParameter(torch.arange(6.0).view(2, 3))
            self.b = bmt.DistributedParameter(torch.ones(2, 3))

        def forward(self, x):
            return ((self.a + self.b + x) ** 2).sum()

    return Two()


def test_gradients_of_two_parameters_are_two_tensors(bmt):
    """The operands of an addition get the same gradient from autograd; each parameter keeps one of its own."""
    m, x = _two(bmt), torch.randn(2, 3)
    m(x).backward()
    once = m._parameters["a"].grad.clone()
    assert torch.equal(m._parameters["b"].grad, once) and once.any()
    assert m._parameters["a"].grad.data_ptr() != m._parameters["b"].grad.data_ptr()
    m(x).backward()                                              # accumulates
    for name in ("a", "b"):
        assert torch.equal(m._parameters[name].grad, 2 * once)


def test_clipping_scales_every_gradient_once(bmt):
    m = _two(bmt)
    opt = bmt.optim.AdamOptimizer(m.parameters(), lr=1e-3)
    manager = bmt.optim.OptimManager(loss_scale=None)
    manager.add_optimizer(opt)
    manager.backward(m(torch.randn(2, 3) + 3))
    manager.clip_grad_norm(opt.param_groups, 1.0)
    norm = torch.stack([p.grad.norm() for p in m.parameters()]).norm()
    assert abs(float(norm) - 1.0) < 1e-4


def test_what_is_done_to_a_gathered_value_stays_there(bmt):
    m = _two(bmt)
    before = m._parameters["a"].detach().clone()
    with torch.no_grad():
        m.a.mul_(2)
        m.a.data.add_(1)
    m._parameters["a"].gather().zero_()
    assert torch.equal(m._parameters["a"].detach(), before)


def test_backward_uses_the_value_of_the_forward_pass(bmt):
    m = _two(bmt)
    x = torch.randn(2, 3, requires_grad=True)
    y = (m.a * x).sum()
    value = m._parameters["a"].detach().clone().view(2, 3)
    m._parameters["a"].data.add_(20)                             # an update between the two passes
    y.backward()
    assert torch.equal(x.grad, value)


def _gpt_block(bmt):
    from bmtrain_b200.models.gpt import TransformerEncoder

    torch.manual_seed(3)
    blk = bmt.Block(TransformerEncoder(16, 8, 2, 32, dtype=torch.float32))
    bmt.init_parameters(blk)
    return blk


def test_state_dict_is_a_snapshot(bmt):
    blk = _gpt_block(bmt)
    saved = blk.state_dict()
    kept = {k: v.clone() for k, v in saved.items()}
    for b in blk._buckets.values():
        b.storage.data.add_(1)                                   # the next optimizer step
    assert all(torch.equal(saved[k], kept[k]) for k in kept)


def test_zero_context_hands_out_a_copy(bmt):
    from bmtrain_b200.zero_context import ZeroContext

    blk = _gpt_block(bmt)
    before = [b.storage.data.clone() for b in blk._buckets.values()]
    with ZeroContext(blk):
        for p in blk._module.parameters():
            p.data.add_(1)
    assert all(torch.equal(b.storage.data, was) for b, was in zip(blk._buckets.values(), before))


def _writer(bmt):
    class Writer(bmt.DistributedModule):
        def __init__(self):
            super().__init__()
            self.lin = bmt.nn.Linear(8, 8, bias=False, dtype=torch.float32)

        def forward(self, x):
            self.lin.weight.detach().clamp_(-0.01, 0.01)         # changes what this pass sees, not the parameter
            return self.lin(x)

    return Writer()


def _partitions(blk):
    return [b.storage.data.clone() for b in blk._buckets.values()]


def test_what_a_block_writes_to_its_parameters_is_dropped(bmt):
    blk = bmt.Block(_writer(bmt))
    bmt.init_parameters(blk)
    before, x = _partitions(blk), torch.randn(4, 8)
    want = x @ before[0].view(-1)[:64].view(8, 8).clamp(-0.01, 0.01).t()
    with torch.no_grad():
        assert torch.allclose(blk(x), want, atol=1e-6)
    y = blk(x.requires_grad_())
    assert torch.allclose(y, want, atol=1e-6)
    y.sum().backward()
    assert all(torch.equal(a, b) for a, b in zip(before, _partitions(blk)))


@pytest.mark.parametrize("how", ["module_hook", "forward", "subclass", "global_hook"])
def test_foreign_code_in_a_known_block_works_on_a_copy(bmt, how):
    blk = _gpt_block(bmt)
    lin = blk._module.ff.w_in
    handle = None

    def write(module, *args):
        module.weight.detach().zero_()

    if how == "module_hook":
        lin.register_forward_pre_hook(write)
    elif how == "global_hook":
        handle = torch.nn.modules.module.register_module_forward_pre_hook(lambda m, a: write(m) if m is lin else None)
    elif how == "forward":
        plain = lin.forward
        lin.forward = lambda x: (write(lin), plain(x))[1]
    else:
        class Own(type(lin)):
            def forward(self, x):
                write(self)
                return super().forward(x)

        lin.__class__ = Own
    before = _partitions(blk)
    blk(torch.randn(2, 4, 16, requires_grad=True)).sum().backward()
    if handle is not None:
        handle.remove()
    assert all(torch.equal(a, b) for a, b in zip(before, _partitions(blk)))


@pytest.mark.parametrize("options", [dict(), dict(zero_level=2), dict(use_checkpoint=False)])
def test_which_blocks_run_in_place(bmt, options):
    from bmtrain_b200.models.gpt import TransformerEncoder
    from bmtrain_b200.models.llama import LlamaBlock

    for module in (TransformerEncoder(16, 8, 2, 32, dtype=torch.float32), LlamaBlock(16, 2, 1, 8, 32, dtype=torch.float32)):
        blk = bmt.Block(module, **options)
        bmt.init_parameters(blk)
        assert blk._may_run_in_place() == (not options)
        blk._enter_forward(in_place=blk._may_run_in_place())
        assert all(b.aliased == (not options) for b in blk._buckets.values())
        blk._release_params()


def test_zero_2_keeps_the_parameters_of_the_forward_pass(bmt):
    from bmtrain_b200.models.gpt import TransformerEncoder

    torch.manual_seed(4)
    blk = bmt.Block(TransformerEncoder(16, 8, 2, 32, dtype=torch.float32), zero_level=2)
    bmt.init_parameters(blk)
    x = torch.randn(2, 4, 16)

    def grad(update):
        a = x.clone().requires_grad_()
        y = blk(a)
        for b in blk._buckets.values():
            b.storage.data.add_(update)
        y.sum().backward()
        for b in blk._buckets.values():
            b.storage.data.sub_(update)
        return a.grad

    assert torch.equal(grad(0.0), grad(0.5))


def _check_tables(bmt, dev, projection):
    """Lookup and projection of a stand-alone table: gradients of a table used twice, of two tables, with hooks, accumulated over
    passes; an update between the two passes; results that share no memory with the table."""
    torch.manual_seed(5)
    dtype = torch.bfloat16 if projection or dev == "cuda" else torch.float32      # fp32 projections on the CPU go through torch
    a, b = (bmt.nn.Embedding(12, 8, dtype=dtype) for _ in range(2))
    bmt.init_parameters(a)
    bmt.init_parameters(b)
    pa, pb = a._parameters["weight"], b._parameters["weight"]
    x = torch.randn(5, 8).to(dtype).to(dev).requires_grad_() if projection else torch.tensor([3, 3, 0, 11, 7], device=dev)
    seen = []
    pa.register_hook(lambda g: seen.append(g))

    def loss():
        return (a(x, projection=projection) * 2 + a(x, projection=projection) + b(x, projection=projection)).float().sum()

    def want():
        wa, wb = (p.detach().clone().view(12, 8).float().requires_grad_() for p in (pa, pb))
        xs = x.detach().float().requires_grad_() if projection else x
        f = lambda w: xs @ w.t() if projection else w[xs]  # noqa: E731
        (f(wa) * 3 + f(wb)).sum().backward()
        return wa.grad.reshape(-1), wb.grad.reshape(-1), xs.grad

    ga, gb, gx = want()
    value = loss()
    for p in (pa, pb):
        p.data.add_(1)                                           # an update between the two passes
    value.backward()
    for p in (pa, pb):
        p.data.sub_(1)
    # bf16: three results of magnitude up to 20 are rounded and added
    tol = dict(rtol=2e-2, atol=2e-1) if dtype == torch.bfloat16 else dict(rtol=1e-6, atol=1e-6)
    assert torch.allclose(pa.grad.float(), ga, **tol) and torch.allclose(pb.grad.float(), gb, **tol)
    if projection:
        assert torch.allclose(x.grad.float(), gx, **tol)
    assert len(seen) == 1 and pa.grad.data_ptr() != pb.grad.data_ptr()
    kept = seen[0].clone()
    once = pb.grad.clone()
    loss().backward()
    assert torch.allclose(pb.grad.float(), 2 * once.float(), **tol)
    assert torch.equal(seen[0], kept)                            # what a hook kept is not added to
    before = pa.detach().clone()
    with torch.no_grad():
        a(x, projection=projection).zero_()
    assert torch.equal(pa.detach(), before)


@pytest.mark.parametrize("projection", [False, True])
def test_tables_are_used_in_place_without_showing(bmt, projection):
    _check_tables(bmt, "cpu", projection)


@pytest.mark.gpu
@pytest.mark.parametrize("projection", [False, True])
def test_tables_are_used_in_place_without_showing_gpu(bmt_gpu, projection):
    _check_tables(bmt_gpu, "cuda", projection)


def test_a_table_with_a_weight_of_its_own_making(bmt):
    class Scaled(bmt.nn.Embedding):
        @property
        def weight(self):
            return self.__getattr__("weight") * 3

    e = Scaled.__new__(Scaled)
    torch.nn.Module.__init__(e)
    e.num_embeddings, e.embedding_dim = 4, 8
    e.register_parameter("weight_", None)
    e._parameters["weight"] = bmt.DistributedParameter(torch.randn(4, 8))
    ids = torch.tensor([1, 2])
    assert torch.allclose(e(ids), 3 * e._parameters["weight"].gather()[ids])


def test_a_dropped_block_is_freed_at_once(bmt):
    """No reference cycle keeps the partition or the gradients of a block until the next garbage collection."""
    import gc
    import weakref

    blk = _gpt_block(bmt)
    blk(torch.randn(2, 4, 16, requires_grad=True)).sum().backward()
    bmt.synchronize()
    gc.collect()
    gc.disable()
    try:
        refs = [weakref.ref(b.storage) for b in blk._buckets.values()] + [weakref.ref(b.storage.grad) for b in blk._buckets.values()]
        refs += [weakref.ref(p) for p in blk._module.parameters()] + [weakref.ref(blk._module)]
        del blk
        assert all(r() is None for r in refs)
    finally:
        gc.enable()


def test_hook_functions_attach_gradient_buffers(bmt):
    """The four moments for code that brackets a block by hand: full-size parameters and gradients are in place in between."""
    from bmtrain_b200 import hook_func

    blk = _gpt_block(bmt)
    before = _partitions(blk)
    hook_func.zero_pre_forward(blk, ())
    for p in blk._module.parameters():
        p.data.mul_(2)                                           # on a copy
    hook_func.zero_post_forward(blk, None, None)
    hook_func.zero_pre_backward(blk, None)
    for s in blk._slots:
        assert s.param.shape == s.shape and s.param.grad.shape == s.shape and not s.param.grad.any()
        s.param.grad.add_(1)
    hook_func.zero_post_backward(blk, None, None)
    bmt.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(before, _partitions(blk)))
    for p in blk.parameters():
        assert torch.equal(p.grad, torch.ones_like(p.grad))
