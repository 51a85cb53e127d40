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
