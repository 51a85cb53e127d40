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
