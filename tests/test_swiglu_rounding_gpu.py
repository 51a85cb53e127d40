"""SwiGLU computes in 32 bits with one rounding for each operation: the same bits as those operations one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_swiglu_operations(bmt_gpu, dtype):
    from bmtrain_b200.ops import elementwise

    gate = torch.arange(-2 ** 15, 2 ** 15, device="cuda", dtype=torch.int32).to(torch.int16).view(dtype)
    gate = gate[(gate.abs() > 2.0 ** -6) & (gate.abs() < 10)]
    gate = gate[:gate.numel() // 8 * 8].expand(64, -1)
    gen = torch.Generator(device="cuda").manual_seed(3)
    up, grad = ((torch.rand(gate.shape, device="cuda", generator=gen) + 0.5).to(dtype) for _ in range(2))
    x = torch.cat([gate, up], 1).requires_grad_()
    y = elementwise.swiglu(x)
    (dx,) = torch.autograd.grad(y, x, grad)
    g = gate.float()
    e = 1 + torch.exp2(g * torch.tensor(-1.4426950408889634, device="cuda"))
    assert torch.equal(y, (g / e * up.float()).to(dtype))
    assert torch.equal(dx[:, gate.shape[1]:], (grad.float() * (g * (1 / e))).to(dtype))
