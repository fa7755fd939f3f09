"""Gradients of gradients through the embedding modules: equal to those of the module's own PyTorch operations, to the bit (the same
comparisons and products).  A batch of gradients (vmap over the backward) as well."""
import pytest
import torch

from pope_pytorch_b200 import AxialPoPE, PoPE

pytestmark = pytest.mark.gpu
DEV = "cuda"
MODULES = [(lambda: PoPE(32, heads=3), 40), (lambda: AxialPoPE(12, heads=2, axial_dims=(4, 8)), (5, 6))]


def spread(module):
    module = module.to(DEV)
    with torch.no_grad():
        module.bias.uniform_(-9.0, 2.0, generator=torch.Generator(DEV).manual_seed(1))
        module.bias.view(-1)[0] = -2 * torch.pi
    return module


def torch_forward(module, where):
    return module._forward_torch(where, 0) if isinstance(module, PoPE) else module._forward_torch(where)


@pytest.mark.parametrize("make,where", MODULES)
def test_gradient_penalty(make, where):
    module = spread(make())
    got = []
    for forward in (lambda: module(where), lambda: torch_forward(module, where)):
        w = torch.linspace(-1, 2, module.bias.numel(), device=DEV).view_as(module.bias).requires_grad_(True)
        g = torch.autograd.grad((w * forward().bias ** 3).sum(), (module.bias, w), create_graph=True)
        got.append((*g, *torch.autograd.grad(sum(x.square().sum() for x in g), (module.bias, w))))
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("make,where", MODULES)
def test_hessian_and_batched_gradients(make, where):
    module = spread(make())
    hessians = []
    for forward in (lambda: module(where), lambda: torch_forward(module, where)):
        g, = torch.autograd.grad(forward().bias.pow(3).sum(), module.bias, create_graph=True)
        hessians.append(torch.stack([torch.autograd.grad(x, module.bias, retain_graph=True)[0] for x in g.flatten()[:20]]))
    assert torch.equal(*hessians) and bool(hessians[0].any())
    bias = module(where).bias
    v = torch.randn(7, *bias.shape, device=DEV, generator=torch.Generator(DEV).manual_seed(2))
    batched, = torch.autograd.grad(bias, module.bias, v, is_grads_batched=True, retain_graph=True)
    for row, x in zip(batched, v):
        assert torch.equal(row, torch.autograd.grad(bias, module.bias, x, retain_graph=True)[0])
