"""The one-launch embedding tables against the module's own PyTorch chain: the same single fp32 multiply per phase and the
same clamp, so every value is bitwise equal; the bias gradient passes exactly where the clamp does."""
import math

import pytest
import torch

from pope_pytorch_b200 import AxialPoPE, PoPE

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("make,where", [
    (lambda: PoPE(1, heads=1), (1,)), (lambda: PoPE(32, heads=3), (257, 5)), (lambda: PoPE(48, heads=16, theta=500.0), (4096, -2.5)),
    (lambda: AxialPoPE(96, heads=8, axial_dims=(32, 32, 32)), ((8, 16, 16),)), (lambda: AxialPoPE(20, heads=2, axial_dims=(4, 16)), ((1, 7),)),
])
def test_tables_equal_the_torch_chain(make, where):
    m = make().to(DEV)
    with torch.no_grad():
        m.bias.uniform_(-9.0, 2.0, generator=torch.Generator(DEV).manual_seed(3))
        m.bias.view(-1)[0] = -2 * math.pi     # the bounds themselves pass their gradient
        m.bias.view(-1)[-1] = 0.0
    got = m(*where)
    ref = m._forward_torch(*where, 0) if isinstance(m, PoPE) and len(where) == 1 else m._forward_torch(*where)
    assert type(got) is type(ref) and torch.equal(got.freqs, ref.freqs) and torch.equal(got.bias, ref.bias)
    for a, b in zip((got.positions, got.inv_freqs, got.axis_of), (ref.positions, ref.inv_freqs, ref.axis_of)):
        assert (a is None) == (b is None) and (a is None or (a.dtype == b.dtype and torch.equal(a, b)))
    w = torch.randn_like(got.bias)
    g1, = torch.autograd.grad((got.bias * w).sum(), m.bias)
    g2, = torch.autograd.grad((ref.bias * w).sum(), m.bias)
    assert torch.equal(g1, g2) and not got.freqs.requires_grad
