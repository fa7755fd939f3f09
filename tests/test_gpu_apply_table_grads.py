"""Gradients of phase tables that the caller broadcast with a stride of 0: every slice of the gradient holds the sum of its own
units, also where one block of the transform takes several units.  Against the CPU oracle, slice by slice, with the bound of the
transform's other table gradients."""
import pytest
import torch

from oracle import pope_oracle as O
from pope_pytorch_b200 import apply_pope_to_qk

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("kind", ["batch", "heads", "both", "plain", "own"])
def test_gradient_of_an_expanded_table(kind):
    b, h, n, d, r = 4, 8, 1500, 32, 16
    g = torch.Generator().manual_seed(1)
    q, k = torch.randn(b, h, n, d, generator=g), torch.randn(b, h, n, d, generator=g)
    gq, gk = torch.randn(b, h, n, d + r, generator=g), torch.randn(b, h, n, d + r, generator=g)
    lead, shape = {"batch": ((1,), (b, n, r)), "heads": ((b, 1), (b, h, n, r)), "both": ((1, 1), (b, h, n, r)), "plain": ((), (n, r)),
                   "own": ((b, h), (b, h, n, r))}[kind]
    base, bias = torch.rand(*lead, n, r, generator=g) * 500, -torch.rand(h, r, generator=g) * 6
    full = base.expand(shape).contiguous().requires_grad_(True)
    ref = [q.requires_grad_(True), k.requires_grad_(True), bias.clone().requires_grad_(True)]
    want = torch.autograd.grad(O.apply_pope(full, ref[2], ref[0], ref[1]), [full, ref[2]], (gq, gk))
    table = base.to(DEV).expand(shape).requires_grad_(True)     # (strides of 0 where it is broadcast)
    bias_gpu = bias.to(DEV).requires_grad_(True)
    out = apply_pope_to_qk((table, bias_gpu), q.detach().to(DEV), k.detach().to(DEV))
    got = torch.autograd.grad(out, [table, bias_gpu], (gq.to(DEV), gk.to(DEV)))
    for x, w in zip(got, want):
        torch.testing.assert_close(x.cpu(), w, rtol=1e-4, atol=1e-4 * max(1.0, float(w.abs().max())))
