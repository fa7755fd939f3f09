"""The stand-alone transform where its pieces change: pairs and quads of features or single ones (widths, strides, addresses), blocks
that span several heads and batch entries, tables that differ by batch entry or head.  Against the CPU oracle with the bounds
of the transform's other tests."""
import pytest
import torch

from oracle import pope_oracle as O
from pope_pytorch_b200 import apply_pope_to_qk

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("b,h,hk,nq,nk,d,r,table,shift,dtype", [
    (3, 16, 8, 2000, 2000, 32, 16, "2d", 0, torch.bfloat16),    # several units per block, across heads
    (5, 12, 12, 1500, 1501, 24, 8, "4d", 0, torch.float16),     # ... each with its own phases
    (4, 16, 4, 1200, 1200, 16, 16, "3d", 0, torch.float32),     # nothing plain, one table per batch entry
    (2, 3, 3, 70, 71, 22, 10, "2d", 0, torch.bfloat16),         # widths that are no multiple of four
    (2, 2, 1, 65, 130, 64, 32, "2d", 1, torch.bfloat16),        # rows that start off a 4-element boundary
    (1, 2, 2, 9, 9, 255, 201, "2d", 0, torch.float32),          # odd, nearly the widest
    (1, 1, 1, 3, 3, 256, 256, "2d", 0, torch.float16),          # the widest
])
def test_pieces_and_groups(b, h, hk, nq, nk, d, r, table, shift, dtype):
    g = torch.Generator().manual_seed(nq + nk + d + r)
    q, k = torch.randn(b, h, nq, d, generator=g).to(dtype), torch.randn(b, hk, nk, d, generator=g).to(dtype)
    lead = {"2d": (), "3d": (b,), "4d": (b, hk)}[table]
    freqs, bias = torch.rand(*lead, nk, r, generator=g) * 500, -torch.rand(hk, r, generator=g) * 6
    gq, gk = torch.randn(b, h, nq, d + r, generator=g), torch.randn(b, hk, nk, d + r, generator=g)
    ref = [t.float().clone().requires_grad_(True) for t in (q, k, freqs, bias)]
    want = O.apply_pope(ref[2], ref[3], ref[0], ref[1])
    torch.autograd.backward(want, (gq, gk))

    def on_gpu(t):   # with `shift`: the same values, one element into a larger buffer
        wide = torch.zeros(*t.shape[:-1], t.shape[-1] + 4 * bool(shift), dtype=t.dtype, device=DEV)
        view = wide[..., shift:shift + t.shape[-1]]
        view.copy_(t)
        return view.requires_grad_(True)

    ins = [on_gpu(q), on_gpu(k), freqs.to(DEV).requires_grad_(True), bias.to(DEV).requires_grad_(True)]
    out = apply_pope_to_qk(tuple(ins[2:]), *ins[:2])
    grads = torch.autograd.grad(out, ins, (gq.to(DEV), gk.to(DEV)))
    rows = dict(rtol=1e-4, atol=1e-5) if dtype == torch.float32 else dict(rtol=1e-2, atol=1e-2)
    for got, w in zip(out, want):
        torch.testing.assert_close(got.cpu(), w.detach(), rtol=1e-5, atol=1e-5)
    for got, w in zip(grads[:2], ref[:2]):
        torch.testing.assert_close(got.float().cpu(), w.grad, **rows)
    for got, w in zip(grads[2:], ref[2:]):
        torch.testing.assert_close(got.cpu(), w.grad, rtol=1e-4, atol=1e-4 * max(1.0, float(w.grad.abs().max())))
