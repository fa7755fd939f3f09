"""The similarity backward sums its even and its odd steps in two accumulators: sweeps of one, two, three and many steps, operands
up to the accumulators' full width, repeated calls equal to the bit.

Bound against 64 bits: an operand kept as two bf16 numbers is off by 2^-17 of itself at most, a product loses lo * lo' on top
(2^-18) and cosine, sine and softplus are good to 1e-6: 2e-5 of the result's 2-norm.  (Key phases are rounded to fp32 by
definition, fl(f + b), and so they are in the reference here.  The rows of the gradient lie on 16 bytes, as these kernels ask.)"""
import pytest
import torch
import torch.nn.functional as F

from pope_pytorch_b200 import _native, compute_attn_similarity

pytestmark = pytest.mark.gpu
DEV = "cuda"


def in_64_bits(q, k, freqs, bias, dsim):
    r = freqs.shape[-1]
    q64, k64 = q.double().requires_grad_(True), k.double().requires_grad_(True)
    phase = (freqs + bias[:, None]).double().requires_grad_(True)   # (hk, n, r); its gradient is the bias gradient, row by row

    def polar(x, ph):
        a = F.softplus(x[..., :r])
        return torch.cat((a * ph.cos(), x[..., r:], a * ph.sin()), -1)

    qe, ke = polar(q64, freqs[-q.shape[2]:].double()), polar(k64, phase[None])
    ke = ke.repeat(1, q.shape[1] // k.shape[1], 1, 1)
    dq, dk, dphase = torch.autograd.grad(qe @ ke.mT, (q64, k64, phase), dsim.double())
    return dq, dk, dphase.sum(1)


@pytest.mark.parametrize("b,h,hk,nq,nk,d,r,repeats", [
    (1, 1, 1, 3, 4, 64, 64, 2),            # one step on either side: the second accumulator is never written
    (1, 2, 1, 64, 68, 64, 32, 4),          # one step per head of a group, two in all; two steps, the second of four keys
    (2, 3, 3, 130, 192, 32, 32, 4),        # three steps
    (1, 2, 2, 200, 300, 128, 0, 4),        # the widest operands: all of them plain ...
    (1, 4, 2, 300, 300, 80, 48, 4),        # ... and partly rotated
    (1, 8, 8, 4096, 4096, 64, 64, 100),    # a long training step
])
def test_two_accumulators(b, h, hk, nq, nk, d, r, repeats):
    g = torch.Generator(DEV).manual_seed(nq + nk + d + r)
    q, k, dsim = (torch.randn(s, generator=g, device=DEV) for s in ((b, h, nq, d), (b, hk, nk, d), (b, h, nq, nk)))
    freqs = torch.arange(nk, device=DEV)[:, None] * 10000.0 ** -(torch.arange(r, device=DEV) / r)
    bias = -6 * torch.rand(hk, r, generator=g, device=DEV)
    got = _native.sim_backward(dsim, q, k, freqs, bias, False, True)
    assert _native.last_path() == "tcgen05" and _native.device_status() == 0
    dq, dk, db = in_64_bits(q, k, freqs, bias, dsim)
    for x, want in ((got[0], dq), (got[1], dk)):
        assert float((x - want).norm()) <= 2e-5 * float(want.norm())
    for _ in range(repeats):
        again = _native.sim_backward(dsim, q, k, freqs, bias, False, True)
        assert torch.equal(again[0], got[0]) and torch.equal(again[1], got[1])
    sim = compute_attn_similarity(q, k, (freqs, bias)) if d in (32, 48, 64, 128) else None
    for _ in range(repeats if sim is not None else 0):
        assert torch.equal(compute_attn_similarity(q, k, (freqs, bias)), sim)


def test_thousands_of_calls_are_equal():
    """A staging buffer that was refilled before its last bytes had been read gave single wrong rows of dq in one call of 600."""
    g = torch.Generator(DEV).manual_seed(5)
    q, k, dsim = (torch.randn(s, generator=g, device=DEV) for s in ((1, 8, 4096, 64), (1, 8, 4096, 64), (1, 8, 4096, 4096)))
    freqs = torch.arange(4096, device=DEV)[:, None] * 10000.0 ** -(torch.arange(64, device=DEV) / 64)
    bias = -6 * torch.rand(8, 64, generator=g, device=DEV)
    first = _native.sim_backward(dsim, q, k, freqs, bias, False, False)
    wrong = torch.zeros((), dtype=torch.int64, device=DEV)
    for _ in range(6000):
        dq, dk = _native.sim_backward(dsim, q, k, freqs, bias, False, False)[:2]
        wrong += (dq != first[0]).sum() + (dk != first[1]).sum()
    assert int(wrong) == 0 and _native.device_status() == 0
