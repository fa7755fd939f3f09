"""fp32 attention with features far below zero, whose magnitudes softplus(x) = e^x have squares outside fp32: the gradients keep
their relative accuracy.  Bound: rtol 1e-4 (expm1, hypot and the division at 1e-7 each; the sums that come before, of 64 terms
and more, at 1e-6 of their largest term, which is what the absolute part scales with, element by element with sigmoid(x))."""
import pytest
import torch
import torch.nn.functional as F

from pope_pytorch_b200 import _native, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("low", [-30.0, -50.0, -70.0])
def test_gradients_of_tiny_magnitudes(low):
    n, d, r = 96, 32, 16
    g = torch.Generator(DEV).manual_seed(int(-low))
    q, k, v, do = (torch.randn(1, 2, n, d, generator=g, device=DEV) for _ in range(4))
    q[..., :r:2] += low
    k[..., 1:r:2] += low
    freqs, bias = torch.rand(n, r, generator=g, device=DEV) * 6, -6 * torch.rand(2, r, generator=g, device=DEV)
    ins = [t.requires_grad_(True) for t in (q, k, v)]
    got = torch.autograd.grad(flash_attn_with_pope(*ins, pos_emb=(freqs, bias)), ins, do)
    assert _native.last_path() == "simt" and _native.device_status() == 0
    r64 = [t.detach().double().requires_grad_(True) for t in (q, k, v)]

    def polar(x, phase):
        a = F.softplus(x[..., :r])
        return torch.cat((a * phase.cos(), x[..., r:], a * phase.sin()), -1)

    p = (polar(r64[0], freqs.double()) @ polar(r64[1], (freqs + bias[:, None]).double()).mT * d ** -0.5).softmax(-1)
    want = torch.autograd.grad(p @ r64[2], r64, do.double())
    for x, w, raw in zip(got, want, (q, k, None)):
        scale = torch.ones_like(w) if raw is None else torch.cat((raw[..., :r].double().sigmoid(), torch.ones_like(w[..., r:])), -1)
        size = float((w / scale).abs().max())
        assert bool(((x - w).abs() <= 1e-4 * w.abs() + 1e-5 * size * scale).all())
