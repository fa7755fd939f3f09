"""The tiled exact-arithmetic attention at the edges of its 64 x 64 tiles, its feature widths and its cluster splits, against
the fp32 CPU oracle: rtol 1e-3 plus 1e-4 of the largest entry, the bound of the other fp32 tests (sums of up to a few hundred
fp32 products on either side differ by 1e-6 relative; the phases reach hundreds of radians, where an fp32 phase is good to
2^-16)."""
import pytest
import torch

from oracle import pope_oracle as O
from pope_pytorch_b200 import PoPE, _native, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("b,h,hk,nq,nk,d,r,causal,masked", [
    (1, 1, 1, 32, 32, 8, 3, True, False),          # half a tile, odd rotate dim
    (2, 2, 2, 63, 65, 33, 33, False, True),        # ragged rows and features
    (1, 4, 2, 64, 64, 64, 64, True, False),        # exactly one tile, grouped heads
    (1, 2, 1, 65, 200, 64, 32, False, True),       # bottom-right positions
    (1, 8, 8, 300, 300, 32, 16, True, True),       # streams cut over clusters
    (3, 6, 2, 130, 257, 128, 64, False, False),    # wide accumulators
    (1, 2, 2, 129, 129, 128, 128, True, True),     # widest operands
    (8, 16, 16, 190, 190, 48, 16, True, False),    # more tiles than SMs: no split
])
def test_tiles_match_the_oracle(b, h, hk, nq, nk, d, r, causal, masked):
    g = torch.Generator().manual_seed(nq + nk + d + r)
    q, k, v, do = (torch.randn(s, generator=g) for s in ((b, h, nq, d), (b, hk, nk, d), (b, hk, nk, d), (b, h, nq, d)))
    freqs, bias = PoPE(r, heads=hk)(nk).freqs, -torch.rand(hk, r, generator=g) * 6
    mask = None
    if masked:
        mask = torch.rand(b, nk, generator=g) > 0.4
        mask[0, 0] = not causal                # with the causal mask: a first row without any visible key
    ref = O.attention_with_grads(q, k, v, freqs, bias, do, mask=mask, causal=causal, want_dfreqs=True)
    ins = [t.to(DEV).requires_grad_(True) for t in (q, k, v, freqs, bias)]
    out = flash_attn_with_pope(*ins[:3], pos_emb=tuple(ins[3:]), mask=None if mask is None else mask.to(DEV), causal=causal)
    grads = torch.autograd.grad(out, ins, do.to(DEV))
    assert _native.device_status() == 0
    for name, got in zip(("out", "dq", "dk", "dv", "dfreqs", "dbias"), (out, *grads)):
        want = ref[name]
        err = (got.detach().cpu() - want).abs() - 1e-3 * want.abs()
        assert float(err.max()) <= 1e-4 * max(1.0, float(want.abs().max())), name
