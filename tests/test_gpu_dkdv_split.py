"""dk / dv of calls with few key blocks, whose query tiles are shared by the CTAs of a cluster: ragged ends, parts without a tile
of their own, key blocks no query sees, every operand width.  Against the fp32 CPU oracle on the rounded inputs, with the
bounds of the other 16-bit tests: 2e-2 plus half an ulp of the element; 1e-2 of the largest entry for the phase gradients."""
import pytest
import torch

from oracle import pope_oracle as O
from pope_pytorch_b200 import PoPE, _native, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("b,h,hk,nq,nk,d,r,causal,masked,dtype", [
    (1, 4, 1, 512, 512, 64, 64, True, False, torch.bfloat16),      # four CTAs a block, one head each
    (3, 8, 2, 777, 777, 64, 32, True, True, torch.float16),        # ragged, padded, grouped
    (1, 4, 1, 130, 130, 128, 128, True, False, torch.bfloat16),    # widest operands
    (1, 2, 1, 129, 129, 64, 64, True, False, torch.bfloat16),      # the last block has one tile per head
    (1, 4, 1, 200, 900, 128, 64, True, False, torch.float16),      # key blocks behind the last query
    (1, 6, 2, 257, 300, 96, 48, False, True, torch.bfloat16),      # six chunks of columns on two CTAs ...
    (1, 4, 1, 600, 600, 96, 96, False, False, torch.float16),      # ... and on four
    (2, 4, 2, 64, 512, 64, 0, False, False, torch.bfloat16),       # nothing rotated, one query tile per head
    (1, 5, 1, 64, 64, 64, 16, True, True, torch.float16),          # five tiles on four CTAs
])
def test_shared_key_blocks_match_the_oracle(b, h, hk, nq, nk, d, r, causal, masked, dtype):
    g = torch.Generator().manual_seed(nq + nk + d + r)
    q, k, v, do = (torch.randn(s, generator=g).to(dtype) for s in ((b, h, nq, d), (b, hk, nk, d), (b, hk, nk, d), (b, h, nq, d)))
    freqs, bias = PoPE(max(r, 1), heads=hk)(nk).freqs[:, :r], -torch.rand(hk, r, generator=g) * 6
    mask = torch.rand(b, nk, generator=g) > 0.3 if masked else None
    ref = O.attention_with_grads(q.float(), k.float(), v.float(), freqs, bias, do.float(), mask=mask, causal=causal, want_dfreqs=True)
    ins = [t.to(DEV).requires_grad_(True) for t in (q, k, v, freqs.contiguous(), bias)]
    out = flash_attn_with_pope(*ins[:3], pos_emb=tuple(ins[3:]), mask=None if mask is None else mask.to(DEV), causal=causal)
    grads = torch.autograd.grad(out, ins, do.to(DEV))
    assert _native.last_path() == "tcgen05" and _native.device_status() == 0
    half_ulp = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    for name, got in zip(("dq", "dk", "dv"), grads):
        want = ref[name]
        assert float(((got.float().cpu() - want).abs() - half_ulp * want.abs()).max()) <= 2e-2, name
    for name, got in zip(("dfreqs", "dbias"), grads[3:]) if r else ():
        want = ref[name]
        assert float((got.cpu() - want).abs().max()) <= 1e-2 * max(1.0, float(want.abs().max())), name
