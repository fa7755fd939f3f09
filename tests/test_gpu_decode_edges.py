"""The decode kernel at the edges of its tiles, key ranges and head groups, against the exact-arithmetic family fed the same
16-bit inputs as fp32.  Bound: half an ulp of the 16-bit output (2^-9 |out| in bf16, 2^-12 in fp16), plus the phase table's
2^-12 per cosine and sine, which moves a score (|score| < 40 here) by at most 40 * 2^-11 = 0.02 and an output, a convex
combination of values with |v| < 4.5, by at most 2 * 0.02 * 4.5 = 0.18 in theory and by its random sum, a tenth of that, in fact."""
import pytest
import torch

from pope_pytorch_b200 import PoPE, _native, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("b,h,hk,nk,d,r,dtype,masked,seq_first", [
    (1, 1, 1, 1, 64, 64, torch.bfloat16, False, False),        # one key
    (2, 4, 1, 63, 128, 64, torch.float16, True, False),        # one partial tile, four heads per CTA
    (1, 4, 2, 64, 96, 48, torch.bfloat16, False, True),        # one whole tile, two heads per CTA, rows apart
    (3, 8, 1, 65, 64, 32, torch.bfloat16, True, False),        # a tile of one key, two blocks of four heads
    (1, 6, 2, 513, 128, 128, torch.float16, False, False),     # three heads per key head: one per CTA
    (2, 16, 4, 777, 128, 64, torch.bfloat16, True, True),      # cluster of eight, ragged tiles
    (16, 32, 8, 700, 128, 64, torch.bfloat16, True, False),    # several waves
    (1, 2, 2, 5000, 96, 96, torch.float16, False, False),      # 64 key ranges merged by the last CTA
    (1, 8, 2, 4099, 64, 0, torch.bfloat16, True, False),       # nothing rotated: counters zeroed by the call itself
    (9, 32, 32, 600, 128, 64, torch.bfloat16, False, False),   # one key range per unit
])
def test_decode_edges(b, h, hk, nk, d, r, dtype, masked, seq_first, monkeypatch):
    g = torch.Generator().manual_seed(nk + d + r)
    q, k, v = (torch.randn(s, generator=g).to(dtype).to(DEV) for s in ((b, h, 1, d), (b, hk, nk, d), (b, hk, nk, d)))
    emb = (PoPE(r, heads=hk)(nk).freqs.to(DEV), (-torch.rand(hk, r, generator=g) * 6).to(DEV)) if r else (
        torch.empty(nk, 0, device=DEV), torch.empty(hk, 0, device=DEV))
    mask = None
    if masked:
        mask = (torch.rand(b, nk, generator=g) > 0.3).to(DEV)
        mask[0] = False                      # an empty row
        k[-1, :, ~mask[-1]] = float("nan")   # what is masked is never touched
        v[-1, :, ~mask[-1]] = float("nan")
    ins = [t.transpose(1, 2).contiguous() for t in (q, k, v)] if seq_first else [q, k, v]
    out = flash_attn_with_pope(*ins, pos_emb=emb, mask=mask, head_dimension_at_first=not seq_first)
    assert _native.last_path() == "decode_stream" and _native.device_status() == 0
    out = out.transpose(1, 2) if seq_first else out
    monkeypatch.setenv("POPE_B200_FORCE_SIMT", "1")
    kc, vc = (torch.nan_to_num(t.float()) for t in (k, v))
    ref = flash_attn_with_pope(q.float(), kc, vc, pos_emb=emb, mask=mask)
    assert _native.last_path() == "simt"
    ulp = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert torch.all((out.float() - ref).abs() <= 2e-2 + ulp * ref.abs())
    if masked:
        assert torch.equal(out[0], torch.zeros_like(out[0]))
