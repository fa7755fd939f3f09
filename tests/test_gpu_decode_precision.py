"""A 16-bit decode below 1024 keys against 64 bits: nearly every output is the nearest 16-bit number to the exact result.  The
arithmetic in front of that rounding (approximate softplus, sine and cosine, 2^-21 each; fp32 sums) moves an output by about
2e-6 of its size, and the spacing of fp16 numbers is 2^-11 to 2^-10 of it: 0.4 to 0.8 % lie near enough to a midpoint to fall on the
other side.  Phases far from zero count too: the position phase of the query and the bias are taken one by one."""
import pytest
import torch
import torch.nn.functional as F

from pope_pytorch_b200 import _native, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("b,h,hk,n,d,r,offset", [(2, 16, 4, 777, 128, 64, 0), (4, 8, 8, 300, 64, 64, 0), (3, 12, 6, 1000, 96, 48, 0),
                                                 (2, 16, 4, 777, 128, 64, 200000)])
def test_short_decode_is_exact_to_the_rounding(b, h, hk, n, d, r, offset):
    g = torch.Generator(DEV).manual_seed(n + d)
    q, k, v = (torch.randn(*s, generator=g, device=DEV).half() for s in ((b, h, 1, d), (b, hk, n, d), (b, hk, n, d)))
    freqs = ((torch.arange(n, device=DEV) + offset)[:, None] * 10000.0 ** -(torch.arange(r, device=DEV) / r)).contiguous()
    bias = -6 * torch.rand(hk, r, generator=g, device=DEV)
    out = flash_attn_with_pope(q, k, v, pos_emb=(freqs, bias))
    assert _native.last_path() == "decode_stream"
    k64, v64 = (t.double().repeat(1, h // hk, 1, 1) for t in (k, v))
    phase = freqs[-1].double() - freqs.double()[None, None] - bias.double().repeat(h // hk, 1)[None, :, None]
    score = (F.softplus(q.double()[..., :r]) * F.softplus(k64[..., :r]) * phase.cos()).sum(-1) + (q.double()[..., r:] * k64[..., r:]).sum(-1)
    want = torch.einsum("bhj,bhjd->bhd", (score * d ** -0.5).softmax(-1), v64)[:, :, None]
    assert float((out != want.half()).double().mean()) <= 0.01
