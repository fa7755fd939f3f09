"""Tensors that do not fit together are refused before a kernel sees their pointers: sizes, types, devices of every operand.  (Each
short tensor here is a view of a longer one and each host tensor is pinned, so that nothing could be read out of range even if
a check were missing.)  Tensors that reach further than is read are taken as before, with zero gradients beyond."""
import pytest
import torch

from pope_pytorch_b200 import PagedKVCache, _native, apply_pope_to_qk, compute_attn_similarity, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"
B, H, HK, N, D, R = 2, 4, 2, 96, 64, 32


def view(*shape, dtype=torch.float32):
    """A tensor inside a buffer that goes on for as much again in every direction, with room for a wider type."""
    return torch.randn(*(2 * s for s in shape[:-1]), 4 * shape[-1], device=DEV).to(dtype)[tuple(slice(0, s) for s in shape)]


def args(dtype=torch.float32, nq=N):
    return dict(q=view(B, H, nq, D, dtype=dtype), k=view(B, HK, N, D, dtype=dtype), v=view(B, HK, N, D, dtype=dtype), freqs=view(N, R),
                bias=view(HK, R), mask=view(B, N) > -1)


def attention(a):
    return flash_attn_with_pope(a["q"], a["k"], a["v"], pos_emb=(a["freqs"], a["bias"]), mask=a["mask"])


def similarity(a):
    return compute_attn_similarity(a["q"], a["k"], (a["freqs"], a["bias"]))


BOTH, ATTENTION = (attention, similarity), (attention,)
WRONG = {
    "k of fewer batch entries": (BOTH, lambda a: dict(k=a["k"][:1])),
    "k of fewer features": (BOTH, lambda a: dict(k=a["k"][..., :32])),
    "a table for fewer batch entries": (BOTH, lambda a: dict(q=view(3, H, N, D), k=view(3, HK, N, D), v=view(3, HK, N, D), mask=None, freqs=view(2, N, R))),
    "a table for fewer heads": (BOTH, lambda a: dict(freqs=view(1, HK, N, R))),
    "bias of fewer heads": (BOTH, lambda a: dict(bias=a["bias"][:1])),
    "bias of fewer features": (BOTH, lambda a: dict(bias=a["bias"][:, :16])),
    "bias without heads": (BOTH, lambda a: dict(bias=a["bias"][0])),
    "freqs on the host": (BOTH, lambda a: dict(freqs=a["freqs"].contiguous().cpu().pin_memory())),
    "bias on the host": (BOTH, lambda a: dict(bias=a["bias"].contiguous().cpu().pin_memory())),
    "v of another type": (ATTENTION, lambda a: dict(v=view(B, HK, N, D, dtype=torch.float16))),
    "v of fewer rows": (ATTENTION, lambda a: dict(v=a["v"][:, :, :95])),
    "v of fewer heads": (ATTENTION, lambda a: dict(v=a["v"][:, :1])),
    "v of fewer batch entries": (ATTENTION, lambda a: dict(v=a["v"][:1])),
    "v of fewer features": (ATTENTION, lambda a: dict(v=a["v"][..., :48])),
    "mask of fewer keys": (ATTENTION, lambda a: dict(mask=a["mask"][:, :95])),
    "mask of fewer batch entries": (ATTENTION, lambda a: dict(mask=a["mask"][:1])),
    "mask with a head axis": (ATTENTION, lambda a: dict(mask=a["mask"][:, None])),
    "mask on the host": (ATTENTION, lambda a: dict(mask=a["mask"].contiguous().cpu().pin_memory())),
}


@pytest.mark.parametrize("wrong", WRONG)
@pytest.mark.parametrize("dtype,nq", [(torch.float32, N), (torch.bfloat16, N), (torch.bfloat16, 1)])
def test_what_does_not_fit_is_refused(wrong, dtype, nq):
    calls, change = WRONG[wrong]
    a = args(dtype, nq)
    change = change(a)
    if "q" in change:
        change.update({name: change[name].to(dtype) for name in "qkv"}, q=change["q"][:, :, :nq].to(dtype))
    for call in calls:
        with pytest.raises((ValueError, TypeError, RuntimeError)):
            call({**a, **change})
    assert _native.device_status() == 0


def test_backward_and_cache_operands():
    a = args(torch.bfloat16)
    rest = (a["freqs"], a["bias"], None, False, 0.125)
    out, lse = _native.attn_forward(a["q"], a["k"], a["v"], *rest)
    good = dict(dout=out, q=a["q"], k=a["k"], v=a["v"], out=out, lse=lse)
    for wrong in (dict(dout=out[:1]), dict(dout=out.float()), dict(out=out[:, :2]), dict(lse=lse[:1]), dict(lse=lse.double())):
        with pytest.raises((ValueError, TypeError)):
            _native.attn_backward(*{**good, **wrong}.values(), *rest, False, False)
    with pytest.raises((ValueError, TypeError)):
        _native.sim_backward(view(B, H, N, N - 1), a["q"].float(), a["k"].float(), a["freqs"], a["bias"], False, False)
    cache = PagedKVCache(B, HK, D, num_pages=8, page_size=64, max_seq_len=128, device=DEV)
    cache.append(a["k"].contiguous(), a["v"].contiguous())
    for emb in ((a["freqs"], a["bias"][:1]), (a["freqs"].contiguous().cpu().pin_memory(), a["bias"]), (a["freqs"], a["bias"][:, :8])):
        with pytest.raises((ValueError, RuntimeError)):
            cache.decode(a["q"][:, :, :1], emb)
    assert _native.device_status() == 0


def test_what_reaches_further_is_read_in_part():
    a = args()
    want = attention({**a, **{n: a[n].contiguous() for n in ("q", "k", "v", "freqs", "bias", "mask")}})
    more = dict(k=torch.cat((a["k"], a["k"][:1])), v=torch.cat((a["v"], a["v"]), 2), bias=torch.cat((a["bias"], a["bias"])), mask=torch.cat((a["mask"], a["mask"]), 1))
    leaves = [t.detach().requires_grad_(True) for t in (a["q"], more["k"], more["v"])]
    out = flash_attn_with_pope(*leaves, pos_emb=(a["freqs"], more["bias"]), mask=more["mask"])
    assert torch.equal(out, want)
    dq, dk, dv = torch.autograd.grad(out, leaves, torch.ones_like(out))
    assert not dk[B:].any() and not dv[:, :, N:].any() and dk[:B].any() and dv[:, :, :N].any()


def test_the_transform_of_what_the_kernel_does_not_take():
    """Batch sizes of their own and a bias shared by the heads: the PyTorch operations, which broadcast."""
    q, k, freqs, bias = torch.randn(2, 4, 10, 16, device=DEV), torch.randn(1, 4, 12, 16, device=DEV), torch.rand(12, 8, device=DEV), -torch.rand(1, 8, device=DEV)
    qo, ko = apply_pope_to_qk((freqs, bias), q, k)
    q2, k2 = apply_pope_to_qk((freqs, bias.expand(4, 8).contiguous()), q, k.expand(2, 4, 12, 16).contiguous())
    torch.testing.assert_close(qo, q2, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(ko, k2[:1], rtol=1e-5, atol=1e-5)
