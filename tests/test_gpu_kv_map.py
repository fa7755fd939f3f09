"""Page-table and length updates that travel as kernel parameters: more entries than one launch carries, and a graph capture
whose first node is a fill in front of the library's kernels."""
import pytest
import torch

from pope_pytorch_b200 import PagedKVCache, PoPE, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [1, 64, 65, 8192 + 3, 20000])   # 20000 keys in 64-key pages: 313 entries per sequence
def test_table_and_lengths_follow_the_host(n):
    cache = PagedKVCache(2, 1, 64, num_pages=1300, page_size=64, max_seq_len=40000, device=DEV)
    k = torch.randn(2, 1, n, 64, device=DEV).bfloat16()
    cache.append(k, k)
    cache.append(k[:, :, :1], k[:, :, :1])
    for b in range(2):
        assert cache.page_table[b, :len(cache.alloc.table[b])].tolist() == cache.alloc.table[b]
        assert torch.equal(cache.gather(b)[0][:, :n], k[b]) and torch.equal(cache.gather(b)[1][:, n], k[b, :, 0])
    assert cache.seq_lens.tolist() == cache.lens == [n + 1, n + 1]
    cache.release(1)
    assert cache.seq_lens.tolist() == [n + 1, 0]


def test_capture_behind_a_fill():
    q, k = torch.randn(1, 4, 1, 64, device=DEV).bfloat16(), torch.randn(1, 4, 300, 64, device=DEV).bfloat16()
    emb = tuple(t.detach() for t in PoPE(32, heads=4).to(DEV)(300))
    want = flash_attn_with_pope(q, k, k, pos_emb=emb)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kk = torch.zeros_like(k)
        kk += k
        got = flash_attn_with_pope(q, kk, kk, pos_emb=emb)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
