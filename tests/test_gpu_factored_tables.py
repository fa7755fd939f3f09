"""Which of the two the kernels read, the table or the factors riding on it: factors that disagree with the values show it."""
import pytest
import torch

from pope_pytorch_b200 import PoPE, _native, compute_attn_similarity, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"
N, R = 1024, 32


@pytest.mark.parametrize("usable", [True, False])
def test_usable_factors_are_read_in_place_of_the_table(usable):
    g = torch.Generator(DEV).manual_seed(1)
    q, k, v = (torch.randn(1, 4, N, 64, generator=g, device=DEV).bfloat16() for _ in range(3))
    emb = PoPE(R, heads=4).to(DEV)(N)
    table, bias = emb.freqs.detach().clone(), emb.bias.detach() - 1
    other = (emb.positions * 2)[:, None] * emb.inv_freqs       # what the attached factors stand for
    mixed = table.clone()
    mixed._pope_factored = (emb.positions * 2, emb.inv_freqs if usable else emb.inv_freqs.double(), None)
    assert (_native._factors_of(mixed) is not None) == usable
    for call in (lambda t: flash_attn_with_pope(q, k, v, pos_emb=(t, bias), causal=True),
                 lambda t: compute_attn_similarity(q.float(), k.float(), (t, bias))):
        got, of_table, of_factors = call(mixed), call(table), call(other)
        assert torch.equal(got, of_factors if usable else of_table) and not torch.equal(of_factors, of_table)


def test_captured_behind_a_fill():
    """Graphs in which a fill is the node directly in front of the library's first kernel."""
    g = torch.Generator(DEV).manual_seed(2)
    q, k = (torch.randn(1, 4, 256, 64, generator=g, device=DEV) for _ in range(2))
    dsim = torch.randn(1, 4, 256, 256, generator=g, device=DEV)
    freqs, bias = PoPE(R, heads=4).to(DEV)(256).freqs, -torch.rand(4, R, generator=g, device=DEV)

    def gradients():   # (the bias gradient is zero-filled just before the launch)
        return _native.sim_backward(dsim, q, k, freqs, bias, False, True)

    def decode():
        keys = torch.empty(1, 4, 256, 64, dtype=torch.bfloat16, device=DEV).fill_(0.5)
        return (flash_attn_with_pope(q[:, :, :1].bfloat16(), keys, keys, pos_emb=(freqs, bias)),)

    for call in (gradients, decode):
        want = [t.clone() for t in call() if t is not None]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = [t for t in call() if t is not None]
        for _ in range(20):
            graph.replay()
            torch.cuda.synchronize()
            for a, b in zip(got, want):
                torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5 * float(b.abs().max()))
