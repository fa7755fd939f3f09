"""Calls whose inputs are written by the kernel just before them, one call after the other without a wait.  The first kernel of
a call may already be on the GPU while that kernel still runs; what it reads must be what was written.  Every result is compared,
on the GPU, with that of the same inputs handed over after a synchronisation: to the bit, or, where atomics sum (gradients of the
phases: their order differs from run to run), to 2^-12 of the largest entry."""
import pytest
import torch

from pope_pytorch_b200 import PagedKVCache, PoPE, _native, apply_pope_to_qk, compute_attn_similarity, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"
VARIANTS = 3


def rand(g, dtype, *shape):
    return torch.randn(*shape, generator=g, device=DEV).to(dtype)


class Call:
    """``ins``: the tensors that are rewritten, ``pool``: what with, ``run``: outputs (exact ones, summed ones)."""

    def __init__(self, shapes, dtype, run, seed, more=()):
        g = torch.Generator(DEV).manual_seed(seed)
        kinds = [(lambda s=s: rand(g, dtype, *s)) for s in shapes] + [(lambda f=f: f(g)) for f in more]
        self.pool = [[make() for make in kinds] for _ in range(VARIANTS)]
        self.ins = [t.clone() for t in self.pool[0]]
        self.run = run

    def write(self, variant, first):
        with torch.no_grad():   # (another input is the last one written each time)
            for i in range(len(self.ins)):
                j = (first + i) % len(self.ins)
                self.ins[j].copy_(self.pool[variant][j])


def phases(n, r):
    return torch.arange(n, device=DEV)[:, None] * 10000.0 ** -(torch.arange(r, device=DEV) / r) if r else torch.empty(n, 0, device=DEV)


def bias_of(hk, r):
    return lambda g: -6 * torch.rand(hk, r, generator=g, device=DEV)


def attention(b, h, hk, nq, nk, d, r, dtype, grad, seed, causal=False, masked=False):
    freqs = phases(nk, r)
    more = [bias_of(hk, r)] + ([lambda g: torch.rand(b, nk, generator=g, device=DEV) > 0.3] if masked else [])

    def run(ins):
        q, k, v, do, bias = ins[:5]
        leaves = [t.detach().requires_grad_(grad) for t in (q, k, v, bias)]
        out = flash_attn_with_pope(*leaves[:3], pos_emb=(freqs, leaves[3]), mask=ins[5] if masked else None, causal=causal)
        if not grad:
            return [out], []
        dq, dk, dv, *db = torch.autograd.grad(out, leaves if r else leaves[:3], do)
        return [out.detach(), dq, dk, dv], db

    return Call([(b, h, nq, d), (b, hk, nk, d), (b, hk, nk, d), (b, h, nq, d)], dtype, run, seed, more)


def similarity(b, h, n, d, r, dtype, grad, seed):
    module = PoPE(r, heads=h).to(DEV)

    def run(ins):
        q, k, ds, bias = ins
        leaves = [t.detach().requires_grad_(grad) for t in (q, k, bias)]
        emb = torch.func.functional_call(module, {"bias": leaves[2]}, (n,))   # table, similarity, its backward, clamp: one chain
        sim = compute_attn_similarity(leaves[0], leaves[1], emb)
        if not grad:
            return [sim], []
        dq, dk, db = torch.autograd.grad(sim, leaves, ds)
        return [sim.detach(), dq, dk], [db]

    return Call([(b, h, n, d), (b, h, n, d), (b, h, n, n)], dtype, run, seed, [bias_of(h, r)])


def transform(b, h, n, d, r, dtype, seed):
    freqs = phases(n, r)

    def run(ins):
        leaves = [t.detach().requires_grad_(True) for t in (ins[0], ins[1], ins[4])]
        out = apply_pope_to_qk((freqs, leaves[2]), leaves[0], leaves[1])
        dq, dk, db = torch.autograd.grad(out, leaves, (ins[2].float(), ins[3].float()))
        return [*(t.detach() for t in out), dq, dk], [db]

    return Call([(b, h, n, d), (b, h, n, d), (b, h, n, d + r), (b, h, n, d + r)], dtype, run, seed, [bias_of(h, r)])


def generate(b, h, hk, n, d, r, seed):
    freqs, page = phases(n + 2, r), 64
    cache = PagedKVCache(b, hk, d, num_pages=b * (-(-(n + 2) // page)), page_size=page, max_seq_len=n + 2, device=DEV)

    def run(ins):
        q, k, v, k1, v1, bias = ins
        outs = []
        for row in range(b):
            cache.release(row)
        cache.append(k, v)
        for _ in range(2):
            cache.append(k1, v1)
            outs.append(cache.decode(q, (freqs, bias)))
        return outs, []

    return Call([(b, h, 1, d), (b, hk, n, d), (b, hk, n, d), (b, hk, 1, d), (b, hk, 1, d)], torch.bfloat16, run, seed, [bias_of(hk, r)])


BF16, FP16, FP32 = torch.bfloat16, torch.float16, torch.float32
CALLS = {
    "similarity": lambda: similarity(1, 8, 1024, 64, 64, FP32, False, 1),
    "similarity_long_with_gradients": lambda: similarity(1, 8, 4096, 64, 64, FP32, True, 2),
    "similarity_bf16": lambda: similarity(1, 4, 640, 64, 32, BF16, False, 3),
    "attention_fp32": lambda: attention(1, 4, 4, 300, 300, 64, 64, FP32, True, 4, causal=True, masked=True),
    "attention_bf16": lambda: attention(2, 8, 8, 1024, 1024, 64, 32, BF16, False, 5, causal=True, masked=True),
    "attention_bf16_with_gradients": lambda: attention(3, 8, 2, 777, 777, 64, 32, FP16, True, 6, causal=True),
    "attention_plain": lambda: attention(1, 4, 4, 512, 512, 96, 0, BF16, False, 7),
    "decode_short": lambda: attention(2, 16, 4, 1, 777, 128, 64, BF16, False, 8, masked=True),
    "decode_long": lambda: attention(2, 16, 16, 1, 9000, 128, 64, BF16, False, 9),
    "decode_plain": lambda: attention(2, 16, 4, 1, 9000, 128, 0, BF16, False, 10),
    "generate": lambda: generate(2, 8, 2, 3000, 128, 64, 11),
    "transform": lambda: transform(2, 4, 500, 64, 32, BF16, 12),
}


@pytest.mark.parametrize("name", CALLS)
def test_results_do_not_depend_on_what_runs_just_before(name):
    call = CALLS[name]()
    want = []
    for variant in range(VARIANTS):
        call.write(variant, 0)
        torch.cuda.synchronize()
        exact, summed = call.run(call.ins)
        torch.cuda.synchronize()
        want.append(([t.clone() for t in exact], [t.clone() for t in summed]))
    differing = torch.zeros((), dtype=torch.int64, device=DEV)
    for i in range(150):
        variant = (i * i + i // 3) % VARIANTS
        call.write(variant, i)
        exact, summed = call.run(call.ins)
        if i % 2:      # every other call has the next one's writes right behind it
            continue
        for got, w in zip(exact, want[variant][0], strict=True):
            differing += (got != w).sum()
        for got, w in zip(summed, want[variant][1], strict=True):
            differing += ((got - w).abs() > 2.0 ** -12 * w.abs().max()).sum()
    assert int(differing) == 0 and _native.device_status() == 0


def test_clamp_gradient_behind_its_producer():
    module = PoPE(64, heads=16).to(DEV)
    with torch.no_grad():
        module.bias.uniform_(-9.0, 2.0, generator=torch.Generator(DEV).manual_seed(0))
    inside = (module.bias >= -2 * torch.pi) & (module.bias <= 0)
    w = torch.empty_like(module.bias)
    differing = torch.zeros((), dtype=torch.int64, device=DEV)
    for i in range(300):
        bias = module(64).bias
        w.fill_(float(i + 1))
        got, = torch.autograd.grad(bias, module.bias, w)
        differing += (got != torch.where(inside, float(i + 1), 0.0)).sum()
    assert int(differing) == 0


@pytest.mark.parametrize("name,calls", [("decode_long", 4000), ("attention_fp32", 1500), ("attention_bf16_with_gradients", 1500)])
def test_repeated_calls_are_equal(name, calls):
    """A ring buffer that is refilled before its last bytes have been read shows in one call of hundreds."""
    call = CALLS[name]()
    first = [t.clone() for t in call.run(call.ins)[0]]
    differing = torch.zeros((), dtype=torch.int64, device=DEV)
    for _ in range(calls):
        for got, w in zip(call.run(call.ins)[0], first, strict=True):
            differing += (got != w).sum()
    assert int(differing) == 0 and _native.device_status() == 0
