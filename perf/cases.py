"""The work that programs have this package do, as cases that can be timed and compared.

A case is a plain dict; ``op`` names the call it makes through the public API:

  forward   flash_attn_with_pope without gradients (prefill, scoring, encoders); the phase table is at hand
  train     PoPE / AxialPoPE -> flash_attn_with_pope -> gradients of q, k, v and the learned phase bias
  decode    flash_attn_with_pope with one query row at the end of a contiguous key / value cache
  generate  PagedKVCache: admit prompts into freed slots, then append + decode token by token
  sim       compute_attn_similarity, forward alone or with the gradients of q, k and the phase bias
  rotate    apply_pope_to_qk with the gradients of q, k and the phase bias (attention done elsewhere)

``listed()`` holds one case for each kind of use; ``draw()`` gives others of the same ranges.  Where a program
trains, the embedding module runs inside the pass, because its bias changes with every step; where it serves, the
weights are fixed and the phase table is made once.
"""
import math

import torch

from pope_pytorch_b200 import (AxialPoPE, PagedKVCache, PoPE, apply_pope_to_qk, compute_attn_similarity,
                               flash_attn_with_pope)

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # Scoring a small batch of padded prompts: a call of a few tens of microseconds, latency and launches count.
        dict(name="forward_small", op="forward", b=2, h=8, hk=8, n=1024, d=64, r=32, dtype="bf16", causal=True, mask=True,
             seq_first=False),
        # Prefill of one long document, the share of one of eight GPUs of a batch of 8: the largest forward.
        dict(name="forward_long", op="forward", b=1, h=32, hk=32, n=32768, d=128, r=64, dtype="bf16", causal=True, mask=False,
             seq_first=False),
        # Fine-tuning step of a small model on padded sequences of an odd length, grouped key heads, (b, n, h, d) layout.
        dict(name="train_small_ragged", op="train", b=3, h=8, hk=2, n=777, d=64, r=32, dtype="fp16", causal=True, mask=True,
             seq_first=True, grid=""),
        # The training step of a language model.
        dict(name="train_large", op="train", b=4, h=16, hk=16, n=4096, d=128, r=128, dtype="bf16", causal=True, mask=False,
             seq_first=False, grid=""),
        # The training step of a video model: positions on a (frame, row, column) grid, every token sees every other.
        dict(name="train_video", op="train", b=2, h=8, hk=8, n=2048, d=96, r=96, dtype="bf16", causal=False, mask=False,
             seq_first=False, grid="8,16,16"),
        # Research code in the default type: fp32 tensors straight into the fused attention.
        dict(name="train_fp32", op="train", b=1, h=8, hk=8, n=1024, d=64, r=64, dtype="fp32", causal=True, mask=False,
             seq_first=False, grid=""),
        # A token of a short chat: a cache of a few hundred keys, padded, grouped key heads; nothing but latency.
        dict(name="decode_short", op="decode", b=2, h=16, hk=4, n=777, d=128, r=64, dtype="bf16", mask=True, seq_first=False),
        # A token against long caches: the key / value stream.
        dict(name="decode_long", op="decode", b=8, h=32, hk=32, n=32768, d=128, r=64, dtype="bf16", mask=False, seq_first=False),
        # A serving turn: four requests of different lengths are admitted and sixteen tokens of each generated.
        dict(name="generate", op="generate", b=4, h=32, hk=8, n=2000, d=128, r=64, dtype="bf16", page=256, steps=16),
        # The similarity matrix by itself, in fp32, for a caller's own softmax; small.
        dict(name="sim_small", op="sim", b=1, h=8, hk=8, nq=1024, nk=1024, d=64, r=64, dtype="fp32", grad=False),
        # The same with gradients over a long sequence: the matrix and its gradient are what moves.
        dict(name="sim_train", op="sim", b=1, h=8, hk=8, nq=4096, nk=4096, d=64, r=64, dtype="fp32", grad=True),
        # The embedding alone, in front of somebody else's attention.
        dict(name="rotate_train", op="rotate", b=4, h=16, hk=16, n=2048, d=64, r=32, dtype="bf16"),
    ]


# ---- more of the same ranges ------------------------------------------------------------------------------------

def _log_int(rng, lo, hi):
    """An integer of [lo, hi], even over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _heads(rng, most):
    hk = rng.choice([x for x in (1, 2, 4, 8, 16, 32) if x <= most])
    return min(most, hk * rng.choice([1, 1, 1, 2, 4])), hk


def draw(rng):
    op = rng.choice(["forward", "forward", "train", "train", "train", "decode", "generate", "sim", "sim", "rotate"])
    d = rng.choice([32, 64, 64, 96, 128, 128])
    r = rng.choice([d, d // 2])
    h, hk = _heads(rng, 32)
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    if op in ("forward", "train"):
        if rng.random() < 0.2:
            dtype = "fp32"
        # fp32 and narrow heads belong to small models; the others go to the listed sizes
        small = dtype == "fp32" or d == 32
        most = 5e10 if small else 3e12 if op == "forward" else 1.5e12
        case = dict(op=op, b=rng.choice([1, 2, 3, 4, 8]), h=h, hk=hk, n=_log_int(rng, 64, 2048 if small else 16384 if op == "forward" else 4096),
                    d=d, r=r, dtype=dtype, causal=rng.random() < 0.6, mask=rng.random() < 0.4, seq_first=rng.random() < 0.3)
        if op == "train":
            case["grid"] = ""
            if d == r and d % 3 == 0 and rng.random() < 0.7:
                f, y, x = rng.choice([2, 4, 8]), rng.choice([8, 12, 16]), rng.choice([8, 14, 16])
                case.update(grid="%d,%d,%d" % (f, y, x), n=f * y * x, causal=False)
        while work(case)["flops"] > most:
            case["b"], case["h"], case["hk"] = 1, max(1, case["h"] // 2), max(1, case["hk"] // 2)
            case["hk"] = math.gcd(case["h"], case["hk"])
            if case["h"] == 1:
                break
        return case
    if op == "decode":
        d = rng.choice([64, 96, 128, 128])
        case = dict(op=op, b=_log_int(rng, 1, 16), h=h, hk=hk, n=_log_int(rng, 128, 32768), d=d, r=rng.choice([d, d // 2]), dtype=dtype,
                    mask=rng.random() < 0.4, seq_first=rng.random() < 0.3)
        while work(case)["bytes"] > 4.3e9:
            case["b"] = max(1, case["b"] // 2)
        return case
    if op == "generate":
        d = rng.choice([64, 96, 128, 128])
        return dict(op=op, b=_log_int(rng, 1, 16), h=h, hk=min(hk, 8) if h % min(hk, 8) == 0 else hk, n=_log_int(rng, 64, 8192), d=d,
                    r=rng.choice([d, d // 2]), dtype=dtype, page=rng.choice([64, 128, 256]), steps=rng.randint(4, 24))
    if op == "sim":
        d = rng.choice([32, 64, 64, 128])
        nk = _log_int(rng, 128, 4096)
        h, hk = _heads(rng, 8)
        case = dict(op=op, b=rng.choice([1, 1, 2]), h=h, hk=hk, nq=nk if rng.random() < 0.7 else rng.randint(nk // 4, nk), nk=nk, d=d,
                    r=rng.choice([d, d // 2]), dtype=rng.choice(["fp32", "fp32", "fp32", "bf16"]), grad=rng.random() < 0.5)
        if case["b"] * h * case["nq"] * nk > 1 << 27:
            case["b"] = 1
        return case
    return dict(op=op, b=rng.choice([1, 2, 4]), h=h, hk=hk, n=_log_int(rng, 64, 4096), d=d, r=r, dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]))


# ---- inputs -----------------------------------------------------------------------------------------------------

def _embedding(case, heads, g):
    """A module whose learned per-head phases are spread over their whole range, as after training."""
    if case.get("grid"):
        m = AxialPoPE(case["r"], heads=heads, axial_dims=(case["r"] // 3,) * 3)
    else:
        m = PoPE(case["r"], heads=heads)
    m = m.to("cuda")
    with torch.no_grad():
        m.bias.uniform_(-2 * math.pi, 0.0, generator=g)
    return m


def _table(module, n):
    """What a serving program keeps: the phase table and the clamped phases of fixed weights."""
    with torch.no_grad():
        return module(n)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt, op, b, h, hk, d = DTYPES[case["dtype"]], case["op"], case["b"], case["h"], case["hk"], case["d"]

    def rand(*shape, dtype=dt, grad=False):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dtype).requires_grad_(grad)

    s = dict(case=case)
    if op in ("forward", "train", "decode"):
        n, nq, grad = case["n"], 1 if op == "decode" else case["n"], op == "train"
        shape = (lambda heads, rows: (b, rows, heads, d)) if case["seq_first"] else (lambda heads, rows: (b, heads, rows, d))
        s["q"], s["k"], s["v"] = rand(*shape(h, nq), grad=grad), rand(*shape(hk, n), grad=grad), rand(*shape(hk, n), grad=grad)
        s["mask"] = None
        if case["mask"]:   # right-padded sequences, each at least half full
            lens = torch.randint(n // 2, n + 1, (b, 1), generator=g, device="cuda")
            s["mask"] = torch.arange(n, device="cuda")[None, :] < lens
        s["pope"] = _embedding(case, hk, g)
        if grad:
            s["dout"] = rand(*shape(h, nq))
            s["where"] = tuple(int(x) for x in case["grid"].split(",")) if case["grid"] else n
        else:
            s["pos_emb"] = _table(s["pope"], n)
        s["how"] = dict(mask=s["mask"], causal=case.get("causal", False), head_dimension_at_first=not case["seq_first"])
    elif op == "generate":
        n, steps, page = case["n"], case["steps"], case["page"]
        lens = torch.randint(n // 2, n + 1, (b,), generator=g, device="cuda").tolist()
        longest = n + steps
        s["cache"] = PagedKVCache(b, hk, d, num_pages=b * -(-longest // page), page_size=page, max_seq_len=longest, dtype=dt, device="cuda")
        s["prompts"] = [(rand(hk, ln, d), rand(hk, ln, d)) for ln in lens]
        s["tokens"] = [(rand(b, h, 1, d), rand(b, hk, 1, d), rand(b, hk, 1, d)) for _ in range(steps)]
        s["pos_emb"] = _table(_embedding(case, hk, g), longest)
    elif op == "sim":
        grad = case["grad"]
        s["q"], s["k"] = rand(b, h, case["nq"], d, grad=grad), rand(b, hk, case["nk"], d, grad=grad)
        s["pope"] = _embedding(case, hk, g)
        if grad:
            s["dsim"] = rand(b, h, case["nq"], case["nk"])
        else:
            s["pos_emb"] = _table(s["pope"], case["nk"])
    else:
        n, r = case["n"], case["r"]
        s["q"], s["k"] = rand(b, h, n, d, grad=True), rand(b, hk, n, d, grad=True)
        s["pope"] = _embedding(case, hk, g)
        s["dq_out"], s["dk_out"] = rand(b, h, n, d + r, dtype=torch.float32), rand(b, hk, n, d + r, dtype=torch.float32)
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    op = case["op"]
    if op in ("forward", "decode"):
        with torch.no_grad():
            return flash_attn_with_pope(s["q"], s["k"], s["v"], pos_emb=s["pos_emb"], **s["how"])
    if op == "train":
        out = flash_attn_with_pope(s["q"], s["k"], s["v"], pos_emb=s["pope"](s["where"]), **s["how"])
        return (out, *torch.autograd.grad(out, (s["q"], s["k"], s["v"], s["pope"].bias), s["dout"]))
    if op == "generate":
        cache, outs = s["cache"], []
        with torch.no_grad():
            for slot, (k, v) in enumerate(s["prompts"]):
                cache.release(slot)
                cache.append_to(slot, k, v)
            for q, k, v in s["tokens"]:
                cache.append(k, v)
                outs.append(cache.decode(q, s["pos_emb"]))
        return outs
    if op == "sim":
        if not case["grad"]:
            with torch.no_grad():
                return compute_attn_similarity(s["q"], s["k"], s["pos_emb"])
        sim = compute_attn_similarity(s["q"], s["k"], s["pope"](case["nk"]))
        return (sim, *torch.autograd.grad(sim, (s["q"], s["k"], s["pope"].bias), s["dsim"]))
    q_out, k_out = apply_pope_to_qk(s["pope"](case["n"]), s["q"], s["k"])
    return (q_out, k_out, *torch.autograd.grad((q_out, k_out), (s["q"], s["k"], s["pope"].bias), (s["dq_out"], s["dk_out"])))


# ---- what a pass cannot do without ------------------------------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once; a multiply and an add for every product of the score matrix's visible
    entries (transcendental and elementwise work counts zero).  Padded sequences are three quarters full on average."""
    op, b, h, hk, d, r = (case[x] for x in ("op", "b", "h", "hk", "d", "r"))
    e = 4 if case["dtype"] == "fp32" else 2
    if op in ("forward", "train", "decode"):
        n, nq = case["n"], 1 if op == "decode" else case["n"]
        kept = 0.75 * n if case["mask"] else n
        pairs = b * h * (kept * n - kept * kept / 2 if case.get("causal") else nq * kept)
        q, kv, small = b * h * nq * d * e, b * hk * kept * d * e, 4 * n * r + 4 * hk * r + (b * n if case["mask"] else 0)
        if op != "train":
            return dict(bytes=2 * q + 2 * kv + small, flops=2 * pairs * (2 * d + r))
        kv_all = b * hk * n * d * e     # the gradients of padding are written too
        # forward q, k, v -> out; backward q, k, v, out, dout -> dq, dk, dv
        return dict(bytes=6 * q + 4 * kv + 2 * kv_all + small, flops=2 * pairs * ((2 * d + r) + (5 * d + 3 * r)))
    if op == "generate":
        prompt, steps = 0.75 * case["n"], case["steps"]
        row = b * hk * d * e * 2        # one cached position of every sequence, k and v
        read = sum(row * (prompt + t + 1) for t in range(steps))
        copied = 2 * row * (prompt + steps)
        return dict(bytes=read + copied + steps * 2 * b * h * d * e, flops=sum(2 * b * h * (prompt + t + 1) * (2 * d + r) for t in range(steps)))
    if op == "sim":
        nq, nk = case["nq"], case["nk"]
        qk, mat, small = (b * h * nq + b * hk * nk) * d * e, b * h * nq * nk * e, 4 * nk * r + 4 * hk * r
        flops = 2 * b * h * nq * nk * (d + r)
        if not case["grad"]:
            return dict(bytes=qk + mat + small, flops=flops)
        return dict(bytes=3 * qk + 2 * mat + 2 * small, flops=3 * flops)
    n = case["n"]
    rows = b * (h + hk) * n
    # forward q, k -> q', k'; backward q, k, dq', dk' -> dq, dk
    return dict(bytes=rows * (3 * d * e + 2 * (d + r) * 4) + 4 * n * r, flops=rows * d * 10)


def tolerance(case):
    """What the types give.  16-bit attention: operands and the probabilities are rounded to 16 bits, and so are the
    score gradients whose sum over all rows, with its cancellation, is the gradient of the phase bias.  fp32: sums of up
    to a few thousand products whose phases reach thousands of radians."""
    if case["dtype"] == "fp32":
        return {"rel": 3e-5}
    if case["op"] == "rotate":
        return {"rel": 3e-3}
    return {"rel": 2e-2 if case["op"] in ("train", "sim") and case.get("grad", True) else 1e-2}
