"""What stands around the operators: forward mode is refused and not dropped, a ``torch.jit.trace`` recording serves other inputs,
function transforms reach the embedding modules.  (No arithmetic is compared across kernels here: results are equal bit for bit,
or, where gradients are summed by atomics, to the last few bits.)"""
import pytest
import torch
import torch.autograd.forward_ad as fwad

from pope_pytorch_b200 import AxialPoPE, PoPE, apply_pope_to_qk, compute_attn_similarity, flash_attn_with_pope

pytestmark = pytest.mark.gpu
DEV = "cuda"


def tensors(n=96, dtype=torch.float32, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(1, 2, n, 64, generator=g, device=DEV, dtype=dtype) for _ in range(3)]


OPS = {
    "flash": lambda emb, q, k, v: flash_attn_with_pope(q, k, v, pos_emb=emb, causal=True),
    "sim": lambda emb, q, k, v: compute_attn_similarity(q, k, emb),
    "apply": lambda emb, q, k, v: torch.cat(apply_pope_to_qk(emb, q, k)),
}


@pytest.mark.parametrize("op", OPS)
def test_forward_mode_is_refused(op):
    q, k, v = tensors()
    emb = tuple(t.detach() for t in PoPE(32, heads=2).to(DEV)(96))
    with fwad.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        OPS[op](emb, fwad.make_dual(q, torch.ones_like(q)), k, v)


@pytest.mark.parametrize("op", ["flash", "apply"])   # (compute_attn_similarity checks sizes in ways a recording refuses)
def test_a_recording_serves_other_inputs(op):
    emb = tuple(t.detach() for t in PoPE(32, heads=2).to(DEV)(96))
    traced = torch.jit.trace(lambda q, k, v: OPS[op](emb, q, k, v), tuple(tensors()), check_trace=False)
    others = tensors(seed=1)
    assert torch.equal(traced(*others), OPS[op](emb, *others))
    ins = [t.requires_grad_(True) for t in others[:2]]
    want = torch.autograd.grad(OPS[op](emb, *others).sum(), ins)
    got = torch.autograd.grad(traced(*others).sum(), ins)
    for a, b in zip(got, want):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("module,arg", [(PoPE(32, heads=2), 96), (AxialPoPE(32, heads=2, axial_dims=(16, 16)), (8, 12))])
def test_function_transforms_reach_the_modules(module, arg):
    module = module.to(DEV)
    params = dict(module.named_parameters())

    def loss(p):
        return torch.func.functional_call(module, p, (arg,)).bias.square().sum()

    got = torch.func.grad(loss)(params)["bias"]
    assert torch.equal(got, 2 * module.bias.detach().clamp(-2 * torch.pi, 0) * ((module.bias >= -2 * torch.pi) & (module.bias <= 0)))
    with fwad.dual_level():
        dual = fwad.make_dual(module.bias.detach(), torch.ones_like(module.bias))
        out = torch.func.functional_call(module, {"bias": dual}, (arg,))
        assert fwad.unpack_dual(out.bias).tangent is not None
