"""Grid lengths that are no Python integers: torch.arange takes them, so the module does."""
import numpy as np
import pytest
import torch

from pope_pytorch_b200 import AxialPoPE

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("where", [(8.0, 6), (2.5, 6), (np.int64(3), 6), (torch.tensor(4), torch.tensor(2.5)), (True, 6)])
def test_lengths_as_torch_takes_them(where):
    m = AxialPoPE(12, heads=2, axial_dims=(4, 8)).to(DEV)
    got, want = m(where), m._forward_torch(where)
    assert torch.equal(got.freqs, want.freqs) and torch.equal(got.bias, want.bias)
