"""The native host path (csrc/ae_host.cpp): what it refuses, and what its autograd nodes owe to the rest of PyTorch."""
import math

import pytest
import torch

import helpers
from attentionengine_b200 import runtime as rt

pytestmark = pytest.mark.gpu


def _mla(B, H, S, dtype=torch.float16):
    return helpers.mla_engine(B, H, S, dtype, 1 / math.sqrt(192))


@pytest.mark.parametrize("B,H,S", [(2, 16, 0), (0, 16, 128), (2, 0, 128)])
def test_mla_of_an_empty_problem_raises(B, H, S):
    """An empty cache must cost a serving loop one request, not its process (the cut into intervals divides by S)."""
    eng = _mla(2, 16, 128)
    args = [torch.zeros(s, dtype=torch.float16, device="cuda") for s in ((B, 1, H, 512), (B, 1, H, 64), (B, S, 1, 512), (B, S, 1, 64))]
    with pytest.raises(rt.AeError, match="empty"):
        eng(*args)
