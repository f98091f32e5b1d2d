"""MLA decode's way out: whole rows and partials through a staging tile, the merge with one head per thread and with four."""
import math

import pytest
import torch

import parity
from attentionengine_b200 import examples as helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,S", [(3, 100, 700), (24, 100, 300), (130, 36, 200), (1, 5, 1)])
def test_mla_outputs_and_merge_at_odd_head_counts(B, H, S):
    g = torch.Generator(device="cuda").manual_seed(B)
    q, qp, kv, kp = (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float16) for shape in
                     ((B, 1, H, 512), (B, 1, H, 64), (B, S, 1, 512), (B, S, 1, 64)))
    scale = 1 / math.sqrt(192)
    eng = helpers.mla_engine(B, H, S, torch.float16, scale)
    o = eng(q, qp, kv, kp)
    eng.check_status()
    s = (torch.einsum("bqhd,bkd->bhqk", q.float(), kv[:, :, 0].float()) + torch.einsum("bqhd,bkd->bhqk", qp.float(), kp[:, :, 0].float())) * scale
    parity.check("o", o, torch.einsum("bhqk,bkd->bqhd", torch.softmax(s, -1), kv[:, :, 0].float()), torch.float16)
