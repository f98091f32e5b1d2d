"""One schedule handed to several decode engines, as layers with other head counts share the lengths of a step."""
import math

import pytest
import torch

import parity
from attentionengine_b200 import examples as helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Sq,Hq,Hkv", [
    (1, 150, 1),   # more than 128 rows per head unit: no kernel for intervals
    (1, 32, 32),   # four times the head units that the intervals were counted for
    (1, 8, 2),
])
def test_schedule_of_another_engine(Sq, Hq, Hkv):
    lens, D, dtype = [8192, 130, 5000, 7000], 128, torch.float16
    B, S = len(lens), max(lens)
    meta = helpers.decode_engine(B, 32, 8, 1, S, D, dtype).decode_schedule(torch.tensor(lens), device="cuda")
    assert meta["intervals"] > 0
    eng = helpers.decode_engine(B, Hq, Hkv, Sq, S, D, dtype)
    g = torch.Generator(device="cuda").manual_seed(Hq)
    q, k, v = (torch.randn(B, n, h, D, generator=g, device="cuda", dtype=dtype) for n, h in ((Sq, Hq), (S, Hkv), (S, Hkv)))
    lengths = torch.tensor(lens, device="cuda")
    o = eng.decode_varlen(q, k, v, lengths, metadata=meta)
    eng.check_status()
    assert eng._decode.last_num_split == meta["n_slots"] / B  # the work list
    kf, vf = (t.float().repeat_interleave(Hq // Hkv, dim=2) for t in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), kf) / math.sqrt(D)
    keep = torch.arange(S, device="cuda")[None, :] < lengths[:, None]
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s.masked_fill(~keep[:, None, None], float("-inf")), -1), vf)
    parity.check("o", o, ref, dtype, stages=2)  # P and the stored O


def test_waves_are_honoured_and_the_count_is_of_the_path_taken():
    lens, D, dtype = [8192, 130, 5000, 7000], 128, torch.float16
    B, S = len(lens), max(lens)
    eng = helpers.decode_engine(B, 32, 8, 1, S, D, dtype)
    q, k, v = (torch.randn(B, n, h, D, device="cuda", dtype=dtype) for n, h in ((1, 32), (S, 8), (S, 8)))
    lengths = torch.tensor(lens, device="cuda")
    cut, twice = eng.decode_schedule(lengths), eng._decode.schedule(lengths, waves=2)
    assert cut["intervals"] == 18 and twice["intervals"] == 0 and twice["n_slots"] > cut["n_slots"]
    eng.decode_varlen(q, k, v, lengths, metadata=cut)
    assert eng._decode.last_num_split == (B + 17) / B
    eng.decode_varlen(q, k, v, lengths, metadata=twice)
    assert eng._decode.last_num_split == twice["n_slots"] / B
