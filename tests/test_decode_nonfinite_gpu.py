"""An infinity among the values of a key whose probability is 0 next to another split's: the merges of decode give what one pass over
all keys gives."""
import math

import pytest
import torch

from attentionengine_b200 import examples as helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["one split", "merge launch", "cluster", "intervals", "shares"])
def test_infinite_value_in_a_split_far_below_the_others(how, monkeypatch):
    B, Hq, Hkv, S, D, dtype = 2, 8, 2, 2000, 64, torch.float16
    eng = helpers.decode_engine(B, Hq, Hkv, 1, S, D, dtype)
    q = torch.zeros(B, 1, Hq, D, dtype=dtype, device="cuda")
    k = torch.zeros(B, S, Hkv, D, dtype=dtype, device="cuda")
    q[..., 0], k[:, 1900, :, 0] = 60, 60  # a score of 450 at one key, 0 at all others: their probability is below fp32's range
    v = torch.randn(B, S, Hkv, D, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(dtype)
    v[1, 10, :, 5], v[1, 10, :, 6] = math.inf, -math.inf
    if how in ("intervals", "shares"):
        lengths = torch.full((B,), S, dtype=torch.int32, device="cuda")
        meta = eng.decode_schedule(lengths)
        meta["intervals"] = 9 if how == "intervals" else 0
        o = eng.decode_varlen(q, k, v, lengths, metadata=meta)
    else:
        pick = {"one split": (1, False), "merge launch": (4, False), "cluster": (4, True)}[how]
        monkeypatch.setattr(eng._decode, "_pick", lambda *_: pick)
        o = eng(q, k, v)
    eng.check_status()
    kf, vf = (t.float().repeat_interleave(Hq // Hkv, dim=2) for t in (k, v))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(torch.einsum("bqhd,bkhd->bhqk", q.float(), kf) / math.sqrt(D), -1), vf)
    assert torch.isnan(ref[1, ..., 5:7]).all()
    assert torch.equal(torch.isnan(o), torch.isnan(ref))
    finite = ~torch.isnan(ref)
    assert torch.equal(o[finite].float(), ref[finite])  # the value of the one key that counts
