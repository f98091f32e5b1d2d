"""Decode on equal intervals of all rows' tiles and with splits that merge in a cluster: rows that begin, end or lie inside an interval,
rows of one key, more rows than a warp has lanes, fewer tiles than intervals, and the merge's layouts, against attention in fp32."""
import math

import pytest
import torch

import parity
from attentionengine_b200 import AttentionEngine, CustomIO, examples as helpers
from attentionengine_b200.attn_engine import attn_decode

pytestmark = pytest.mark.gpu


def _attention(q, k, v, lens):
    B, Sq, Hq, D = q.shape
    k, v = (t.float().repeat_interleave(Hq // t.shape[2], dim=2) for t in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), k) / math.sqrt(D)
    keep = torch.arange(k.shape[1], device=q.device)[None, :] < lens[:, None].to(q.device)
    return torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s.masked_fill(~keep[:, None, None], float("-inf")), -1), v)


def _inputs(B, Sq, Hq, Hkv, S, D, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(*shape, generator=g, device="cuda", dtype=dtype) for shape in ((B, Sq, Hq, D), (B, S, Hkv, D), (B, S, Hkv, D))]


@pytest.mark.parametrize("B,Sq,Hq,Hkv,S,D,dtype,n", [
    (5, 1, 32, 8, 4200, 128, torch.float16, 18),    # 5 rows of 33 tiles, shares of 10
    (3, 1, 8, 4, 1000, 64, torch.bfloat16, 7),      # rows longer and shorter than what is left of an interval
    (2, 3, 4, 4, 700, 128, torch.bfloat16, 5),      # several query positions: a unit's rows are not neighbours in the output
    (1, 100, 2, 2, 2000, 64, torch.float16, 3),
    (2, 1, 8, 2, 100, 128, torch.float16, 74),      # fewer tiles than intervals: nothing to merge
    (1, 1, 16, 4, 128 * 70, 128, torch.bfloat16, 70),  # a row spans 32 intervals at most
])
def test_rows_of_one_length_in_intervals(B, Sq, Hq, Hkv, S, D, dtype, n):
    eng = helpers.decode_engine(B, Hq, Hkv, Sq, S, D, dtype)
    q, k, v = _inputs(B, Sq, Hq, Hkv, S, D, dtype, S)
    meta = eng.decode_schedule(torch.full((B,), S))
    meta["intervals"] = n
    o = eng.decode_varlen(q, k, v, torch.full((B,), S), metadata=meta)
    eng.check_status()
    parity.check("o", o, _attention(q, k, v, torch.full((B,), S)), dtype, stages=2)  # P and the stored O


@pytest.mark.parametrize("lens,Hq,Hkv,D,dtype,paged,intervals", [
    ([1, 128, 129, 5000, 127, 700, 256, 2048, 1], 32, 8, 128, torch.float16, True, 18),
    ([300] * 40 + [1] * 30, 16, 4, 64, torch.bfloat16, False, 37),  # more rows than a warp has lanes, several rows per interval
    ([6000], 8, 8, 128, torch.bfloat16, True, 18),
])
def test_ragged_rows_in_intervals(lens, Hq, Hkv, D, dtype, paged, intervals):
    B, S = len(lens), max(lens)
    eng = helpers.decode_engine(B, Hq, Hkv, 1, S, D, dtype)
    q, k, v = _inputs(B, 1, Hq, Hkv, -(-S // 128) * 128, D, dtype, B)
    lengths = torch.tensor(lens, dtype=torch.int32)
    ref = _attention(q, k, v, lengths)
    table = None
    if paged:
        pages = k.shape[1] // 128
        table = torch.randperm(B * pages, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(B, pages).cuda()
        pools = []
        for t in (k, v):
            pool = torch.empty(B * pages, 128, Hkv, D, dtype=dtype, device="cuda")
            pool[table.flatten().long()] = t.view(B * pages, 128, Hkv, D)
            pools.append(pool)
        k, v = pools
    meta = eng.decode_schedule(lengths.cuda())
    meta["intervals"] = intervals
    o = eng.decode_varlen(q, k, v, lengths.cuda(), block_table=table, metadata=meta)
    eng.check_status()
    parity.check("o", o, ref, dtype, stages=2)


@pytest.mark.parametrize("B,Sq,Hq,Hkv,S,D,dtype,n", [
    (2, 1, 32, 8, 1000, 128, torch.float16, 4), (1, 1, 8, 8, 1000, 64, torch.bfloat16, 3), (3, 100, 2, 2, 300, 128, torch.bfloat16, 3),
    (1, 3, 4, 4, 2000, 64, torch.float16, 2), (2, 1, 64, 1, 900, 128, torch.bfloat16, 4)])
def test_splits_that_merge_in_a_cluster(B, Sq, Hq, Hkv, S, D, dtype, n, monkeypatch):
    """Fewer rows than warps and more, a last split that is shorter, both layouts of a unit's rows."""
    eng = helpers.decode_engine(B, Hq, Hkv, Sq, S, D, dtype)
    monkeypatch.setattr(eng._decode, "_pick", lambda *_: (n, True))
    q, k, v = _inputs(B, Sq, Hq, Hkv, S, D, dtype, S)
    o = eng(q, k, v)
    eng.check_status()
    parity.check("o", o, _attention(q, k, v, torch.full((B,), S)), dtype, stages=2)


def test_a_split_without_a_kept_key_weighs_nothing(monkeypatch):
    """A mask that leaves whole splits empty: their partial is 0 / 0, in the launch that merges and in the cluster."""
    B, H, S, D, dtype = 1, 2, 1024, 64, torch.float16
    metas = (helpers.meta_tensor(B, H, 1, D, dtype=dtype), *(helpers.meta_tensor(B, H, S, D, dtype=dtype),) * 2)
    eng = AttentionEngine(metas, CustomIO({}), score_mod=lambda s, c, b, h, q, kv: s * 0.125, mask_mod=lambda b, h, q, kv: kv >= 700,
                          online_func=helpers.OnlineSoftmaxSplit())
    q, k, v = _inputs(B, 1, H, H, S, D, dtype, 3)
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float()) * 0.125
    s[..., :700] = float("-inf")
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v.float())
    for cut in ((8, False), (4, True)):
        monkeypatch.setattr(eng._decode, "_pick", lambda *_: cut)
        parity.check(str(cut), eng(q, k, v), ref, dtype)
    meta = eng.decode_schedule(torch.full((B,), S))
    meta["intervals"] = 5
    parity.check("intervals", eng.decode_varlen(q, k, v, torch.full((B,), S), metadata=meta), ref, dtype)


def test_how_a_call_is_cut():
    dec = helpers.decode_engine(16, 32, 8, 1, 8192, 128, torch.float16)._decode
    assert dec._pick(16, 8192) == (1, False) and dec._pick(2, 1000) == (4, True) and dec._pick(1, 16384)[1] is False
    assert dec.schedule(torch.tensor([8192, 1, 5000]))["intervals"] == attn_decode.N_SM // 8
    assert dec.schedule(torch.tensor([300] * 8))["intervals"] == 0 and dec.schedule(torch.tensor([8192]))["intervals"] == 0
