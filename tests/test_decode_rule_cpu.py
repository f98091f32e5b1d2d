"""Which calls merge in a cluster: short splits of few rows whose clusters run all at once.  Which schedules are cut into intervals: long rows of head units that fill the SMs, never where one CTA per unit and wave would leave
many of them idle, and not when the caller asks for waves of shares."""
import pytest
import torch

from attentionengine_b200 import examples as helpers
from attentionengine_b200.attn_engine.attn_decode import N_SM


@pytest.mark.parametrize("Hkv,D,lens,cut", [
    (8, 128, [8192, 1, 5000, 7000] * 16, True), (32, 128, [8192, 3000, 4000, 1], True), (8, 64, [8192, 1, 5000, 7000] * 6, True),
    (80, 128, [4096] * 16, False), (80, 128, [8192, 1, 5000, 7000], False), (100, 128, [4096, 100, 2000, 3000] * 4, False),
    (50, 128, [2560] * 16, False), (32, 128, [4096] * 64, False), (1, 128, [8192, 1, 5000, 7000], False),
    (48, 64, [16384] * 6, False), (149, 128, [8192, 1, 5000], False)])
def test_which_schedules_are_cut_into_intervals(Hkv, D, lens, cut):
    dec = helpers.decode_engine(len(lens), Hkv, Hkv, 1, max(lens), D, torch.float16)._decode
    meta = dec.schedule(torch.tensor(lens), device="cpu")
    assert meta["intervals"] == (N_SM // Hkv if cut else 0)
    assert dec.schedule(torch.tensor(lens), device="cpu", waves=2)["intervals"] == 0


@pytest.mark.parametrize("Hq,Hkv,B,S,pick", [
    (32, 8, 1, 1000, (8, True)), (32, 8, 2, 1000, (4, True)), (32, 8, 2, 700, (6, True)), (32, 8, 4, 300, (3, True)),
    (32, 8, 4, 1000, (4, False)), (32, 8, 8, 250, (2, False)), (32, 32, 1, 1500, (4, False)), (32, 8, 1, 2000, (16, False)),
    (32, 8, 2, 2000, (8, False)), (16, 1, 1, 250, (2, True)), (64, 1, 1, 250, (2, False)), (150, 1, 1, 1000, (8, False)),
    (32, 8, 16, 8192, (1, False)), (32, 8, 1, 100, (1, False))])
def test_which_calls_merge_in_a_cluster(Hq, Hkv, B, S, pick):
    dec = helpers.decode_engine(B, Hq, Hkv, 1, S, 128, torch.float16)._decode
    assert dec._pick(B, S) == pick and dec.pick_splits(B, S) == pick[0]
