"""Splits that merge in a cluster give bit for bit what the launch that merges gives: captured calls take the launch, calls made one by
one the cluster."""
import pytest
import torch

from attentionengine_b200 import AttentionEngine, CustomIO, examples as helpers

pytestmark = pytest.mark.gpu


def _inputs(B, Sq, Hq, Hkv, S, D, dtype, seed=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(*shape, generator=g, device="cuda").to(dtype) for shape in ((B, Sq, Hq, D), (B, S, Hkv, D), (B, S, Hkv, D))]


@pytest.mark.parametrize("B,Sq,Hq,Hkv,S,D,dtype,n", [
    (1, 1, 32, 8, 1000, 128, torch.float16, 8), (2, 1, 32, 8, 700, 64, torch.bfloat16, 6), (3, 100, 2, 2, 300, 128, torch.bfloat16, 3),
    (1, 1, 128, 1, 900, 64, torch.float16, 8), (2, 3, 4, 4, 600, 128, torch.bfloat16, 5), (1, 1, 1, 1, 129, 64, torch.float16, 2)])
def test_cluster_and_launch_agree(B, Sq, Hq, Hkv, S, D, dtype, n, monkeypatch):
    eng = helpers.decode_engine(B, Hq, Hkv, Sq, S, D, dtype)
    args = _inputs(B, Sq, Hq, Hkv, S, D, dtype)
    outs = []
    for cut in (False, True):
        monkeypatch.setattr(eng._decode, "_pick", lambda *_: (n, cut))
        outs.append(eng(*args))
        eng.check_status()
    assert torch.equal(*outs)


def test_cluster_and_launch_agree_without_row_state(monkeypatch):
    B, Hq, Hkv, S, D, dtype = 2, 8, 2, 900, 64, torch.float16
    metas = (helpers.meta_tensor(B, Hq, 1, D, dtype=dtype), *(helpers.meta_tensor(B, Hkv, S, D, dtype=dtype),) * 2)
    eng = AttentionEngine(metas, CustomIO({}), score_mod=lambda s, c, b, h, q, kv: (s * 0.125).max(0) * (1.0 / S),
                          mask_mod=None, online_func=helpers.OnlineIdentity(), mask_value="0")
    args = _inputs(B, 1, Hq, Hkv, S, D, dtype)
    outs = []
    for cut in (False, True):
        monkeypatch.setattr(eng._decode, "_pick", lambda *_: (8, cut))
        outs.append(eng(*args))
        eng.check_status()
    assert torch.equal(*outs)


@pytest.mark.parametrize("B,S", [(1, 1000), (2, 1000), (4, 250)])
def test_captured_call_gives_the_bits_of_a_direct_one(B, S):
    eng = helpers.decode_engine(B, 32, 8, 1, S, 128, torch.float16)
    assert eng._decode._pick(B, S)[1]
    args = _inputs(B, 1, 32, 8, S, 128, torch.float16)
    want = eng(*args)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = eng(*args)
    graph.replay()
    torch.cuda.synchronize()
    eng.check_status()
    assert torch.equal(got, want)
