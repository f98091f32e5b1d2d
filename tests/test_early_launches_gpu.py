"""Kernels launched to come up under the one in front of them, captured in a graph and replayed on new inputs: they still follow it."""
import math

import pytest
import torch

from attentionengine_b200 import CustomIO, LinearAttentionEngine, examples as helpers, meta_tensor

pytestmark = pytest.mark.gpu


def _replays_as_called(call, inputs, fill, check, same=torch.equal):
    want = call()  # builds and loads what the call takes
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = call()
    for _ in range(3):
        for t in inputs:
            t.data.copy_(fill(t))
        graph.replay()
        torch.cuda.synchronize()
        check()
        want = call()
        for name, x, y in zip(("first", "second", "third", "fourth"), got if isinstance(got, tuple) else (got,), want if isinstance(want, tuple) else (want,)):
            assert same(x, y), name


def _normal(gen):
    return lambda t: torch.randn(t.shape, generator=gen, device="cuda", dtype=torch.float32).to(t.dtype)


@pytest.mark.parametrize("how", ["merge", "intervals", "shares"])
def test_decode_with_its_merge_in_a_graph(how):
    B, Hq, Hkv, D, dtype = (1 if how == "merge" else 3), 32, 8, 128, torch.float16
    S = 16384 if how == "merge" else 6000
    eng = helpers.decode_engine(B, Hq, Hkv, 1, S, D, dtype)
    fill = _normal(torch.Generator(device="cuda").manual_seed(1))
    q, k, v = (fill(torch.empty(B, n, h, D, dtype=dtype, device="cuda")) for n, h in ((1, Hq), (S, Hkv), (S, Hkv)))
    if how == "merge":
        assert eng._decode._pick(B, S)[0] > 1 and not eng._decode._pick(B, S)[1]
        call = lambda: eng(q, k, v)  # noqa: E731
    else:
        lengths = torch.tensor([6000, 1, 4100], device="cuda")
        meta = eng.decode_schedule(lengths)
        meta["intervals"] = 18 if how == "intervals" else 0
        assert meta["n_slots"] > B
        call = lambda: eng.decode_varlen(q, k, v, lengths, metadata=meta)  # noqa: E731
    _replays_as_called(call, (q, k, v), fill, eng.check_status)


@pytest.mark.parametrize("B,H,S", [(8, 128, 3000), (40, 128, 700)])  # one head and four heads by a thread of the merge
def test_mla_with_its_merge_in_a_graph(B, H, S):
    dtype = torch.bfloat16
    eng = helpers.mla_engine(B, H, S, dtype, 1 / math.sqrt(192))
    fill = _normal(torch.Generator(device="cuda").manual_seed(2))
    args = [fill(torch.empty(s, dtype=dtype, device="cuda")) for s in ((B, 1, H, 512), (B, 1, H, 64), (B, S, 1, 512), (B, S, 1, 64))]
    _replays_as_called(lambda: eng(*args), args, fill, eng.check_status)


@pytest.mark.parametrize("B,Hkv,S", [(2, 8, 1300), (1, 2, 300)])  # the main kernel under the pre-pass, and behind it
def test_training_step_in_a_graph(B, Hkv, S):
    D, dtype = 128, torch.float16
    eng = helpers.softmax_engine(B, Hkv, Hkv, S, D, D, dtype, True)
    fill = _normal(torch.Generator(device="cuda").manual_seed(3))
    q, k, v, d_o = (fill(torch.empty(B, S, Hkv, D, dtype=dtype, device="cuda")) for _ in range(4))
    for t in (q, k, v):
        t.requires_grad_()

    def call():
        o = eng(q, k, v)
        dq, dk, dv = torch.autograd.grad(o, (q, k, v), d_o)
        return o.detach(), dk, dv, dq

    def same(x, y):  # dQ is a sum of fp32 atomics, its order differs from run to run
        return torch.equal(x, y) or torch.allclose(x.float(), y.float(), rtol=2e-3, atol=2e-4)

    side = torch.cuda.Stream()  # autograd's first step off the capturing stream
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    _replays_as_called(call, (q, k, v, d_o), fill, eng.check_status, same)


def test_scan_in_segments_in_a_graph():
    B, H, T, dtype = 1, 4, 2500, torch.bfloat16
    eng = LinearAttentionEngine(tuple(meta_tensor(B, H, T, n, dtype=dtype) for n in (128, 128, 64)), custom_io=CustomIO({}))
    fill = _normal(torch.Generator(device="cuda").manual_seed(4))
    q, k, v = (fill(torch.empty(B, H, T, n, dtype=dtype, device="cuda")) for n in (128, 128, 64))
    a = -0.01 * torch.rand(B, H, T, device="cuda")
    with torch.no_grad():
        _replays_as_called(lambda: eng(q, k, v, a), (q, k, v), fill, eng.check_status)
    assert eng._native_plan().fwd_cut64  # it was cut
