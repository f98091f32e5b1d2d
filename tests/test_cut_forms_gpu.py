"""Forms of the kernels for cut calls that the engines' own rules do not take, or take for online functions of other kinds: splits that
simply add up, clusters of up to eight, intervals of one length given to the C interface, a cut scan that hands out its states,
key heads of two blocks."""
import ctypes as C
import math

import pytest
import torch

import parity
from attentionengine_b200 import AttentionEngine, CustomIO, LinearAttentionEngine, examples as helpers, meta_tensor, runtime as rt
from oracle.linear_oracle import linear_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["one split", "merge launch", "cluster", "intervals", "shares"])
def test_decode_without_row_state(how, monkeypatch):
    """ReLU scores: no row scales, the splits' partials add up; what lies behind a row's end counts for nothing."""
    lens, Hq, Hkv, D, dtype = [3001, 1, 2500, 129], 8, 2, 128, torch.float16
    B, S = len(lens), max(lens)
    if how in ("one split", "merge launch", "cluster"):
        lens = [S] * B
    scale = 1 / math.sqrt(D)
    metas = (helpers.meta_tensor(B, Hq, 1, D, dtype=dtype), *(helpers.meta_tensor(B, Hkv, S, D, dtype=dtype),) * 2)
    eng = AttentionEngine(metas, CustomIO({}), score_mod=lambda s, c, b, h, q, kv: (s * scale).max(0) * (1.0 / S),
                          mask_mod=None, online_func=helpers.OnlineIdentity(), mask_value="0")
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(B, n, h, D, generator=g, device="cuda").to(dtype) for n, h in ((1, Hq), (S, Hkv), (S, Hkv)))
    lengths = torch.tensor(lens, device="cuda")
    keep = torch.arange(S, device="cuda")[None, :] < lengths[:, None]
    k[~keep], v[~keep] = 50.0, 1000.0
    if how in ("intervals", "shares"):
        meta = eng.decode_schedule(lengths)
        meta["intervals"] = 11 if how == "intervals" else 0
        o = eng.decode_varlen(q, k, v, lengths, metadata=meta)
    else:
        pick = {"one split": (1, False), "merge launch": (5, False), "cluster": (4, True)}[how]
        monkeypatch.setattr(eng._decode, "_pick", lambda *_: pick)
        o = eng(q, k, v)
    eng.check_status()
    kf, vf = (t.double().repeat_interleave(Hq // Hkv, dim=2) for t in (k, v))
    p = torch.relu(torch.einsum("bqhd,bkhd->bhqk", q.double(), kf) * scale) / S
    ref = torch.einsum("bhqk,bkhd->bqhd", p.masked_fill(~keep[:, None, None], 0.0), vf)
    parity.check("o", o, ref, dtype, stages=2)  # P and the stored O


@pytest.mark.parametrize("n,S", [(5, 600), (8, 1000)])
def test_clusters_of_more_than_four(n, S, monkeypatch):
    B, Hq, Hkv, D, dtype = 1, 8, 2, 64, torch.bfloat16
    eng = helpers.decode_engine(B, Hq, Hkv, 1, S, D, dtype)
    monkeypatch.setattr(eng._decode, "_pick", lambda *_: (n, True))
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn(B, m, h, D, generator=g, device="cuda").to(dtype) for m, h in ((1, Hq), (S, Hkv), (S, Hkv)))
    o = eng(q, k, v)
    eng.check_status()
    kf, vf = (t.float().repeat_interleave(Hq // Hkv, dim=2) for t in (k, v))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(torch.einsum("bqhd,bkhd->bhqk", q.float(), kf) / math.sqrt(D), -1), vf)
    parity.check("o", o, ref, dtype, stages=2)


def test_intervals_without_lengths():
    """C interface: rows of one length, Skv keys, without `seqlens`."""
    B, Hq, Hkv, S, D, dtype, n = 3, 8, 2, 1000, 128, torch.float16, 7
    dec = helpers.decode_engine(B, Hq, Hkv, 1, S, D, dtype)._decode
    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn(B, m, h, D, generator=g, device="cuda").to(dtype) for m, h in ((1, Hq), (S, Hkv), (S, Hkv)))
    o = torch.empty(B, 1, Hq, D, dtype=dtype, device="cuda")
    rows = Hq // Hkv
    part = torch.empty(Hkv, 2 * n, rows, D, device="cuda")
    scales = torch.empty(Hkv, 2 * n, rows, device="cuda")
    info = torch.empty(B * Hkv, 2, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = rt.DecodeParams()
    p.q, p.k, p.v, p.o = (t.data_ptr() for t in (q, k, v, o))
    p.q_stride, p.k_stride, p.v_stride = ((C.c_int64 * 3)(*t.stride()[:3]) for t in (q, k, v))
    p.o_partial, p.rowscale_partial[0], p.row_info, p.status = part.data_ptr(), scales.data_ptr(), info.data_ptr(), status.data_ptr()
    p.B, p.Hq, p.Hkv, p.Sq, p.Skv, p.n_split, p.n_intervals = B, Hq, Hkv, 1, S, 1, n
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rt.check(rt.lib().ae_launch_attn_decode(dec.cut_kernel.handle, C.byref(p), stream), "ae_launch_attn_decode")
    rt.check(rt.lib().ae_launch_decode_combine(dec.combine.handle, C.byref(p), stream), "ae_launch_decode_combine")
    torch.cuda.synchronize()
    assert status.item() == 0
    kf, vf = (t.float().repeat_interleave(rows, dim=2) for t in (k, v))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(torch.einsum("bqhd,bkhd->bhqk", q.float(), kf) / math.sqrt(D), -1), vf)
    parity.check("o", o, ref, dtype, stages=2)


@pytest.mark.parametrize("T,seg_chunks", [(1000, 3), (700, 1)])
def test_cut_scan_hands_out_its_states(T, seg_chunks):
    """C interface: h_states_out and v_out of a cut launch are those of one walk, the states up to one rounding to 16 bits (their fp32 sums
    come in another order)."""
    B, H, dtype = 2, 3, torch.bfloat16
    x, dt, _, Bm, Cm = (t.cuda() for t in helpers.mamba2_inputs(B, H, T, 128, 64, dtype, seed=T))
    s, d = dt.to(dtype), torch.randn(H, device="cuda")
    a = -0.05 * dt
    eng = helpers.mamba2_engine(B, H, T, 128, 64, dtype, d_skip=True)
    n = -(-T // 128)
    parts, scan = eng._segment_kernels(64, True)
    states = [torch.full((B, H, n, 128, 64), float("nan"), dtype=dtype, device="cuda") for _ in range(2)]
    scaled = [torch.full_like(x, float("nan")) for _ in range(2)]
    one = eng._launch(Cm, Bm, x, a, s, d, scaled[0], states[0])
    o, status = torch.empty_like(x), torch.zeros(1, dtype=torch.int32, device="cuda")
    n_seg = -(-n // seg_chunks)
    st, dec = torch.empty(B, H, n_seg - 1, 128 * 64, device="cuda"), torch.empty(B, H, n_seg - 1, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = rt.LinearSegParams()
    g.k, g.v, g.a, g.vscale, g.vscale_16bit = Bm.data_ptr(), x.data_ptr(), a.data_ptr(), s.data_ptr(), 1
    p = rt.LinearParams()
    p.q, p.k, p.v, p.a, p.o = (t.data_ptr() for t in (Cm, Bm, x, a, o))
    p.vscale, p.vscale_16bit, p.dskip, p.v_out, p.h_states_out = s.data_ptr(), 1, d.data_ptr(), scaled[1].data_ptr(), states[1].data_ptr()
    p.B, p.H, p.HQ, p.HK, p.T = B, H, 1, 1, T
    g.B, g.H, g.HK, g.T = B, H, 1, T
    for r in (g, p):
        r.seg_chunks, r.seg_state, r.seg_decay, r.status = seg_chunks, st.data_ptr(), dec.data_ptr(), status.data_ptr()
    rt.check(rt.lib().ae_launch_linear_segments(parts.handle, C.byref(g), stream), "ae_launch_linear_segments")
    rt.check(rt.lib().ae_launch_linear_fwd(scan.handle, C.byref(p), stream), "ae_launch_linear_fwd")
    torch.cuda.synchronize()
    assert status.item() == 0 and torch.equal(*scaled)
    for got, want in ((o, one), (states[1], states[0])):
        assert (got.double() - want.double()).norm() / want.double().norm() <= 2.0 ** -8


def test_key_heads_of_two_blocks_in_segments():
    """Gated linear attention with 256 key dims: the scans of two key blocks, each cut, summed."""
    B, H, T, DK, DV, dtype = 1, 2, 1000, 256, 128, torch.float16
    gen = torch.Generator().manual_seed(7)
    q, k, v = ((0.3 * torch.randn(B, H, T, n, generator=gen)).to(dtype) for n in (DK, DK, DV))
    a = torch.nn.functional.logsigmoid(torch.randn(B, H, T, generator=gen)) / 16
    eng = LinearAttentionEngine(tuple(meta_tensor(B, H, T, n, dtype=dtype) for n in (DK, DK, DV)), custom_io=CustomIO({}))
    eng._native_plan().segments = 3
    with torch.no_grad():
        o = eng(*(t.cuda() for t in (q, k, v, a)))
    eng.check_status()
    assert eng._native_plan().fwd_cut128
    parity.check("o", o, linear_scan(q, k, v, a), dtype, stages=4, unnormalised=True)
