"""The native host path (csrc/ae_host.cpp): what it refuses, and what its autograd nodes owe to the rest of PyTorch."""
import math
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch
import torch.autograd.forward_ad as fwAD
import torch.utils.checkpoint

import helpers
from attentionengine_b200 import AttentionEngine, CustomIO, meta_tensor, runtime as rt
from attentionengine_b200.attn_engine import OnlineFunc
from attentionengine_b200.core import SymbolScalar, Var

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


# ---------------------------------------------------------------------------------------------------- nodes
def _attention(mask="causal", S=300, D=64, dtype=torch.float16):
    """An attention call: (engine, q, k, v, d_o) with GQA heads."""
    B, Hq, Hkv = 2, 4, 2
    if mask == "window":
        eng = AttentionEngine(helpers.metas(B, Hq, Hkv, S, D, D, dtype), CustomIO({}), score_mod=lambda s, c, b, h, q, kv: s * D ** -0.5,
                              mask_mod=lambda b, h, q, kv: torch.logical_and(q >= kv, q - kv <= 130), online_func=helpers.OnlineSoftmax())
        assert eng.mask_mode == 2
    else:
        eng = helpers.softmax_engine(B, Hq, Hkv, S, D, D, dtype, True)
    return (eng, *helpers.seeded_qkv(B, Hq, Hkv, S, D, D, dtype, seed=1, device="cuda"))


def _block(T=200, H=4, dtype=torch.bfloat16, seed=2):
    """A Mamba2 block call: (engine, [C, B, x, step, A, step16, skip], d_o)."""
    x, step, A, Bm, Cm = (t.cuda() for t in helpers.mamba2_inputs(2, H, T, 128, 64, dtype, seed=seed))
    g = torch.Generator(device="cuda").manual_seed(seed)
    eng = helpers.mamba2_engine(2, H, T, 128, 64, dtype, d_skip=True)
    return eng, [Cm, Bm, x, step, A.view(1, H), step.to(dtype), torch.randn(1, H, generator=g, device="cuda")], torch.randn(x.shape, generator=g, device="cuda", dtype=dtype)


def test_forward_mode_is_refused():
    """Neither kernel has a forward-mode rule: a dual tensor among the inputs raises, it does not lose its tangent."""
    eng, q, k, v, _ = _attention()
    scan, args, _ = _block()
    with fwAD.dual_level():
        for i in range(3):
            a = [q, k, v]
            a[i] = fwAD.make_dual(a[i], torch.ones_like(a[i]))
            with pytest.raises(NotImplementedError, match="jvp"):
                eng(*a)
        for i in range(len(args)):
            a = list(args)
            a[i] = fwAD.make_dual(a[i], torch.ones_like(a[i]))
            with pytest.raises(NotImplementedError, match="jvp"):
                scan(*a)


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("mask", ["causal", "window"])
def test_traced_attention_runs_its_kernel(mask):
    """torch.jit.trace records the call: on other inputs the traced function computes, with gradients."""
    eng, q, k, v, d_o = _attention(mask)
    f = torch.jit.trace(lambda a, b, c: eng(a, b, c) * 2, (q, k, v), check_trace=False)
    q2, k2, v2 = (torch.randn_like(t).requires_grad_() for t in (q, k, v))
    o = f(q2, k2, v2)
    got = (o, *torch.autograd.grad(o, (q2, k2, v2), d_o))
    o = eng(q2, k2, v2) * 2
    want = (o, *torch.autograd.grad(o, (q2, k2, v2), d_o))
    assert torch.equal(got[0], want[0])
    for x, y in zip(got[1:], want[1:]):  # dQ: fp32 additions in any order, rounded to fp16
        torch.testing.assert_close(x, y, rtol=2 ** -9, atol=2 ** -9)


@pytest.mark.filterwarnings("ignore")
def test_traced_scan_runs_its_kernel():
    """The same for the Mamba2 block, whose mods then run one by one: their results are rounded to bf16 in between."""
    eng, args, _ = _block()
    f = torch.jit.trace(lambda *a: eng(*a), tuple(args), check_trace=False)
    other = _block(seed=3)[1]
    o = eng(*other)
    err = (f(*other).float() - o.float()).norm() / o.float().norm()
    assert err < 4 * 2 ** -8  # v * step and the output before the skip, each rounded once more


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, g):
        return None


def test_undefined_gradient_counts_as_zero():
    eng, q, k, v, _ = _attention()
    scan, args, _ = _block()
    for f, leaves in ((eng, [q, k, v]), (scan, args)):
        for t in leaves:
            t.requires_grad_()
        _NoGradient.apply(f(*leaves)).sum().backward()
        assert all(t.grad is not None and not t.grad.any() for t in leaves)


# ---------------------------------------------------------------------------------------------------- paged MLA
def _paged(B=2, H=16, pages=4):
    g = torch.Generator(device="cuda").manual_seed(7)
    q = torch.randn(B, 1, H, 576, generator=g, device="cuda", dtype=torch.float16)
    pool = torch.randn(B * pages, 64, 1, 576, generator=g, device="cuda", dtype=torch.float16)
    return _mla(B, H, pages * 64), q, pool, torch.arange(B * pages, dtype=torch.int32, device="cuda").view(B, pages), \
        torch.tensor([100, pages * 64], dtype=torch.int32, device="cuda")


def test_paged_mla_waits_for_its_lengths_when_a_launch_fails():
    """The copy of the lengths into the thread's landing place is queued in front of the launches: a call that fails there
    returns behind the copy, so that the next one, on any stream, has the place to itself."""
    eng, q, pool, table, lens = _paged()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)  # ten milliseconds or so in front of the copy
        before = side.record_event()
        with pytest.raises(rt.AeError):
            eng.decode_paged(q, pool[:0], table, lens)
        assert before.query()
    with pytest.raises(ValueError, match="cache_seqlens"):
        eng.decode_paged(q, pool, table[:, :0], lens)
    with pytest.raises(rt.AeError, match="empty"):
        eng.decode_paged(q[:0], pool, table[:0], lens[:0])
    o, _ = eng.decode_paged(q, pool, table, lens)
    torch.cuda.synchronize()
    assert torch.isfinite(o).all()


def test_paged_mla_is_refused_under_capture():
    eng, q, pool, table, lens = _paged()
    want = eng.decode_paged(q, pool, table, lens)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(RuntimeError, match="captured"):
            eng.decode_paged(q, pool, table, lens)
        q.add_(0)
    got = eng.decode_paged(q, pool, table, lens)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_paged_mla_takes_any_layout_of_q():
    """q with another stride order, or on a base that TMA cannot read, is copied; a block table may have trailing ones."""
    eng, q, pool, table, lens = _paged()
    want = eng.decode_paged(q, pool, table, lens)
    odd = torch.empty(q.numel() + 1, dtype=q.dtype, device="cuda")[1:].view(q.shape).copy_(q)
    turned = q.transpose(2, 3).contiguous().transpose(2, 3)
    assert odd.data_ptr() % 16 and turned.stride(3) != 1
    for got in (eng.decode_paged(odd, pool, table, lens), eng.decode_paged(turned, pool, table, lens),
                eng.decode_paged(q, pool, table[..., None], lens)):
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_decode_takes_custom_inputs_by_the_dims_it_indexes():
    """A decode call reads a custom input by its named dims: it may lack dims that are not indexed and have more at the end."""
    B, H, S, D, dtype = 2, 4, 300, 64, torch.float16
    eng = AttentionEngine(tuple(meta_tensor(B, H, n, D, dtype=dtype) for n in (1, S, S)), CustomIO({"scale": (1,), "slope": (1, "heads")}),
                          score_mod=lambda s, c, b, h, q, kv: s * c.input_tensors["scale"] + c.input_tensors["slope"] * s, mask_mod=None,
                          online_func=helpers.OnlineSoftmaxSplit())
    g = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn(B, n, H, D, generator=g, device="cuda", dtype=dtype) for n in (1, S, S))
    scale, slope = torch.tensor([0.1], device="cuda"), torch.rand(1, H, generator=g, device="cuda")
    want = eng(q, k, v, scale, slope)
    assert torch.equal(eng(q, k, v, scale[0], slope[..., None]), want)
    with pytest.raises(ValueError, match="slope"):
        eng(q, k, v, scale, slope[0])
    with pytest.raises(ValueError, match="contiguous last dimension"):
        eng(q, k[0, 0], v, scale, slope)


class _PlainExp(helpers.OnlineSoftmaxSplit):
    """Softmax without the running maximum: its sums under- and overflow."""

    def __init__(self):
        OnlineFunc.__init__(self, {"r": SymbolScalar("r", Var("0.0"))}, {"lse": SymbolScalar("lse", Var("0.0"))}, CustomIO())

    @staticmethod
    def online_fwd(scores, online_rowscales, b, h, q_idx):
        scores = scores.exp()
        return scores, {"r": online_rowscales["r"] + scores.get_reduce("sum")}, SymbolScalar("o_scale", Var("1"))

    @staticmethod
    def online_fwd_epilogue(o, online_rowscales, b, h, q_idx):
        return o, {"lse": online_rowscales["r"].log()}


@pytest.mark.parametrize("shift", [-1000.0, 1000.0])
def test_paged_mla_infinite_log_sum_exp(shift):
    """Rows whose sums are all 0 or infinite have the log-sum-exp -inf or inf, merged (second row) or not (first row)."""
    B, H, S, dtype = 2, 16, 2048, torch.float16
    metas = (meta_tensor(B, H, 1, 576, dtype=dtype), meta_tensor(B, 1, S, 576, dtype=dtype), meta_tensor(B, 1, S, 512, dtype=dtype))
    eng = AttentionEngine(metas, CustomIO({}), score_mod=lambda s, c, b, h, q, kv: s * 0.01 + shift, mask_mod=None, online_func=_PlainExp(),
                          kv_shared=True)
    _, q, pool, table, _ = _paged(B, H, S // 64)
    _, lse = eng.decode_paged(q, pool, table, torch.tensor([100, S], dtype=torch.int32, device="cuda"))
    assert (lse == math.copysign(math.inf, shift)).all()


@pytest.mark.parametrize("H,pages,lens,most", [
    (16, 310, [128, 19840], 32),       # 156 tiles: intervals of 5, so that no row touches more than 32; the second begins inside one
    (16, 4, [100, 256], 2),            # 3 tiles in two intervals of 2
    (16, 2, [128, 128, 128], 1),       # whole rows
    (16, 64, [1, 4096, 300], 17),      # 1 + 32 + 3 tiles in intervals of 2
])
def test_last_num_split_counts_the_shares_of_a_row(H, pages, lens, most):
    B = len(lens)
    eng, q, pool, table, _ = _paged(B, H, pages)
    eng.decode_paged(q, pool, table, torch.tensor(lens, dtype=torch.int32, device="cuda"))
    assert eng._mla.last_num_split == most
    if len(set(lens)) == 1:
        kv = pool.view(B, pages * 64, 1, 576)[:, :lens[0]]
        eng(q[..., :512], q[..., 512:], kv[..., :512], kv[..., 512:])
        assert eng._mla.last_num_split == most


# ---------------------------------------------------------------------------------------------------- what nodes owe autograd
@pytest.fixture(params=["attention", "block", "scan"])
def call(request):
    """(f, leaves, output gradient) of an attention call, of the Mamba2 block and of the plain scan."""
    if request.param == "attention":
        eng, q, k, v, d_o = _attention()
        return eng, [t.requires_grad_() for t in (q, k, v)], d_o
    eng, args, d_o = _block()
    if request.param == "scan":
        eng = helpers.mamba2_engine(2, 4, 200, 128, 64, torch.bfloat16)
        args = args[:-1]
    return eng, [t.requires_grad_() for t in args], d_o


def _same(got, want):
    """The outputs bit for bit; gradients up to the order of dQ's fp32 additions and a rounding to 16 bits."""
    assert torch.equal(got[0], want[0])
    for x, y in zip(got[1:], want[1:]):
        assert (x.float() - y.float()).norm() <= 2 ** -8 * y.float().norm()


def _once(f, leaves, d_o):
    o = f(*leaves)
    return (o, *torch.autograd.grad(o, leaves, d_o))


def test_saved_tensors_go_through_hooks(call):
    f, leaves, d_o = call
    want = _once(*call)
    packed, unpacked = [], []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t), t.detach().cpu())[1],
                                                  lambda t: (unpacked.append(t), t.cuda())[1]):
        o = f(*leaves)
    _same((o, *torch.autograd.grad(o, leaves, d_o)), want)
    assert len(packed) == len(unpacked) >= len(leaves)


def test_checkpointed_call(call):
    f, leaves, d_o = call
    o = torch.utils.checkpoint.checkpoint(f, *leaves, use_reentrant=False)
    _same((o, *torch.autograd.grad(o, leaves, d_o)), _once(*call))


def test_backward_from_another_thread_and_a_second_one(call):
    f, leaves, d_o = call
    want = _once(*call)
    o = f(*leaves)
    with ThreadPoolExecutor(1) as pool:
        _same((o, *pool.submit(torch.autograd.grad, o, leaves, d_o, True).result()), want)
    _same((o, *torch.autograd.grad(o, leaves, d_o)), want)  # the graph was kept once, and is released now
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(o, leaves, d_o)


def test_call_on_a_side_stream(call):
    """The call and its backward run on the stream that is current, behind what is queued there."""
    f, leaves, d_o = call
    want = _once(*call)
    late = [torch.zeros_like(t) for t in leaves]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        for t, u in zip(late, leaves):
            t.copy_(u.detach())
        got = _once(f, [t.requires_grad_() for t in late], d_o)
    side.synchronize()
    _same(got, want)


def test_modified_input_is_noticed(call):
    f, leaves, d_o = call
    mid = [t * 1 for t in leaves]
    o = f(*mid)
    with torch.no_grad():
        mid[0].add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        o.backward(d_o)


def test_empty_inputs_raise(call):
    f, leaves, _ = call
    with pytest.raises((rt.AeError, ValueError)):
        f(*(t[:0] if t.shape[0] > 1 else t for t in leaves))


def test_calls_in_threads():
    """One new engine, several threads with a stream each, and its status word looked at while their first calls make it."""
    eng, q, k, v, _ = _attention()
    want = eng(q, k, v)
    torch.cuda.synchronize()
    eng, *_ = _attention()

    def work(_):
        with torch.cuda.stream(torch.cuda.Stream()):
            outs = [eng(q, k, v) for _ in range(20)]
            torch.cuda.current_stream().synchronize()
            return all(torch.equal(o, want) for o in outs)

    with ThreadPoolExecutor(4) as pool:
        jobs = [pool.submit(work, i) for i in range(8)]
        seen = [eng._status for _ in range(1000)]
        assert all(j.result() for j in jobs)
    torch.cuda.synchronize()
    eng.check_status()
    assert all(s is None or s.is_cuda for s in seen)
