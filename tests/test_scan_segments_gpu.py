"""A scan cut into segments along the sequence against one walk over it, at the sizes where a cut can go wrong: one chunk per
segment, a last segment that is shorter, a last chunk that is nearly empty, and decays slow enough that the state of the first
segment still counts in the last."""
import pytest
import torch

import parity
from attentionengine_b200 import CustomIO, LinearAttentionEngine, examples as helpers, meta_tensor

pytestmark = pytest.mark.gpu


def _run(make, args, segments):
    eng = make()
    eng._native_plan().segments = segments
    with torch.no_grad():
        o = eng(*args)
    torch.cuda.synchronize()
    eng.check_status()
    return o


def _same(got, ref, dtype):
    # Both round the same weighted values to 16 bits; they differ where a state, carried in another order of fp32 sums,
    # falls on the other side of a rounding edge: below one unit of the 16-bit type on the whole tensor.
    rel = (got.double() - ref.double()).norm() / ref.double().norm()
    assert rel <= 2.0 ** (-8 if dtype == torch.bfloat16 else -11), rel.item()


@pytest.mark.parametrize("T,segments,dtype", [(129, 2, torch.bfloat16), (1000, 8, torch.float16), (1000, 3, torch.bfloat16),
                                              (1153, 5, torch.float16), (2048, 16, torch.bfloat16)])
def test_block_in_segments_against_one_walk(T, segments, dtype):
    B, H = 2, 3
    x, dt, _, Bm, Cm = helpers.mamba2_inputs(B, H, T, 128, 64, dtype, seed=T)
    gen = torch.Generator().manual_seed(T)
    A = -torch.rand(1, H, generator=gen) * 0.05
    args = [t.cuda() for t in (Cm, Bm, x, dt, A, dt.to(dtype), torch.randn(1, H, generator=gen))]
    make = lambda: helpers.mamba2_engine(B, H, T, 128, 64, dtype, d_skip=True)  # noqa: E731
    _same(_run(make, args, segments), _run(make, args, 1), dtype)


@pytest.mark.parametrize("T,segments,DV", [(300, 3, 128), (650, 2, 128), (1024, 4, 64)])
def test_plain_scan_in_segments_against_one_walk(T, segments, DV):
    """Value blocks of 64 and of 128; one q / k head per value head."""
    B, H, dtype = 1, 2, torch.float16
    gen = torch.Generator().manual_seed(T)
    q, k, v = ((0.3 * torch.randn(B, H, T, n, generator=gen)).to(dtype).cuda() for n in (128, 128, DV))
    a = -0.01 * torch.rand(B, H, T, generator=gen).cuda()
    metas = tuple(meta_tensor(B, H, T, n, dtype=dtype) for n in (128, 128, DV))
    make = lambda: LinearAttentionEngine(metas, custom_io=CustomIO({}))  # noqa: E731
    _same(_run(make, [q, k, v, a], segments), _run(make, [q, k, v, a], 1), dtype)


def test_segments_against_oracle():
    from oracle.linear_oracle import linear_scan
    B, H, T, dtype = 1, 2, 520, torch.float16
    gen = torch.Generator().manual_seed(1)
    q, k, v = ((0.3 * torch.randn(B, H, T, n, generator=gen)).to(dtype) for n in (128, 128, 64))
    a = -0.01 * torch.rand(B, H, T, generator=gen)
    metas = tuple(meta_tensor(B, H, T, n, dtype=dtype) for n in (128, 128, 64))
    o = _run(lambda: LinearAttentionEngine(metas, custom_io=CustomIO({})), [t.cuda() for t in (q, k, v, a)], 4)
    parity.check("o", o, linear_scan(*(t.double() for t in (q, k, v, a))), dtype, stages=4, unnormalised=True)


def test_rule_cuts_only_where_sms_would_idle():
    """Few long walks are cut, unless gradients are wanted; a problem that fills the GPU is one walk per head, bit for bit as
    without the rule."""
    for H, T, cut in ((2, 2048, True), (160, 256, False)):
        gen = torch.Generator().manual_seed(H)
        q, k, v = ((0.3 * torch.randn(1, H, T, n, generator=gen)).to(torch.bfloat16).cuda() for n in (128, 128, 64))
        a = -0.01 * torch.rand(1, H, T, generator=gen).cuda()
        metas = tuple(meta_tensor(1, H, T, n, dtype=torch.bfloat16) for n in (128, 128, 64))
        eng = LinearAttentionEngine(metas, custom_io=CustomIO({}))
        with torch.no_grad():
            o = eng(q, k, v, a)
            eng._native_plan().segments = 1
            one = eng(q, k, v, a)
            eng._native_plan().segments = 0
        assert torch.equal(o, one) != cut
        assert torch.equal(eng(q.requires_grad_(), k, v, a), one)
