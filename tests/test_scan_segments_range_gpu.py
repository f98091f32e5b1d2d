"""Segments of a scan in fp16 where a value times all the decay to the end of its segment is far below fp16's range, or far above it, while
state and output are not: against the scan in fp64."""
import pytest
import torch

from attentionengine_b200 import CustomIO, LinearAttentionEngine, meta_tensor
from oracle.linear_oracle import linear_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("DV", [64, 128])
@pytest.mark.parametrize("folds,k_size,v_size", [(-7.0, 16.0, 5e-4), (12.0, 1e-3, 1.0)])
def test_values_keep_their_bits_over_a_segment(folds, k_size, v_size, DV):
    B, H, T, dtype = 1, 2, 1024, torch.float16  # two segments of 512 steps
    gen = torch.Generator().manual_seed(DV)
    q, k, v = ((size * torch.randn(B, H, T, n, generator=gen)).to(dtype) for size, n in ((0.3, 128), (k_size, 128), (v_size, DV)))
    v[:, :, 128:] = 0  # what the second segment puts out came in with the first chunk
    a = torch.full((B, H, T), folds / 512)
    a[:, :, 512:] = -0.01
    eng = LinearAttentionEngine(tuple(meta_tensor(B, H, T, n, dtype=dtype) for n in (128, 128, DV)), custom_io=CustomIO({}))
    ref = linear_scan(q, k, v, a)[:, :, 512:640]
    eng._native_plan().segments = 2
    with torch.no_grad():
        o = eng(*(t.cuda() for t in (q, k, v, a)))[:, :, 512:640].cpu().double()
    eng.check_status()
    # one rounding to fp16 each of the weighted value, the state's copy and the output
    assert (o - ref).norm() / ref.norm() <= 3 * 2.0 ** -11
