"""The pre-pass of the one-pass backward clears the dQ buffer on its way: head dims that differ, rows that do not fill a block, and a
buffer that holds the sums of the step before."""
import pytest
import torch

import parity
from attentionengine_b200 import examples as helpers
from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hkv,S,D,DV,causal", [(1, 2, 1, 130, 64, 128, True), (2, 4, 4, 200, 128, 64, False), (1, 3, 3, 77, 128, 128, True),
                                                    (2, 2, 2, 5, 64, 64, False)])
def test_gradients_do_not_see_the_buffer_of_the_step_before(B, Hq, Hkv, S, D, DV, causal):
    dtype = torch.float16
    eng = helpers.softmax_engine(B, Hq, Hkv, S, D, DV, dtype, causal)
    q, k, v, d_o = helpers.seeded_qkv(B, Hq, Hkv, S, D, DV, dtype, seed=S, device="cuda")
    for t in (q, k, v):
        t.requires_grad_()
    for _ in range(2):
        for t in (q, k, v):
            t.grad = None
        o = eng(q, k, v)
        o.backward(d_o)
    torch.cuda.synchronize()
    eng.check_status()
    ref_o, ref_g = orc.fwd_bwd(lambda a, b, c: orc.softmax_attention(a, b, c, causal), tuple(t.detach().cpu() for t in (q, k, v)), d_o.cpu())
    for name, got, ref in (("o", o, ref_o), ("dq", q.grad, ref_g[0]), ("dk", k.grad, ref_g[1]), ("dv", v.grad, ref_g[2])):
        parity.check(name, got, ref, dtype)
