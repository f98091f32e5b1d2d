"""MLA (kv_shared) decode path of AttentionEngine: ``mod(q, q_pe, kv, k_pe) -> o``.

Reference: shape-class dispatch ``kv_shared`` (attention_engine/attn_engine/attn_engine.py:235-250),
lowering core/lower/lower_decode_mla.py:25-38 and template core/template/tl_template/attn/mla_decode_tl.py.
Unlike the reference, which ignores ``score_mod`` / ``online_func`` on this path and hard-codes
softmax with scale 1/sqrt(576) (mla_decode_tl.py:30), the traced callables are honoured here, so the
user's ``score * softmax_scale`` decides the scale.  Forward only, as in the reference (:337-339).
"""
from __future__ import annotations

import torch

from .. import runtime as rt
from ..lower.cuda_lower import lower_attention, lower_combine

N_SM = 148


class MlaDecode:
    def __init__(self, score_mod, online_func, custom_fwd_inputs, H: int, D: int, DV: int, dtype):
        if (D, DV) != (576, 512):
            raise NotImplementedError(f"MLA decode is built for D = 512 + 64, DV = 512; got D={D}, DV={DV}")
        if H > 128:
            raise NotImplementedError("MLA decode handles up to 128 query heads per latent KV")
        if custom_fwd_inputs.input_tensors:
            raise NotImplementedError("custom inputs are not wired into the MLA decode kernel")
        self.dtype = dtype
        bf16 = dtype == torch.bfloat16
        self.low = lower_attention(score_mod, None, online_func, custom_fwd_inputs, D=D, DV=DV, bf16=bf16, mask_mode=0)
        tag = rt.DTYPE_BF16 if bf16 else rt.DTYPE_F16
        # Q and K (9 blocks of 64 x 128 B each), V (4 blocks of 128 x 128 B), P, barriers, exchanged row reductions, alignment
        smem = 18 * 64 * 128 + 4 * 128 * 128 + 2 * 64 * 128 + 512 + 1024 + 1024
        cfg = rt.KernelConfig(kind=rt.KIND_MLA_DECODE, dtype=tag, head_dim=D, head_dim_v=DV, threads=192,
                              smem_bytes=smem, stages=1, mask_mode=0)
        self.src = rt.kernel_source("mla_decode.cuh", prelude=self.low.prelude_fwd, defines={"AE_RSPLIT": 2, "AE_XCH_ROWS": 64})
        self.decode = rt.compile_module(self.src, "ae_mla_decode", cfg)
        comb = (rt.KERNEL_DIR / "mla_combine.cuh").read_text().replace("//%%AE_COMBINE_FUNCTOR%%", lower_combine(online_func))
        cfg2 = rt.KernelConfig(kind=rt.KIND_MLA_COMBINE, dtype=tag, head_dim=D, head_dim_v=DV, threads=128, smem_bytes=0)
        head = (rt.KERNEL_DIR / "ae_sm100.cuh").read_text().replace("#pragma once\n", "") + (rt.KERNEL_DIR / "ae_args.h").read_text()
        defs = f"#define AE_BF16 {int(bf16)}\n#define AE_NFINAL {len(self.low.final_names)}\n#define AE_DV {DV}\n"
        self.combine_src = head + defs + comb
        self.combine = rt.compile_module(self.combine_src, "ae_mla_combine", cfg2)
        # None = the kernel cuts the tiles of all rows into equal intervals, one per CTA pair (its split 0); n = n shares per row
        self.num_split = None
        from .attn_engine import OnlineFunc
        overridden = getattr(type(online_func), "combine", None) is not OnlineFunc.combine
        self._auto_split = 0 if overridden or not self.low.final_names else 1  # row state without a combine: rows stay whole
        self.last_num_split = None  # of the last call: the most shares that a row was cut into
        self._plan = None  # the native side, made at the first call

    def _native_plan(self):
        if self._plan is None:
            self._plan = rt.host().MlaPlan(self.decode.handle.value, self.combine.handle.value, self.dtype == torch.bfloat16,
                                           len(self.low.final_names), N_SM // 2)
        return self._plan

    @property
    def status(self):
        return self._plan.status if self._plan is not None else None

    def __call__(self, q, q_pe, kv, k_pe):
        res = rt.host().mla(self._plan or self._native_plan(), q, q_pe, kv, k_pe, self.num_split or self._auto_split)
        if res is None:  # not launched: say what does not fit
            for name, t in (("q", q), ("q_pe", q_pe), ("kv", kv), ("k_pe", k_pe)):
                if not t.is_cuda:
                    raise rt.AeError(f"{name} must be a CUDA tensor: this back end has no CPU path")
                if t.dtype != self.dtype:
                    raise TypeError(f"{name} has dtype {t.dtype}, engine was built for {self.dtype}")
            if q.dim() == kv.dim() == 4 and 0 in (q.shape[0], q.shape[2], kv.shape[1]):
                raise rt.AeError(f"MLA decode of an empty problem: q {tuple(q.shape)}, kv {tuple(kv.shape)}")
            raise ValueError("expected q [B,1,H,512], q_pe [B,1,H,64], kv [B,S,1,512], k_pe [B,S,1,64]")
        o, self.last_num_split = res
        return o

    def paged(self, q, kcache, block_table, cache_seqlens, num_split=None):
        """Decode over a paged KV pool with one length per batch row; returns (o [B, 1, H, 512], lse [B, H] fp32).

        The call of the reference's CuTe kv-shared path (core/template/cute_template_kvshared/flash_mla_interface.py:73-113,
        attn_script/mla_decode_cute.py:295-303): q [B, 1, H, 576] (latent 512 + rope 64), kcache [num_pages, 64, 1, 576]
        or [num_pages, 64, 576], block_table [B, max_pages] int32 (page of each 64-key tile), cache_seqlens [B] int32.
        The kernel cuts the work by the lengths itself, so the launch needs none on the host; they are read back behind the
        launches only to raise on one outside the table."""
        if list(self.low.final_names) != ["lse"]:
            raise NotImplementedError("the paged call returns the log-sum-exp: the online function must have the final row scale 'lse'")
        res = rt.host().mla_paged(self._plan or self._native_plan(), q, kcache, block_table, cache_seqlens,
                                  num_split or self.num_split or self._auto_split)
        if res is None:
            self._refuse_paged(q, kcache, block_table, cache_seqlens)
        if not res:
            raise ValueError("cache_seqlens must lie in [1, max_pages * 64]")
        o, lse, self.last_num_split = res
        return o, lse

    def _refuse_paged(self, q, kcache, block_table, cache_seqlens):
        for name, t in (("q", q), ("kcache", kcache)):
            if not t.is_cuda:
                raise rt.AeError(f"{name} must be a CUDA tensor: this back end has no CPU path")
            if t.dtype != self.dtype:
                raise TypeError(f"{name} has dtype {t.dtype}, engine was built for {self.dtype}")
        B, one, H, D = q.shape
        if one != 1 or D != 576 or H > 128:
            raise ValueError("expected q [B, 1, H <= 128, 576]")
        if B == 0 or H == 0:
            raise rt.AeError(f"MLA decode of an empty problem: q {tuple(q.shape)}")
        if kcache.dim() == 4:
            if kcache.shape[2] != 1:
                raise ValueError("expected kcache [num_pages, 64, 1, 576]")
            kcache = kcache[:, :, 0]
        if kcache.shape[1:] != (64, 576) or not kcache.is_contiguous():
            raise ValueError("expected a contiguous kcache of 64-key pages, [num_pages, 64, (1,) 576]")
        if block_table.shape[0] != q.shape[0] or cache_seqlens.shape != (q.shape[0],):
            raise ValueError("block_table is [B, max_pages], cache_seqlens is [B]")
        raise ValueError("tensors do not fit this engine")
