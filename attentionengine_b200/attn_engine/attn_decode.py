"""Split-KV decode for MHA / GQA: ``mod(q, k, v, *custom) -> o`` with ``q_len != kv_len``.

Reference: shape-class dispatch attention_engine/attn_engine/attn_engine.py:252-286 (GQA decode needs
``q_len == 1``), lowering core/lower/lower_decode.py / lower_decode_gqa.py, templates
core/template/tl_template/attn/attn_decode_tl.py:34-206 (split kernel + ``combine``), scripts
attn_script/gqa_inference.py and mha_inference.py.  Forward only, as in the reference.

The kernel is the forward attention kernel built with ``AE_DECODE``: the query rows of one head unit (the
query heads of a kv head's group, or the positions of one head) fill one tile, so K / V of a kv head are read
once per split whatever the group size; the splits' results are merged by the traced ``OnlineFunc.combine``.
The reference fixes ``num_split = 4`` (attn_decode_tl.py:230-236); here it is chosen so that the CTAs cover the
GPU once.

Rows of different lengths and paged K / V (the serving call of the reference's kv-shared path,
core/template/cute_template_kvshared/flash_mla_interface.py:73-113 with its scheduler
kernels/get_mla_metadata.cu:8-75) are ``decode_varlen``: ``schedule(cache_seqlens)`` cuts every row into shares of
about equal size, one CTA each, or for each head unit the line of all rows' tiles into equal intervals (attn_decode.cuh), and the
result is reused by every layer of a decode step.
A ``mask_mod`` is applied element by element (mask mode 3), the dense mask input of the reference's TL decode
(core/lower/lower_decode_gqa.py:390-396); the query position it sees is the row's index among the engine's q_len
positions.
"""
from __future__ import annotations

import torch

from .. import runtime as rt
from ..lower.cuda_lower import lower_attention, lower_combine

N_SM = 148
MAX_ROWS = 256  # two 128-row tiles per CTA


class AttnDecode:
    def __init__(self, score_mod, mask_mod, online_func, custom_fwd_inputs, Hq: int, Hkv: int, Sq: int, D: int, DV: int,
                 dtype, mask_value="-inf"):
        if Hq % Hkv:
            raise ValueError("query heads must be a multiple of kv heads")
        if Hq > Hkv and Sq != 1:
            raise NotImplementedError("decode with grouped query heads takes q_len == 1 (as the reference does)")
        self.rows = Hq // Hkv if Hq > Hkv else Sq
        if self.rows > MAX_ROWS:
            raise NotImplementedError(f"decode packs at most {MAX_ROWS} query rows per head unit, got {self.rows}")
        if D % 64 or DV % 64 or D > 128 or DV > 128:
            raise NotImplementedError(f"head dims D={D}, DV={DV}: multiples of 64 up to 128 are supported")
        self.Hq, self.Hkv, self.Sq, self.D, self.DV, self.dtype = Hq, Hkv, Sq, D, DV, dtype
        bf16 = dtype == torch.bfloat16
        tag = rt.DTYPE_BF16 if bf16 else rt.DTYPE_F16
        mask_mode = 0 if mask_mod is None else 3
        self.low = lower_attention(score_mod, mask_mod, online_func, custom_fwd_inputs, D=D, DV=DV, bf16=bf16,
                                   mask_mode=mask_mode, stages=2, mask_value=mask_value)
        # at most 128 rows: one q tile in shared memory, its space goes to a third K / V stage
        nq, stages = (1, 3) if self.rows <= 128 else (2, 2)
        smem = nq * 128 * D * 2 + stages * 128 * (D + DV) * 2 + 512 + 1024
        cfg = rt.KernelConfig(kind=rt.KIND_ATTN_DECODE, dtype=tag, head_dim=D, head_dim_v=DV, threads=192 if nq == 1 else 384,
                              smem_bytes=smem, stages=stages, mask_mode=mask_mode)
        cfg.reserved[1] = len(self.low.final_names)
        prelude = self.low.prelude_fwd.replace("#define AE_STAGES 2\n", f"#define AE_STAGES {stages}\n")
        assert f"#define AE_STAGES {stages}\n" in prelude
        self.src = rt.kernel_source("attn_fwd.cuh", prelude=prelude + f"#define AE_DECODE 1\n#define AE_NQ {nq}\n")
        self.kernel = rt.compile_module(self.src, "ae_attn_fwd", cfg)
        self.combine = None
        self.combine_src = None
        self.cut_kernel = None  # for intervals and clusters
        from .attn_engine import OnlineFunc
        overridden = getattr(type(online_func), "combine", None) is not OnlineFunc.combine
        # OnlineFunc.combine left at its default gives every split the weight 1: right for online functions without
        # row state (their partial outputs add up); with row state and no combine of its own the engine keeps one split.
        if overridden or not self.low.final_names:
            functor = lower_combine(online_func)
            if functor is not None:
                if nq == 1:  # built here like the others: lengths decide at run time, and a serving call should not wait for a compiler
                    cut_src = rt.kernel_source("attn_decode.cuh", prelude=prelude).replace("//%%AE_COMBINE_FUNCTOR%%", functor)
                    self.cut_kernel = rt.compile_module(cut_src, "ae_attn_decode", rt.KernelConfig.from_buffer_copy(bytes(cfg)))
                comb = (rt.KERNEL_DIR / "mla_combine.cuh").read_text().replace("//%%AE_COMBINE_FUNCTOR%%", functor)
                head = (rt.KERNEL_DIR / "ae_sm100.cuh").read_text().replace("#pragma once\n", "") + \
                    (rt.KERNEL_DIR / "ae_args.h").read_text()
                defs = f"#define AE_BF16 {int(bf16)}\n#define AE_NFINAL {len(self.low.final_names)}\n#define AE_DV {DV}\n"
                self.combine_src = head + defs + comb
                cfg2 = rt.KernelConfig(kind=rt.KIND_MLA_COMBINE, dtype=tag, head_dim=D, head_dim_v=DV, threads=128,
                                       smem_bytes=0)
                self.combine = rt.compile_module(self.combine_src, "ae_mla_combine", cfg2)
        self.num_split = None  # None = choose per call
        self.last_num_split = None
        self._plan = None  # the native side, made at the first call
        self._splits = {}  # (batch rows, kv tiles) -> (split count, whether the splits merge in a cluster)

    @property
    def units(self):
        return self.Hkv if self.Hq > self.Hkv else self.Hq

    def pick_splits(self, B: int, Skv: int) -> int:
        """How many splits a call of one length takes, see ``_pick``.  One when the online function has row state but no combine of
        its own."""
        return self._pick(B, Skv)[0]

    def _pick(self, B: int, Skv: int):
        """(splits, whether they merge in a cluster), by tile periods: a CTA occupies an SM alone, so the CTAs run in waves of 148,
        and each pays about three periods to fill its pipeline and write its partials (measured at B = 16: 2 splits 0.131 ms,
        8 splits 0.139 ms).  No empty split.

        Up to eight short splits of few rows are a cluster and merge in it: one launch, 6.6 us of the host's time instead of
        9.8.  The GPU takes 0.3 to 0.5 us longer than with the launch that merges, 8 to 12 us a call of up to two tiles a split, less than
        the host needs for what surrounds it; longer splits are the GPU's time alone, and captured calls take the launch (same
        bits, see attn_decode.cuh).  At most 16 rows a unit (64 rows: 10.3 -> 11.7 us).  All clusters at once, a whole SM's shared memory a
        CTA: 112 CTAs in clusters of seven and eight (16 clusters of eight took two rounds, 9.8 -> 16.4 us), and up to 96 of the
        smaller ones (32 clusters of four 12.8 -> 13.8); seven or eight splits that are more are four, of two tiles."""
        if self.combine is None:
            return 1, False
        n_tiles = -(-Skv // 128)
        known = self._splits.get((B, n_tiles))  # one look: another thread may clear the table
        if known is not None:
            return known
        units = B * self.units
        best, cost = 1, None
        for n in range(1, min(32, n_tiles) + 1):
            tps = -(-n_tiles // n)
            if (n - 1) * tps >= n_tiles:
                continue
            c = -(-units * n // N_SM) * (tps + 3)
            if cost is None or c < cost:
                best, cost = n, c
        pick = best, False
        n = 4 if 6 < best <= 8 and units * best > 112 else best
        if 1 < n <= 8 and self.cut_kernel is not None and self.rows <= 16 and -(-n_tiles // n) <= 2 and \
                units * n <= (112 if n > 6 else 96):
            pick = n, True
        if len(self._splits) >= 4096:  # a serving loop over many batch sizes and lengths must not grow without bound
            self._splits.clear()
        self._splits[B, n_tiles] = pick
        return pick

    # ------------------------------------------------------------------------------------------------------
    # rows of different lengths
    # ------------------------------------------------------------------------------------------------------
    def schedule(self, cache_seqlens, device=None, waves: int = 1):
        """Work list for a batch whose rows hold ``cache_seqlens[b]`` keys: every row is cut into shares of at most
        ``g`` 128-key tiles, ``g`` chosen so that the shares of all rows and head units fill the GPU ``waves`` times
        (at least 2 tiles per share, at most 32 shares per row); or, for long rows, the number of equal intervals that all
        rows' tiles are cut into for each head unit (``_pick_intervals``).  Returns a dict of device tensors that
        ``decode_varlen`` takes; compute it once per decode step and reuse it for every layer (the reference's
        ``get_mla_metadata`` is used the same way).  Reads the lengths on the host (one small copy)."""
        lens = torch.as_tensor(cache_seqlens).to("cpu", torch.int64)
        if lens.dim() != 1 or int(lens.min()) < 1:
            raise ValueError("cache_seqlens must be a 1-D tensor of positive lengths")
        B = lens.numel()
        units = self.units
        tiles = (lens + 127) // 128
        if self.combine is None:
            g = int(tiles.max())  # no combine: one share per row
        else:
            total = int(tiles.sum()) * units
            g = max(2, -(-total // (N_SM * waves)))
            g = max(g, -(-int(tiles.max()) // 32))
        items, part_off = [], [0]
        for b in range(B):
            nt = int(tiles[b])
            n = -(-nt // g)
            per = -(-nt // n)
            n = -(-nt // per)  # no empty share
            for sidx in range(n):
                items.append((b, sidx, sidx * per, min(per, nt - sidx * per)))
            part_off.append(part_off[-1] + n)
        # Waves asked for by the caller are shares' alone.  The work list is made in any case: an engine with other head units that is
        # handed the schedule takes it (see _run).
        intervals = self._pick_intervals(B, tiles, items) if waves == 1 else 0
        dev = device if device is not None else (cache_seqlens.device if isinstance(cache_seqlens, torch.Tensor)
                                                 and cache_seqlens.is_cuda else torch.device("cuda"))
        return {"work": torch.tensor(items, dtype=torch.int32).to(dev), "n_items": len(items),
                "part_off": torch.tensor(part_off, dtype=torch.int32).to(dev), "n_slots": part_off[-1],
                "seqlens": lens.to(torch.int32).to(dev), "max_seqlen": int(lens.max()), "tiles_per_share": g, "B": B,
                "intervals": intervals, "units": units}

    def _pick_intervals(self, B, tiles, items) -> int:
        """Intervals per head unit for long rows (the kernel cuts all rows' tiles into them by its own reading of the lengths), or 0
        where the shares ``items`` are expected to be faster.  Microseconds, as measured over 1 to 128 units, 2 to 64 rows, even,
        uniform and skewed lengths, dense and paged: a tile takes a CTA 1.3 (in shares 1.15 at 64 dims) and all CTAs together 0.0101 of
        HBM; a share costs three tiles more than it holds, an interval 2 us for every row that it begins.  Intervals are one
        wave of N_SM // units CTAs a unit, so they leave SMs idle where the units do not divide N_SM.  In shares / in intervals:
        64 rows up to 8192 keys over 8 units (144 CTAs) 216 / 189; 16 rows of 4096 over 80 units (80 CTAs) 436 / 659; 64 of 4096 over 32
        units (128 CTAs) 670 / 704; 4 rows up to 8192 over 1 unit 17 / 21; 6 rows of 16384 over 48 units of 64 dims 277 / 329."""
        n, total, units = N_SM // self.units, int(tiles.sum()), self.units
        if self.cut_kernel is None or n == 0 or B == 1 or total < 16 * B:
            return 0
        size = (self.D + self.DV) / 256
        together = 0.0101 * size * total * units
        longest = max(x[3] for x in items) + 3
        in_turn = min(-(-units * len(items) // N_SM) * longest, units * (total + 3 * len(items)) / N_SM + 0.7 * longest)
        shares = 10 + max(together, (1 + 0.3 * size) * in_turn)
        per_cta = max(-(-total // n), -(-int(tiles.max()) // 31))
        return n if 16 + max(together, 1.3 * per_cta + 2 * (1 - (-B // n))) < shares else 0

    def decode_varlen(self, q, k, v, cache_seqlens, *custom, block_table=None, metadata=None):
        """``q`` [B, q_len, Hq, D]; dense ``k`` / ``v`` [B, S_max, Hkv, D] of which row b uses its first
        ``cache_seqlens[b]`` keys, or, with ``block_table`` [B, max_pages] int32, pools [num_pages, 128, Hkv, D]
        whose pages a row lists in order.  ``metadata`` = ``schedule(cache_seqlens)`` (computed here when absent)."""
        meta = metadata if metadata is not None else self.schedule(cache_seqlens, q.device)
        return self._run(q, k, v, custom, meta, block_table)

    def __call__(self, q, k, v, *custom):
        return self._run(q, k, v, custom, None, None)

    def _native_plan(self):
        if self._plan is None:
            from .attn_engine import custom_slots
            self._plan = rt.host().DecodePlan(self.kernel.handle.value, self.combine.handle.value if self.combine else 0,
                                              self.dtype == torch.bfloat16, self.Hq, self.Hkv, self.Sq, self.D, self.DV,
                                              len(self.low.final_names), custom_slots(self.low.custom),
                                              self.cut_kernel.handle.value if self.cut_kernel else 0)
        return self._plan

    @property
    def status(self):
        return self._plan.status if self._plan is not None else None

    def _run(self, q, k, v, custom, meta, block_table):
        if meta is None:
            cut, n_split, in_cluster = 0, self.num_split, False
            if not n_split:
                n_split, in_cluster = self._pick(q.shape[0], k.shape[1]) if q.dim() == k.dim() == 4 else (1, False)
            m = None
        else:
            # the work list serves any engine, intervals only one with the head units they were counted for and the kernel for them
            cut = meta.get("intervals", 0) if self.cut_kernel is not None and meta.get("units") == self.units else 0
            n_split, in_cluster = 1, False
            m = (meta["work"], meta["n_items"], meta["seqlens"], meta["part_off"], meta["n_slots"], meta["max_seqlen"], meta["B"])
        o = rt.host().decode(self._plan or self._native_plan(), q, k, v, custom, n_split, m, block_table, cut, in_cluster)
        if o is None:
            self._refuse(q, k, v, custom, meta, block_table, n_split)
        if meta is None:
            self.last_num_split = n_split
        else:  # pieces of a row on average; every end of an interval but the last counted as a cut
            self.last_num_split = (meta["B"] + cut - 1 if cut else meta["n_slots"]) / meta["B"]
        return o

    def _refuse(self, q, k, v, custom, meta, block_table, n_split):
        """The native path did not take these tensors: raise what is wrong with them."""
        for name, t in (("q", q), ("k", k), ("v", v)):
            if not t.is_cuda:
                raise rt.AeError(f"{name} must be a CUDA tensor: this back end has no CPU path")
            if t.dtype != self.dtype:
                raise TypeError(f"{name} has dtype {t.dtype}, engine was built for {self.dtype}")
            if t.dim() != 4 or t.stride(3) != 1:
                raise ValueError(f"{name} must be [B, S, H, D] with a contiguous last dimension")
        B, Sq, Hq, D = q.shape
        _, Skv, Hkv, _ = k.shape
        if (Sq, Hq, Hkv, D, v.shape[3]) != (self.Sq, self.Hq, self.Hkv, self.D, self.DV) or v.shape[:3] != k.shape[:3]:
            raise ValueError("q / k / v shapes differ from the engine's")
        if block_table is not None:
            if meta is None:
                raise ValueError("paged K / V go through decode_varlen")
            if Skv != 128 or k.stride(0) != 128 * k.stride(1) or v.stride(0) != 128 * v.stride(1):
                raise ValueError("paged K / V pools are [num_pages, 128, Hkv, D] with the keys of a page contiguous")
            if block_table.dtype != torch.int32 or block_table.dim() != 2 or block_table.shape[0] != B or \
                    not block_table.is_contiguous() or block_table.shape[1] * 128 < meta["max_seqlen"]:
                raise ValueError("block_table must be contiguous int32 [B, max_pages] covering the longest row")
        elif k.shape[0] != B:
            raise ValueError("q / k / v shapes differ from the engine's")
        if meta is not None and (meta["B"] != B or (block_table is None and meta["max_seqlen"] > Skv)):
            raise ValueError("the schedule was made for other lengths than these tensors hold")
        specs = self.low.custom
        if len(custom) != len(specs):
            raise TypeError(f"expected {len(specs)} custom input(s) {[s.name for s in specs]}, got {len(custom)}")
        if n_split > 1 and self.combine is None:
            raise ValueError("more than one split needs OnlineFunc.combine")
        for sp, t in zip(specs, custom):
            if sp.is_16bit:
                raise NotImplementedError("tile-shaped custom inputs are not wired into the decode kernel")
            if not t.is_cuda:
                raise rt.AeError("custom inputs must be CUDA tensors: this back end has no CPU path")
            if any(slot >= 0 for slot in sp.dim_slots[t.dim():]):
                raise ValueError(f"custom input {sp.name}: expected {len(sp.shape)} dims, got {tuple(t.shape)}")
        if block_table is not None and not block_table.is_cuda:
            raise rt.AeError("block_table must be a CUDA tensor: this back end has no CPU path")
        raise ValueError("tensors do not fit this engine")
