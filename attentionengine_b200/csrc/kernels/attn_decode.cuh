// Split-KV decode for sm_100a with at most 128 query rows per head unit (reference: attn_decode_tl.py:34-141,
// attn_gqa_decode_tl.py; varlen scheduling get_mla_metadata.cu:8-75), for two kinds of calls that the plain splits of
// attn_fwd.cuh (AE_DECODE: one CTA per row, unit and split) serve less well.  A unit is a kv head (its group's query heads are
// the rows) or a head with its own K / V (its query positions are).
//   args.n_intervals > 0: long rows of different lengths.  For every unit, the 128-key tiles of all rows in one line, cut into
//     equal intervals, one per CTA (grid: unit, interval); an interval may hold the end of a row, whole rows and the beginning
//     of one.  The kernel finds it from the lengths itself.  What bounds decode is HBM; shares of single rows left SMs uneven,
//     each with the fill and drain of its pipeline: 64 rows up to 8192 keys over pages 210 us in shares, 199 in intervals; 11 rows
//     up to 10490 keys 70 and 56.  K and V of the next row stream in under the tail of the one before.  All units walk the same
//     keys at the same time, side by side as the heads of a key lie in memory: with the units of a row one after the other the 64
//     rows took 217.  Rows of one length are as even in plain splits and read faster there (16 rows of 8192 keys 96 us, 102 in
//     intervals).
//   args.in_cluster: short calls made one by one.  The splits of a unit (grid: split, unit, batch row) are the CTAs of one cluster,
//     which leave their partials in shared memory and merge them there: one launch for the host instead of two (6.6 us a call instead of
//     9.8).  The GPU itself is 0.3 to 0.5 us quicker with the launch that merges, brought up under its split kernel (2 rows of 1000 keys
//     in four splits 10.2 us, in clusters 10.5), so captured calls take that.
// A segment is a stretch of tiles of one row; a row inside one interval is written directly, others leave normalised fp32 partials
// for ae_mla_combine.
//
// Roles: warps 0-3 row threads (thread i = row i), warp 4 TMA producer of K and V, warp 5 MMA issuer, which also loads Q.
// TMEM columns: S0 | S1 | O.  The scores of the CTA's n-th tile go to region n & 1 and the S GEMM runs two tiles ahead of P V, so
// the row threads find the next tile's scores ready when they finish a tile.
// Expects the forward prelude (AE_D, AE_DV, AE_BF16, AE_STAGES >= 3, AE_MASK_MODE 0 or 3, ...) and the traced merge.

AE_DEVICE float ae_warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
AE_DEVICE float ae_warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
//%%AE_COMBINE_FUNCTOR%%
AE_DEVICE float ld_cluster_f32(u32 addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
AE_DEVICE void ld_cluster(float (&v)[2], u32 addr) {
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(addr) : "memory");
}
AE_DEVICE void ld_cluster(float (&v)[4], u32 addr) {
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(addr)
               : "memory");
}

#define AE_BM 128
#define AE_BN 128
#if AE_MASK_MODE != 0 && AE_MASK_MODE != 3
#error "the decode build takes no mask, or an element-wise one (mask mode 3)"
#endif
#if AE_STAGES < 3
#error "the two-ahead S GEMM needs three K / V stages"
#endif
#define AE_NTHREADS 192
#define AE_Q_BYTES (AE_BM * AE_D * 2)
#define AE_K_BYTES (AE_BN * AE_D * 2)
#define AE_V_BYTES (AE_BN * AE_DV * 2)
#define AE_SMEM_Q 0
#define AE_SMEM_K AE_Q_BYTES
#define AE_SMEM_V (AE_SMEM_K + AE_STAGES * AE_K_BYTES)
#define AE_SMEM_BAR (AE_SMEM_V + AE_STAGES * AE_V_BYTES)
#define AE_PART_LD (AE_DV + 4)  // floats from row to row of a cluster's partials: the threads of a warp, a row each, in different banks
static_assert(128 * (AE_PART_LD + AE_NFINAL) * 4 <= AE_STAGES * (AE_K_BYTES + AE_V_BYTES), "a cluster's partials lie in the K / V ring");

struct AeDecBars {
  u64 q_full, q_free;  // Q of a segment has landed; its last S GEMM has read it
  u64 k_full[AE_STAGES], k_empty[AE_STAGES];
  u64 v_full[AE_STAGES], v_empty[AE_STAGES];
  u64 s_full[2], p_full[2];
  u64 o_done;  // one phase per tile
  AeCtaCtl ctl;
  int row0, tile0, share, total;
};
static_assert(sizeof(AeDecBars) <= 512, "barrier block");

struct AeDecSeg {
  int b;      // batch row
  int kt, n;  // tiles [kt, kt + n)
  int keys;   // of the row
  bool whole;
};

extern "C" __global__ void __launch_bounds__(AE_NTHREADS, 1) ae_attn_decode(const __grid_constant__ AeAttnFwdArgs args) {
  extern __shared__ u8 smem_raw[];
  u8* smem = smem_align1024(smem_raw);
  AeDecBars* bars = (AeDecBars*)(smem + AE_SMEM_BAR);
  AeCtaCtl* ctl = &bars->ctl;
  const u32 warp = threadIdx.x >> 5;
  const u32 lane = threadIdx.x & 31;
  auto keys_of = [&](int b) { return args.seqlens ? args.seqlens[b] : args.Skv; };
  auto tiles_of = [](int keys) { return (keys + AE_BN - 1) / AE_BN; };

  if (threadIdx.x == 0) {
    ctl->abort = 0;
    mbar_init(&bars->q_full, 1);
    mbar_init(&bars->q_free, 1);
    for (int i = 0; i < AE_STAGES; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], 1);
      mbar_init(&bars->v_full[i], 1);
      mbar_init(&bars->v_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->p_full[i], 4);
    }
    mbar_init(&bars->o_done, 1);
    mbar_fence_init();
  }
  if (warp == 0 && args.n_intervals > 0) {
    // this CTA's interval: all tiles, equal shares (a row spans at most 32 of them), the row and tile it begins at
    int total = 0, longest = 0;
    const int n_mine = args.seqlens && (int)lane < args.B ? tiles_of(keys_of((int)lane)) : 0;  // the first 32 rows are read once
    if (args.seqlens) {
      for (int b = (int)lane; b < args.B; b += 32) {
        const int n = b < 32 ? n_mine : tiles_of(keys_of(b));
        total += n;
        longest = n > longest ? n : longest;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        total += __shfl_xor_sync(0xffffffffu, total, o);
        const int l = __shfl_xor_sync(0xffffffffu, longest, o);
        longest = l > longest ? l : longest;
      }
    } else {
      longest = tiles_of(args.Skv);
      total = longest * args.B;
    }
    int share = (total + args.n_intervals - 1) / args.n_intervals;
    if (share < (longest + 30) / 31) share = (longest + 30) / 31;
    const int g0 = (int)blockIdx.y * share;
    int row0 = 0, tile0 = 0;
    if (!args.seqlens) {
      row0 = g0 / longest;
      tile0 = g0 % longest;
    } else if (g0 < total) {
      int before = 0;
      for (int base = 0; base < args.B; base += 32) {
        const int b = base + (int)lane;
        const int n = base == 0 ? n_mine : b < args.B ? tiles_of(keys_of(b)) : 0;
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o);
          if ((int)lane >= o) incl += y;
        }
        const u32 hit = __ballot_sync(0xffffffffu, b < args.B && before + incl > g0);
        if (hit) {
          const int src = __ffs(hit) - 1;
          row0 = base + src;
          tile0 = g0 - (before + __shfl_sync(0xffffffffu, incl - n, src));
          break;
        }
        before += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    if (lane == 0) {
      bars->row0 = row0;
      bars->tile0 = tile0;
      bars->share = share;
      bars->total = total;
    }
  }
  if (warp == 5) {
    tmem_alloc(&ctl->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const u32 tmem = ctl->tmem_base;
  ae_grid_trigger();
  const u32 TM_S = 0, TM_O = 256;  // S region i at TM_S + 128 i

  // ---- the CTA's segments, the same walk in every role ----
  struct Walk {
    int b, tile, left;
  } w0;
  int unit;
  if (args.n_intervals > 0) {
    unit = (int)blockIdx.x;
    const int left = bars->total - (int)blockIdx.y * bars->share;
    w0 = {bars->row0, bars->tile0, left < bars->share ? left : bars->share};
  } else {
    unit = (int)blockIdx.y;
    const int kt = (int)blockIdx.x * args.tiles_per_split, n = args.n_kt - kt;
    w0 = {(int)blockIdx.z, kt, n < args.tiles_per_split ? n : args.tiles_per_split};
  }
  const int n_all = w0.left > 0 ? w0.left : 0;  // tiles of this CTA
  auto next_seg = [&](Walk& w, AeDecSeg& s) -> bool {
    if (w.left <= 0) return false;
    s.b = w.b++;
    s.kt = w.tile;
    s.keys = keys_of(s.b);
    const int n_t = tiles_of(s.keys);
    s.n = n_t - w.tile < w.left ? n_t - w.tile : w.left;
    s.whole = s.n == n_t;
    w.left -= s.n;
    w.tile = 0;
    return true;
  };

  if (warp == 4) {
    // =============================== TMA producer: K and V ===============================
    if (lane == 0) {
      tma_prefetch_desc(&args.tm_k);
      tma_prefetch_desc(&args.tm_v);
      Walk w = w0;
      AeDecSeg s;
      bool ok = true;
      int it = 0;
      while (ok && next_seg(w, s)) {
        // paged K / V (args.block_table): the pool is one batch of num_pages * 128 rows, a tile is a page
        const int kv_b = args.block_table ? 0 : s.b;
        for (int j = 0; j < s.n; ++j, ++it) {
          const int stage = it % AE_STAGES;
          const u32 par = ((it / AE_STAGES) & 1) ^ 1;
          const int row0 = (args.block_table ? args.block_table[(i64)s.b * args.max_pages + s.kt + j] : s.kt + j) * AE_BN;
          if (!(ok = mbar_wait(&bars->k_empty[stage], par, ctl, args.status, 1))) break;
          mbar_arrive_expect_tx(&bars->k_full[stage], AE_K_BYTES);
          for (int dh = 0; dh < AE_D / 64; ++dh)
            tma_load_bshd(smem + AE_SMEM_K + stage * AE_K_BYTES + dh * (AE_BN * 128), &args.tm_k, &bars->k_full[stage], dh * 64,
                          unit, row0, kv_b);
          if (!(ok = mbar_wait(&bars->v_empty[stage], par, ctl, args.status, 2))) break;
          mbar_arrive_expect_tx(&bars->v_full[stage], AE_V_BYTES);
          for (int dh = 0; dh < AE_DV / 64; ++dh)
            tma_load_bshd(smem + AE_SMEM_V + stage * AE_V_BYTES + dh * (AE_BN * 128), &args.tm_v, &bars->v_full[stage], dh * 64,
                          unit, row0, kv_b);
        }
      }
    }
  } else if (warp == 5) {
    // =============================== MMA issuer, Q loads =================================
    if (lane == 0 && n_all > 0) {
      tma_prefetch_desc(&args.tm_q);
      const u32 idesc_s = umma_idesc_f16(AE_BM, AE_BN, AE_BF16, 0, 0);
      const u32 idesc_o = umma_idesc_f16(AE_BM, AE_DV, AE_BF16, 0, 1);
      const u64 da = umma_base_k(smem_u32(smem + AE_SMEM_Q));
      const u64 dk0 = umma_base_k(smem_u32(smem + AE_SMEM_K));
      const u64 dv0 = umma_base_mn(smem_u32(smem + AE_SMEM_V), AE_BN);
      bool ok = true;
      Walk wq = w0, wp = w0;
      AeDecSeg sq, sp;
      int n_q = 0;             // segments whose Q has been requested
      int ns = 0, s_left = 0;  // tiles whose S has been issued; S to go in the segment they are in
      int p_left = 0;          // P V to go in the segment they are in
      auto load_q = [&]() -> bool {  // Q of the next segment, once the S GEMMs of the one before have read theirs
        if (!next_seg(wq, sq)) return true;
        if (n_q > 0 && !mbar_wait(&bars->q_free, (n_q - 1) & 1, ctl, args.status, 3)) return false;
        mbar_arrive_expect_tx(&bars->q_full, AE_Q_BYTES);
        for (int dh = 0; dh < AE_D / 64; ++dh)
          tma_load_bshd(smem + AE_SMEM_Q + dh * (AE_BM * 128), &args.tm_q, &bars->q_full, dh * 64, unit, 0, sq.b);
        s_left = sq.n;
        ++n_q;
        return true;
      };
      bool fresh = true;  // the segment's Q has not been waited for
      auto issue_s = [&]() -> bool {
        const int stage = ns % AE_STAGES;
        if (fresh && !mbar_wait(&bars->q_full, (n_q - 1) & 1, ctl, args.status, 4)) return false;
        if (!mbar_wait(&bars->k_full[stage], (ns / AE_STAGES) & 1, ctl, args.status, 7)) return false;
        tc_fence_after_sync();
        const u64 db = dk0 + (u64)((stage * AE_K_BYTES) >> 4);
        const u32 d = tmem + TM_S + (ns & 1) * 128;
#pragma unroll
        for (int kk = 0; kk < AE_D / 16; ++kk)
          umma_ss(d, umma_step_k(da, kk, AE_BM), umma_step_k(db, kk, AE_BN), idesc_s, kk > 0);
        umma_commit(&bars->s_full[ns & 1]);
        umma_commit(&bars->k_empty[stage]);
        ++ns;
        fresh = --s_left == 0;
        if (fresh) umma_commit(&bars->q_free);
        return true;
      };
      ok = load_q() && issue_s();
      if (ok && ns < n_all) ok = (s_left > 0 || load_q()) && issue_s();
      for (int n = 0; n < n_all && ok; ++n) {
        const int stage = n % AE_STAGES;
        if (s_left == 0 && ns < n_all && !(ok = load_q())) break;  // under the row threads' pass
        ok = mbar_wait(&bars->p_full[n & 1], (n >> 1) & 1, ctl, args.status, 5) &&
             mbar_wait(&bars->v_full[stage], (n / AE_STAGES) & 1, ctl, args.status, 6);
        if (!ok) break;
        tc_fence_after_sync();
        const bool first = p_left == 0;
        if (first) {
          next_seg(wp, sp);
          p_left = sp.n;
        }
        --p_left;
        const u64 db = dv0 + (u64)((stage * AE_V_BYTES) >> 4);
        const u32 a = tmem + TM_S + (n & 1) * 128;
#pragma unroll
        for (int kk = 0; kk < AE_BN / 16; ++kk)
          umma_ts(tmem + TM_O, a + kk * 8, umma_step_mn(db, kk), idesc_o, (u32)(!first) | (kk > 0));
        umma_commit(&bars->o_done);
        umma_commit(&bars->v_empty[stage]);
        // the region of tile n is free once its P V (just issued) has read P: MMAs run in issue order
        if (ns < n_all) ok = issue_s();
      }
      // every commit of this thread has arrived before the CTA may retire (the last releases have no other waiter)
      if (ok) {
        const int l = n_all - 1;
        ok = mbar_wait(&bars->v_empty[l % AE_STAGES], (l / AE_STAGES) & 1, ctl, args.status, 12) &&
             mbar_wait(&bars->k_empty[l % AE_STAGES], (l / AE_STAGES) & 1, ctl, args.status, 13) &&
             mbar_wait(&bars->q_free, (n_q - 1) & 1, ctl, args.status, 15);
      }
    }
  } else {
    // =============================== row threads =============================
    const u32 row = threadIdx.x;  // row of the unit == TMEM lane
    const u32 lane_base = (warp * 32) << 16;
    const u32 tm_o = tmem + TM_O + lane_base;
    // rows past the last valid one compute on zero-filled Q with the indices of row 0 and are never stored
    const bool row_valid = (int)row < args.rows;
    const int q_idx = (args.gq > 1 || !row_valid) ? 0 : (int)row;
    const int h_row = (args.gq > 1) ? unit * args.gq + (row_valid ? (int)row : 0) : unit;
    AeCustom cu;
#pragma unroll
    for (int i = 0; i < AE_MAX_CUSTOM; ++i) {
      cu.p[i] = args.custom[i];
#pragma unroll
      for (int k = 0; k < 4; ++k) cu.st[i][k] = args.custom_st[i][k];
    }
    AeRow st;
    Walk w = w0;
    AeDecSeg s;
    u32 n_done = 0;  // tiles of this CTA
    int pos = 0;     // ... in front of the segment
    bool ok = true;
    for (int n_seg = 0; next_seg(w, s); ++n_seg) {
      const int b = s.b;
      st.init();
      for (int j = 0; j < s.n; ++j) {
        // scores of the CTA's n-th tile: region n & 1, phase n >> 1 of that region's barriers
        const u32 rgn = n_done & 1u;
        const u32 tm_s = tmem + TM_S + rgn * 128 + lane_base;
        ok = mbar_wait_row(ok, &bars->s_full[rgn], (n_done >> 1) & 1u, ctl, args.status, 9);
        tc_fence_after_sync();
        float sc[AE_BN];
        tmem_ld_f32x128(tm_s, sc);
        const int kv0 = (s.kt + j) * AE_BN;
        if (kv0 + AE_BN > s.keys) {
          const int lim = s.keys - kv0;
#pragma unroll
          for (int c = 0; c < AE_BN; ++c) sc[c] = c < lim ? sc[c] : (AE_MASK_NEG_INF ? -__int_as_float(0x7f800000) : 0.f);
        }
#if AE_MASK_MODE != 0 && AE_MASK_NEG_INF  // (additive mask value 0: scores stay as they are)
#pragma unroll
        for (int c = 0; c < AE_BN; ++c) sc[c] = ae_mask(b, h_row, q_idx, kv0 + c) ? sc[c] : -__int_as_float(0x7f800000);
#endif
        const bool last = j == s.n - 1;
        ae_online_tile<1>(sc, st, b, h_row, q_idx, kv0, cu, [&](auto K, float o_scale, float (&p)[AE_BN]) {
          if constexpr (decltype(K)::value == -1) {
#if !AE_O_SCALE_ONE
            // O is rescaled only when some row of the warp needs it; only then must P V of the tile before have completed.  (A
            // skipped wait cannot alias: o_done runs at most one phase ahead of this warp's arrivals.)
            if (j > 0 && __any_sync(0xffffffffu, o_scale != 1.0f)) {
              ok = mbar_wait_row(ok, &bars->o_done, (n_done - 1) & 1, ctl, args.status, 10);
              tc_fence_after_sync();
#pragma unroll
              for (int c = 0; c < AE_DV / 32; ++c) {
                float f[32];
                u32 r[32];
                tmem_ld_f32x32(tm_o + c * 32, f);
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(f[i] * o_scale);
                tmem_st32(tm_o + c * 32, r);
              }
            }
#endif
          } else {
            // The wait after the segment names the last tile's phase: the one before it has to be over by then, and before this
            // arrival it cannot be further than that.
            if (last && n_done > 0) ok = mbar_wait_row(ok, &bars->o_done, (n_done - 1) & 1, ctl, args.status, 14);
            // P -> TMEM (16-bit pairs, column c/2 holds kv columns c, c+1)
            u32 pk[32];
#pragma unroll
            for (int hh = 0; hh < AE_BN / 64; ++hh) {
#pragma unroll
              for (int i = 0; i < 32; ++i) pk[i] = pack2<AE_BF16>(p[hh * 64 + 2 * i], p[hh * 64 + 2 * i + 1]);
              tmem_st32(tm_s + hh * 32, pk);
            }
            tc_wait_st();
            tc_fence_before_sync();
            mbar_arrive_warp(&bars->p_full[rgn]);
          }
        });
        ++n_done;
      }
      // ---- the segment's rows out: under the next one's loads and S GEMMs; its first P V waits for this warp's P ----
      ok = mbar_wait_row(ok, &bars->o_done, (n_done - 1) & 1, ctl, args.status, 11);
      tc_fence_after_sync();
      const bool store = row_valid && ok;
      // a partial: fp32 slots of a unit's rows; in a cluster this CTA's K / V ring, whose last tile has been read (rows, then their
      // final row scales)
      const bool staged = args.in_cluster || !s.whole;
      const int slot = 2 * (unit * args.n_intervals + (int)blockIdx.y) + (n_seg > 0);
      const i64 part_row = (i64)slot * args.rows + row;
      u16* orow = (u16*)args.o + (i64)b * args.o_sb + (i64)(store ? q_idx : 0) * args.o_ss + (i64)h_row * args.o_sh;
      float* prow = args.in_cluster ? (float*)(smem + AE_SMEM_K) + (row_valid ? row : 0) * AE_PART_LD : args.o_part + part_row * AE_DV;
      // tcgen05.ld is warp-collective: every lane of the warp runs it; only the stores are per-row.
      if ((int)(warp * 32) < args.rows) {
#pragma unroll
        for (int c = 0; c < AE_DV / 32; ++c) {
          float r[32];
          tmem_ld_f32x32(tm_o + c * 32, r);
          if (store && staged) {
            float4* dst = (float4*)(prow + c * 32);
#pragma unroll
            for (int v = 0; v < 8; ++v)
              dst[v] = make_float4(ae_epilogue_o(r[v * 4 + 0], st), ae_epilogue_o(r[v * 4 + 1], st),
                                   ae_epilogue_o(r[v * 4 + 2], st), ae_epilogue_o(r[v * 4 + 3], st));
          } else if (store) {
            uint4* dst = (uint4*)(orow + c * 32);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4 x;
              x.x = pack2<AE_BF16>(ae_epilogue_o(r[v * 8 + 0], st), ae_epilogue_o(r[v * 8 + 1], st));
              x.y = pack2<AE_BF16>(ae_epilogue_o(r[v * 8 + 2], st), ae_epilogue_o(r[v * 8 + 3], st));
              x.z = pack2<AE_BF16>(ae_epilogue_o(r[v * 8 + 4], st), ae_epilogue_o(r[v * 8 + 5], st));
              x.w = pack2<AE_BF16>(ae_epilogue_o(r[v * 8 + 6], st), ae_epilogue_o(r[v * 8 + 7], st));
              dst[v] = x;
            }
          }
        }
      }
      tc_fence_before_sync();  // ordered before this warp's next arrival: the next segment's P V overwrites O
#if AE_NFINAL > 0
      if (store && staged) {
        float fr[AE_NFINAL];
        ae_final_rowscales(st, fr);
#pragma unroll
        for (int i = 0; i < AE_NFINAL; ++i) {
          if (args.in_cluster)
            ((float*)(smem + AE_SMEM_K))[args.rows * (AE_PART_LD + i) + (int)row] = fr[i];
          else
            args.fr_part[i][part_row] = fr[i];
        }
      }
#endif
      if (args.n_intervals > 0 && s.kt == 0 && row == 0) {
        // for the merge: first partial slot of the unit's row and the number of intervals it touches (1 = written directly)
        int* info = args.row_info + 2 * ((i64)b * args.units + unit);
        info[0] = slot;
        info[1] = (pos + tiles_of(s.keys) - 1) / bars->share + 1;
      }
      pos += s.n;
    }
  }

  if (args.in_cluster) {
    // ---- the unit's splits meet: lane k holds what split k left (see mla_combine.cuh), a row per warp, all
    // its dims at once: with 32 of them per step, a unit of 8 rows in two splits was four steps of two trips to other SMs each, and
    // with the threads' rows 512 bytes apart their stores met in one bank (8 rows of 256 keys 9.98 -> 7.6 us, 8 units of 1000 keys
    // 10.24 -> 10.16).  Bit for bit what the launch that merges gives for the same splits. ----
    __syncthreads();  // the producer's and the issuer's warps whole again
    cluster_sync_all();
    if (warp < 4) {
      constexpr int VEC = AE_DV / 32;  // dims of a lane
      const int n = args.n_split, b = (int)blockIdx.z;
      const u32 part = smem_u32(smem + AE_SMEM_K);
      for (int x = (int)(cluster_ctarank() * 4 + warp); x < args.rows; x += n * 4) {
        float fr[AE_NFINAL > 0 ? AE_NFINAL : 1];
#pragma unroll
        for (int i = 0; i < AE_NFINAL; ++i) {
          const float far = ld_cluster_f32(mapa_u32(part + 4 * (args.rows * (AE_PART_LD + i) + x), (int)lane < n ? lane : 0));
          fr[i] = (int)lane < n ? far : -__int_as_float(0x7f800000);
        }
        float v[8][VEC];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < n) ld_cluster(v[k], mapa_u32(part + 4 * (x * AE_PART_LD + (int)lane * VEC), k));
        float w = ae_combine(fr);
        if ((int)lane >= n) w = 0.f;
        const u32 empty = AE_NFINAL > 0 ? ae_empty_splits(fr, w) : 0u;
        float acc[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float wk = __shfl_sync(0xffffffffu, w, k);
          if (k < n && !(empty >> k & 1u)) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[e] += wk * v[k][e];
          }
        }
        const int h = args.gq > 1 ? unit * args.gq + x : unit, q = args.gq > 1 ? 0 : x;
        u32* dst = (u32*)((u16*)args.o + (i64)b * args.o_sb + (i64)q * args.o_ss + (i64)h * args.o_sh + lane * VEC);
#pragma unroll
        for (int e = 0; e < VEC; e += 2) dst[e / 2] = pack2<AE_BF16>(acc[e], acc[e + 1]);
      }
    }
    cluster_sync_all();  // no CTA leaves while another reads its shared memory
  }
  // ---- teardown --------------------------------------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}
