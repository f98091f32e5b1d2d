// MLA (multi-head latent attention) decode for sm_100a over CTA pairs.  Replaces the reference's `flash_attn` /
// `flash_attn_split` kernels (attention_engine/core/template/tl_template/attn/mla_decode_tl.py:38-177; CuTe variant
// cute_template_kvshared/kernels/splitkv_mla.cu:1061-1391) and the scheduler of the latter (get_mla_metadata.cu:8-75).
//
// All H <= 128 query heads of one batch row share one latent KV stream: rows of the MMAs are heads.  Per 128-key tile
//   S = [q | q_pe] [kv | k_pe]^T   over 512 + 64 dims (9 blocks of 64)
//   row threads: fused score_mod + online recurrence, P (16 bit) -> shared memory
//   O += P kv[:, :512]
// A cluster of two CTAs does it with tcgen05.mma.cta_group::2, M = 128: each CTA owns 64 heads, its O [64 x 512] fp32 takes
// 256 TMEM columns (64 rows lie on 128 lanes: row r's first half of the columns on lane r, the second on lane r + 64), and
// each B operand is split between the two: 64 of the 128 keys for S, half of the value dims for P V.  One CTA per head
// block with M = 128 cannot hold O and S; splitting the value dims over two CTAs instead computed S twice.  Here the MMAs of a
// 128-key tile take about 1,400 (S) and 1,200 clk (P V) of the 4,300 to 5,400 clk between tiles; the rest is the loads, 136 KB
// per CTA and tile (V comes a second time, by value dims, out of L2), 7 TB/s into shared memory over the chip.
//
// Work: the tiles of all batch rows in one line, cut into equal intervals, one per cluster (args.n_clusters; an interval may
// cover the end of a row, whole rows, the beginning of a row).  A row that lies in one interval is written directly,
// others as normalised partials that ae_mla_combine merges.  One CTA per row, split and value half left 108 of 148 SMs
// without work in the second wave of 128 rows: 549 us for 128 rows of 8192 keys against 295 (353 under the power cap) now,
// 147 -> 39 us for a paged call of 8 rows up to 4096 keys, 274 -> 141 us for a batch that just missed a wave.  With
// args.n_split > 0 (the caller's choice) cluster (b, s) takes share s of row b instead.
//
// Shared memory per CTA: Q 72 KB | K 72 KB (9 blocks of 64 keys) | V 64 KB (2 x 2 blocks of 64 dims, 128 keys) | P 16 KB.
// K and V are one tile deep but released in parts (three K blocks, half of V), which are refilled while the MMAs of the
// other parts run.  No L2 prefetch: 74 pairs with 136 KB slots cover the latency, and prefetches one or two tiles ahead, which
// share the bulk-copy queue with the loads, took 322 us where none take 295 (128 rows of 8192), 125 / 111 (32 rows).
// TMEM columns: O dims 0-255 (128) | O dims 256-511 (128) | S0 64 | S1 64.
// Roles per CTA: warps 0-3 row threads (two per row), warp 4 TMA producer, warp 5 of rank 0 the MMA issuer.
// Barriers that both CTAs' loads or row warps complete live in rank 0; every tcgen05.commit arrives in both CTAs.
// Expects the forward prelude built with AE_RSPLIT = 2, AE_XCH_ROWS = 64.

#define AE_MLA_DV 512
#define AE_MLA_NBK 9       // 64-wide blocks of the 576 dims
#define AE_MLA_BN 128      // keys per tile
#define AE_MLA_KBLK (64 * 128)           // bytes of a K or Q block: 64 rows of 128 B
#define AE_MLA_VBLK (AE_MLA_BN * 128)    // bytes of a V block: 128 keys of 64 dims
#define AE_MLA_SMEM_Q 0
#define AE_MLA_SMEM_K (AE_MLA_NBK * AE_MLA_KBLK)
#define AE_MLA_SMEM_V (AE_MLA_SMEM_K + AE_MLA_NBK * AE_MLA_KBLK)
#define AE_MLA_SMEM_P (AE_MLA_SMEM_V + 4 * AE_MLA_VBLK)
#define AE_MLA_SMEM_BAR (AE_MLA_SMEM_P + 2 * AE_MLA_KBLK)
#define AE_MLA_SMEM_XCH (AE_MLA_SMEM_BAR + 512)  // [phase][half][row] of ae_row_xchg

struct AeMlaBars {
  u64 q_full, q_empty;
  u64 k_full[3], k_empty[3];  // three K blocks each
  u64 v_full[2], v_empty[2];  // value dims 0-255 / 256-511
  u64 s_full[2];
  u64 p_full;   // the row warps of both CTAs
  u64 pv_done;
  AeCtaCtl ctl;
  int row0, tile0, share, total;
};
static_assert(sizeof(AeMlaBars) <= 512, "barrier block");

// Load with the byte count going to a barrier of the pair's rank 0 (cluster address `bar`).  Rank 0 alone arrives there and
// expects the bytes of both CTAs: rank 1's loads may complete before that, but never for a phase whose slot is not free in
// both.  A remote arrive.expect_tx.release.cluster per load group held the producers up for 1,200 clk each (562 us).
AE_DEVICE void mla_load(void* dst, const AeTmaDesc* d, u32 bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"((u64)d), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// Arrival at a barrier of the pair's rank 0.  Release at CTA scope, the default: what it announces (P, written and fenced
// towards the async proxy) is read by this CTA's own tensor core, the barrier's CTA only issues the MMA.  That is a reliance
// on the hardware: the PTX memory model orders rank 1's writes before rank 0's MMA only with a release at cluster scope.  With
// .release.cluster in rank 1 alone an arrival takes about 1,200 clk under load, on the chain of the rows: 128 rows of 8192
// keys 291 -> 340 us, 32 rows 99 -> 127, 8 rows of 4096 35.5 -> 39.1.
AE_DEVICE void mla_arrive(u32 bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

struct AeMlaSeg {
  int b, t0, t1;   // tiles [t0, t1) of batch row b
  int n_t, len;    // tiles and keys of the row
};

extern "C" __global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(192, 1) ae_mla_decode(const __grid_constant__ AeMlaArgs args) {
  extern __shared__ u8 smem_raw[];
  u8* smem = smem_align1024(smem_raw);
  AeMlaBars* bars = (AeMlaBars*)(smem + AE_MLA_SMEM_BAR);
  AeCtaCtl* ctl = &bars->ctl;
  const u32 warp = threadIdx.x >> 5;
  const u32 lane = threadIdx.x & 31;
  const u32 rank = cluster_ctarank();
  const int cl = (int)(blockIdx.x >> 1);

  // keys of a row, clamped to the table; a row has at least one tile (an empty one is all masked)
  auto row_len = [&](int b) {
    if (!args.seqlens) return args.S;
    const int len = args.seqlens[b];
    return len < 0 ? 0 : (len < args.S ? len : args.S);
  };
  auto tiles_of = [](int len) { return len > 0 ? (len + AE_MLA_BN - 1) / AE_MLA_BN : 1; };

  if (threadIdx.x == 0) {
    ctl->abort = 0;
    mbar_init(&bars->q_full, 1);
    mbar_init(&bars->q_empty, 1);
    for (int i = 0; i < 3; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->v_full[i], 1);
      mbar_init(&bars->v_empty[i], 1);
      mbar_init(&bars->s_full[i], 1);
    }
    mbar_init(&bars->p_full, 8);
    mbar_init(&bars->pv_done, 1);
    mbar_fence_init();
  }
  if (warp == 0 && args.n_split == 0) {
    // this cluster's interval: total tiles, equal shares (a row spans at most 32 of them), the row and tile it begins at
    int total = 0, longest = 0;
    const int n_mine = args.seqlens && (int)lane < args.B ? tiles_of(row_len((int)lane)) : 0;  // the first 32 rows are read once
    if (args.seqlens) {
      for (int b = (int)lane; b < args.B; b += 32) {
        const int n = b < 32 ? n_mine : tiles_of(row_len(b));
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
      longest = tiles_of(args.S);
      total = longest * args.B;
    }
    int share = (total + args.n_clusters - 1) / args.n_clusters;
    if (share < (longest + 30) / 31) share = (longest + 30) / 31;
    const int g0 = cl * share;
    int row0 = 0, tile0 = 0;
    if (!args.seqlens) {
      row0 = g0 / longest;
      tile0 = g0 % longest;
    } else if (g0 < total) {
      int before = 0;
      for (int base = 0; base < args.B; base += 32) {
        const int b = base + (int)lane;
        const int n = base == 0 ? n_mine : b < args.B ? tiles_of(row_len(b)) : 0;
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
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anything can arrive on them
  if (warp == 5) {
    tmem_alloc2(&ctl->tmem_base, 512);
    tmem_relinquish2();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const u32 tmem = ctl->tmem_base;
  if (args.lens_host && blockIdx.x == 1 && warp == 5) {
    // The row lengths for the caller, who checks them on the host: written to its pinned memory by a warp that has no other
    // work, then the call's number, which the caller waits for.  A copy in front of the kernel held it up for 6 us.
    for (int b = (int)lane; b < args.B; b += 32) ((volatile int*)args.lens_host)[1 + b] = args.seqlens[b];
    __threadfence_system();
    __syncwarp();
    if (lane == 0) ((volatile int*)args.lens_host)[0] = args.lens_call;
  }
  const u32 TM_O = 0, TM_S = 256;  // S region i at TM_S + 64 i

  // ---- the cluster's segments, the same walk in every role ----
  int w_row, w_tile, w_left;
  if (args.n_split == 0) {
    w_row = bars->row0;
    w_tile = bars->tile0;
    w_left = bars->total - cl * bars->share;
    if (w_left > bars->share) w_left = bars->share;
  } else {
    w_row = cl / args.n_split;
    const int n_t = tiles_of(row_len(w_row));
    const int per = (n_t + args.n_split - 1) / args.n_split;
    w_tile = (cl % args.n_split) * per;
    w_left = n_t - w_tile < per ? n_t - w_tile : per;
  }
  auto next_seg = [&](AeMlaSeg& sg) -> bool {
    if (w_left <= 0) return false;
    sg.b = w_row;
    sg.len = row_len(w_row);
    sg.n_t = tiles_of(sg.len);
    sg.t0 = w_tile;
    const int n = sg.n_t - w_tile < w_left ? sg.n_t - w_tile : w_left;
    sg.t1 = w_tile + n;
    w_left -= n;
    w_row++;
    w_tile = 0;
    return true;
  };
  AeMlaSeg sg;

  if (warp == 4) {
    // =============================== TMA producer (both CTAs) ===============================
    if (lane == 0) {
      tma_prefetch_desc(&args.tm_q);
      tma_prefetch_desc(&args.tm_qpe);
      tma_prefetch_desc(&args.tm_kv);
      tma_prefetch_desc(&args.tm_kpe);
      const u32 q_bar = mapa_u32(smem_u32(&bars->q_full), 0);
      u32 k_bar[3], v_bar[2];
      for (int g = 0; g < 3; ++g) k_bar[g] = mapa_u32(smem_u32(&bars->k_full[g]), 0);
      for (int i = 0; i < 2; ++i) v_bar[i] = mapa_u32(smem_u32(&bars->v_full[i]), 0);
      // row of the `half`-th 64 keys of tile t; keys that the row does not have come from outside the tensor (zeros), so
      // that a page index is only read where the row has keys
      auto kv_row = [&](const AeMlaSeg& s, int t, int half) -> int {
        const int key = t * AE_MLA_BN + half * 64;
        if (!args.block_table) return key;
        if (key >= s.len) return 1 << 30;
        return args.block_table[(i64)s.b * args.max_pages + 2 * t + half] * 64;
      };
      bool ok = true;
      int it = 0, n_seg = 0;
      auto load_v = [&](const AeMlaSeg& s, int t, int n) {
        const int r0 = kv_row(s, t, 0), r1 = kv_row(s, t, 1), kb = args.block_table ? 0 : s.b;
        for (int i = 0; i < 2 && ok; ++i) {
          ok = mbar_wait_cl(&bars->v_empty[i], (n & 1) ^ 1, ctl, args.status, 41);
          if (!ok) return;
          if (rank == 0) mbar_arrive_expect_tx(&bars->v_full[i], 4 * AE_MLA_VBLK);
          for (int j = 0; j < 2; ++j) {
            const int d0 = i * 256 + (int)rank * 128 + j * 64;
            u8* dst = smem + AE_MLA_SMEM_V + (i * 2 + j) * AE_MLA_VBLK;
            mla_load(dst, &args.tm_kv, v_bar[i], d0, r0, kb);
            mla_load(dst + AE_MLA_KBLK, &args.tm_kv, v_bar[i], d0, r1, kb);
          }
        }
      };
      while (ok && next_seg(sg)) {
        ok = mbar_wait_cl(&bars->q_empty, (n_seg & 1) ^ 1, ctl, args.status, 40);
        if (!ok) break;
        if (rank == 0) mbar_arrive_expect_tx(&bars->q_full, 2 * AE_MLA_NBK * AE_MLA_KBLK);
        for (int blk = 0; blk < AE_MLA_NBK; ++blk)
          mla_load(smem + AE_MLA_SMEM_Q + blk * AE_MLA_KBLK, blk < 8 ? &args.tm_q : &args.tm_qpe, q_bar, blk < 8 ? blk * 64 : 0,
                   (int)rank * 64, sg.b);
        for (int t = sg.t0; t < sg.t1 && ok; ++t, ++it) {
          const int r = kv_row(sg, t, (int)rank), kb = args.block_table ? 0 : sg.b;
          for (int g = 0; g < 3 && ok; ++g) {
            ok = mbar_wait_cl(&bars->k_empty[g], (it & 1) ^ 1, ctl, args.status, 42);
            if (!ok) break;
            if (rank == 0) mbar_arrive_expect_tx(&bars->k_full[g], 6 * AE_MLA_KBLK);
            for (int blk = 3 * g; blk < 3 * g + 3; ++blk)
              mla_load(smem + AE_MLA_SMEM_K + blk * AE_MLA_KBLK, blk < 8 ? &args.tm_kv : &args.tm_kpe, k_bar[g],
                       blk < 8 ? blk * 64 : 0, r, kb);
          }
          // V follows the K of the tile after it, the order in which the MMAs free the slots
          if (t > sg.t0 && ok) load_v(sg, t - 1, it - 1);
        }
        if (ok) load_v(sg, sg.t1 - 1, it - 1);
        ++n_seg;
      }
      // the last release of every slot has arrived in this CTA before it may retire
      if (ok && it > 0) {
        ok = mbar_wait_cl(&bars->q_empty, (n_seg - 1) & 1, ctl, args.status, 50);
        for (int g = 0; g < 3 && ok; ++g) ok = mbar_wait_cl(&bars->k_empty[g], (it - 1) & 1, ctl, args.status, 51);
        for (int i = 0; i < 2 && ok; ++i) ok = mbar_wait_cl(&bars->v_empty[i], (it - 1) & 1, ctl, args.status, 52);
      }
    }
  } else if (warp == 5) {
    // =============================== MMA issuer (rank 0) ====================================
    if (rank == 0) {  // all 32 lanes run the control flow, one elected lane issues
      const u32 idesc_s = umma_idesc_f16(128, AE_MLA_BN, AE_BF16, 0, 0);
      const u32 idesc_o = umma_idesc_f16(128, 256, AE_BF16, 0, 1);
      const u64 dq = umma_base_k(smem_u32(smem + AE_MLA_SMEM_Q));
      const u64 dk = umma_base_k(smem_u32(smem + AE_MLA_SMEM_K));
      const u64 dv = umma_base_mn(smem_u32(smem + AE_MLA_SMEM_V), AE_MLA_BN);
      const u64 dp = umma_base_k(smem_u32(smem + AE_MLA_SMEM_P));
      auto wait = [&](u64* bar, u32 parity, u32 site) -> bool {
        return __all_sync(0xffffffffu, mbar_wait_cl(bar, parity, ctl, args.status, site));
      };
      auto issue_s = [&](int n) -> bool {  // S of the cluster's n-th tile into region n & 1
        const u32 d = tmem + TM_S + (n & 1) * 64;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          if (!wait(&bars->k_full[g], n & 1, 43)) return false;
          if (elect_one()) {
#pragma unroll
            for (int blk = 3 * g; blk < 3 * g + 3; ++blk)
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                const u64 off = (u64)((blk * AE_MLA_KBLK + kk * 32) >> 4);
                umma_ss2(d, dq + off, dk + off, idesc_s, (blk | kk) > 0);
              }
            umma_commit2(&bars->k_empty[g]);
            if (g == 2) umma_commit2(&bars->s_full[n & 1]);
          }
        }
        return true;
      };
      bool ok = true;
      int it = 0, n_seg = 0;
      while (ok && next_seg(sg)) {
        ok = wait(&bars->q_full, n_seg & 1, 44) && issue_s(it);
        for (int t = sg.t0; t < sg.t1 && ok; ++t, ++it) {
          // the S GEMM runs one tile ahead; the other region held S of tile it - 1, whose P has been handed over
          if (t + 1 < sg.t1) ok = issue_s(it + 1);
          if (!ok) break;
          if (t + 2 >= sg.t1 && (t + 1 < sg.t1 || sg.t1 - sg.t0 == 1)) {
            if (elect_one()) umma_commit2(&bars->q_empty);  // that was the segment's last S
          }
          ok = wait(&bars->p_full, it & 1, 45);
          if (!ok) break;
          tc_fence_after_sync();
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (!(ok = wait(&bars->v_full[i], it & 1, 46))) break;
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < AE_MLA_BN / 16; ++kk)
                umma_ss2(tmem + TM_O + i * 128, umma_step_k(dp, kk, 64), umma_step_mn(dv + (u64)((i * 2 * AE_MLA_VBLK) >> 4), kk), idesc_o,
                         (t > sg.t0) | (kk > 0));
              umma_commit2(&bars->v_empty[i]);
              if (i == 1) umma_commit2(&bars->pv_done);
            }
          }
        }
        ++n_seg;
      }
    }
  } else {
    // =============================== row threads (two per head) =============================
    const u32 row = threadIdx.x & 63;        // head inside this CTA's block
    const u32 half = (threadIdx.x >> 6) & 1;  // which half of the columns of every accumulator
    const u32 lane_base = ((warp & 3) * 32) << 16;
    const u32 tm_o = tmem + TM_O + lane_base;
    const int h = (int)(rank * 64 + row);
    const u32 p_bar = mapa_u32(smem_u32(&bars->p_full), 0);
    AeCustom cu;
#pragma unroll
    for (int i = 0; i < AE_MAX_CUSTOM; ++i) {
      cu.p[i] = nullptr;
#pragma unroll
      for (int k = 0; k < 4; ++k) cu.st[i][k] = 0;
    }
    AeRow st;
    st.xch = (volatile float*)(smem + AE_MLA_SMEM_XCH);
    st.xme = half * 64 + row;
    st.xother = (half ^ 1u) * 64 + row;
    st.xbar = 1 + (warp & 1);  // warps w and w + 2 share their rows
    st.xn = 64;
    st.xphase = 0;
    bool ok = true;
    int it = 0, pos = 0;
    // 32 columns of this warp's rows on their way out: 4 KB of the P tile, free once P V of a segment's last tile has read it
    u8* const stg = smem + AE_MLA_SMEM_P + warp * 4096;
    for (int n_seg = 0; next_seg(sg); ++n_seg) {
      st.init();
      for (int t = sg.t0; t < sg.t1; ++t, ++it) {
        const u32 tm_s = tmem + TM_S + (it & 1) * 64 + lane_base;
        ok = mbar_wait_row(ok, &bars->s_full[it & 1], (it >> 1) & 1, ctl, args.status, 47);
        tc_fence_after_sync();
        float sc[64];
        tmem_ld_f32x64(tm_s, sc);
        const int kv0 = t * AE_MLA_BN + (int)half * 64;
        if (t * AE_MLA_BN + AE_MLA_BN > sg.len) {
          const int lim = sg.len - kv0;
#pragma unroll
          for (int c = 0; c < 64; ++c) sc[c] = c < lim ? sc[c] : -__int_as_float(0x7f800000);
        }
        float osc = 1.f;
        ae_online_tile<1>(sc, st, sg.b, h, 0, kv0, cu, [&](auto K, float o_scale, float (&p)[64]) {
          if constexpr (decltype(K)::value == -1) {
            osc = o_scale;
          } else {
            // P V of the tile before has read P, and O is up to date
            if (it > 0) ok = mbar_wait_row(ok, &bars->pv_done, (it - 1) & 1, ctl, args.status, 48);
            u8* dst = smem + AE_MLA_SMEM_P + half * AE_MLA_KBLK;
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) {
              uint4 w;
              w.x = pack2<AE_BF16>(p[ch * 8 + 0], p[ch * 8 + 1]);
              w.y = pack2<AE_BF16>(p[ch * 8 + 2], p[ch * 8 + 3]);
              w.z = pack2<AE_BF16>(p[ch * 8 + 4], p[ch * 8 + 5]);
              w.w = pack2<AE_BF16>(p[ch * 8 + 6], p[ch * 8 + 7]);
              *(uint4*)(dst + swz128(row, ch)) = w;
            }
#if !AE_O_SCALE_ONE
            if (t > sg.t0 && __any_sync(0xffffffffu, osc != 1.0f)) {
              tc_fence_after_sync();
#pragma unroll
              for (int c = 0; c < 8; ++c) {
                float f[32];
                u32 r[32];
                tmem_ld_f32x32(tm_o + c * 32, f);
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(f[i] * osc);
                tmem_st32(tm_o + c * 32, r);
              }
              tc_wait_st();
            }
#endif
            fence_proxy_async_smem();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mla_arrive(p_bar);
          }
        });
      }
      if (w_left <= 0) ae_grid_trigger();  // the merge may be brought up; earlier its blocks cost this kernel 2 %
      ok = mbar_wait_row(ok, &bars->pv_done, (it - 1) & 1, ctl, args.status, 49);
      tc_fence_after_sync();
      const bool store = ok && h < args.H;
      const bool whole = args.n_split > 0 ? args.n_split == 1 : (sg.t0 == 0 && sg.t1 == sg.n_t);
      const i64 slot = args.n_split > 0 ? cl : 2 * cl + (n_seg > 0);
      // This thread's dims: 128 of each half of the value dims, 32 at a time.  A thread that stored its own row wrote 16 bytes
      // of 32 lines with each instruction (8,192 L2 requests a segment, about 4 us); through the staging tile a warp writes
      // whole lines of a few rows.
      const bool all_ok = __all_sync(0xffffffffu, ok);
      const int h_first = (int)(rank * 64 + (warp & 1) * 32);  // head of this warp's first row
      // One chunk's code for all eight: unrolled, they were instructions fetched anew for every segment (microseconds, unrolled ->
      // not: 40 rows of 2000 keys and 128 heads 45.4 -> 42.9, 16 heads 37.1 -> 33.7).
      const int n_out = h_first < args.H ? 8 : 0;  // a warp without a head of the call has nothing to write
#pragma unroll 1
      for (int c = 0; c < n_out; ++c) {
        float r[32];
        tmem_ld_f32x32(tm_o + c * 32, r);
        const int d0 = (c >> 2) * 256 + (int)half * 128 + (c & 3) * 32;
        __syncwarp();  // the chunk before has been read
        if (whole) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 w;
            w.x = pack2<AE_BF16>(ae_epilogue_o(r[v * 8 + 0], st), ae_epilogue_o(r[v * 8 + 1], st));
            w.y = pack2<AE_BF16>(ae_epilogue_o(r[v * 8 + 2], st), ae_epilogue_o(r[v * 8 + 3], st));
            w.z = pack2<AE_BF16>(ae_epilogue_o(r[v * 8 + 4], st), ae_epilogue_o(r[v * 8 + 5], st));
            w.w = pack2<AE_BF16>(ae_epilogue_o(r[v * 8 + 6], st), ae_epilogue_o(r[v * 8 + 7], st));
            *(uint4*)(stg + lane * 64 + ((v ^ ((lane >> 1) & 3)) * 16)) = w;
          }
          __syncwarp();
          u16* dst = (u16*)args.o + (i64)sg.b * args.H * AE_MLA_DV + d0 + (lane & 3) * 8;
#pragma unroll
          for (int i = 0; i < 4; ++i) {  // eight rows of 64 bytes
            const u32 rr = i * 8 + (lane >> 2);
            if (all_ok && h_first + (int)rr < args.H)
              *(uint4*)(dst + (i64)(h_first + (int)rr) * AE_MLA_DV) = *(const uint4*)(stg + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) * 16));
          }
        } else {
#pragma unroll
          for (int v = 0; v < 8; ++v)
            *(float4*)(stg + lane * 128 + ((v ^ (lane & 7)) * 16)) =
                make_float4(ae_epilogue_o(r[v * 4 + 0], st), ae_epilogue_o(r[v * 4 + 1], st),
                            ae_epilogue_o(r[v * 4 + 2], st), ae_epilogue_o(r[v * 4 + 3], st));
          __syncwarp();
          float* dst = args.o_part + slot * args.H * AE_MLA_DV + d0 + (lane & 7) * 4;
#pragma unroll
          for (int i = 0; i < 8; ++i) {  // four rows of 128 bytes
            const u32 rr = i * 4 + (lane >> 3);
            if (all_ok && h_first + (int)rr < args.H)
              *(float4*)(dst + (i64)(h_first + (int)rr) * AE_MLA_DV) = *(const float4*)(stg + rr * 128 + (((lane & 7) ^ (rr & 7)) * 16));
          }
        }
      }
      __syncwarp();  // the next segment writes P here
      tc_fence_before_sync();  // ordered before this warp's next arrival: the next segment's P V overwrites O
#if AE_NFINAL > 0
      if (store && half == 0) {
        float fr[AE_NFINAL];
        ae_final_rowscales(st, fr);
        if (whole) {
          if (args.lse_out) args.lse_out[(i64)sg.b * args.H + h] = fr[0];
        } else {
#pragma unroll
          for (int i = 0; i < AE_NFINAL; ++i) args.fr_part[i][slot * args.H + h] = fr[i];
        }
      }
#endif
      if (args.n_split == 0 && args.row_info && sg.t0 == 0 && rank == 0 && threadIdx.x == 0) {
        // for the merge: first partial slot of the row and the number of intervals it touches (1 = written directly)
        args.row_info[2 * sg.b] = (int)slot;
        args.row_info[2 * sg.b + 1] = (pos + sg.n_t - 1) / bars->share + 1;
      }
      pos += sg.t1 - sg.t0;
    }
    if (args.n_split > 1 && it == 0 && h < args.H) {
      // a share past the row's last tile: a zero partial with -inf row scales, which the merge weighs with exp(-inf - ...) = 0
      float4* dst = (float4*)(args.o_part + ((i64)cl * args.H + h) * AE_MLA_DV + half * 256);
      for (int v = 0; v < 64; ++v) dst[v] = make_float4(0.f, 0.f, 0.f, 0.f);
#if AE_NFINAL > 0
      if (half == 0)
        for (int i = 0; i < AE_NFINAL; ++i) args.fr_part[i][(i64)cl * args.H + h] = -__int_as_float(0x7f800000);
#endif
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc2(tmem, 512);
  }
}
