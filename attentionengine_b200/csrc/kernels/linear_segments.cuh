// State contributions of the segments of a linear-attention / SSD scan, for sm_100a.
//
// The scan kernels walk a head's chunks one after the other, so a problem with fewer (batch, head) walks than SMs leaves the
// rest idle for the whole walk.  Such a problem is cut into segments of whole chunks along the sequence: this kernel
// computes what every segment adds to the state on its own, all segments at once, and the scan kernel (one CTA per
// batch, head and segment) starts from the decayed sum over the segments in front of its own.
//
//     L = sum_t exp(sum of a over the segment's steps behind t) k_t^T v_t
//
// A chunk's own contribution is one accumulation in TMEM, with the weights of the scan kernels: exp of the decay to the end of
// the chunk, the weighted values rounded to 16 bits.  The decay from there on is applied in fp32, chunk by chunk to the sum that
// the row threads keep in registers: rounding v times the decay to the end of the segment lost the bits of small values in fp16.  The
// sum of one chunk is read while the next chunk's MMAs run (two accumulators), so nothing waits for the chunk before; what bounds
// it is the pass over the V tile and the loads, and two CTAs share an SM (1.3 us a chunk, the scan 2.95).  A CTA takes 64 value
// dims (128 sums a thread would not fit): two CTAs per head of 128, which load k twice.
// Roles: warps 0-3 row threads (thread r = step r of the chunk, then state row r), warp 4 TMA producer, warp 5 MMA issuer.
// Expects AE_BF16, AE_LIN_DV (64 or 128), AE_LIN_STAGES (at least 2).

#define AE_LG_C 128
#define AE_LG_DK 128
#define AE_LG_K_BYTES (AE_LG_C * AE_LG_DK * 2)
#define AE_LG_DV 64  // value dims of a CTA
#define AE_LG_V_BYTES (AE_LG_C * AE_LG_DV * 2)
#define AE_LG_STAGE_BYTES (AE_LG_K_BYTES + AE_LG_V_BYTES)
#define AE_LG_SMEM_BAR (AE_LIN_STAGES * AE_LG_STAGE_BYTES)

struct AeLgBars {
  u64 full[AE_LIN_STAGES];
  u64 prep[AE_LIN_STAGES];   // the stage's V tile carries the weights
  u64 empty[AE_LIN_STAGES];  // the MMAs have read the stage
  u64 l_full[2];             // the sum of a chunk is complete, by chunk parity
  float tot[2][4];  // warp totals of the chunk's log-decays, by chunk parity
  AeCtaCtl ctl;
};

extern "C" __global__ void __launch_bounds__(192, 2) ae_linear_segments(const __grid_constant__ AeLinearSegArgs args) {
  extern __shared__ u8 smem_raw[];
  u8* smem = smem_align1024(smem_raw);
  AeLgBars* bars = (AeLgBars*)(smem + AE_LG_SMEM_BAR);
  AeCtaCtl* ctl = &bars->ctl;
  const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = (int)blockIdx.x / (AE_LIN_DV / AE_LG_DV), b = blockIdx.y;
  const int d0 = (int)blockIdx.x % (AE_LIN_DV / AE_LG_DV) * AE_LG_DV;
  const int hk = h / (args.H / args.HK);
  const int n_total = (args.T + AE_LG_C - 1) / AE_LG_C;
  const int c_begin = (int)blockIdx.z * args.seg_chunks;  // the last segment has no reader
  const int n_chunks = min(args.seg_chunks, n_total - c_begin);

  ae_grid_trigger();  // the scan kernel may be brought up
  if (threadIdx.x == 0) {
    ctl->abort = 0;
    for (int i = 0; i < AE_LIN_STAGES; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->prep[i], 4);
      mbar_init(&bars->empty[i], 1);
    }
    mbar_init(&bars->l_full[0], 1);
    mbar_init(&bars->l_full[1], 1);
    mbar_fence_init();
  }
  if (warp == 5) {
    tmem_alloc(&ctl->tmem_base, 2 * AE_LG_DV);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const u32 tmem = ctl->tmem_base;

  if (warp == 4) {
    if (lane == 0) {
      tma_prefetch_desc(&args.tm_k);
      tma_prefetch_desc(&args.tm_v);
      for (int i = 0; i < n_chunks; ++i) {
        const int stage = i % AE_LIN_STAGES, c = c_begin + i;
        if (!mbar_wait(&bars->empty[stage], ((i / AE_LIN_STAGES) & 1) ^ 1, ctl, args.status, 91)) break;
        u8* st = smem + stage * AE_LG_STAGE_BYTES;
        mbar_arrive_expect_tx(&bars->full[stage], AE_LG_STAGE_BYTES);
        tma_load_4d(st + AE_LG_K_BYTES, &args.tm_v, &bars->full[stage], d0, c * AE_LG_C, h, b);
        for (int dh = 0; dh < AE_LG_DK / 64; ++dh)
          tma_load_4d(st + dh * (AE_LG_C * 128), &args.tm_k, &bars->full[stage], dh * 64, c * AE_LG_C, hk, b);
      }
    }
  } else if (warp == 5) {
    const u32 idesc = umma_idesc_f16(AE_LG_DK, AE_LG_DV, AE_BF16, 1, 1);
    const u64 bk_mn = umma_base_mn(smem_u32(smem), AE_LG_C);
    const u64 bv_mn = umma_base_mn(smem_u32(smem + AE_LG_K_BYTES), AE_LG_C);
    bool ok = true;
    for (int i = 0; i < n_chunks && ok; ++i) {
      const int stage = i % AE_LIN_STAGES;
      const u64 so = (u64)((stage * AE_LG_STAGE_BYTES) >> 4);
      ok = mbar_wait_w(&bars->full[stage], (i / AE_LIN_STAGES) & 1, ctl, args.status, 92) &&
           mbar_wait_w(&bars->prep[stage], (i / AE_LIN_STAGES) & 1, ctl, args.status, 93);
      if (!ok) break;
      tc_fence_after_sync();
      // the accumulator of chunk i - 2: its readers arrived at prep for chunk i after they had read it
#pragma unroll
      for (int kk = 0; kk < AE_LG_C / 16; ++kk)
        umma_ss_w(tmem + (u32)(i & 1) * AE_LG_DV, umma_step_mn(bk_mn + so, kk), umma_step_mn(bv_mn + so, kk), idesc, kk > 0);
      umma_commit_w(&bars->empty[stage]);
      umma_commit_w(&bars->l_full[i & 1]);
    }
    // no commit may still be on its way into the shared memory of a CTA that has retired: the last ones of the ring
    for (int i = max(0, n_chunks - AE_LIN_STAGES); i < n_chunks && ok; ++i)
      ok = mbar_wait_w(&bars->empty[i % AE_LIN_STAGES], (i / AE_LIN_STAGES) & 1, ctl, args.status, 94);
  } else {
    const u32 r = threadIdx.x;
    const u32 lane_base = (warp * 32) << 16;
    const i64 bh = (i64)b * args.H + h;
    const float* a_row = args.a + bh * args.T;
    const float asc = args.ascale ? args.ascale[h] : 1.f;
    const bool vs16 = args.vscale_16 != 0;
    auto step_of = [&](int i) { return (c_begin + i) * AE_LG_C + (int)r; };
    auto load_a = [&](int i) { return i < n_chunks && step_of(i) < args.T ? a_row[step_of(i)] : 0.f; };
    auto load_vs = [&](int i) -> u32 {  // raw bits: converting at once would wait for the load
      if (!args.vscale || i >= n_chunks || step_of(i) >= args.T) return vs16 ? (AE_BF16 ? 0x3f80u : 0x3c00u) : 0x3f800000u;
      const i64 si = bh * args.T + step_of(i);
      return vs16 ? (u32)((const u16*)args.vscale)[si] : ((const u32*)args.vscale)[si];
    };
    float a_next = load_a(0), decay = 0.f, dec = 0.f;
    u32 vs_next = load_vs(0);
    bool ok = true;
    float sum[AE_LG_DV];
#pragma unroll
    for (int e = 0; e < AE_LG_DV; ++e) sum[e] = 0.f;
    auto add_chunk = [&](int i, float dec) {  // row r of the state: chunk i's decay over it, then its own contribution
      ok = ok && mbar_wait(&bars->l_full[i & 1], (i >> 1) & 1, ctl, args.status, 96);
      tc_fence_after_sync();
#pragma unroll
      for (int cc = 0; cc < AE_LG_DV / 32; ++cc) {
        float f[32];
        tmem_ld_f32x32(tmem + (u32)(i & 1) * AE_LG_DV + lane_base + cc * 32, f);
#pragma unroll
        for (int e = 0; e < 32; ++e) sum[cc * 32 + e] = fmaf(sum[cc * 32 + e], dec, f[e]);
      }
    };
    for (int i = 0; i < n_chunks; ++i) {
      const int stage = i % AE_LIN_STAGES;
      float g = a_next * asc;
      const float vsc = vs16 ? unpack_lo<AE_BF16>(vs_next) : __uint_as_float(vs_next);
      a_next = load_a(i + 1);
      vs_next = load_vs(i + 1);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_up_sync(0xffffffffu, g, o);
        if (lane >= (u32)o) g += n;
      }
      float* tot = bars->tot[i & 1];
      if (lane == 31) tot[warp] = g;
      named_bar_sync(1, 128);
      float all = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        if ((u32)w < warp) g += tot[w];
        all += tot[w];
      }
      const float wgt = ae_exp(all - g);
      decay += all;
      ok = ok && mbar_wait(&bars->full[stage], (i / AE_LIN_STAGES) & 1, ctl, args.status, 95);
      u8* vt = smem + stage * AE_LG_STAGE_BYTES + AE_LG_K_BYTES;  // row r of the tile is this thread's alone
#pragma unroll
      for (int ch = 0; ch < AE_LG_DV / 8; ++ch) {
        const u32 off = tile_off(r, ch * 8, AE_LG_C);
        uint4 x = *(const uint4*)(vt + off);
        u32* xw = (u32*)&x;
        if (args.vscale) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            xw[e] = pack2<AE_BF16>(unpack_lo<AE_BF16>(xw[e]) * vsc, unpack_hi<AE_BF16>(xw[e]) * vsc);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
          xw[e] = pack2<AE_BF16>(unpack_lo<AE_BF16>(xw[e]) * wgt, unpack_hi<AE_BF16>(xw[e]) * wgt);
        *(uint4*)(vt + off) = x;
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive_warp(&bars->prep[stage]);
      if (i > 0) add_chunk(i - 1, dec);
      dec = i > 0 ? ae_exp(all) : 0.f;  // nothing in front of the first chunk: its decay may be out of range
    }
    add_chunk(n_chunks - 1, dec);
    const i64 slot = bh * gridDim.z + blockIdx.z;
    float4* out = (float4*)args.seg_state + (slot * AE_LIN_DV + d0) * (AE_LG_DK / 4);  // [DV / 4][DK] of float4: lanes side by side
#pragma unroll
    for (int e = 0; e < AE_LG_DV / 4; ++e)
      out[e * AE_LG_DK + r] = make_float4(sum[e * 4], sum[e * 4 + 1], sum[e * 4 + 2], sum[e * 4 + 3]);
    if (r == 0 && d0 == 0) args.seg_decay[slot] = decay;
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 2 * AE_LG_DV);
  }
}
