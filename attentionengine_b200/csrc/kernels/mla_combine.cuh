// Split-KV merge for the decode kernels (reference: `combine` prim_func, mla_decode_tl.py:181-216; CuTe variant
// cute_template_kvshared/kernels/mla_combine.cu:14-152).  Lane k of every warp holds the final row scales of split k
// (n_split <= 32; absent splits hold -inf), the traced OnlineFunc.combine runs with its reductions over the split dimension
// as warp-shuffle reductions and leaves each lane with the weight of its split.  A thread sums four value dims over the
// splits, AE_DV / 4 threads (at least a warp) per (batch row, head): latency-bound, so the loads of several splits are in flight
// (one warp per head, one split after the other, took 11.6 us for 8 x 128 heads of 512 dims and 10 splits).
// Expects AE_BF16, AE_NFINAL, AE_DV and ae_combine(const float* fr_of_this_lane) -> weight of this lane's split.

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

#define AE_CMB_TPH (AE_DV / 4 > 32 ? AE_DV / 4 : 32)  // threads per head
#define AE_CMB_HPB (128 / AE_CMB_TPH)                 // heads per block
static_assert(AE_DV % 4 == 0 && AE_DV <= 512, "value head dim");

// HPT heads of a row by one thread: four where the blocks would otherwise come in several rounds, each a chain of four dependent
// loads (128 rows of 128 heads, most of them in two splits).
template <int HPT>
AE_DEVICE void ae_combine_heads(const AeMlaCombineArgs& args, int h0, int n_split, i64 slot0, i64 slot1, i64 step, int in_slot, int per_slot) {
  constexpr int FLY = HPT == 1 ? 8 : 4;  // splits in flight
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.y;
  const i64 my_slot = lane == 0 ? slot0 : slot1 + (lane - 1) * step;
  float fr[HPT][AE_NFINAL > 0 ? AE_NFINAL : 1], w[HPT];
  u32 empty[HPT];  // splits without a kept key
#pragma unroll
  for (int e = 0; e < HPT; ++e) {
    const int x = h0 + e < args.H ? in_slot + e : in_slot;
#pragma unroll
    for (int i = 0; i < AE_NFINAL; ++i) fr[e][i] = lane < n_split ? args.fr_part[i][my_slot * per_slot + x] : -__int_as_float(0x7f800000);
  }
#pragma unroll
  for (int e = 0; e < HPT; ++e) {
#if AE_NFINAL > 0
    if (args.lse_out) {
      float m = ae_warp_max(fr[e][0]);
      if (fabsf(m) == __int_as_float(0x7f800000)) m = 0.f;  // all -inf stays -inf, an inf stays inf
      const float sum = ae_warp_sum(lane < n_split ? expf(fr[e][0] - m) : 0.f);
      if (threadIdx.x % AE_CMB_TPH == 0 && h0 + e < args.H) args.lse_out[(i64)b * args.H + h0 + e] = m + logf(sum);
    }
#endif
    w[e] = ae_combine(fr[e]);
    if (lane >= n_split) w[e] = 0.f;
    empty[e] = AE_NFINAL > 0 ? ae_empty_splits(fr[e], w[e]) : 0u;
  }
  const int d0 = (threadIdx.x % AE_CMB_TPH) * 4;
  const bool active = d0 < AE_DV;
  const float* src = args.o_part + (i64)in_slot * AE_DV + (active ? d0 : 0);
  const i64 row = (i64)per_slot * AE_DV;
  float4 acc[HPT];
#pragma unroll
  for (int e = 0; e < HPT; ++e) acc[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < n_split; k0 += FLY) {
    float4 v[HPT][FLY];
#pragma unroll
    for (int j = 0; j < FLY; ++j) {
      const int k = k0 + j;
      const float* from = src + (k == 0 ? slot0 : slot1 + (k - 1) * step) * row;
#pragma unroll
      for (int e = 0; e < HPT; ++e) {
        v[e][j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < n_split && h0 + e < args.H) v[e][j] = *(const float4*)(from + e * AE_DV);
      }
    }
#pragma unroll
    for (int j = 0; j < FLY; ++j) {
#pragma unroll
      for (int e = 0; e < HPT; ++e) {
        const float wk = __shfl_sync(0xffffffffu, w[e], (k0 + j) & 31);
        if (k0 + j >= n_split || (empty[e] >> ((k0 + j) & 31) & 1u)) continue;
        acc[e].x += wk * v[e][j].x;
        acc[e].y += wk * v[e][j].y;
        acc[e].z += wk * v[e][j].z;
        acc[e].w += wk * v[e][j].w;
      }
    }
  }
#pragma unroll
  for (int e = 0; e < HPT; ++e) {
    if (!active || h0 + e >= args.H) continue;
    uint2 o2;
    o2.x = pack2<AE_BF16>(acc[e].x, acc[e].y);
    o2.y = pack2<AE_BF16>(acc[e].z, acc[e].w);
    *(uint2*)((u16*)args.o + ((i64)b * args.H + h0 + e) * AE_DV + d0) = o2;
  }
}

extern "C" __global__ void __launch_bounds__(128) ae_mla_combine(const AeMlaCombineArgs args) {
  const int b = blockIdx.y;
#if AE_DV == 512
  const int hpt = args.heads_per_thread;
#else
  const int hpt = 1;
#endif
  const int h0 = (int)(blockIdx.x * AE_CMB_HPB + threadIdx.x / AE_CMB_TPH) * hpt;
  ae_grid_wait();  // brought up under the split kernel; everything read below is in place from here on
  if (h0 >= args.H) return;  // warp-uniform
  int n_split = args.n_split, in_slot = h0, per_slot = args.H;
  i64 slot0 = (i64)b * n_split, slot1 = slot0 + 1, step = 1;  // slots slot0, slot1, slot1 + step, ...
  if (args.part_off) {
    slot0 = args.part_off[b];
    slot1 = slot0 + 1;
    n_split = args.part_off[b + 1] - args.part_off[b];
  } else if (args.row_info) {
    i64 at = b;
    if (args.units) {
      const int unit = args.gq > 1 ? h0 / args.gq : h0 % args.units;
      in_slot = args.gq > 1 ? h0 % args.gq : h0 / args.units;
      per_slot = args.unit_rows;
      at = (i64)b * args.units + unit;
    }
    slot0 = args.row_info[2 * at];
    n_split = args.row_info[2 * at + 1];
    slot1 = 2 * (slot0 / 2 + 1);
    step = 2;
  }
  if ((args.part_off || args.row_info) && n_split <= 1) return;  // written directly by the split kernel
#if AE_DV == 512
  if (hpt == 4) return ae_combine_heads<4>(args, h0, n_split, slot0, slot1, step, in_slot, per_slot);
#endif
  ae_combine_heads<1>(args, h0, n_split, slot0, slot1, step, in_slot, per_slot);
}
