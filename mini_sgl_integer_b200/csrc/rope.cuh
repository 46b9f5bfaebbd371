// q/k-norm + RoPE + Hadamard rotation of one 128-wide head row by one warp (shared by the stand-alone
// RoPE kernel and the fused q/k/v preparation of a decode or prefill step).
#pragma once
#include "common.cuh"
#include "luts.cuh"

namespace b200 {

__device__ __forceinline__ int fwht_scale(int y, int kq15) {
  return sat32(rsr15((long long)y * (long long)kq15));
}

// The n = 128 scale rsr15(y * 2896).  2896 = 16 * 181, so (16a +- 2^14) >> 15 == (a +- 2^10) >> 11 with a = y * 181
// (64 bits), and for y < 0 floor((a - 2^10) / 2^11) == floor((a + 2^10) / 2^11) - 1: one wide multiply-add, one
// funnel shift (the result fits: |result| < |y|) and the sign word.
__device__ __forceinline__ int fwht_scale128(int y) {
  const long long a = (long long)y * 181LL + 1024LL;
  return (int)__funnelshift_r((unsigned)a, (unsigned)(a >> 32), 11) + (y >> 31);
}

// rsr15 of a product sum that fits 32 bits afterwards: for v < 0, (v - 2^14) >> 15 = ((v + 2^14) >> 15) - 1.
__device__ __forceinline__ int rsr15_small(long long v) { return (int)((v + 16384) >> 15) + (int)(v >> 63); }

__device__ __forceinline__ unsigned abs_u(int v) { return v < 0 ? 0u - (unsigned)v : (unsigned)v; }

// Lane l ends up with elements 2l, 2l+1 (a0, a1) and 64+2l, 64+2l+1 (b0, b1) of the row, so that the
// rotate-half pairs (j, j+64) sit in one thread.  nw: per-head RMSNorm weight (nullable).
// (lo, hi): the lane's four values of the row as loaded.
// What bounds it is issue.  Values below 2^22 with cos and sin of at most 1 (nearly every row: 2^22 is 64.0) cannot
// saturate anywhere - the rotation stays below 2^23, seven butterfly stages below 2^30 - and take plain adds; the saturating
// stages cost six times as many instructions.  The sum of squares is added up in two 16-bit halves by the warp's reduction
// instruction instead of ten shuffles.  8244 tokens x 48 heads: 210 us, 347 us before; it issues on 78 % of the cycles.
struct RopeConstants {      // of a lane: cos and sin of its pairs, norm gains of its four values
  int2 c, s, wl, wh;
};
// FRESH: read as in common.cuh, for kernels with loads in front of their wait (others leave the order to the compiler: 8244 tokens x 48 heads
// 215 us, 237 fresh).
template <bool FRESH = false>
__device__ __forceinline__ RopeConstants rope_constants(const int32_t* __restrict__ nw, int pos, const int32_t* __restrict__ cos_sin, int max_pos,
                                                        int lane) {
  pos = max(0, min(max_pos - 1, pos));
  auto load = [](const int32_t* p) { return FRESH ? fresh2(p) : *reinterpret_cast<const int2*>(p); };
  RopeConstants r;
  r.c = load(cos_sin + (int64_t)pos * 128 + 2 * lane);
  r.s = load(cos_sin + (int64_t)pos * 128 + 64 + 2 * lane);
  r.wl = r.wh = make_int2(0, 0);
  if (nw != nullptr) {
    r.wl = load(nw + 2 * lane);
    r.wh = load(nw + 64 + 2 * lane);
  }
  return r;
}

__device__ __forceinline__ void rope_row_vals(int2 lo, int2 hi, bool norm, const RopeConstants& k, const int32_t* __restrict__ lut, int with_fwht,
                                              int lane, int& a0, int& a1, int& b0, int& b1) {
  const int2 c = k.c, s = k.s;
  if (norm) {  // per-head fixed-point RMSNorm over the 128 values
    const int2 wl = k.wl, wh = k.wh;
    int m = max(max(0, abs_wrap(lo.x)), max(abs_wrap(lo.y), max(abs_wrap(hi.x), abs_wrap(hi.y))));
    m = __reduce_max_sync(FULL_MASK, m);
    const NormRow nr = norm_row_from_absmax(m);
    // (each square is at most 2^30, four of them at most 2^32)
    const unsigned long long sq = (unsigned long long)(unsigned)norm_normalised_sq(lo.x, nr.p) + (unsigned)norm_normalised_sq(lo.y, nr.p) +
                                  (unsigned)norm_normalised_sq(hi.x, nr.p) + (unsigned)norm_normalised_sq(hi.y, nr.p);
    const unsigned s_lo = __reduce_add_sync(FULL_MASK, (unsigned)sq & 0xffffu), s_hi = __reduce_add_sync(FULL_MASK, (unsigned)(sq >> 16));
    const long long S = ((long long)s_hi << 16) + (long long)s_lo;
    const int inv = norm_inv_sqrt(S, 128, lut);
    lo.x = nr.zero ? 0 : norm_apply(lo.x, inv, wl.x, nr.p);
    lo.y = nr.zero ? 0 : norm_apply(lo.y, inv, wl.y, nr.p);
    hi.x = nr.zero ? 0 : norm_apply(hi.x, inv, wh.x, nr.p);
    hi.y = nr.zero ? 0 : norm_apply(hi.y, inv, wh.y, nr.p);
  }

  const bool unit = max(max(abs_u(c.x), abs_u(c.y)), max(abs_u(s.x), abs_u(s.y))) <= 32768u;
  const unsigned top = max(max(abs_u(lo.x), abs_u(lo.y)), max(abs_u(hi.x), abs_u(hi.y)));
  if (__all_sync(FULL_MASK, unit && top < (1u << 22))) {
    a0 = rsr15_small((long long)lo.x * c.x - (long long)hi.x * s.x);
    b0 = rsr15_small((long long)lo.x * s.x + (long long)hi.x * c.x);
    a1 = rsr15_small((long long)lo.y * c.y - (long long)hi.y * s.y);
    b1 = rsr15_small((long long)lo.y * s.y + (long long)hi.y * c.y);
    if (with_fwht) {
      int t0 = a0 + a1, t1 = a0 - a1, u0 = b0 + b1, u1 = b0 - b1;
#pragma unroll
      for (int bit = 0; bit < 5; ++bit) {
        const int sign = ((lane >> bit) & 1) ? -1 : 1;
        t0 = __shfl_xor_sync(FULL_MASK, t0, 1 << bit) + sign * t0;
        t1 = __shfl_xor_sync(FULL_MASK, t1, 1 << bit) + sign * t1;
        u0 = __shfl_xor_sync(FULL_MASK, u0, 1 << bit) + sign * u0;
        u1 = __shfl_xor_sync(FULL_MASK, u1, 1 << bit) + sign * u1;
      }
      a0 = fwht_scale128(t0 + u0); b0 = fwht_scale128(t0 - u0);
      a1 = fwht_scale128(t1 + u1); b1 = fwht_scale128(t1 - u1);
    }
    return;
  }
  a0 = sat32(rsr15((long long)lo.x * c.x - (long long)hi.x * s.x));
  b0 = sat32(rsr15((long long)lo.x * s.x + (long long)hi.x * c.x));
  a1 = sat32(rsr15((long long)lo.y * c.y - (long long)hi.y * s.y));
  b1 = sat32(rsr15((long long)lo.y * s.y + (long long)hi.y * c.y));

  if (with_fwht) {
    // step 1: (2l, 2l+1) pairs
    int t0 = add_sat(a0, a1), t1 = sub_sat(a0, a1), u0 = add_sat(b0, b1), u1 = sub_sat(b0, b1);
    a0 = t0; a1 = t1; b0 = u0; b1 = u1;
#pragma unroll
    for (int bit = 0; bit < 5; ++bit) {  // steps 2..32: lane bits
      const bool lower = ((lane >> bit) & 1) == 0;
      int p;
      p = __shfl_xor_sync(FULL_MASK, a0, 1 << bit); a0 = lower ? add_sat(a0, p) : sub_sat(p, a0);
      p = __shfl_xor_sync(FULL_MASK, a1, 1 << bit); a1 = lower ? add_sat(a1, p) : sub_sat(p, a1);
      p = __shfl_xor_sync(FULL_MASK, b0, 1 << bit); b0 = lower ? add_sat(b0, p) : sub_sat(p, b0);
      p = __shfl_xor_sync(FULL_MASK, b1, 1 << bit); b1 = lower ? add_sat(b1, p) : sub_sat(p, b1);
    }
    // step 64: (j, j+64)
    t0 = add_sat(a0, b0); u0 = sub_sat(a0, b0); t1 = add_sat(a1, b1); u1 = sub_sat(a1, b1);
    a0 = fwht_scale(t0, 2896); b0 = fwht_scale(u0, 2896);
    a1 = fwht_scale(t1, 2896); b1 = fwht_scale(u1, 2896);
  }
}

__device__ __forceinline__ void rope_row(const int32_t* __restrict__ src, const int32_t* __restrict__ nw, int pos_in,
                                         const int32_t* __restrict__ cos_sin, int max_pos, int with_fwht, int lane,
                                         int& a0, int& a1, int& b0, int& b1) {
  const int2 lo = *reinterpret_cast<const int2*>(src + 2 * lane);
  const int2 hi = *reinterpret_cast<const int2*>(src + 64 + 2 * lane);
  rope_row_vals(lo, hi, nw != nullptr, rope_constants(nw, pos_in, cos_sin, max_pos, lane), g_inv_sqrt_lut, with_fwht, lane, a0, a1, b0, b1);
}

}  // namespace b200
