// 32-bit linears whose sums may be taken in any order: closer to the exact ones than a chain over K, but rounded otherwise for
// other numbers of rows.  (float_gemm.cu has the chains.)
//
//   out[b][t, j] = act( sum_k x[b][t, k] * w[b][j, k] )          operands, products and result in 32 bits
//
// Up to eight rows stream the weights through the fp32 units (gemv_f32_kernel); more run on the bf16 tensor cores.
//
// An fp32 number is the sum of three bf16 numbers (8 + 8 + 8 bits of fraction, each rounded to nearest); of the nine products of
// two such sums the six above 2^-24 of the largest are formed: hi hi, hi mid, mid hi, mid mid, hi lo, lo hi.  split_parts_kernel
// writes the parts of both operands, gemm_f32x3_kernel multiplies them: tcgen05.mma kind::f16 with fp32 accumulators in
// tensor memory, operands staged by TMA, small products first.  The tensor core's accumulation rounds less well than an
// fma (a chain over K = 1024 loses a factor of two against fp32 units; so does one over 128 that comes back to small products), so
// the accumulator starts afresh with every 64 of K and the pieces are added in registers, rounded to nearest.  Error against 64
// bits, standard normal operands, 2-norm over 2-norm: K = 64 0.8e-7 (fp32 units 1.4e-7), 256 0.9e-7 (2.9e-7), 1024 1.1e-7 (5.7e-7),
// 4096 1.7e-7 (11e-7).
//
// What bounds it: six bf16 products are a sixth of the bf16 peak, four times what the fp32 units can do; below that, the
// operands' way from L2 (96 KB for 24 instructions of 128 x 128 x 16).
//
// What the parts cannot give is computed again on the fp32 units, as the chain over K of float_gemm.cu: outputs that are not finite (an
// operand that is not, inf = inf + NaN + NaN, or finite products of leading parts above the largest number) or almost
// subnormal, and the rows and columns of operands below 2^-110, whose lowest part bf16 cannot hold.  Each output is judged by
// itself, so such a row leaves the other rows' bits alone; a block of 64 x 64 outputs that holds one costs a CTA what it costs
// gemm_f32_kernel.  1400 x 4608 x 1024: 87 us, 239 with one NaN, 787 with nothing else (gemm_f32_kernel 419).
#include "float_common.cuh"
#include "umma.cuh"

namespace b200 {

constexpr int kXM = 128, kXN = 128, kXK = 64;       // tile; values of K per stage
constexpr int kXPlane = 128 * 128;                  // bytes of one operand part in a stage: 128 rows x 64 bf16
constexpr int kXStageBytes = 6 * kXPlane;
constexpr int kXStages = 2;
constexpr int kXEpiWarps = 8;
constexpr int kXThreads = 64 + 32 * kXEpiWarps;
constexpr int kXPitch = 20;                         // words per staged row of 16: 16-byte aligned, conflict-free both ways
constexpr unsigned kXTiny = (127u - 110u) << 23;    // 2^-110: from here on three bf16 numbers hold all 24 bits
constexpr unsigned kXInf = 0x7f800000u;

struct X3Operand {
  const float* src;
  int64_t rows, pitch, bstride;                     // rows of one batch
  bf16* dst;                                        // [3][batch][rows][dst_pitch]
  unsigned* odd;                                    // [batch][rows] the parts of one of the row's values do not add up to it; a byte for each
                                                    // of `pieces` warps that split the row
  int vec;                                          // rows start on 16-byte boundaries
};
struct X3Params {
  X3Operand x, w;
  float* out;
  int M, N, K, batch, kp;                           // kp: pitch of the parts
  int64_t out_pitch, out_bstride;
  int act;
  float act_a, act_b;
  int vec;
  int pieces;                                       // 1 or 4: few rows are split by four warps each
  unsigned odd_mask;
};

// Neither zero nor within [2^-110, infinity).
__device__ __forceinline__ bool odd_value(float v) {
  const unsigned u = __float_as_uint(v) & 0x7fffffffu;
  return u != 0u && u - kXTiny >= kXInf - kXTiny;
}

// Three bf16 numbers whose sum is v to 24 bits.  (Rounding up to infinity: the truncated number instead.)
__device__ __forceinline__ void split3(float v, unsigned short (&o)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    bf16 h = __float2bfloat16_rn(v);
    if (i == 0 && (__bfloat16_as_ushort(h) & 0x7fff) == 0x7f80) h = __ushort_as_bfloat16((unsigned short)(__float_as_uint(v) >> 16));
    o[i] = __bfloat16_as_ushort(h);
    v -= __bfloat162float(h);
  }
}

// A warp per row; four for each of few rows, half a warp for short ones.
__global__ void __launch_bounds__(256)
split_parts_kernel(const X3Params p) {
  pdl_launch_dependents();
  pdl_wait();
  const int quads = (p.K + 3) / 4, lanes = quads <= 16 ? 16 : 32, per = 256 / lanes, lane = threadIdx.x & (lanes - 1);
  const int64_t nx = (int64_t)p.batch * p.x.rows, total = (nx + (int64_t)p.batch * p.w.rows) * p.pieces;
  for (int64_t base = (int64_t)blockIdx.x * per; base < total; base += (int64_t)gridDim.x * per) {
    const int64_t at = min(base + threadIdx.x / lanes, total - 1);      // (behind the end: the last one again, to the same values)
    const int64_t i = p.pieces == 1 ? at : at >> 2;
    const int piece = p.pieces == 1 ? 0 : (int)(at & 3);
    const X3Operand& o = i >= nx ? p.w : p.x;
    const int64_t r = i >= nx ? i - nx : i, b = r / o.rows, plane = (int64_t)p.batch * o.rows * p.kp;
    const float* src = o.src + b * o.bstride + (r - b * o.rows) * o.pitch;
    bf16* dst = o.dst + r * p.kp;
    bool odd = false;
#pragma unroll 4
    for (int q = lane + lanes * piece; q < quads; q += lanes * p.pieces) {
      const int k = 4 * q;
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (o.vec && k + 3 < p.K) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(src + k));
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (k + c < p.K) v[c] = __ldg(src + k + c);
      }
      unsigned short part[4][3];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        odd |= odd_value(v[c]);
        split3(v[c], part[c]);
      }
#pragma unroll
      for (int s = 0; s < 3; ++s)                   // (kp is a multiple of 8: the quad fits its row)
        *reinterpret_cast<uint2*>(dst + s * plane + k) = make_uint2(part[0][s] | ((unsigned)part[1][s] << 16), part[2][s] | ((unsigned)part[3][s] << 16));
    }
    const unsigned votes = __ballot_sync(FULL_MASK, odd) >> (threadIdx.x & 31 & ~(lanes - 1)) & (lanes == 16 ? 0xffffu : ~0u);
    if (lane == 0) reinterpret_cast<unsigned char*>(o.odd + r)[piece] = votes != 0;
  }
}

__device__ __forceinline__ void umma_bf16x3(unsigned tmem_d, uint64_t desc_a, uint64_t desc_b, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kXEpiWarps) : "memory"); }
__device__ __forceinline__ bool epilogue_any(bool v) {
  unsigned r;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %1, 0;\nbar.red.or.pred p, 1, %2, q;\nselp.u32 %0, 1, 0, p;\n}"
               : "=r"(r) : "r"((unsigned)v), "n"(32 * kXEpiWarps) : "memory");
  return r != 0;
}

// The epilogue warps go over this CTA's tiles once more, 64 x 64 outputs at a time with 4 x 4 per thread as in gemm_f32_kernel, and
// replace the outputs that the parts could not give.
__device__ __forceinline__ void chain_again(const X3Params& p, int* smem, int et, int num_tiles, int m_tiles, int n_tiles) {
  float(*xs)[68] = reinterpret_cast<float(*)[68]>(smem), (*ws)[68] = xs + 16;
  static_assert(2 * 16 * 68 <= kXEpiWarps * 32 * kXPitch, "two tiles of 16 x 64 in the staging area");
  const int tx = et & 15, ty = et >> 4;
  for (int block = 4 * blockIdx.x; block < 4 * num_tiles; block = (block & 3) < 3 ? block + 1 : block - 3 + 4 * (int)gridDim.x) {
    const int tile = block >> 2, m_blk = tile % m_tiles, r = tile / m_tiles, n_blk = r % n_tiles, b = r / n_tiles;
    const int m0 = m_blk * kXM + 64 * (block & 1), n0 = n_blk * kXN + 32 * (block & 2);
    if (m0 >= p.M || n0 >= p.N) continue;            // (the same for all threads)
    float* out = p.out + (int64_t)b * p.out_bstride;
    unsigned need = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
        if (m < p.M && n < p.N && (((p.x.odd[(int64_t)b * p.M + m] | p.w.odd[(int64_t)b * p.N + n]) & p.odd_mask) || odd_value(out[(int64_t)m * p.out_pitch + n])))
          need |= 1u << (4 * i + j);
      }
    if (!epilogue_any(need != 0)) continue;
    // a thread fetches four columns of one row of either operand, a step ahead
    const int fr = et >> 2, fk = 4 * (et & 3);
    auto fetch = [&](const X3Operand& o, int row, int k) {
      float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (row >= o.rows || k >= p.K) return f;
      const float* src = o.src + (int64_t)b * o.bstride + row * o.pitch + k;
      if (o.vec && k + 3 < p.K) return __ldg(reinterpret_cast<const float4*>(src));
      f.x = src[0];
      if (k + 1 < p.K) f.y = src[1];
      if (k + 2 < p.K) f.z = src[2];
      if (k + 3 < p.K) f.w = src[3];
      return f;
    };
    float4 fx = fetch(p.x, m0 + fr, fk), fw = fetch(p.w, n0 + fr, fk);
    float acc[4][4] = {};
    for (int k0 = 0; k0 < p.K; k0 += 16) {
      xs[fk][fr] = fx.x; xs[fk + 1][fr] = fx.y; xs[fk + 2][fr] = fx.z; xs[fk + 3][fr] = fx.w;
      ws[fk][fr] = fw.x; ws[fk + 1][fr] = fw.y; ws[fk + 2][fr] = fw.z; ws[fk + 3][fr] = fw.w;
      epilogue_barrier();
      fx = fetch(p.x, m0 + fr, k0 + 16 + fk);
      fw = fetch(p.w, n0 + fr, k0 + 16 + fk);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(&xs[k][ty * 4]), c = *reinterpret_cast<const float4*>(&ws[k][tx * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w}, cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], cv[j], acc[i][j]);
      }
      epilogue_barrier();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((need >> (4 * i + j)) & 1u)
          out[(int64_t)(m0 + ty * 4 + i) * p.out_pitch + n0 + tx * 4 + j] = p.act == B200F_ACT_XIELU ? xielu_f32(acc[i][j], p.act_a, p.act_b) : acc[i][j];
  }
}

__global__ void __launch_bounds__(kXThreads, 1)
gemm_f32x3_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ X3Params p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + kXStages * kXStageBytes);   // full[S], empty[S], tfull[2], tempty[2]
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * kXStages + 4);
  int* stage_all = reinterpret_cast<int*>(tmem_slot + 4);
  __shared__ int again_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.K + kXK - 1) / kXK;
  const int m_tiles = (p.M + kXM - 1) / kXM, n_tiles = (p.N + kXN - 1) / kXN;
  const int num_tiles = p.batch * n_tiles * m_tiles;
  const unsigned full0 = smem_u32(bars), empty0 = smem_u32(bars + kXStages);
  const unsigned tfull0 = smem_u32(bars + 2 * kXStages), tempty0 = smem_u32(bars + 2 * kXStages + 2);

  if (warp == 0 && lane == 0) {
    for (int s = 0; s < kXStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(tfull0 + 8 * s, 1);
      mbar_init(tempty0 + 8 * s, kXEpiWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    again_s = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * kXN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_launch_dependents();
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const unsigned tmem_base = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      unsigned it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const int m_blk = tile % m_tiles, r = tile / m_tiles, n_blk = r % n_tiles, b = r / n_tiles;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const unsigned s = it % kXStages, ph = (it / kXStages) & 1;
          ok = mbar_wait(empty0 + 8 * s, ph ^ 1, 1);
          if (!ok) break;
          mbar_expect_tx(full0 + 8 * s, kXStageBytes);
          const unsigned dst = smem_u32(tiles + s * kXStageBytes);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            tma_load_3d(dst + i * kXPlane, &map_x, kb * kXK, m_blk * kXM, i * p.batch + b, full0 + 8 * s);
            tma_load_3d(dst + (3 + i) * kXPlane, &map_w, kb * kXK, n_blk * kXN, i * p.batch + b, full0 + 8 * s);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // D = f32, A = B = bf16, both K-major
      constexpr unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(kXN >> 3) << 17) | ((unsigned)(kXM >> 4) << 24);
      unsigned it = 0;                               // one accumulation per stage
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const unsigned slot = it & 1, aph = (it >> 1) & 1, s = it % kXStages, ph = (it / kXStages) & 1;
          ok = mbar_wait(tempty0 + 8 * slot, aph ^ 1, 4) && mbar_wait(full0 + 8 * s, ph, 2);
          if (!ok) break;
          tcgen05_fence_after();
          const unsigned tmem_d = tmem_base + slot * kXN, base = smem_u32(tiles + s * kXStageBytes);
          constexpr int ax[6] = {2, 1, 0, 1, 0, 0}, bw[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
          for (int t = 0; t < 6; ++t) {
            const uint64_t da = make_smem_desc(base + ax[t] * kXPlane), db = make_smem_desc(base + (3 + bw[t]) * kXPlane);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16x3(tmem_d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (t > 0 || k > 0) ? 1u : 0u);
          }
          tcgen05_commit(empty0 + 8 * s);
          tcgen05_commit(tfull0 + 8 * slot);
        }
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2, et = threadIdx.x - 64;
    int* stage = stage_all + (warp - 2) * (32 * kXPitch);
    unsigned lc = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const int m_blk = tile % m_tiles, r = tile / m_tiles, n_blk = r % n_tiles, b = r / n_tiles;
      const int row0 = m_blk * kXM + q * 32, col0 = n_blk * kXN + half * 64;
      const unsigned *ox = p.x.odd + (int64_t)b * p.M, *ow = p.w.odd + (int64_t)b * p.N;
      const unsigned odd = (row0 + lane < p.M ? ox[row0 + lane] : 0u) | (col0 + lane < p.N ? ow[col0 + lane] : 0u) |
                           (col0 + 32 + lane < p.N ? ow[col0 + 32 + lane] : 0u);
      float acc[2][32];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[h][j] = 0.0f;
      for (int kb = 0; kb < num_kb; ++kb, ++lc) {
        const unsigned slot = lc & 1, aph = (lc >> 1) & 1;
        if (ok) ok = mbar_wait(tfull0 + 8 * slot, aph, 3);
        __syncwarp();
        tcgen05_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          int v[32];
          tmem_ld_32x32(tmem_base + ((unsigned)(q * 32) << 16) + slot * kXN + (unsigned)(half * 64 + h * 32), v);
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[h][j] += __int_as_float(v[j]);
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty0 + 8 * slot);
      }
      if (p.act == B200F_ACT_XIELU) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[h][j] = xielu_f32(acc[h][j], p.act_a, p.act_b);
      }
      bool again = (odd & p.odd_mask) != 0;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 32; ++j) again |= odd_value(acc[h][j]);
      if (again) again_s = 1;
      float* out = p.out + (int64_t)b * p.out_bstride;
      const int rr = lane >> 2, cc = (lane & 3) * 4;
#pragma unroll
      for (int h = 0; h < 4; ++h) {                  // 16 columns at a time through the warp's staging tile
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          *reinterpret_cast<float4*>(stage + lane * kXPitch + j) =
              make_float4(acc[h >> 1][16 * (h & 1) + j], acc[h >> 1][16 * (h & 1) + j + 1], acc[h >> 1][16 * (h & 1) + j + 2], acc[h >> 1][16 * (h & 1) + j + 3]);
        __syncwarp();
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const int row = row0 + it * 8 + rr, col = col0 + 16 * h + cc;
          if (!ok || row >= p.M || col >= p.N) continue;
          const float4 o = *reinterpret_cast<const float4*>(stage + (it * 8 + rr) * kXPitch + cc);
          float* dst = out + (int64_t)row * p.out_pitch + col;
          if (p.vec && col + 3 < p.N) {
            *reinterpret_cast<float4*>(dst) = o;
          } else {
            dst[0] = o.x;
            if (col + 1 < p.N) dst[1] = o.y;
            if (col + 2 < p.N) dst[2] = o.z;
            if (col + 3 < p.N) dst[3] = o.w;
          }
        }
      }
    }
    epilogue_barrier();
    if (again_s) chain_again(p, stage_all, et, num_tiles, m_tiles, n_tiles);      // behind all tiles: no wait of the pipeline spans it
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * kXN) : "memory");
  }
}

// Up to eight rows in 32 bits: what counts is streaming the weights once, which tiles of 64 x 64 on few CTAs did at a tenth of the
// memory's rate and the split into bf16 parts at a third (it writes and reads 6 bytes for each 4).  A CTA has four weight
// rows; its threads stride over K, so every lane has four loads of 16 bytes in flight, and the sums meet in the end.  One row,
// 1024 x 4096 weights: 357 -> 8.5 us; 32768 x 1024: 153 -> 21.5 (20.6 at the memory's rate); eight rows: 370 -> 9.4 and 154 -> 59 us, where the
// loads of x bound it.
constexpr int kGemvRows = 4, kGemvThreads = 128;

template <int M, int VEC>
__global__ void __launch_bounds__(kGemvThreads)
gemv_f32_kernel(const X3Params p) {
  constexpr int R = kGemvRows;
  __shared__ float part[kGemvThreads / 32][R * M];
  pdl_launch_dependents();
  pdl_wait();
  const int n0 = blockIdx.x * R, b = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float *xr[M], *wr[R];
#pragma unroll
  for (int m = 0; m < M; ++m) xr[m] = p.x.src + (int64_t)b * p.x.bstride + min(m, p.M - 1) * p.x.pitch;
#pragma unroll
  for (int r = 0; r < R; ++r) wr[r] = p.w.src + (int64_t)b * p.w.bstride + min(n0 + r, p.N - 1) * p.w.pitch;
  float acc[R][M] = {};
  const int body = p.K / VEC * VEC;
#pragma unroll 2
  for (int c = threadIdx.x * VEC; c < body; c += kGemvThreads * VEC) {
    float wv[R][VEC];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (VEC == 4) *reinterpret_cast<float4*>(wv[r]) = __ldg(reinterpret_cast<const float4*>(wr[r] + c));
      else wv[r][0] = __ldg(wr[r] + c);
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
      float xv[VEC];
      if (VEC == 4) *reinterpret_cast<float4*>(xv) = *reinterpret_cast<const float4*>(xr[m] + c);
      else xv[0] = xr[m][c];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc[r][m] = fmaf(wv[r][k], xv[k], acc[r][m]);
    }
  }
  if (VEC > 1 && body + (int)threadIdx.x < p.K) {          // the columns behind the last group of four
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r][m] = fmaf(wr[r][body + threadIdx.x], xr[m][body + threadIdx.x], acc[r][m]);
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const float v = warp_sum(acc[r][m]);
      if (lane == 0) part[warp][r * M + m] = v;
    }
  __syncthreads();
  if (threadIdx.x >= R * M) return;
  const int r = threadIdx.x / M, m = threadIdx.x % M;
  if (m >= p.M || n0 + r >= p.N) return;
  float v = (part[0][threadIdx.x] + part[1][threadIdx.x]) + (part[2][threadIdx.x] + part[3][threadIdx.x]);
  if (p.act == B200F_ACT_XIELU) v = xielu_f32(v, p.act_a, p.act_b);
  p.out[(int64_t)b * p.out_bstride + m * p.out_pitch + n0 + r] = v;
}

template <int M>
static int launch_gemv(const X3Params& p, cudaStream_t st) {
  const dim3 grid((unsigned)((p.N + kGemvRows - 1) / kGemvRows), (unsigned)p.batch);
  if (p.x.vec && p.w.vec) launch_pdl(gemv_f32_kernel<M, 4>, grid, dim3(kGemvThreads), 0, st, p);
  else launch_pdl(gemv_f32_kernel<M, 1>, grid, dim3(kGemvThreads), 0, st, p);
  return check_launch("gemm_f32 (few rows)");
}

// ----------------------------------------------------------------------------- host side
static int64_t x3_pitch(int64_t k) { return (k + 7) / 8 * 8; }
static int64_t x3_bytes(int64_t rows, int64_t k, int64_t batch) { return (3 * batch * rows * x3_pitch(k) * 2 + 127) / 128 * 128; }

static bool x3_map(CUtensorMap* map, const bf16* base, int64_t rows, int64_t K, int64_t kp, int64_t batch) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)(3 * batch)};
  const cuuint64_t strides[2] = {(cuuint64_t)kp * 2, (cuuint64_t)(rows * kp) * 2};
  const cuuint32_t box[3] = {(cuuint32_t)kXK, 128, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace b200

using namespace b200;

extern "C" int64_t b200f_gemm_f32_ws_bytes(int64_t m, int64_t n, int64_t k, int64_t batch) {
  if (m <= 0 || n <= 0 || k <= 0 || batch <= 0 || batch > 65535 / 3 || m >= (1ll << 31) || n >= (1ll << 31) || k >= (1ll << 31)) return -1;
  // Short sums: the chains' kernels have little to do and no second launch (16 of K: 2 .. 4 us, 7 .. 13 here; 9 x 4096 with 64 of K: 5.9,
  // 7.9; 2048 x 256: 7.3, 8.6; 300 x 4096, of more tiles than SMs: 12.4, 10.0; five rows, 16384 weight rows with 64 of K: 6.3, 18.2).
  if (k <= 32 || (k <= 64 && (m > 8 ? batch * ((m + 63) / 64) * ((n + 63) / 64) <= sm_count() : m > 4 && batch * n >= 8192))) return -1;
  if (m <= 8) return 0;
  // Few rows against many weight rows: the fp32 units read the weights once (4 bytes each) and fill the GPU with a tile of 64 x 64
  // per CTA, the split moves 10 bytes of each (m = 16, n = 32768, k = 1024: 155 us against 177).  Everywhere else that kernel has too
  // few CTAs (m = 16, n = 4608: 70 us against 51; n = 1024, k = 4096: 265 against 90) or too many products (m = 1400, n = 4608: 406
  // against 92).
  if (m <= 64 && batch * ((n + 63) / 64) >= 2 * sm_count()) return -1;
  return x3_bytes(m, k, batch) + x3_bytes(n, k, batch) + 4 * batch * (m + n);
}

extern "C" int b200f_gemm_f32(const float* x, const float* w, float* out, int64_t m, int64_t n, int64_t k, int64_t batch, int64_t x_pitch,
                              int64_t x_bstride, int64_t w_pitch, int64_t w_bstride, int64_t out_pitch, int64_t out_bstride, int act,
                              float act_a, float act_b, void* ws, b200_stream_t s) {
  B200_REQUIRE(x && w && out, B200_E_NULL, "gemm_f32: null pointer");
  const int64_t need = b200f_gemm_f32_ws_bytes(m, n, k, batch);
  B200_REQUIRE(need >= 0, B200_E_SHAPE, "gemm_f32: m=%lld n=%lld k=%lld batch=%lld", (long long)m,
               (long long)n, (long long)k, (long long)batch);
  B200_REQUIRE(x_pitch >= k && w_pitch >= k && out_pitch >= n, B200_E_SHAPE, "gemm_f32: a row pitch is shorter than its row");
  B200_REQUIRE(act == B200F_ACT_NONE || act == B200F_ACT_XIELU, B200_E_UNSUPPORTED, "gemm_f32: activation %d", act);
  B200_REQUIRE(need == 0 || ws, B200_E_NULL, "gemm_f32: no workspace");
  B200_REQUIRE((reinterpret_cast<uintptr_t>(ws) & 127u) == 0, B200_E_ALIGN, "gemm_f32: the workspace must be 128-byte aligned");
  cudaStream_t st = (cudaStream_t)s;
  unsigned char* at = (unsigned char*)ws;
  X3Params p;
  auto rows16 = [&](const float* base, int64_t pitch, int64_t bstride) { return aligned16(base) && pitch % 4 == 0 && (batch == 1 || bstride % 4 == 0); };
  p.x = {x, m, x_pitch, x_bstride, (bf16*)at, nullptr, rows16(x, x_pitch, x_bstride)};
  at += x3_bytes(m, k, batch);
  p.w = {w, n, w_pitch, w_bstride, (bf16*)at, nullptr, rows16(w, w_pitch, w_bstride)};
  at += x3_bytes(n, k, batch);
  p.x.odd = (unsigned*)at;
  p.w.odd = p.x.odd + batch * m;
  p.out = out; p.M = (int)m; p.N = (int)n; p.K = (int)k; p.batch = (int)batch; p.kp = (int)x3_pitch(k);
  p.out_pitch = out_pitch; p.out_bstride = out_bstride; p.act = act; p.act_a = act_a; p.act_b = act_b;
  p.vec = rows16(out, out_pitch, out_bstride);
  if (need == 0) return m == 1 ? launch_gemv<1>(p, st) : m == 2 ? launch_gemv<2>(p, st) : m <= 4 ? launch_gemv<4>(p, st) : launch_gemv<8>(p, st);
  // a few thousand warps keep the memory busy; below that, rows of several hundred values are worth four
  p.pieces = batch * (m + n) <= 16 * sm_count() && k > 256 ? 4 : 1;
  p.odd_mask = p.pieces == 4 ? ~0u : 0xffu;
  const int64_t blocks = (batch * (m + n) * p.pieces + (k <= 64 ? 15 : 7)) / (k <= 64 ? 16 : 8), most = 16 * sm_count();
  CUtensorMap mx, mw;
  B200_REQUIRE(x3_map(&mx, p.x.dst, m, k, p.kp, batch) && x3_map(&mw, p.w.dst, n, k, p.kp, batch), B200_E_CUDA, "gemm_f32: cuTensorMapEncodeTiled failed");
  launch_pdl(split_parts_kernel, dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, st, p);
  if (const int rc = check_launch("gemm_f32 (parts)")) return rc;
  constexpr size_t smem = (size_t)kXStages * kXStageBytes + 1024 + (2 * kXStages + 4) * 8 + 16 + kXEpiWarps * 32 * kXPitch * 4;
  static_assert(smem <= 227 * 1024, "shared memory budget");
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32x3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  B200_REQUIRE(e == cudaSuccess, B200_E_CUDA, "gemm_f32: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  const int64_t tiles = batch * ((m + kXM - 1) / kXM) * ((n + kXN - 1) / kXN);
  launch_pdl(gemm_f32x3_kernel, dim3((unsigned)(tiles < sm_count() ? tiles : sm_count())), dim3(kXThreads), smem, st, mx, mw, p);
  return check_launch("gemm_f32");
}

extern "C" int b200f_gemm_f32_status(int* out_host, int reset) {
  B200_REQUIRE(out_host, B200_E_NULL, "gemm_f32_status: null pointer");
  cudaError_t e = cudaMemcpyFromSymbol(out_host, g_gemm_status, sizeof(int));
  if (e == cudaSuccess && reset) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(int));
  }
  B200_REQUIRE(e == cudaSuccess, B200_E_CUDA, "gemm_f32_status: %s", cudaGetErrorString(e));
  return B200_OK;
}
