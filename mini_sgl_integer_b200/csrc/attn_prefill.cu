// Prefill / extend attention over the int8 paged pool: many new tokens per sequence, causal inside the new
// tokens, a cached prefix in front of them.  Same arithmetic as the decode kernel (attn.cu), bit for bit.
//
// A CTA owns one (sequence, KV head, tile of 64 / G consecutive new tokens): 64 query rows = tokens x the G query
// heads of the KV head, 16 rows per PAIR of warps.  The integer MMA runs with the QUERY rows on M:
//   scores [16 rows x 8 keys]  = Q [16 x 128] . K^T [128 x 8]        (4 k-steps of 32 d; Q stays in registers)
//   out    [16 rows x 8 d]     = W [16 x 32 keys] . V [32 x 8]       (one k-step per pair of pages, 16 d-tiles)
// The 8 columns of a score tile are mapped to the keys {4c, 4c+1} (first tile of a page) and {4c+2, 4c+3} (second
// tile) for column pair c, so a lane ends up with the scores of the keys 4c .. 4c+3 of a page for its two rows:
// exactly the bytes its A operand of the PV product needs, and the V page is read as the B operand straight from the
// pool's operand order (v_chunk_offset).  Of every 64 keys the two warps of a pair score 32 each; their probability
// limbs meet in shared memory, and each warp multiplies all 64 with its half of d.  (One warp per 16 rows needs 128
// accumulator registers: two CTAs per SM then spill.)
//
// The softmax is exact (LUT exponential with truncation), so nothing can be rescaled on the fly: the keys are
// walked three times per tile - row maxima, sums of exponentials, then probabilities and PV.  Tensor memory, which
// the integer MMA does not need, keeps what the next walk wants of the first kPfKept stages (512 keys): a lane's 16
// scores per stage behind the first walk, their exponentials behind the second, in columns of its own lane.  Those stages read K
// once and V once; behind them the scores are recomputed in each walk.
//
// What bounds it is the latency of dependent integer steps on four warps per scheduler (128 registers a thread, 8 words of it
// spilled).  Recomputing every score in every walk took 115 thread instructions per causal score (masked corners of tiles and set-up
// included); of a kept score the second walk is an exponential and a sum, the third a product and the limbs.  The general steps (64-bit
// rounding shifts with saturation, clamps, a table in global memory) remain for scales whose scores could saturate.  Otherwise a score is one wide multiply, one shift and a rounding
// step, and its exponential one wide multiply-add: with nx = max - score, P = 94548 nx - 1 + 2^32 has the shift in
// its high word and, read backwards, the table index on top of its low word (tests/test_kernel_identities.py).
// 32 / 8 heads: 15 prompts of 100 .. 1000 tokens 0.59 ms a layer, 0.82 with every score recomputed; one of 333 tokens 27.8 us, 41.3.
#include "attn_common.cuh"
#include "luts.cuh"

namespace b200 {

struct PrefillParams {
  const int8_t* q;
  const int32_t* q_mul;
  const int32_t* q_shift;
  const int8_t* k_codes;
  const int8_t* v_codes;
  const int32_t* meta;
  const int32_t* page_table;
  int64_t table_pitch;
  const int32_t* kv_lens;   // [batch] keys per sequence including the new tokens
  const int32_t* q_lens;    // [batch] new tokens per sequence
  const int32_t* q_start;   // [batch] row of the sequence's first new token in q / out
  int32_t* out_q15;
  int8_t* out_codes;
  int32_t* out_absmax;
  int q_heads, kv_heads;
  int64_t num_pages;
  int max_kv_len;
};

constexpr int kPfWarps = 8;
constexpr int kPfThreads = kPfWarps * 32;
constexpr int kPfGroups = kPfWarps / 2;            // pairs of warps
constexpr int kPfRows = kPfGroups * 16;            // query rows per CTA
constexpr int kPfKeys = 64;                        // keys per stage: four pages, two for either warp of a pair
constexpr int kPfStages = 4;
constexpr int kPfV = 8192, kPfMeta = 16384;        // in a stage: K pages (swizzled rows), V pages (operand order), scale blocks
constexpr int kPfStageBytes = kPfMeta + 4 * 192;
constexpr int kPfNeg = (int)(-2147483647 - 1);
constexpr int kPfListPages = 8192;                 // page ids kept in shared memory; those of longer contexts are read where they are
constexpr int kPfMaxPages = 42624;                 // of a sequence
// Tensor memory of a CTA: 256 of 512 columns, for two CTAs per SM.  A warp reaches the 32 lanes of its quarter; two warps share
// each and have half of the columns, 16 for each stage.
constexpr int kPfColumns = 256, kPfKept = kPfColumns / 2 / 16;

// Shared memory behind the ring.
struct PfShared {
  int exp_lut[1024];                               // entry 1023 - j of the table, shifted right by 13
  uint4 limbs[kPfWarps][32][2];                    // probability limbs of a warp's 32 keys as A operands: high, low
  int red[kPfGroups][2][16];
  int rel[2][kPfKeys];                             // relative V scales of this stage's and the next one's keys
  unsigned long long vref;
  int ks_min, ks_max;
  unsigned tmem;
};

// 16 words of every lane to and from its own columns.
__device__ __forceinline__ void pf_keep(unsigned taddr, const int (&v)[2][2][4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
               ::"r"(taddr), "r"(v[0][0][0]), "r"(v[0][0][1]), "r"(v[0][0][2]), "r"(v[0][0][3]), "r"(v[0][1][0]), "r"(v[0][1][1]), "r"(v[0][1][2]),
                 "r"(v[0][1][3]), "r"(v[1][0][0]), "r"(v[1][0][1]), "r"(v[1][0][2]), "r"(v[1][0][3]), "r"(v[1][1][0]), "r"(v[1][1][1]), "r"(v[1][1][2]),
                 "r"(v[1][1][3])
               : "memory");
}
__device__ __forceinline__ void pf_kept(unsigned taddr, int (&v)[2][2][4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(v[0][0][0]), "=r"(v[0][0][1]), "=r"(v[0][0][2]), "=r"(v[0][0][3]), "=r"(v[0][1][0]), "=r"(v[0][1][1]), "=r"(v[0][1][2]),
                 "=r"(v[0][1][3]), "=r"(v[1][0][0]), "=r"(v[1][0][1]), "=r"(v[1][0][2]), "=r"(v[1][0][3]), "=r"(v[1][1][0]), "=r"(v[1][1][1]),
                 "=r"(v[1][1][2]), "=r"(v[1][1][3])
               : "r"(taddr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pf_keep_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void mma_u8s8(int (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ unsigned shr_clamp(unsigned v, unsigned n) {   // 0 from 32 on
  unsigned r;
  asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));
  return r;
}

// exp of the decode kernel, LUT[(y & 0xffff) >> 6] >> min(31, 13 - (y >> 16)) with y = (x * 94548) >> 16 and x = max(score -
// row_max, -2^30); `c` = 94548 row_max - 1 + 2^32.
__device__ __forceinline__ unsigned pf_exp(int score, long long c, const int* lut) {
  const long long v = (long long)score * -94548LL + c;
  return shr_clamp((unsigned)lut[(unsigned)v >> 22], (unsigned)(v >> 32));
}

template <int G>
__global__ void __launch_bounds__(kPfThreads, 2)
attn_prefill_kernel(const PrefillParams p) {
  constexpr int TQ = kPfRows / G;                    // new tokens per tile
  const int b = blockIdx.z, kh = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = warp >> 1, side = warp & 1;
  const int fr = lane >> 2, fc = lane & 3;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* ring = smem_raw;                                                    // [stages][kPfStageBytes]
  PfShared& sh = *reinterpret_cast<PfShared*>(smem_raw + kPfStages * kPfStageBytes);
  int32_t* pages = reinterpret_cast<int32_t*>(smem_raw + kPfStages * kPfStageBytes + sizeof(PfShared));
  // In front of the trigger: a GEMM behind this kernel allocates all columns and keeps them while it waits for it, so it may
  // start only when every CTA here has its own.
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(&sh.tmem)), "r"(kPfColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned kept = sh.tmem + ((unsigned)((warp & 3) * 32) << 16) + (warp >> 2) * (kPfColumns / 2);
  auto release = [&]() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem), "r"(kPfColumns) : "memory");
    }
  };
  pdl_launch_dependents();
  for (int i = tid; i < 1024; i += kPfThreads) sh.exp_lut[i] = g_exp2_attn_lut[1023 - i] >> 13;
  if (tid == 0) {
    sh.vref = ~0ull;
    sh.ks_min = 127;
    sh.ks_max = -128;
  }
  pdl_wait();

  const int L_all = max(0, min(p.kv_lens[b], p.max_kv_len));
  const int n_q = max(0, min(p.q_lens[b], L_all));
  const int n_tiles = (n_q + TQ - 1) / TQ;
  if ((int)blockIdx.x >= n_tiles) {                  // whole CTA: this sequence has fewer tiles
    release();
    return;
  }
  const int tile = n_tiles - 1 - (int)blockIdx.x;    // the tiles with the most keys start first
  const int t0 = tile * TQ;
  const int64_t q_row0 = p.q_start[b];
  const int prefix = L_all - n_q;                    // keys in front of the new tokens
  const int Lt = min(L_all, prefix + min(n_q, t0 + TQ));   // keys the last row of the tile sees
  const int n_stages = (Lt + kPfKeys - 1) / kPfKeys;
  const int n_pages = (Lt + kPage - 1) / kPage;
  const int32_t* table = p.page_table + (int64_t)b * p.table_pitch;
  auto read_page = [&](int i) {
    const int64_t pid = __ldg(table + i);
    return (int)(pid < 0 ? 0 : (pid >= p.num_pages ? p.num_pages - 1 : pid));
  };
  const bool listed = n_pages <= kPfListPages;
  auto page_id = [&](int i) { return listed ? pages[i] : read_page(i); };
  if (listed)
    for (int i = tid; i < n_pages; i += kPfThreads) pages[i] = read_page(i);
  __syncthreads();

  // ---- the ring: one stage = four pages.  Thread t copies 16-byte chunk t & 127 of two pages' K (and V) bytes.
  const unsigned ring_base = (unsigned)__cvta_generic_to_shared(ring);
  const int c_page = tid >> 7, c_chunk = tid & 127;
  const unsigned k_dst = ((c_chunk >> 3) << 7) + ((((c_chunk & 7) ^ ((c_chunk >> 3) & 1))) << 4);   // row-parity swizzle
  const int64_t chunk_off = (int64_t)kh * (kPage * kD) + (c_chunk << 4);
  const int64_t page_stride = (int64_t)p.kv_heads * (kPage * kD);
  auto issue = [&](int stage, bool with_k, bool with_v) {
    if (stage < n_stages) {
      const unsigned st = ring_base + (stage % kPfStages) * kPfStageBytes;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int pi = c_page + 2 * i, pg = 4 * stage + pi;
        if (pg < n_pages) {
          const int64_t off = page_id(pg) * page_stride + chunk_off;
          if (with_k) cp_async16(st + pi * 2048 + k_dst, reinterpret_cast<const unsigned char*>(p.k_codes) + off);
          if (with_v) cp_async16(st + kPfV + pi * 2048 + (c_chunk << 4), reinterpret_cast<const unsigned char*>(p.v_codes) + off);
        }
      }
      if (tid < 40) {
        const int pi = tid / 10, c16 = tid - 10 * pi;
        if (4 * stage + pi < n_pages)
          cp_async16(st + kPfMeta + pi * 192 + c16 * 16,
                     reinterpret_cast<const unsigned char*>(p.meta + ((int64_t)page_id(4 * stage + pi) * p.kv_heads + kh) * kMetaWords) + c16 * 16);
      }
    }
    cp_async_commit();
  };
  for (int j = 0; j < kPfStages - 1; ++j) issue(j, true, false);

  // ---- over ALL keys of the sequence: the reference V scale, and the range of the K shifts
  {
    unsigned long long lv = ~0ull;
    int lo = 127, hi = -128;
    for (int key = tid; key < L_all; key += kPfThreads) {
      const int32_t* mt = p.meta + ((int64_t)read_page(key >> 4) * p.kv_heads + kh) * kMetaWords;
      const unsigned vm = (unsigned)__ldg(mt + 16 + (key & 15));
      const int ks = __ldg(reinterpret_cast<const int8_t*>(mt + 32) + (key & 15)), vs = __ldg(reinterpret_cast<const int8_t*>(mt + 36) + (key & 15));
      const unsigned long long vkey = ((unsigned long long)(unsigned)(vs + 128) << 32) | (unsigned long long)(0xFFFFFFFFu - vm);
      lv = vkey < lv ? vkey : lv;
      lo = min(lo, ks);
      hi = max(hi, ks);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(FULL_MASK, lv, o);
      lv = other < lv ? other : lv;
    }
    lo = __reduce_min_sync(FULL_MASK, lo);
    hi = __reduce_max_sync(FULL_MASK, hi);
    if (lane == 0) {
      atomicMin(&sh.vref, lv);
      atomicMin(&sh.ks_min, lo);
      atomicMax(&sh.ks_max, hi);
    }
  }

  // ---- this lane's two query rows: row r of the CTA is new token t0 + r / G, query head kh * G + r % G
  int lim[2], qm[2], qs[2];
  bool valid[2];
  int64_t orow[2];                                   // element offset of the row in q / out
  unsigned qa[2][8];                                 // Q bytes [32 fc, 32 fc + 32) of the row: A operand words
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = group * 16 + fr + 8 * h;
    const int tok = t0 + r / G, g = r % G;
    valid[h] = tok < n_q;                            // a row past the sequence's last token stands for that one and is not stored
    const int t = min(tok, n_q - 1);
    lim[h] = prefix + t + 1;                         // keys the row sees
    const int64_t hrow = (q_row0 + t) * p.q_heads + kh * G + g;
    orow[h] = hrow * kD;
    qm[h] = p.q_mul[hrow];
    qs[h] = p.q_shift[hrow] - 48;
    const uint4* qp = reinterpret_cast<const uint4*>(p.q + hrow * kD + fc * 32);
    const uint4 x0 = __ldg(qp), x1 = __ldg(qp + 1);
    qa[h][0] = x0.x; qa[h][1] = x0.y; qa[h][2] = x0.z; qa[h][3] = x0.w;
    qa[h][4] = x1.x; qa[h][5] = x1.y; qa[h][6] = x1.z; qa[h][7] = x1.w;
  }
  // the fewest and the most keys that a row of this pair of warps sees (rows are in the order of their tokens)
  const int lim_all = __reduce_min_sync(FULL_MASK, lim[0]), lim_any = __reduce_max_sync(FULL_MASK, lim[1]);
  __syncthreads();
  const int v_shift_ref = (int)(sh.vref >> 32) - 128;
  const int v_mul_ref = (int)(0xFFFFFFFFu - (unsigned)(sh.vref & 0xFFFFFFFFull));
  // |dot| <= 2^21 and |(q_mul k_mul) >> 32| <= 2^30: from a shift of 22 on nothing saturates and a shift by one less fits 32 bits
  const int qs_min = __reduce_min_sync(FULL_MASK, min(qs[0], qs[1])), qs_max = __reduce_max_sync(FULL_MASK, max(qs[0], qs[1]));
  const bool plain = qs_min > -1024 && qs_max < 1024 && qs_min + sh.ks_min >= 22 && qs_max + sh.ks_max <= 62;

  // Scores of this warp's pair of pages for this lane: sc[h][pg][e] = row h, key stage * 64 + side * 32 + pg * 16 + 4 fc + e
  auto scores = [&](const unsigned char* st, int (&sc)[2][2][4]) {
#pragma unroll
    for (int pg = 0; pg < 2; ++pg) {
      const int32_t* mt = reinterpret_cast<const int32_t*>(st + kPfMeta + (2 * side + pg) * 192);
      const int4 km = *reinterpret_cast<const int4*>(mt + 4 * fc);
      const unsigned ksw = reinterpret_cast<const unsigned*>(mt + 32)[fc];
      const int kmv[4] = {km.x, km.y, km.z, km.w};
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const int tok = 4 * (fr >> 1) + 2 * jj + (fr & 1);                   // the key row this lane feeds as column fr
        const unsigned char* kr = st + (2 * side + pg) * 2048 + tok * 128;
        const uint4 k0 = *reinterpret_cast<const uint4*>(kr + (((2 * fc) ^ (tok & 1)) << 4));
        const uint4 k1 = *reinterpret_cast<const uint4*>(kr + (((2 * fc + 1) ^ (tok & 1)) << 4));
        int c[4] = {0, 0, 0, 0};
        mma_s8s8(c, qa[0][0], qa[1][0], qa[0][1], qa[1][1], k0.x, k0.y);
        mma_s8s8(c, qa[0][2], qa[1][2], qa[0][3], qa[1][3], k0.z, k0.w);
        mma_s8s8(c, qa[0][4], qa[1][4], qa[0][5], qa[1][5], k1.x, k1.y);
        mma_s8s8(c, qa[0][6], qa[1][6], qa[0][7], qa[1][7], k1.z, k1.w);
        // c[0]: (row fr, key 4 fc + 2 jj)  c[1]: (row fr, + 1)  c[2]: (row fr + 8, key 4 fc + 2 jj)  c[3]: (row fr + 8, + 1)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
          const int e = 2 * jj + e2;
          const int ks = (int)(signed char)((ksw >> (8 * e)) & 0xff);
#pragma unroll
          for (int h = 0; h < 2; ++h) sc[h][pg][e] = c[2 * h + e2];
          if (plain) {                                 // floor((x + 2^(s-1)) / 2^s) = floor((floor(x / 2^(s-1)) + 1) / 2)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              sc[h][pg][e] = ((int)(((long long)sc[h][pg][e] * (long long)__mulhi(qm[h], kmv[e])) >> (qs[h] + ks - 1)) + 1) >> 1;
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) sc[h][pg][e] = mul_shift_sat32(sc[h][pg][e], __mulhi(qm[h], kmv[e]), qs[h] + ks);
          }
        }
      }
    }
  };
  // Walks the stages; body(stage's shared memory, first key of this warp's pair of pages).
  auto walk = [&](int first, bool with_v, auto&& ahead, auto&& body) {
    for (int stage = first; stage < n_stages; ++stage) {
      cp_async_wait<kPfStages - 3>();                    // this stage and the next one
      __syncthreads();                                   // ... have landed for everybody; the stage before is free
      issue(stage + kPfStages - 1, !with_v || stage + kPfStages - 1 >= kPfKept, with_v);
      ahead(stage);
      if (stage * kPfKeys < lim_any) body(ring + (stage % kPfStages) * kPfStageBytes, stage * kPfKeys + side * 32, stage);
    }
    cp_async_wait<0>();
    __syncthreads();
  };

  // ---- pass 1: row maxima
  int row_max[2] = {kPfNeg, kPfNeg};
  walk(0, false, [](int) {}, [&](const unsigned char* st, int key0, int stage) {
    if (key0 >= lim_any) return;
    int sc[2][2][4];
    scores(st, sc);
    if (stage < kPfKept) pf_keep(kept + 16 * stage, sc);
    const bool all = key0 + 32 <= lim_all;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int pg = 0; pg < 2; ++pg)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (all || key0 + pg * 16 + 4 * fc + e < lim[h]) row_max[h] = max(row_max[h], sc[h][pg][e]);
  });
  pf_keep_done();
  for (int j = 0; j < kPfStages - 1; ++j) issue(kPfKept + j, true, false);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    row_max[h] = max(row_max[h], __shfl_xor_sync(FULL_MASK, row_max[h], 1));
    row_max[h] = max(row_max[h], __shfl_xor_sync(FULL_MASK, row_max[h], 2));
    if (fc == 0) sh.red[group][side][fr + 8 * h] = row_max[h];
  }
  __syncthreads();
  long long exp_c[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    row_max[h] = max(row_max[h], sh.red[group][side ^ 1][fr + 8 * h]);
    // keys behind the causal limit take part in the reference's maximum as -2^30
    if (lim[h] < L_all) row_max[h] = max(row_max[h], -(1 << 30));
    exp_c[h] = (long long)row_max[h] * 94548LL - 1LL + (1LL << 32);
  }

  // ---- pass 2: sums of exponentials; sc becomes the exponentials, 0 for keys that the row does not see
  unsigned row_sum[2] = {0u, 0u};
  auto exponentials = [&](int (&sc)[2][2][4], int key0) {
    const bool all = key0 + 32 <= lim_all;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int pg = 0; pg < 2; ++pg)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const unsigned v = pf_exp(sc[h][pg][e], exp_c[h], sh.exp_lut);
          sc[h][pg][e] = all || key0 + pg * 16 + 4 * fc + e < lim[h] ? (int)v : 0;
        }
  };
  auto add_up = [&](const int (&sc)[2][2][4]) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int pg = 0; pg < 2; ++pg)
#pragma unroll
        for (int e = 0; e < 4; ++e) row_sum[h] += (unsigned)sc[h][pg][e];
  };
#pragma unroll 1
  for (int stage = 0; stage < min(n_stages, kPfKept); ++stage) {
    const int key0 = stage * kPfKeys + side * 32;
    if (key0 >= lim_any) break;
    int sc[2][2][4];
    pf_kept(kept + 16 * stage, sc);
    exponentials(sc, key0);
    pf_keep(kept + 16 * stage, sc);
    add_up(sc);
  }
  walk(kPfKept, false, [](int) {}, [&](const unsigned char* st, int key0, int) {
    if (key0 >= lim_any) return;
    int sc[2][2][4];
    scores(st, sc);
    exponentials(sc, key0);
    add_up(sc);
  });
  pf_keep_done();
  for (int j = 0; j < kPfStages - 1; ++j) issue(j, j >= kPfKept, true);
  unsigned inv[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    // (a lane adds at most 2^16 for each eighth key: 32 bits last for half a million equal keys)
    unsigned long long tot = row_sum[h];
    tot += __shfl_xor_sync(FULL_MASK, tot, 1);
    tot += __shfl_xor_sync(FULL_MASK, tot, 2);
    if (fc == 0) *reinterpret_cast<unsigned long long*>(&sh.limbs[warp][fr + 8 * h][0]) = tot;
    row_sum[h] = 0;
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    unsigned long long tot = *reinterpret_cast<unsigned long long*>(&sh.limbs[warp][fr + 8 * h][0]) +
                             *reinterpret_cast<unsigned long long*>(&sh.limbs[warp ^ 1][fr + 8 * h][0]);
    if (tot < 1ull) tot = 1ull;
    inv[h] = (unsigned)(2147483647ull / tot);
  }

  // ---- pass 3: probabilities (Q0.15) folded with the relative V scale, as two byte limbs, times V
  int acc_hi[8][4], acc_lo[8][4];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc_hi[nt][j] = acc_lo[nt][j] = 0;
  // two warps work out the relative V scales of a stage while the one before is multiplied
  auto rel_scales = [&](int stage, int i) {
    const int32_t* mt = reinterpret_cast<const int32_t*>(ring + (stage % kPfStages) * kPfStageBytes + kPfMeta + (i >> 4) * 192);
    const int vs = reinterpret_cast<const int8_t*>(mt + 36)[i & 15];
    if (stage * kPfKeys + i < Lt) sh.rel[stage & 1][i] = (int)rel_scale_q15((unsigned)mt[16 + (i & 15)], (unsigned)v_mul_ref, vs - v_shift_ref);
  };
  cp_async_wait<kPfStages - 2>();
  __syncthreads();                                       // the first stage; and the sums have been read
  if (tid < kPfKeys) rel_scales(0, tid);
  walk(0, true, [&](int stage) {
    if (stage + 1 < n_stages && group == (stage & (kPfGroups - 1))) rel_scales(stage + 1, tid & (kPfKeys - 1));
  }, [&](const unsigned char* st, int key0, int stage) {
    uint4 own_hi = make_uint4(0, 0, 0, 0), own_lo = make_uint4(0, 0, 0, 0);      // [row h, page]: keys 4 fc .. 4 fc + 3 as bytes
    if (key0 < lim_any) {
      int sc[2][2][4];
      if (stage < kPfKept) {
        pf_kept(kept + 16 * stage, sc);
      } else {
        scores(st, sc);
        exponentials(sc, key0);
      }
      unsigned ah[2][2], al[2][2];
#pragma unroll
      for (int pg = 0; pg < 2; ++pg) {
        const int4 rv = *reinterpret_cast<const int4*>(&sh.rel[stage & 1][side * 32 + pg * 16 + 4 * fc]);
        const unsigned r[4] = {(unsigned)rv.x, (unsigned)rv.y, (unsigned)rv.z, (unsigned)rv.w};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          unsigned w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const unsigned pr = ((unsigned)sc[h][pg][e] * inv[h]) >> 16;
            w[e] = (pr * r[e] + 16384u) >> 15;
          }
          const unsigned w01 = __byte_perm(w[0], w[1], 0x5410), w23 = __byte_perm(w[2], w[3], 0x5410);
          ah[h][pg] = __byte_perm(w01, w23, 0x7531);
          al[h][pg] = __byte_perm(w01, w23, 0x6420);
        }
      }
      own_hi = make_uint4(ah[0][0], ah[1][0], ah[0][1], ah[1][1]);
      own_lo = make_uint4(al[0][0], al[1][0], al[0][1], al[1][1]);
    }
    sh.limbs[warp][lane][0] = own_hi;
    sh.limbs[warp][lane][1] = own_lo;
    asm volatile("bar.sync %0, 64;" ::"r"(group + 1) : "memory");
#pragma unroll
    for (int pp = 0; pp < 2; ++pp) {
      if (stage * kPfKeys + pp * 32 >= lim_any) break;
      const uint4 wh = sh.limbs[(warp & ~1) + pp][lane][0], wl = sh.limbs[(warp & ~1) + pp][lane][1];
      const unsigned char* vp = st + kPfV + pp * 4096 + side * 1024 + lane * 16;      // d-tiles 8 side .. 8 side + 7
#pragma unroll
      for (int qd = 0; qd < 2; ++qd) {
        // (pages past the last one hold leftovers: their limbs are zero)
        const uint4 va = *reinterpret_cast<const uint4*>(vp + qd * 512), vb = *reinterpret_cast<const uint4*>(vp + 2048 + qd * 512);
        const unsigned wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          mma_u8s8(acc_hi[4 * qd + i], wh.x, wh.y, wh.z, wh.w, wa[i], wb[i]);
          mma_u8s8(acc_lo[4 * qd + i], wl.x, wl.y, wl.z, wl.w, wa[i], wb[i]);
        }
      }
    }
  });

  // ---- output: acc -> Q15.16, optionally the per-row int8 codes.  C tile: [0] (row fr, d = 64 side + 8 nt + 2 fc)  [1] (row fr,
  // d + 1)  [2] (row fr + 8, d)  [3] (row fr + 8, d + 1)
  int o[2][16], m[2] = {0, 0};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int a = acc_hi[nt][2 * h + j] * 256 + acc_lo[nt][2 * h + j];
        const int v = mul_shift_sat32_wide((long long)a, v_mul_ref, v_shift_ref - 1);
        o[h][2 * nt + j] = v;
        m[h] = max(m[h], abs_wrap(v));
      }
    if (p.out_q15 && valid[h]) {
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
        *reinterpret_cast<int2*>(p.out_q15 + orow[h] + 64 * side + 8 * nt + 2 * fc) = make_int2(o[h][2 * nt], o[h][2 * nt + 1]);
    }
  }
  if (p.out_codes) {                                     // (the same for the whole launch)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      m[h] = max(m[h], __shfl_xor_sync(FULL_MASK, m[h], 1));
      m[h] = max(m[h], __shfl_xor_sync(FULL_MASK, m[h], 2));
      if (fc == 0) sh.red[group][side][fr + 8 * h] = m[h];
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int am = max(1, max(m[h], sh.red[group][side ^ 1][fr + 8 * h]));
      if (valid[h]) {
        const float mf = __int2float_rn(am);
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          const unsigned short c2 = (unsigned short)((quant_code(o[h][2 * nt], mf) & 0xff) | ((quant_code(o[h][2 * nt + 1], mf) & 0xff) << 8));
          *reinterpret_cast<unsigned short*>(p.out_codes + orow[h] + 64 * side + 8 * nt + 2 * fc) = c2;
        }
        if (fc == 0 && side == 0) p.out_absmax[orow[h] / kD] = am;
      }
    }
  }
  release();
}

template <int G>
static int launch_prefill(const PrefillParams& p, int batch, int max_q_len, cudaStream_t st) {
  constexpr int TQ = kPfRows / G;
  const int pages = (p.max_kv_len + kPage - 1) / kPage;
  if (pages > kPfMaxPages) {
    set_error("attn_prefill: max_kv_len=%d is more than %d pages", p.max_kv_len, kPfMaxPages);
    return B200_E_UNSUPPORTED;
  }
  const size_t smem = (size_t)kPfStages * kPfStageBytes + sizeof(PfShared) + (size_t)(pages < kPfListPages ? pages : kPfListPages) * 4;
  const int tiles = (max_q_len + TQ - 1) / TQ;
  cudaError_t e = cudaFuncSetAttribute(attn_prefill_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    set_error("attn_prefill: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return B200_E_CUDA;
  }
  launch_pdl(attn_prefill_kernel<G>, dim3(tiles, p.kv_heads, batch), dim3(kPfThreads), smem, st, p);
  return check_launch("attn_prefill");
}

}  // namespace b200

using namespace b200;

extern "C" int b200_attn_prefill(const int8_t* q, const int32_t* q_mul, const int32_t* q_shift, const int8_t* k_codes,
                                 const int8_t* v_codes, const int32_t* meta, const int32_t* page_table, int64_t table_pitch,
                                 const int32_t* kv_lens, const int32_t* q_lens, const int32_t* q_start, int32_t* out_q15,
                                 int8_t* out_codes, int32_t* out_absmax, int batch, int max_q_len, int q_heads, int kv_heads,
                                 int64_t num_pages, int max_kv_len, b200_stream_t s) {
  B200_REQUIRE(q && q_mul && q_shift && k_codes && v_codes && meta && page_table && kv_lens && q_lens && q_start, B200_E_NULL,
               "attn_prefill: null pointer");
  B200_REQUIRE((out_codes == nullptr) == (out_absmax == nullptr), B200_E_NULL,
               "attn_prefill: out_codes and out_absmax must be given together");
  B200_REQUIRE(out_q15 || out_codes, B200_E_NULL, "attn_prefill: no output requested");
  B200_REQUIRE(batch >= 0 && batch <= 65535 && max_q_len >= 0 && q_heads > 0 && kv_heads > 0 && kv_heads <= 65535 &&
                   num_pages > 0 && max_kv_len > 0,
               B200_E_SHAPE, "attn_prefill: batch=%d max_q_len=%d q_heads=%d kv_heads=%d num_pages=%lld max_kv_len=%d", batch,
               max_q_len, q_heads, kv_heads, (long long)num_pages, max_kv_len);
  B200_REQUIRE(q_heads % kv_heads == 0, B200_E_SHAPE, "attn_prefill: q_heads=%d not a multiple of kv_heads=%d", q_heads, kv_heads);
  const int G = q_heads / kv_heads;
  B200_REQUIRE(G == 1 || G == 2 || G == 4 || G == 8, B200_E_UNSUPPORTED, "attn_prefill: group size %d (1, 2, 4 or 8)", G);
  B200_REQUIRE(table_pitch >= (max_kv_len + kPage - 1) / kPage, B200_E_SHAPE,
               "attn_prefill: table_pitch=%lld < pages for max_kv_len (%d)", (long long)table_pitch, (max_kv_len + kPage - 1) / kPage);
  B200_REQUIRE(aligned16(q) && aligned16(k_codes) && aligned16(v_codes) && aligned16(meta) &&
                   (reinterpret_cast<uintptr_t>(out_q15) & 7u) == 0 && (reinterpret_cast<uintptr_t>(out_codes) & 1u) == 0,
               B200_E_ALIGN, "attn_prefill: q and pool buffers must be 16-byte aligned, out_q15 8-byte");
  if (batch == 0 || max_q_len == 0) return B200_OK;
  B200_REQUIRE((int64_t)((max_q_len + 15) / 16) <= 65535 * 8, B200_E_SHAPE, "attn_prefill: max_q_len=%d", max_q_len);
  PrefillParams p;
  p.q = q; p.q_mul = q_mul; p.q_shift = q_shift; p.k_codes = k_codes; p.v_codes = v_codes; p.meta = meta;
  p.page_table = page_table; p.table_pitch = table_pitch; p.kv_lens = kv_lens; p.q_lens = q_lens; p.q_start = q_start;
  p.out_q15 = out_q15; p.out_codes = out_codes; p.out_absmax = out_absmax; p.q_heads = q_heads; p.kv_heads = kv_heads;
  p.num_pages = num_pages; p.max_kv_len = max_kv_len;
  cudaStream_t st = (cudaStream_t)s;
  switch (G) {
    case 1: return launch_prefill<1>(p, batch, max_q_len, st);
    case 2: return launch_prefill<2>(p, batch, max_q_len, st);
    case 4: return launch_prefill<4>(p, batch, max_q_len, st);
    default: return launch_prefill<8>(p, batch, max_q_len, st);
  }
}
