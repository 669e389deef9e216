// Causal GQA flash prefill, head_dim 256, 16-bit operands, fp32 accumulation, with the
// sigmoid-gate epilogue fused:  out = softmax(scale * Q K^T + causal) V * sigmoid(gate).
//
// Work comes in items: 128 query rows of one query head, over the 64-key tiles they see; items are numbered longest
// first (every head's latest query tile first), because causal items differ 64-fold in length.  Two ways to deal
// them out (flash_plan, below the kernel):
//   one CTA per item, when the items fill the SMs evenly;
//   one CTA per SM, each with an equal stretch of the concatenated tiles of all items, when they would not (a short
//   chunk over a long past is 16 CTAs; 256 equal items on 148 SMs are two waves, the second half empty).  A CTA
//   walks the segments of its stretch; an item that a boundary cuts leaves (O, max, sum) partials in fp32, which
//   flash_merge_kernel joins, gate included.
// Twelve warps:
//   warps 0-7  softmax + drain; warp w owns query rows 32 * (w % 4) .. (= its TMEM lanes) and keys
//              32 * (w / 4) .. of every 64-key tile; the two halves of a row swap maxima and sums through
//              shared memory behind a 64-thread barrier
//   warp  8    issues the first half of the S = Q K^T MMAs (feature slabs 0-1, one lane)
//   warp  9    TMA producer for Q and K (one lane)
//   warp 10    issues the O += P V MMAs and fetches the next V tile behind them (one lane)
//   warp 11    issues the second half of the S MMAs (feature slabs 2-3) into a second accumulator
// Per 64-key tile:  S = Q K^T (M128 x N64 x K256) into one of two TMEM buffers, each made of two
// accumulators that the softmax adds (one thread sustains only one tcgen05.mma per ~85 cycles, so
// the 16 MMAs of a tile are split between two issuers);
// the softmax warps read S from TMEM, keep a running maximum with lazy rescaling of
// the TMEM-resident O (only when the maximum grew by more than 2^8), write P as a
// 16-bit K-major swizzled tile to one of two shared-memory buffers; O += P V (M128 x N256 x K64)
// with V read in place as an MN-major B operand (no transposed copy).
// S of tile j+1 is issued before P of tile j is consumed and P of tile j+1 is written while P V of
// tile j runs, so the tensor pipe overlaps the softmax.
// Drain: the gate tile arrives by TMA in the Q buffer during the last tile; each thread normalises its half row,
// applies the sigmoid and writes the output chunks in place; TMA stores write the tile.
// TMEM: S0a [0,64) S0b [64,128) S1a [128,192) S1b [192,256) O [256,512).
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace mxb {

constexpr int FB_M = 128, FB_N = 64, FB_D = 256;
constexpr int kMaxBins = 160;
#ifndef MXB_FLASH_POLY
#define MXB_FLASH_POLY 1
#endif
constexpr int kPolyOf8 = MXB_FLASH_POLY;   // of every eight exponentials, this many (0 .. 4) run on the FMA pipe


struct FlashSmem {
  static constexpr int q_off = 0;                       // 4 slabs x [128 x 128 B]
  static constexpr int k_off = q_off + 4 * 16384;       // 2 stages x 4 slabs x [64 x 128 B]
  static constexpr int v_off = k_off + 2 * 32768;       // 2 stages x 4 slabs x [64 keys x 128 B]
  static constexpr int p_off = v_off + 2 * 32768;       // 2 buffers x [128 x 128 B]
  static constexpr int bar_off = p_off + 2 * 16384;
  static constexpr int rowmax_off = bar_off + 256;      // [2 tiles][2 halves][128 rows] bf16 (1 KB); reused for the row sums
  static constexpr int total = rowmax_off + 1024;
};

struct FlashParams {
  const void* gate;
  int64_t g_ss, g_sh;
  void* out;
  int64_t o_ss, o_sh;
  int32_t S, Skv, Hq, Hkv;
  float scale_log2;  // scale * log2(e)
  int32_t q_head_inner, k_head_inner;  // tensor-map dimension order: (D, head, row) instead of (D, row, head)
  int32_t g_head_inner, o_head_inner, v_head_inner;
  int32_t tma_drain;   // gate tile in and output tile out by TMA through the (then idle) Q buffer
  int32_t* status;
  // Stretches of tiles, one per CTA (n_bins = 0: one item per CTA).  Bin i covers the tiles from bin_start[i] up to
  // bin_start[i + 1], both (item << 16 | tile of the item).
  float4* part_o;      // [2 n_bins][64 groups of 4 features][128 rows]
  float2* part_ml;     // [2 n_bins][128 rows]: reference maximum (log2 units), sum
  int32_t n_bins;
  uint32_t bin_start[kMaxBins + 1];
};

// 64-key tiles that the 128 rows of query tile qt see
__host__ __device__ inline int flash_tiles(int qt, int S, int Skv) {
  const int64_t end = (int64_t)qt * FB_M + FB_M + (Skv - S);
  return (int)(((end < Skv ? end : (int64_t)Skv) + FB_N - 1) / FB_N);
}
// where a cut item's segment leaves its partial: a bin holds at most one segment that starts inside an item, and
// one that starts an item and does not finish it
__device__ __forceinline__ int part_slot(int bin, bool starts_inside) { return 2 * bin + (starts_inside ? 0 : 1); }
// The reference maximum a cut segment starts from: finite, so that a row that sees none of the segment's first tile
// (the rows above the diagonal) gets weights of 0 and not of exp(-inf + inf).
constexpr float kNoMax = -3e38f;

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (BF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}
__device__ __forceinline__ float fast_ex2(float x) {   // 2^x, x <= 0 here; -inf -> 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^x on the FMA pipe for x <= ~8: round-to-nearest split x = n + f with the 1.5 * 2^23 trick, a cubic for 2^f on
// [-0.5, 0.5] (relative error 7.5e-5, below the rounding of a 16-bit P), n added into the exponent field.  One in
// eight of a tile's exponentials goes this way (measured best among 0 to 4 in eight): it takes the edge off the
// special-function unit's 16 results per clock per SM.  Inputs below -126 (masked keys) give 2^-126 instead of 0.
__device__ __forceinline__ float poly_ex2(float x) {
  x = fmaxf(x, -126.f);
  const float kMagic = 12582912.f;
  const float xr = x + kMagic;
  const float f = x - (xr - kMagic);
  float r = fmaf(0.0551716685295105f, f, 0.2426111251115799f);
  r = fmaf(r, f, 0.6932609677314758f);
  r = fmaf(r, f, 0.9999280571937561f);
  return __int_as_float(__float_as_int(r) + (__float_as_int(xr) << 23));
}

__device__ __forceinline__ float fast_tanh(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool BF16>
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  if constexpr (BF16) return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
  else return __half22float2(*reinterpret_cast<__half2*>(&u));
}

template <bool BF16, bool BINS>
__global__ void __launch_bounds__(384, 1) flash_prefill_kernel(const __grid_constant__ CUtensorMap tm_q,
                                                               const __grid_constant__ CUtensorMap tm_k,
                                                               const __grid_constant__ CUtensorMap tm_vt,
                                                               const __grid_constant__ CUtensorMap tm_g,
                                                               const __grid_constant__ CUtensorMap tm_o,
                                                               const __grid_constant__ FlashParams p) {
  using L = FlashSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* q_s = smem + L::q_off;
  uint8_t* k_s = smem + L::k_off;
  uint8_t* v_s = smem + L::v_off;
  uint8_t* p_s = smem + L::p_off;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bar_off);
  uint16_t* rowmax_s = reinterpret_cast<uint16_t*>(smem + L::rowmax_off);
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;   // [2]
  uint64_t* k_empty = bars + 3;  // [2]
  uint64_t* v_full = bars + 5;   // [2]
  uint64_t* s_ready = bars + 9;  // [2]
  uint64_t* p_ready = bars + 11;  // [2], one per P buffer (the softmax warps may be a tile apart)
  uint64_t* pv_done = bars + 13;  // [2], one per P buffer
  uint64_t* s_free = bars + 15;   // [2]
  uint64_t* g_full = bars + 17;   // gate tile landed
  uint64_t* q_free = bars + 18;   // the Q buffer may take the next segment's rows
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Items in longest-first order: every head's latest (heaviest) query tile, then the next tile of every head, ...;
  // items that run at the same time share their K/V stream across the query heads of a KV head.
  const int n_qt = (p.S + FB_M - 1) / FB_M;
  const int past = p.Skv - p.S;
  int it_first = (int)blockIdx.x, j_first = 0, it_stop = it_first + 1, j_stop = 0;
  if constexpr (BINS) {
    const uint32_t at = p.bin_start[blockIdx.x], stop = p.bin_start[blockIdx.x + 1];
    it_first = (int)(at >> 16); j_first = (int)(at & 0xFFFFu);
    it_stop = (int)(stop >> 16); j_stop = (int)(stop & 0xFFFFu);
  }
  // The walk over this CTA's segments, identical in every role: item `it`, its tiles [lo, hi) of nt.
  struct Seg { int it, lo, hi, nt, head, kvh, m0; };
  auto seg_at = [&](int it) {
    Seg g;
    const int qt = n_qt - 1 - it / p.Hq;
    g.it = it;
    g.head = it % p.Hq;
    g.kvh = g.head / (p.Hq / p.Hkv);
    g.m0 = qt * FB_M;
    g.nt = flash_tiles(qt, p.S, p.Skv);
    g.lo = BINS && it == it_first ? j_first : 0;
    g.hi = BINS && it == it_stop ? j_stop : g.nt;
    return g;
  };
  const int it_end = BINS && j_stop > 0 ? it_stop + 1 : it_stop;
  if (tid == 0) {
    ptx::mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&k_full[i], 1);
      ptx::mbar_init(&k_empty[i], 2);   // both S issuers release a K stage
      ptx::mbar_init(&v_full[i], 1);
      ptx::mbar_init(&s_ready[i], 2);   // both halves of S
      ptx::mbar_init(&pv_done[i], 1);
      ptx::mbar_init(&p_ready[i], 256);
    }
    ptx::mbar_init(g_full, 1);
    ptx::mbar_init(q_free, 1);
    ptx::mbar_init(&s_free[0], 256);
    ptx::mbar_init(&s_free[1], 256);
    *abort_flag = 0;
    ptx::mbar_fence_init();
  }
  __syncwarp();
  if (warp == 0) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_o = tmem_base + 256;

  if (warp == 9) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      ptx::tma_prefetch_desc(&tm_q);
      ptx::tma_prefetch_desc(&tm_k);
      int n = 0, r = 0;   // segments and tiles so far: they give the barriers' phases
      for (int it = it_first; it < (BINS ? it_end : it_first + 1); ++it, ++n) {
        const Seg g = seg_at(it);
        if (n > 0) ptx::mbar_wait(q_free, (uint32_t)((n - 1) & 1), abort_flag);
        ptx::mbar_expect_tx(q_full, 4 * 16384);
        for (int kb = 0; kb < 4; ++kb)
          ptx::tma_load_3d(q_s + kb * 16384, &tm_q, q_full, kb * 64, p.q_head_inner ? g.head : g.m0,
                           p.q_head_inner ? g.m0 : g.head);
        for (int j = g.lo; j < g.hi; ++j, ++r) {   // K tiles only: V is fetched by the P V issuer, behind its own MMAs
          const int s = r & 1;
          if (r >= 2) ptx::mbar_wait(&k_empty[s], (uint32_t)(((r >> 1) - 1) & 1), abort_flag);
          ptx::mbar_expect_tx(&k_full[s], 32768);
          for (int kb = 0; kb < 4; ++kb)
            ptx::tma_load_3d(k_s + s * 32768 + kb * 8192, &tm_k, &k_full[s], kb * 64, p.k_head_inner ? g.kvh : j * FB_N,
                             p.k_head_inner ? j * FB_N : g.kvh);
        }
      }
    }
  } else if (warp == 8 || warp == 11) {
    // ------------------------------------------------------------ S = Q K^T issuers
    // Warp 8 accumulates feature slabs 0-1 into S(s)a, warp 11 slabs 2-3 into S(s)b; P V (4 MMAs) is a third
    // issuer.  All write different TMEM columns, so none waits for another.
    if (lane == 0) {
      const int half = warp == 8 ? 0 : 1;
      constexpr uint32_t fmt = BF16 ? ptx::kFmtBF16 : ptx::kFmtF16;
      const uint32_t idesc_s = ptx::idesc_f16(fmt, fmt, FB_M, FB_N, 0, 0);
      const uint64_t q_desc = ptx::smem_desc_sw128(ptx::smem_u32(q_s), 16, 1024);
      const uint64_t k_desc = ptx::smem_desc_sw128(ptx::smem_u32(k_s), 16, 1024);
      int n = 0, j = 0;   // segments and tiles so far
      for (int it = it_first; it < (BINS ? it_end : it_first + 1); ++it, ++n) {
        const Seg g = seg_at(it);
        ptx::mbar_wait(q_full, (uint32_t)(n & 1), abort_flag);
        for (int i = g.lo; i < g.hi; ++i, ++j) {
          const int s = j & 1;
          ptx::mbar_wait(&k_full[s], (uint32_t)((j >> 1) & 1), abort_flag);
          if (j >= 2) ptx::mbar_wait(&s_free[s], (uint32_t)(((j >> 1) - 1) & 1), abort_flag);  // softmax read S(j-2)
          ptx::tc_fence_after_sync();
          const uint32_t d = tmem_base + (uint32_t)(s * 2 * FB_N + half * FB_N);
          const uint64_t kd = ptx::desc_advance(k_desc, s * 32768);
#pragma unroll
          for (int kb2 = 0; kb2 < 2; ++kb2) {
            const int kb = half * 2 + kb2;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              ptx::mma_f16_ss(d, ptx::desc_advance(q_desc, kb * 16384 + ks * 32),
                              ptx::desc_advance(kd, kb * 8192 + ks * 32), idesc_s, (kb2 | ks) ? 1u : 0u);
          }
          ptx::mma_commit(&s_ready[s]);
          ptx::mma_commit(&k_empty[s]);
        }
      }
    }
  } else if (warp == 10) {
    // ------------------------------------------------------------ O += P V issuer
    if (lane == 0) {
      constexpr uint32_t fmt = BF16 ? ptx::kFmtBF16 : ptx::kFmtF16;
      // V is read as it lies in memory ([key][feature]): as the B operand that is MN-major, four 64-feature slabs of
      // [64 keys x 128 B] (8 KB apart = LBO), groups of 8 keys 1 KB apart (SBO), 16 keys per K step
      const uint32_t idesc_o = ptx::idesc_f16(fmt, fmt, FB_M, FB_D, 0, 1);
      const uint64_t v_desc = ptx::smem_desc_sw128(ptx::smem_u32(v_s), 8192, 1024);
      const uint64_t p_desc = ptx::smem_desc_sw128(ptx::smem_u32(p_s), 16, 1024);
      ptx::tma_prefetch_desc(&tm_vt);
      // V tiles are fetched in the order of the walk, across the segments' boundaries
      Seg vg = seg_at(it_first);
      int vj = vg.lo, vr = 0;
      auto load_next_v = [&]() {
        if (BINS ? vg.it >= it_end : vj >= vg.hi) return;
        const int s = vr & 1;
        ptx::mbar_expect_tx(&v_full[s], 32768);
        for (int kb = 0; kb < 4; ++kb)
          ptx::tma_load_3d(v_s + s * 32768 + kb * 8192, &tm_vt, &v_full[s], kb * 64, p.v_head_inner ? vg.kvh : vj * FB_N,
                           p.v_head_inner ? vj * FB_N : vg.kvh);
        ++vr;
        if (++vj == vg.hi && BINS) {
          vg = seg_at(vg.it + 1);
          vj = vg.lo;
        }
      };
      load_next_v();
      load_next_v();
      int j = 0;   // tiles so far
      for (int it = it_first; it < (BINS ? it_end : it_first + 1); ++it) {
        const Seg g = seg_at(it);
        for (int i = g.lo; i < g.hi; ++i, ++j) {
          const int s = j & 1;
          ptx::mbar_wait(&p_ready[s], (uint32_t)((j >> 1) & 1), abort_flag);
          ptx::mbar_wait(&v_full[s], (uint32_t)((j >> 1) & 1), abort_flag);
          ptx::tc_fence_after_sync();
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            ptx::mma_f16_ss(tmem_o, ptx::desc_advance(p_desc, s * 16384 + ks * 32),
                            ptx::desc_advance(v_desc, s * 32768 + ks * 2048), idesc_o, (i > g.lo || ks > 0) ? 1u : 0u);
          ptx::mma_commit(&pv_done[s]);
          // V of the next tile goes where P V of the previous tile read; that one was issued a whole tile ago
          if (j >= 1 && (BINS || j + 1 < g.hi)) {
            ptx::mbar_wait(&pv_done[s ^ 1], (uint32_t)(((j - 1) >> 1) & 1), abort_flag);
            load_next_v();
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ softmax + epilogue (warps 0-7)
    // Thread = (query row, half of the tile's 64 keys): warps 0-3 take keys 0-31, warps 4-7 keys 32-63 of the
    // same 128 rows (a warp reaches the TMEM lanes 32 * (warp % 4) ..).  The two halves of a row swap their
    // maxima through shared memory, so both keep the same running reference; each rescales and writes out its
    // half of the 256 output features.
    const int quad = warp & 3, half = warp >> 2;
    const int row = quad * 32 + lane;   // 0..127
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    int j = 0, n_gates = 0;             // tiles and gate loads so far
    for (int it = it_first; it < (BINS ? it_end : it_first + 1); ++it) {
      const Seg g = seg_at(it);
      const int m0 = g.m0, head = g.head;
      const int qi = m0 + row;            // query row
      const bool cut = BINS && (g.lo > 0 || g.hi < g.nt);
      const bool gate_tile = p.tma_drain && p.gate && !cut, out_tile = p.tma_drain && !cut;
      float m_used = -INFINITY, l = 0.f;
      for (int i = g.lo; i < g.hi; ++i, ++j) {
        const int s = j & 1;
        ptx::mbar_wait(&s_ready[s], (uint32_t)((j >> 1) & 1), abort_flag);
        ptx::tc_fence_after_sync();
        // the last S has been computed, so nothing reads Q any more
        if (BINS && i == g.hi - 1 && !out_tile && tid == 0) ptx::mbar_arrive(q_free);
        if (i == g.hi - 1 && gate_tile && tid == 0) {
          // its buffer receives the gate tile ([128 rows x 256] as four 64-feature slabs, swizzled like an operand)
          // while the last tile is finished
          ptx::mbar_expect_tx(g_full, 4 * 16384);
          for (int kb = 0; kb < 4; ++kb)
            ptx::tma_load_3d(q_s + kb * 16384, &tm_g, g_full, kb * 64, p.g_head_inner ? head : m0,
                             p.g_head_inner ? m0 : head);
        }
        uint32_t sv[32];
        {
          uint32_t sb[32];
          const uint32_t sa = tmem_base + lane_off + (uint32_t)(s * 2 * FB_N + half * 32);
          ptx::tmem_ld32(sa, sv);
          ptx::tmem_ld32(sa + FB_N, sb);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 32; ++c) sv[c] = __float_as_uint(__uint_as_float(sv[c]) + __uint_as_float(sb[c]));
        }
        ptx::tc_fence_before_sync();
        ptx::mbar_arrive(&s_free[s]);
        const int key0 = i * FB_N + half * 32;
        const bool need_mask = i * FB_N + FB_N - 1 > m0 + past;  // tile reaches past the first row's diagonal
        // sv keeps the raw dot products; the (positive) scale is applied once to the maximum here and inside the
        // exponent's fused multiply-add below
        if (need_mask) {
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (key0 + c > qi + past) sv[c] = 0xff800000u;   // -inf
        }
        float tm4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // four independent chains
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
#pragma unroll
          for (int i = 0; i < 4; ++i) tm4[i] = fmaxf(tm4[i], __uint_as_float(sv[c + i]));
        }
        float tmax = fmaxf(fmaxf(tm4[0], tm4[1]), fmaxf(tm4[2], tm4[3])) * p.scale_log2;
        // Both halves of a row must use the SAME reference, and any upper bound of the tile's maximum will do:
        // each half publishes its maximum rounded UP to bfloat16 and both take the larger of the two rounded values.
        {
          const uint32_t tb = __float_as_uint(tmax);
          const uint16_t up = (uint16_t)(((tb >> 31) ? tb : tb + 0xFFFFu) >> 16);   // toward +inf; -inf stays -inf
          rowmax_s[(s * 2 + half) * FB_M + row] = up;
          asm volatile("bar.sync %0, 64;" ::"r"(quad + 1) : "memory");   // the two warps that share these rows
          const uint16_t other = rowmax_s[(s * 2 + (half ^ 1)) * FB_M + row];
          tmax = fmaxf(__uint_as_float((uint32_t)up << 16), __uint_as_float((uint32_t)other << 16));
        }
        float factor = 1.f;
        bool grow = false;
        const bool first = i == g.lo;
        if (first) {
          m_used = cut ? fmaxf(tmax, kNoMax) : tmax;  // an item's key 0 is visible to every row: finite unless cut
        } else {
          grow = tmax > m_used + 8.f;
        }
        // P buffer s is free once P V of tile j-2 has read it
        if (j >= 2) ptx::mbar_wait(&pv_done[s], (uint32_t)(((j >> 1) - 1) & 1), abort_flag);
        if (!first) {
          if (__any_sync(0xffffffffu, grow)) {   // the same answer in both warps of a row quarter
            // O is final only after the previous P V finished
            ptx::mbar_wait(&pv_done[(j - 1) & 1], (uint32_t)(((j - 1) >> 1) & 1), abort_flag);
            ptx::tc_fence_after_sync();
            if (grow) {
              factor = exp2f(m_used - tmax);
              m_used = tmax;
            }
#pragma unroll 1
            for (int c0 = half * (FB_D / 2); c0 < (half + 1) * (FB_D / 2); c0 += 32) {
              uint32_t ov[32];
              ptx::tmem_ld32(tmem_o + lane_off + (uint32_t)c0, ov);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * factor);
              ptx::tmem_st32(tmem_o + lane_off + (uint32_t)c0, ov);
            }
            ptx::tmem_st_wait();
            l *= factor;
          }
        }
        float psum = 0.f;
        uint8_t* prow = p_s + s * 16384 + row * 128;
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float xa = fmaf(__uint_as_float(sv[c8 * 8 + 2 * i]), p.scale_log2, -m_used);
            const float xb = fmaf(__uint_as_float(sv[c8 * 8 + 2 * i + 1]), p.scale_log2, -m_used);
            const float a = fast_ex2(xa);
            const bool on_fma = kPolyOf8 == 1 ? i == 0 : kPolyOf8 == 2 ? (i & 1) == 0 : kPolyOf8 == 3 ? i < 3 : kPolyOf8 >= 4;
            const float b = on_fma ? poly_ex2(xb) : fast_ex2(xb);
            psum += a + b;
            w[i] = pack2<BF16>(a, b);
          }
          *reinterpret_cast<uint4*>(prow + (((half * 4 + c8) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        l += psum;
        ptx::fence_proxy_async_smem();
        ptx::tc_fence_before_sync();
        ptx::mbar_arrive(&p_ready[s]);
      }
      // epilogue: the row sum over both halves, then each half writes its 128 output features
      if (cut) {
        // partial: O as it stands, four features of the 128 rows side by side (a warp stores 512 bytes at a time)
        float* rowsum_s = reinterpret_cast<float*>(rowmax_s);   // [2 halves][128 rows]
        asm volatile("bar.sync 5, 256;" ::: "memory");   // all eight warps: every maximum of the last tile has been read
        rowsum_s[half * FB_M + row] = l;
        const int slot = part_slot((int)blockIdx.x, g.lo > 0);
        float4* po = p.part_o + ((int64_t)slot * (FB_D / 4) + half * (FB_D / 8)) * FB_M + row;
        ptx::mbar_wait(&pv_done[(j - 1) & 1], (uint32_t)(((j - 1) >> 1) & 1), abort_flag);
        ptx::tc_fence_after_sync();
#pragma unroll 1
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t ov[32];
          ptx::tmem_ld32(tmem_o + lane_off + (uint32_t)(half * (FB_D / 2) + cc * 32), ov);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4)
            po[(cc * 8 + c4) * FB_M] = make_float4(__uint_as_float(ov[4 * c4]), __uint_as_float(ov[4 * c4 + 1]),
                                                   __uint_as_float(ov[4 * c4 + 2]), __uint_as_float(ov[4 * c4 + 3]));
        }
        asm volatile("bar.sync 5, 256;" ::: "memory");   // every row sum is there
        if (half == 0)
          p.part_ml[(int64_t)slot * FB_M + row] = make_float2(m_used == kNoMax ? -INFINITY : m_used, l + rowsum_s[FB_M + row]);
        asm volatile("bar.sync 5, 256;" ::: "memory");   // read: the next segment's maxima may overwrite them
      } else if (out_tile) {
        // Drain through shared memory so that global memory sees whole tiles: the gate tile arrived by TMA in the Q
        // buffer; each thread turns the 16-byte chunks of its half row into output chunks in place; one TMA store
        // per slab writes the tile (rows past the end of the sequence are clipped by the tensor map).
        float* rowsum_s = reinterpret_cast<float*>(rowmax_s);   // [2 halves][128 rows]
        asm volatile("bar.sync 5, 256;" ::: "memory");   // all eight warps: every maximum of the last tile has been read
        rowsum_s[half * FB_M + row] = l;
        asm volatile("bar.sync %0, 64;" ::"r"(quad + 1) : "memory");
        l += rowsum_s[(half ^ 1) * FB_M + row];
        ptx::mbar_wait(&pv_done[(j - 1) & 1], (uint32_t)(((j - 1) >> 1) & 1), abort_flag);
        if (p.gate) ptx::mbar_wait(g_full, (uint32_t)(n_gates++ & 1), abort_flag);
        ptx::tc_fence_after_sync();
        const float inv_l = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t ov[32];
          ptx::tmem_ld32(tmem_o + lane_off + (uint32_t)(half * (FB_D / 2) + cc * 32), ov);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int c8 = 0; c8 < 4; ++c8) {
            const int chunk = half * 16 + cc * 4 + c8;   // 16-byte chunk of the 512-byte row
            uint4* cell = reinterpret_cast<uint4*>(q_s + (chunk >> 3) * 16384 + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
            uint32_t w[4];
            if (p.gate) {
              const uint4 g = *cell;
              const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 gg = unpack2<BF16>(gw[i]);
                // sigmoid(g) = 0.5 + 0.5 * tanh(g / 2): one special-function result per element
                const float sa = fmaf(0.5f, fast_tanh(0.5f * gg.x), 0.5f), sb = fmaf(0.5f, fast_tanh(0.5f * gg.y), 0.5f);
                w[i] = pack2<BF16>(__uint_as_float(ov[c8 * 8 + 2 * i]) * inv_l * sa,
                                   __uint_as_float(ov[c8 * 8 + 2 * i + 1]) * inv_l * sb);
              }
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                w[i] = pack2<BF16>(__uint_as_float(ov[c8 * 8 + 2 * i]) * inv_l, __uint_as_float(ov[c8 * 8 + 2 * i + 1]) * inv_l);
            }
            *cell = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        ptx::fence_proxy_async_smem();
        asm volatile("bar.sync 5, 256;" ::: "memory");
        if (tid == 0) {
          for (int kb = 0; kb < 4; ++kb)
            ptx::tma_store_3d(&tm_o, q_s + kb * 16384, kb * 64, p.o_head_inner ? head : m0, p.o_head_inner ? m0 : head);
          ptx::tma_store_commit();
          ptx::tma_store_wait_read();
          if (BINS) ptx::mbar_arrive(q_free);
        }
      } else {
      // The gate values of this thread's half row (16 x 16 bytes) are requested first, all at once: they travel
        // while the last P V finishes and the row sums are exchanged (one load per use would put 16 round trips
        // to L2 on the drain's critical path).
        const bool row_ok = qi < p.S;
        const uint16_t* gptr = (p.gate && row_ok) ? reinterpret_cast<const uint16_t*>(p.gate) + (int64_t)qi * p.g_ss +
                                                        (int64_t)head * p.g_sh + half * (FB_D / 2)
                                                  : nullptr;
        uint4 gv[16];
    #pragma unroll
        for (int i = 0; i < 16; ++i) gv[i] = gptr ? __ldg(reinterpret_cast<const uint4*>(gptr) + i) : make_uint4(0, 0, 0, 0);
        float* rowsum_s = reinterpret_cast<float*>(rowmax_s);   // [2 halves][128 rows]
        asm volatile("bar.sync 5, 256;" ::: "memory");   // all eight warps: every maximum of the last tile has been read
        rowsum_s[half * FB_M + row] = l;
        asm volatile("bar.sync %0, 64;" ::"r"(quad + 1) : "memory");
        l += rowsum_s[(half ^ 1) * FB_M + row];
        ptx::mbar_wait(&pv_done[(j - 1) & 1], (uint32_t)(((j - 1) >> 1) & 1), abort_flag);
        ptx::tc_fence_after_sync();
        const float inv_l = l > 0.f ? 1.f / l : 0.f;
        uint16_t* optr = reinterpret_cast<uint16_t*>(p.out) + (int64_t)qi * p.o_ss + (int64_t)head * p.o_sh + half * (FB_D / 2);
    #pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t ov[32];
          ptx::tmem_ld32(tmem_o + lane_off + (uint32_t)(half * (FB_D / 2) + cc * 32), ov);
          ptx::tmem_ld_wait();
          if (row_ok) {
    #pragma unroll
            for (int c8 = 0; c8 < 4; ++c8) {
              const uint4 g = gv[cc * 4 + c8];
              const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
              uint32_t w[4];
    #pragma unroll
              for (int i = 0; i < 4; ++i) {
                float a = __uint_as_float(ov[c8 * 8 + 2 * i]) * inv_l;
                float b = __uint_as_float(ov[c8 * 8 + 2 * i + 1]) * inv_l;
                if (p.gate) {
                  const float2 gg = unpack2<BF16>(gw[i]);
                  a = __fdividef(a, 1.f + __expf(-gg.x));
                  b = __fdividef(b, 1.f + __expf(-gg.y));
                }
                w[i] = pack2<BF16>(a, b);
              }
              *reinterpret_cast<uint4*>(optr + cc * 32 + c8 * 8) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
        asm volatile("bar.sync 5, 256;" ::: "memory");   // the row sums have been read
      }
      ptx::tc_fence_before_sync();
    }
  }

  __syncthreads();
  if (warp == 0) ptx::tmem_dealloc(tmem_base, 512);
  if (tid == 0 && *abort_flag && p.status) atomicExch(p.status, 1);
}

// Joins the partials of the items that a bin boundary cut, and finishes them as the drain above would (division by
// the sum, gate, rounding).  Block (bin - 1, 32 features): the block of the bin in which an item's second piece lies does
// the item, the others leave.  Thread = (row, 16 features): the partials are read 512 bytes a warp, the output in
// whole 32-byte sectors.
template <bool BF16>
__global__ void __launch_bounds__(256) flash_merge_kernel(const __grid_constant__ FlashParams p) {
  const int bin = (int)blockIdx.x + 1;
  const uint32_t at = p.bin_start[bin], before = p.bin_start[bin - 1];
  const int it = (int)(at >> 16);
  if ((at & 0xFFFFu) == 0 || ((before >> 16) == (uint32_t)it && (before & 0xFFFFu) != 0)) return;
  int last = bin;   // bins bin .. last start inside the item
  while (last + 1 < p.n_bins && (int)(p.bin_start[last + 1] >> 16) == it) ++last;
  const int n_qt = (p.S + FB_M - 1) / FB_M;
  const int row = threadIdx.x & (FB_M - 1), f16 = (int)blockIdx.y * 2 + (threadIdx.x >> 7);
  const int qi = (n_qt - 1 - it / p.Hq) * FB_M + row, head = it % p.Hq;
  if (qi >= p.S) return;
  float m = -INFINITY;
#pragma unroll 8
  for (int b = bin - 1; b <= last; ++b) m = fmaxf(m, __ldg(&p.part_ml[(int64_t)part_slot(b, b >= bin) * FB_M + row].x));
  float l = 0.f;
  float4 o[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) o[c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int b = bin - 1; b <= last; ++b) {   // in the order of the keys
    const int slot = part_slot(b, b >= bin);
    const float2 ml = __ldg(p.part_ml + (int64_t)slot * FB_M + row);
    const float4* po = p.part_o + ((int64_t)slot * (FB_D / 4) + f16 * 4) * FB_M + row;
    float4 v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = __ldg(po + c * FB_M);
    // a row without a finite maximum anywhere has no weights: (-inf) - (-inf), as in an item that is not cut
    const float w = exp2f(ml.x - m);
    l = fmaf(ml.y, w, l);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      o[c].x = fmaf(v[c].x, w, o[c].x);
      o[c].y = fmaf(v[c].y, w, o[c].y);
      o[c].z = fmaf(v[c].z, w, o[c].z);
      o[c].w = fmaf(v[c].w, w, o[c].w);
    }
  }
  const float inv_l = l > 0.f ? 1.f / l : 0.f;
  uint4* optr = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (int64_t)qi * p.o_ss + (int64_t)head * p.o_sh + f16 * 16);
  const uint4* gptr = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.gate) + (int64_t)qi * p.g_ss +
                                                     (int64_t)head * p.g_sh + f16 * 16);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float x[8] = {o[2 * h].x, o[2 * h].y, o[2 * h].z, o[2 * h].w, o[2 * h + 1].x, o[2 * h + 1].y, o[2 * h + 1].z, o[2 * h + 1].w};
    uint32_t gw[4] = {0, 0, 0, 0}, w[4];
    if (p.gate) {
      const uint4 g = __ldg(gptr + h);
      gw[0] = g.x; gw[1] = g.y; gw[2] = g.z; gw[3] = g.w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float a = x[2 * i] * inv_l, c = x[2 * i + 1] * inv_l;
      if (p.gate) {
        const float2 gg = unpack2<BF16>(gw[i]);
        a = __fdividef(a, 1.f + __expf(-gg.x));
        c = __fdividef(c, 1.f + __expf(-gg.y));
      }
      w[i] = pack2<BF16>(a, c);
    }
    optr[h] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

}  // namespace mxb

using namespace mxb;

// How the items are dealt out.  Costs are in tiles (0.9 to 1.05 us each on a B200): a segment costs its tiles and
// kSegCost for its Q load, first scores and drain; cutting costs kCutCost (partials out, merge launch, partials in), and
// the stretches must be kSaving percent shorter than the SM with the most whole items works.  That much, because tiles
// take a tenth longer when every SM streams K and V at once, and because a cut saves time and not energy: back to back,
// under the power cap, the SMs that idle behind whole items leave the others a higher clock.  Stretches of less than
// kMinShare are not worth an SM of their own.  Measured (16 query / 2 KV heads, bf16, gated; tokens over past, us, one
// CTA per item against equal stretches, alone / back to back for half a second):
//   64 over 3,000 51.1 -> 27.6 and 64 over 30,000 404 -> 74.4 alone; 500 over 30,000 531 -> 264 / 508 -> 290;
//   1,200 over 30,000 1,082 -> 633 / 1,011 -> 692; 1,700 over 30,000 (saving 29 %) 1,092 -> 864 / 1,073 -> 958;
//   1,900 over 30,000 (21 %) 1,112 -> 936 / 1,106 -> 1,037;
// below the line 2,048 over 30,720 (13 %) 1,136 -> 1,038 / 1,154 -> 1,140; 3,000 over 8,000 (11 %) 458 -> 429 / 477 -> 495;
//   5,000 over 8,000 (10 %) 808 -> 778 / 871 -> 898; 704 over 2,000 (12 %) 63 -> 66 / 48 -> 53; 1,728 over 4,000 (13 %)
//   185 -> 168 / 161 -> 165; 1,024 over 12,000 (10 %) 240 -> 219 / 214 -> 227; 2,048 over 24,000 (13 %) 913 -> 762 / 893 -> 847;
//   32 heads, 2,048 over 30,720 (14 %) 2,267 -> 2,442; 700 over 1,365 39.8 -> 44.2 and 1,000 over 1,000 40.5 -> 47.5 alone.
// A cut changes the results in the last bits (P is rounded to 16 bits against each segment's own reference; the error
// against float64 stays the same, 2.31e-3 relative in bf16 on either side).  The partials take up to 39 MB (296 slots).
constexpr int kSegCost = 4, kCutCost = 16, kMinShare = 12, kSaving = 15;

// Fills p.n_bins / p.bin_start (n_bins = 0: one CTA per item) and returns the bytes of partials the plan needs.
static int64_t flash_plan(FlashParams& p, int sms) {
  p.n_bins = 0;
  if (sms > kMaxBins) sms = kMaxBins;
  const int n_qt = (int)ceil_div(p.S, FB_M);
  const int64_t items = (int64_t)n_qt * p.Hq;
  // more than eight rounds of items even out by themselves; bin_start holds 16 bits of tile
  if (items > 8 * sms || flash_tiles(n_qt - 1, p.S, p.Skv) > 0xFFFF) return 0;
  // One CTA per item: the hardware hands the next item to the SM that is done first.  Dealt back and forth over the
  // SMs, longest first, that ends with the largest of these sums.
  int load[kMaxBins] = {0}, longest = 0, k = 0, step = 1;
  int64_t total = 0;
  for (int qt = n_qt - 1; qt >= 0; --qt) {
    const int cost = flash_tiles(qt, p.S, p.Skv) + kSegCost;
    total += (int64_t)cost * p.Hq;
    for (int h = 0; h < p.Hq; ++h) {
      load[k] += cost;
      if (load[k] > longest) longest = load[k];
      k += step;
      if (k == sms || k < 0) {
        step = -step;
        k += step;
      }
    }
  }
  const int bins = (int)(total / kMinShare < sms ? total / kMinShare : sms);
  if (bins < 2 || 100 * (int64_t)longest <= (100 + kSaving) * (total / bins) + 100 * kCutCost) return 0;
  // Equal stretches of the items' costs.  A piece of fewer than kSegCost tiles is not worth a segment: the boundary
  // moves to the item's edge.
  uint32_t* start = p.bin_start;
  int n = 0, qt = n_qt - 1, h = 0, nt = flash_tiles(qt, p.S, p.Skv);
  int64_t c0 = 0;     // where item (qt, h) starts
  uint32_t item = 0;
  start[n++] = 0;
  for (int b = 1; b < bins; ++b) {
    const int64_t x = total * b / bins;
    while (x >= c0 + nt + kSegCost) {
      c0 += nt + kSegCost;
      ++item;
      if (++h == p.Hq) {
        h = 0;
        nt = flash_tiles(--qt, p.S, p.Skv);
      }
    }
    const int64_t j = x - c0 - kSegCost / 2;
    const uint32_t at = j < kSegCost ? item << 16 : j > nt - kSegCost ? (item + 1) << 16 : item << 16 | (uint32_t)j;
    if (at > start[n - 1] && at < (uint32_t)items << 16) start[n++] = at;
  }
  start[n] = (uint32_t)items << 16;
  p.n_bins = n;
  return (int64_t)2 * n * FB_M * (FB_D * 4 + 8);
}

static int flash_validate(const mxb_flash_prefill_args* a) {
  MXB_REQUIRE(a != nullptr, MXB_ERR_INVALID, "flash prefill: null args");
  MXB_REQUIRE(a->D == 256, MXB_ERR_INVALID, "flash prefill requires head_dim=256");
  MXB_REQUIRE(a->dtype == MXB_BF16 || a->dtype == MXB_F16, MXB_ERR_INVALID,
              "flash prefill requires bfloat16 or float16 operands");
  MXB_REQUIRE(a->S > 0 && a->Skv >= a->S, MXB_ERR_INVALID, "flash prefill requires 1 <= S <= Skv");
  MXB_REQUIRE(a->Hq > 0 && a->Hkv > 0 && a->Hq % a->Hkv == 0, MXB_ERR_INVALID,
              "query heads must be a multiple of kv heads");
  MXB_REQUIRE(a->q && a->k && a->v && a->out, MXB_ERR_INVALID, "flash prefill: null tensor");
  return MXB_OK;
}

extern "C" int64_t mxb_flash_prefill_workspace_bytes(const mxb_flash_prefill_args* a) {
  if (flash_validate(a) != MXB_OK) return 0;
  FlashParams p{};
  p.S = a->S; p.Skv = a->Skv; p.Hq = a->Hq;
  return flash_plan(p, sm_count());
}

extern "C" int mxb_flash_prefill(const mxb_flash_prefill_args* a, void* stream) {
  int rc = flash_validate(a);
  if (rc != MXB_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  MXB_REQUIRE((reinterpret_cast<uintptr_t>(a->out) & 15) == 0 && a->out_stride_s % 8 == 0 && a->out_stride_h % 8 == 0,
              MXB_ERR_INVALID, "out must be 16-byte aligned with strides that are multiples of 8 elements");
  MXB_REQUIRE(!a->gate || ((reinterpret_cast<uintptr_t>(a->gate) & 15) == 0 && a->gate_stride_s % 8 == 0 &&
                           a->gate_stride_h % 8 == 0),
              MXB_ERR_INVALID, "gate must be 16-byte aligned with strides that are multiples of 8 elements");
  const CUtensorMapDataType dt = a->dtype == MXB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tq, tk, tv;
  // cuTensorMapEncodeTiled wants ascending strides: put the head axis before the row axis when its
  // stride is the smaller one ([rows, heads, D] layouts); the box is one head wide either way.
  const bool q_hin = a->q_stride_h < a->q_stride_s, k_hin = a->k_stride_h < a->k_stride_s;
  {
    uint64_t dims[3] = {(uint64_t)a->D, (uint64_t)(q_hin ? a->Hq : a->S), (uint64_t)(q_hin ? a->S : a->Hq)};
    uint64_t str[2] = {(uint64_t)(q_hin ? a->q_stride_h : a->q_stride_s) * 2,
                       (uint64_t)(q_hin ? a->q_stride_s : a->q_stride_h) * 2};
    uint32_t box[3] = {64, q_hin ? 1u : (uint32_t)FB_M, q_hin ? (uint32_t)FB_M : 1u};
    rc = make_tensor_map(&tq, dt, 3, a->q, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != MXB_OK) return rc;
  }
  {
    uint64_t dims[3] = {(uint64_t)a->D, (uint64_t)(k_hin ? a->Hkv : a->Skv), (uint64_t)(k_hin ? a->Skv : a->Hkv)};
    uint64_t str[2] = {(uint64_t)(k_hin ? a->k_stride_h : a->k_stride_s) * 2,
                       (uint64_t)(k_hin ? a->k_stride_s : a->k_stride_h) * 2};
    uint32_t box[3] = {64, k_hin ? 1u : (uint32_t)FB_N, k_hin ? (uint32_t)FB_N : 1u};
    rc = make_tensor_map(&tk, dt, 3, a->k, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != MXB_OK) return rc;
  }
  const bool v_hin = a->v_stride_h < a->v_stride_s;
  {
    uint64_t dims[3] = {(uint64_t)a->D, (uint64_t)(v_hin ? a->Hkv : a->Skv), (uint64_t)(v_hin ? a->Skv : a->Hkv)};
    uint64_t str[2] = {(uint64_t)(v_hin ? a->v_stride_h : a->v_stride_s) * 2,
                       (uint64_t)(v_hin ? a->v_stride_s : a->v_stride_h) * 2};
    uint32_t box[3] = {64, v_hin ? 1u : (uint32_t)FB_N, v_hin ? (uint32_t)FB_N : 1u};
    rc = make_tensor_map(&tv, dt, 3, a->v, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != MXB_OK) return rc;
  }

  // gate and output tiles travel by TMA when their layouts allow a tensor map (rows and heads at distinct,
  // 16-byte aligned strides); otherwise the kernel reads and writes them with per-thread accesses
  CUtensorMap tg, to;
  memset(&tg, 0, sizeof(tg));
  memset(&to, 0, sizeof(to));
  const bool g_hin = a->gate_stride_h < a->gate_stride_s, o_hin = a->out_stride_h < a->out_stride_s;
  auto tile_map = [&](CUtensorMap* m, const void* base, int64_t ss, int64_t sh, bool hin) -> bool {
    if (ss <= 0 || sh <= 0 || ss == sh) return false;
    uint64_t dims[3] = {(uint64_t)a->D, (uint64_t)(hin ? a->Hq : a->S), (uint64_t)(hin ? a->S : a->Hq)};
    uint64_t str[2] = {(uint64_t)(hin ? sh : ss) * 2, (uint64_t)(hin ? ss : sh) * 2};
    uint32_t box[3] = {64, hin ? 1u : (uint32_t)FB_M, hin ? (uint32_t)FB_M : 1u};
    if (str[0] > str[1] || str[1] % str[0] != 0) return false;   // plain nested layouts only
    return make_tensor_map(m, dt, 3, base, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B) == MXB_OK;
  };
  bool tma_drain = tile_map(&to, a->out, a->out_stride_s, a->out_stride_h, o_hin);
  if (tma_drain && a->gate) tma_drain = tile_map(&tg, a->gate, a->gate_stride_s, a->gate_stride_h, g_hin);

  MXB_REQUIRE(a->scale > 0.f, MXB_ERR_INVALID, "flash prefill: scale must be positive");
  FlashParams p{};
  p.g_head_inner = g_hin ? 1 : 0; p.o_head_inner = o_hin ? 1 : 0; p.tma_drain = tma_drain ? 1 : 0;
  p.v_head_inner = v_hin ? 1 : 0;
  p.gate = a->gate; p.g_ss = a->gate_stride_s; p.g_sh = a->gate_stride_h;
  p.out = a->out; p.o_ss = a->out_stride_s; p.o_sh = a->out_stride_h;
  p.S = a->S; p.Skv = a->Skv; p.Hq = a->Hq; p.Hkv = a->Hkv;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.status = a->status;
  p.q_head_inner = q_hin ? 1 : 0;
  p.k_head_inner = k_hin ? 1 : 0;
  const int smem = FlashSmem::total + 1024;
  // the partials of cut items need the workspace; without it every item is one CTA's
  const int64_t need = flash_plan(p, sm_count());
  if (!a->workspace || a->workspace_bytes < need || (reinterpret_cast<uintptr_t>(a->workspace) & 15) != 0) p.n_bins = 0;
  p.part_o = reinterpret_cast<float4*>(a->workspace);
  p.part_ml = reinterpret_cast<float2*>(p.part_o + (int64_t)2 * p.n_bins * (FB_D / 4) * FB_M);
  const dim3 grid(p.n_bins > 0 ? (unsigned)p.n_bins : (unsigned)(ceil_div(a->S, FB_M) * a->Hq));
  const dim3 merge_grid((unsigned)(p.n_bins - 1), FB_D / 32);
  auto go = [&](auto* whole, auto* binned, auto* merge) -> int {
    auto* kernel = p.n_bins > 0 ? binned : whole;
    MXB_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kernel<<<grid, 384, smem, st>>>(tq, tk, tv, tg, to, p);
    note_launch();
    if (p.n_bins > 1) {
      merge<<<merge_grid, 256, 0, st>>>(p);
      note_launch();
    }
    MXB_CUDA_OK(cudaGetLastError());
    return MXB_OK;
  };
  return a->dtype == MXB_BF16 ? go(flash_prefill_kernel<true, false>, flash_prefill_kernel<true, true>, flash_merge_kernel<true>)
                              : go(flash_prefill_kernel<false, false>, flash_prefill_kernel<false, true>, flash_merge_kernel<false>);
}
