// Causal GQA flash prefill, head_dim 256, 16-bit operands, fp32 accumulation, with the
// sigmoid-gate epilogue fused:  out = softmax(scale * Q K^T + causal) V * sigmoid(gate).
//
// Work comes in items: 128 query rows in each CTA of a pair (a cluster of two on neighbouring SMs), over the 128-key
// tiles they see: the same rows of two query heads of one KV head, or 256 rows of one head where heads do not pair up.
// Items are numbered longest first (every head's latest query tile first), because causal items differ 64-fold in
// length.  Two ways to deal them out (flash_plan, below the kernel):
//   one pair per item, when the items fill the SMs evenly;
//   one pair per two SMs, each with an equal stretch of the concatenated tiles of all items, when they would not (a
//   short chunk over a long past is 8 pairs; 128 equal items on 74 pairs of SMs are two waves, the second part-empty).
//   A pair walks the segments of its stretch; an item that a boundary cuts leaves (O, max, sum) partials in fp32, which
//   flash_merge_kernel joins, gate included.
// The MMAs are pair MMAs (cta_group::2, M = 256): each CTA holds its own 128 query rows and half of every K and V tile,
// and gets the other half's data from its neighbour.  That halves the operand bytes per SM, which is what bounded one CTA
// on its own: S = Q K^T with 64 keys moved 6 KB of shared memory per MMA of 32 tensor cycles (48 cycles at 128 B a
// clock), the K and V tiles' arrival 64 KB per 64 keys, P 16 KB in and 16 KB out; 1,750 of the 1,890 cycles a 64-key tile
// took.  Here 128 keys cost 96 KB of Q and K, 32 KB of V and 64 KB of arrivals in 2,048 tensor cycles, and P travels
// through tensor memory.  8,192 tokens of 16 heads, gated bf16: 560 -> 477 us back to back under the power cap, 2,048
// over a past of 30,720: 1,080 -> 850.
// Twelve warps per CTA:
//   warps 0-7  softmax + drain, in two groups of four that take the key tiles in turn; thread = query row
//   warp  8    issues the S = Q K^T MMAs for the pair (one lane of the even CTA)
//   warp  9    TMA producer for this CTA's halves of Q, K and V (one lane)
//   warp 10    issues the O += P V MMAs for the pair (one lane of the even CTA)
// Per 128-key tile:  S = Q K^T (M256 x N128 x K256) into one of two TMEM buffers; the softmax warps read S, keep a
// running maximum with lazy rescaling of the TMEM-resident O (only when the maximum grew by more than 2^8) and write P
// over the S it came from, 16 bits an element; O += P V (M256 x N256 x K128) with P read from TMEM and V in place as an
// MN-major B operand (no transposed copy).  S of tile j + 1 runs before P V of tile j, so the tensor pipe works while the
// softmax of tile j + 1 does; what a tile takes beyond its tensor cycles (2,680 measured) is the wait for P V of tile j
// before S of tile j + 2 may overwrite its P, and shared memory at its limit while K and V tiles arrive under S.
// Drain: the gate tile arrives by TMA in the Q buffer during the last tile; each thread normalises its half row,
// applies the sigmoid and writes the output chunks in place; TMA stores write the tile.
// TMEM: S0 / P0 [0,128) S1 / P1 [128,256) O [256,512).
#include "flash_common.cuh"

namespace mxb {

constexpr int FB_N = 128;
constexpr int kStages = 5;

struct FlashSmem {
  static constexpr int stage_bytes = 32768;             // a CTA's half of a K or V tile
  static constexpr int q_off = 0;                       // 4 slabs x [128 x 128 B]
  static constexpr int ring_off = q_off + 4 * 16384;    // K: 4 slabs x [64 keys x 128 B]; V: 2 slabs x [128 keys x 128 B]
  static constexpr int bar_off = ring_off + kStages * stage_bytes;
  static constexpr int rowmax_off = bar_off + 256;      // [128 rows] reference maximum
  static constexpr int rowsum_off = rowmax_off + 512;   // [2 groups][128 rows]
  static constexpr int total = rowsum_off + 1024;
};

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

__device__ __forceinline__ float bf16_up(float x) {   // rounded toward +inf; -inf stays
  const uint32_t b = __float_as_uint(x);
  return __uint_as_float(((b >> 31) ? b : b + 0xFFFFu) & 0xFFFF0000u);
}

template <bool BF16, bool BINS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
flash_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_g,
                     const __grid_constant__ CUtensorMap tm_o, const __grid_constant__ FlashParams p) {
  using L = FlashSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* q_s = smem + L::q_off;
  uint8_t* ring = smem + L::ring_off;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bar_off);
  float* rowmax_s = reinterpret_cast<float*>(smem + L::rowmax_off);
  float* rowsum_s = reinterpret_cast<float*>(smem + L::rowsum_off);
  uint64_t* full = bars + 0;       // [kStages] even CTA: both halves of a tile have landed
  uint64_t* empty = bars + 5;      // [kStages] the MMAs that read a tile are done
  uint64_t* q_full = bars + 10;    // even CTA: both query tiles have landed
  uint64_t* q_free = bars + 11;    // the Q buffer may take the next segment's rows
  uint64_t* s_ready = bars + 12;   // [2]
  uint64_t* p_ready = bars + 14;   // [2 buffers][2 halves] even CTA: both CTAs' P of 64 keys of a tile
  uint64_t* pv_done = bars + 18;   // [2]
  uint64_t* g_full = bars + 20;    // gate tile landed
  uint64_t* qk_issued = bars + 21; // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 23);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)ptx::cluster_ctarank(), pair = (int)blockIdx.x >> 1;
  const FlashItems items = flash_items(p.S, p.Hq, p.pair_heads);
  const int past = p.Skv - p.S;
  int it_first = pair, j_first = 0, it_stop = it_first + 1, j_stop = 0;
  if constexpr (BINS) {
    const uint32_t at = p.bin_start[pair], stop = p.bin_start[pair + 1];
    it_first = (int)(at >> 16); j_first = (int)(at & 0xFFFFu);
    it_stop = (int)(stop >> 16); j_stop = (int)(stop & 0xFFFFu);
  }
  // The walk over this pair's segments, identical in every role of both CTAs: item `it`, its tiles [lo, hi) of nt.
  struct Seg { int lo, hi, nt, head, kvh, m0; };
  auto seg_at = [&](int it) {
    Seg g;
    flash_item_at(items, it, p.pair_heads, rank, g.head, g.m0);
    g.kvh = g.head / (p.Hq / p.Hkv);
    g.nt = flash_tiles<FB_N>(items.n_qt - 1 - it / items.per_qt, p.pair_heads ? FB_M : 2 * FB_M, p.S, p.Skv);
    g.lo = BINS && it == it_first ? j_first : 0;
    g.hi = BINS && it == it_stop ? j_stop : g.nt;
    return g;
  };
  const int it_end = BINS ? (j_stop > 0 ? it_stop + 1 : it_stop) : it_first + 1;
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      ptx::mbar_init(&full[i], 1);
      ptx::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&s_ready[i], 1);
      ptx::mbar_init(&pv_done[i], 1);
      ptx::mbar_init(&qk_issued[i], 1);
      for (int h = 0; h < 2; ++h) ptx::mbar_init(&p_ready[2 * i + h], 8);   // the four warps of a group, in both CTAs
    }
    ptx::mbar_init(q_full, 1);
    ptx::mbar_init(q_free, 1);
    ptx::mbar_init(g_full, 1);
    *abort_flag = 0;
    ptx::mbar_fence_init();
  }
  __syncwarp();
  if (warp == 0) {
    ptx::tmem_alloc_pair(tmem_slot, 512);
    ptx::tmem_relinquish_pair();
  }
  if (tid == 288) {
    ptx::tma_prefetch_desc(&tm_q);
    ptx::tma_prefetch_desc(&tm_k);
    ptx::tma_prefetch_desc(&tm_v);
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_arrive();   // the neighbour's barriers are set up before anything arrives on them
  ptx::cluster_wait();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_o = tmem_base + 256;

  if (warp == 9) {
    // ------------------------------------------------------------ TMA producer: this CTA's halves, in the order of use
    if (lane == 0) {
      const uint32_t full0 = ptx::cluster_map(ptx::smem_u32(full), 0), q_full0 = ptx::cluster_map(ptx::smem_u32(q_full), 0);
      int n = 0, c = 0;   // segments and tiles so far: they give the barriers' phases
      for (int it = it_first; it < it_end; ++it, ++n) {
        const Seg g = seg_at(it);
        auto stage = [&]() -> uint8_t* {
          const int s = c % kStages;
          if (c >= kStages) ptx::mbar_wait(&empty[s], (uint32_t)((c / kStages - 1) & 1), abort_flag);
          if (rank == 0) ptx::mbar_expect_tx(&full[s], 2 * L::stage_bytes);
          return ring + s * L::stage_bytes;
        };
        auto load_k = [&](int j) {
          uint8_t* dst = stage();
          const uint32_t bar = full0 + (uint32_t)(c % kStages) * 8;
          const int key = j * FB_N + rank * (FB_N / 2);
          for (int kb = 0; kb < 4; ++kb)
            ptx::tma_load_3d_pair(dst + kb * 8192, &tm_k, bar, kb * 64, p.k_head_inner ? g.kvh : key, p.k_head_inner ? key : g.kvh);
          ++c;
        };
        auto load_v = [&](int j) {
          uint8_t* dst = stage();
          const uint32_t bar = full0 + (uint32_t)(c % kStages) * 8;
          const int key = j * FB_N;
          for (int kb = 0; kb < 2; ++kb)
            ptx::tma_load_3d_pair(dst + kb * 16384, &tm_v, bar, rank * (FB_D / 2) + kb * 64, p.v_head_inner ? g.kvh : key,
                                  p.v_head_inner ? key : g.kvh);
          ++c;
        };
        if (n > 0) ptx::mbar_wait(q_free, (uint32_t)((n - 1) & 1), abort_flag);
        if (rank == 0) ptx::mbar_expect_tx(q_full, 2 * 4 * 16384);
        for (int kb = 0; kb < 4; ++kb)
          ptx::tma_load_3d_pair(q_s + kb * 16384, &tm_q, q_full0, kb * 64, p.q_head_inner ? g.head : g.m0,
                                p.q_head_inner ? g.m0 : g.head);
        load_k(g.lo);
        for (int j = g.lo; j < g.hi; ++j) {
          if (j + 1 < g.hi) load_k(j + 1);
          load_v(j);
        }
      }
    }
  } else if (warp == 8) {
    // ------------------------------------------------------------ S = Q K^T issuer (the even CTA's thread works for the pair)
    if (rank == 0 && lane == 0) {
      constexpr uint32_t fmt = BF16 ? ptx::kFmtBF16 : ptx::kFmtF16;
      const uint32_t idesc_s = ptx::idesc_f16(fmt, fmt, 2 * FB_M, FB_N, 0, 0);
      const uint64_t q_desc = ptx::smem_desc_sw128(ptx::smem_u32(q_s), 16, 1024);
      const uint64_t k_desc = ptx::smem_desc_sw128(ptx::smem_u32(ring), 16, 1024);
      int n = 0, r = 0, c0 = 0;   // segments, tiles and loads so far
      for (int it = it_first; it < it_end; ++it, ++n) {
        const Seg g = seg_at(it);
        ptx::mbar_wait(q_full, (uint32_t)(n & 1), abort_flag);
        for (int i = g.lo; i < g.hi; ++i, ++r) {
          const int x = i - g.lo, c = c0 + (x == 0 ? 0 : 2 * x - 1), st = c % kStages;   // (K and V alternate, a K ahead)
          ptx::mbar_wait(&full[st], (uint32_t)((c / kStages) & 1), abort_flag);
          // S goes over P of the tile before last
          if (r >= 2) ptx::mbar_wait(&pv_done[r & 1], (uint32_t)(((r >> 1) - 1) & 1), abort_flag);
          ptx::tc_fence_after_sync();
          const uint64_t kd = ptx::desc_advance(k_desc, st * L::stage_bytes);
          const uint32_t d = tmem_base + (uint32_t)((r & 1) * FB_N);
#pragma unroll
          for (int kb = 0; kb < 4; ++kb)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              ptx::mma_f16_ss_pair(d, ptx::desc_advance(q_desc, kb * 16384 + ks * 32),
                                   ptx::desc_advance(kd, kb * 8192 + ks * 32), idesc_s, (kb | ks) ? 1u : 0u);
          ptx::mbar_arrive(&qk_issued[r & 1]);
          ptx::mma_commit_pair(&s_ready[r & 1]);
          ptx::mma_commit_pair(&empty[st]);
        }
        c0 += 2 * (g.hi - g.lo);
      }
    }
  } else if (warp == 10) {
    // ------------------------------------------------------------ O += P V issuer (the same)
    if (rank == 0 && lane == 0) {
      constexpr uint32_t fmt = BF16 ? ptx::kFmtBF16 : ptx::kFmtF16;
      // V is read as it lies in memory ([key][feature]): as the B operand that is MN-major, 64-feature slabs of
      // [128 keys x 128 B] (16 KB apart = LBO), groups of 8 keys 1 KB apart (SBO), 16 keys per K step
      const uint32_t idesc_o = ptx::idesc_f16(fmt, fmt, 2 * FB_M, FB_D, 0, 1);
      const uint64_t v_desc = ptx::smem_desc_sw128(ptx::smem_u32(ring), 16384, 1024);
      int r = 0, c0 = 0;
      for (int it = it_first; it < it_end; ++it) {
        const Seg g = seg_at(it);
        for (int i = g.lo; i < g.hi; ++i, ++r) {
          const int x = i - g.lo, c = c0 + (i + 1 < g.hi ? 2 * x + 2 : 2 * x + 1), st = c % kStages;
          ptx::mbar_wait(&full[st], (uint32_t)((c / kStages) & 1), abort_flag);
          const uint64_t vd = ptx::desc_advance(v_desc, st * L::stage_bytes);
          // the next tile's S goes first: interleaved with this P V it would be late, and the softmax behind it
          if (i + 1 < g.hi) ptx::mbar_wait(&qk_issued[(r + 1) & 1], (uint32_t)(((r + 1) >> 1) & 1), abort_flag);
#pragma unroll
          for (int h = 0; h < 2; ++h) {   // 64 keys as soon as their P is there
            ptx::mbar_wait(&p_ready[2 * (r & 1) + h], (uint32_t)((r >> 1) & 1), abort_flag);
            ptx::tc_fence_after_sync();
#pragma unroll
            for (int ks = 4 * h; ks < 4 * h + 4; ++ks)
              ptx::mma_f16_ts_pair(tmem_o, tmem_base + (uint32_t)((r & 1) * FB_N + ks * 8), ptx::desc_advance(vd, ks * 2048),
                                   idesc_o, (i > g.lo || ks > 0) ? 1u : 0u);
          }
          ptx::mma_commit_pair(&pv_done[r & 1]);
          ptx::mma_commit_pair(&empty[st]);
        }
        c0 += 2 * (g.hi - g.lo);
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------ softmax + drain (warps 0-7)
    // Two groups of four warps take the tiles in turn, thread = query row (warp w reaches the TMEM lanes 32 (w % 4) ..):
    // while one group evaluates a tile's exponentials the other loads the next tile and finds its maxima.  The
    // reference maximum travels from tile to tile through shared memory, warp to warp.
    const int quad = warp & 3, grp = warp >> 2;
    const int row = quad * 32 + lane;   // 0..127
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t p_ready0 = ptx::cluster_map(ptx::smem_u32(p_ready + 2 * grp), 0);
    const int bar_mine = 1 + grp * 4 + quad, bar_other = 1 + (grp ^ 1) * 4 + quad;   // where this warp hears, and tells
    int r0 = 0, n_gates = 0;            // tiles of the segments before, gate loads so far
    for (int it = it_first; it < it_end; ++it) {
      const Seg g = seg_at(it);
      const int m0 = g.m0, head = g.head;
      const int qi = m0 + row;            // query row
      const bool cut = BINS && (g.lo > 0 || g.hi < g.nt);
      const bool gate_tile = p.tma_drain && p.gate && !cut, out_tile = p.tma_drain && !cut;
      float m_used = -INFINITY, l = 0.f;   // of this group's tiles
      for (int i = g.lo + ((r0 ^ grp) & 1); i < g.hi; i += 2) {
        const int r = r0 + i - g.lo;       // r & 1 == grp
        const bool first = i == g.lo, last = i == g.hi - 1;
        const uint32_t ph = (uint32_t)((r >> 1) & 1);
        const uint32_t sa = tmem_base + lane_off + (uint32_t)(grp * FB_N);
        float before = -INFINITY;
        if (!first) {   // the reference as the tile before has left it, which was known long before this tile's scores
          asm volatile("bar.sync %0, 64;" ::"r"(bar_mine) : "memory");
          before = rowmax_s[row];
        }
        ptx::mbar_wait(&s_ready[grp], ph, abort_flag);
        ptx::tc_fence_after_sync();
        // the last S has been computed, so nothing reads Q any more
        if (last && (tid & 127) == 0) {
          if (BINS && !out_tile) ptx::mbar_arrive(q_free);
          if (gate_tile) {
            // its buffer receives the gate tile ([128 rows x 256] as four 64-feature slabs, swizzled like an operand)
            // while the last tile is finished
            ptx::mbar_expect_tx(g_full, 4 * 16384);
            for (int kb = 0; kb < 4; ++kb)
              ptx::tma_load_3d(q_s + kb * 16384, &tm_g, g_full, kb * 64, p.g_head_inner ? head : m0,
                               p.g_head_inner ? m0 : head);
          }
        }
        __syncwarp();
        uint32_t sv[FB_N];
#pragma unroll
        for (int c = 0; c < FB_N; c += 32) ptx::tmem_ld32(sa + (uint32_t)c, sv + c);
        ptx::tmem_ld_wait();
        // sv keeps the raw dot products; the (positive) scale is applied once to the maximum here and inside the
        // exponent's fused multiply-add below
        const int key0 = i * FB_N;
        if (key0 + FB_N - 1 > m0 + past) {   // the tile reaches past the first row's diagonal
          const int seen = qi + past - key0;
#pragma unroll
          for (int c = 0; c < FB_N; ++c)
            if (c > seen) sv[c] = 0xff800000u;   // -inf
        }
        float tm4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // four independent chains, two for each half of the keys
#pragma unroll
        for (int c = 0; c < FB_N / 2; c += 4) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int k = (e >> 1) * (FB_N / 2) + c + 2 * (e & 1);
            tm4[e] = max3(tm4[e], __uint_as_float(sv[k]), __uint_as_float(sv[k + 1]));
          }
        }
        // Any value near the maximum will do as the reference; it is taken as if tiles were 64 keys long, their maxima
        // rounded up to bfloat16: the 16-bit roundings of P do not depend on how the tiles are cut, then.
        const float ta = bf16_up(fmaxf(tm4[0], tm4[1]) * p.scale_log2), tb = bf16_up(fmaxf(tm4[2], tm4[3]) * p.scale_log2);
        float m;
        if (first) {
          m = cut ? fmaxf(ta, kNoMax) : ta;      // an item's key 0 is visible to every row: finite unless cut
          if (tb > m + kGrow) m = tb;
          rowmax_s[row] = m;
          if (!last) asm volatile("bar.arrive %0, 64;" ::"r"(bar_other) : "memory");
        } else {
          m = ta > before + kGrow ? ta : before;
          if (tb > m + kGrow) m = tb;
          const bool grow = m != before;
          rowmax_s[row] = m;
          if (!last) asm volatile("bar.arrive %0, 64;" ::"r"(bar_other) : "memory");
          if (__any_sync(0xffffffffu, grow)) {
            // O belongs to the old reference; it is final for the tiles so far once the previous P V has finished
            ptx::mbar_wait(&pv_done[grp ^ 1], (uint32_t)(((r - 1) >> 1) & 1), abort_flag);
            ptx::tc_fence_after_sync();
            const float factor = grow ? exp2f(before - m) : 1.f;
#pragma unroll 1
            for (int c0 = 0; c0 < FB_D; c0 += 16) {
              uint32_t ov[16];
              ptx::tmem_ld16(tmem_o + lane_off + (uint32_t)c0, ov);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < 16; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * factor);
              ptx::tmem_st16(tmem_o + lane_off + (uint32_t)c0, ov);
            }
          }
        }
        if (m != m_used) {   // moved since this group's last tile
          l *= exp2f(m_used - m);
          m_used = m;
        }
        float2 psum = make_float2(0.f, 0.f);
        const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), nm2 = make_float2(-m, -m);
#pragma unroll
        for (int c = 0; c < FB_N; c += 32) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[c + 2 * e]), __uint_as_float(sv[c + 2 * e + 1])), sc2, nm2);
            const int i4 = e & 3;
            const bool on_fma = kPolyOf8 == 1 ? i4 == 0 : kPolyOf8 == 2 ? (i4 & 1) == 0 : kPolyOf8 == 3 ? i4 < 3 : kPolyOf8 >= 4;
            const float2 w = make_float2(fast_ex2(x.x), on_fma ? poly_ex2(x.y) : fast_ex2(x.y));
            psum = __fadd2_rn(psum, w);
            sv[c + e] = pack2<BF16>(w.x, w.y);
          }
          // P of keys c .. c + 31 over columns of S that have been read
          ptx::tmem_st16(sa + (uint32_t)(c >> 1), sv + c);
          if ((c & 32) != 0) {   // the first 64 keys may be multiplied while the others' exponentials are evaluated
            ptx::tmem_st_wait();
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive_cluster(p_ready0 + (uint32_t)(c >> 6) * 8);
          }
        }
        l += psum.x + psum.y;
      }
      const int r_last = r0 + g.hi - g.lo - 1;
      r0 += g.hi - g.lo;
      // epilogue: the row sum over both groups at the last reference, then each group writes 128 output features
      asm volatile("bar.sync 9, 256;" ::: "memory");   // the last tile's reference is there
      const float m_fin = rowmax_s[row];
      if (m_used != m_fin) l *= exp2f(m_used - m_fin);
      rowsum_s[grp * FB_M + row] = l;
      asm volatile("bar.sync 9, 256;" ::: "memory");
      l = rowsum_s[row] + rowsum_s[FB_M + row];
      const uint32_t oa = tmem_o + lane_off + (uint32_t)(grp * (FB_D / 2));
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      if (cut) {
        // partial: O as it stands, four features of the 128 rows side by side (a warp stores 512 bytes at a time)
        const int slot = part_slot(pair, g.lo > 0) * 2 + rank;
        float4* po = p.part_o + ((int64_t)slot * (FB_D / 4) + grp * (FB_D / 8)) * FB_M + row;
        ptx::mbar_wait(&pv_done[r_last & 1], (uint32_t)((r_last >> 1) & 1), abort_flag);
        ptx::tc_fence_after_sync();
#pragma unroll 1
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t ov[32];
          ptx::tmem_ld32(oa + (uint32_t)(cc * 32), ov);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4)
            po[(cc * 8 + c4) * FB_M] = make_float4(__uint_as_float(ov[4 * c4]), __uint_as_float(ov[4 * c4 + 1]),
                                                   __uint_as_float(ov[4 * c4 + 2]), __uint_as_float(ov[4 * c4 + 3]));
        }
        if (grp == 0) p.part_ml[(int64_t)slot * FB_M + row] = make_float2(m_fin == kNoMax ? -INFINITY : m_fin, l);
      } else if (out_tile) {
        // Drain through shared memory so that global memory sees whole tiles: the gate tile arrived by TMA in the Q
        // buffer; each thread turns the 16-byte chunks of its half row into output chunks in place; one TMA store
        // per slab writes the tile (rows past the end of the sequence are clipped by the tensor map).
        ptx::mbar_wait(&pv_done[r_last & 1], (uint32_t)((r_last >> 1) & 1), abort_flag);
        if (p.gate) ptx::mbar_wait(g_full, (uint32_t)(n_gates++ & 1), abort_flag);
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t ov[32];
          ptx::tmem_ld32(oa + (uint32_t)(cc * 32), ov);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int c8 = 0; c8 < 4; ++c8) {
            const int chunk = grp * 16 + cc * 4 + c8;   // 16-byte chunk of the 512-byte row
            uint4* cell = reinterpret_cast<uint4*>(q_s + (chunk >> 3) * 16384 + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
            uint32_t w[4];
            if (p.gate) {
              const uint4 gt = *cell;
              const uint32_t gw[4] = {gt.x, gt.y, gt.z, gt.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 gg = unpack2<BF16>(gw[i]);
                // sigmoid(g) = 0.5 + 0.5 * tanh(g / 2): one special-function result per element
                const float sga = fmaf(0.5f, fast_tanh(0.5f * gg.x), 0.5f), sgb = fmaf(0.5f, fast_tanh(0.5f * gg.y), 0.5f);
                w[i] = pack2<BF16>(__uint_as_float(ov[c8 * 8 + 2 * i]) * inv_l * sga,
                                   __uint_as_float(ov[c8 * 8 + 2 * i + 1]) * inv_l * sgb);
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
        asm volatile("bar.sync 9, 256;" ::: "memory");
        if (tid == 0) {
          if (m0 < p.S) {   // (the second query tile of a pair of rows may lie past the end)
            for (int kb = 0; kb < 4; ++kb)
              ptx::tma_store_3d(&tm_o, q_s + kb * 16384, kb * 64, p.o_head_inner ? head : m0, p.o_head_inner ? m0 : head);
            ptx::tma_store_commit();
            ptx::tma_store_wait_read();
          }
          if (BINS) ptx::mbar_arrive(q_free);
        }
      } else {
        // The gate values of this thread's half row (16 x 16 bytes) are requested first, all at once: they travel
        // while the last P V finishes (one load per use would put 16 round trips to L2 on the drain's critical path).
        const bool row_ok = qi < p.S;
        const uint16_t* gptr = (p.gate && row_ok) ? reinterpret_cast<const uint16_t*>(p.gate) + (int64_t)qi * p.g_ss +
                                                        (int64_t)head * p.g_sh + grp * (FB_D / 2)
                                                  : nullptr;
        uint4 gv[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) gv[i] = gptr ? __ldg(reinterpret_cast<const uint4*>(gptr) + i) : make_uint4(0, 0, 0, 0);
        ptx::mbar_wait(&pv_done[r_last & 1], (uint32_t)((r_last >> 1) & 1), abort_flag);
        ptx::tc_fence_after_sync();
        uint16_t* optr = reinterpret_cast<uint16_t*>(p.out) + (int64_t)qi * p.o_ss + (int64_t)head * p.o_sh + grp * (FB_D / 2);
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t ov[32];
          ptx::tmem_ld32(oa + (uint32_t)(cc * 32), ov);
          ptx::tmem_ld_wait();
          if (row_ok) {
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8) {
              const uint4 gt = gv[cc * 4 + c8];
              const uint32_t gw[4] = {gt.x, gt.y, gt.z, gt.w};
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
      }
      ptx::tc_fence_before_sync();
      if (BINS) asm volatile("bar.sync 9, 256;" ::: "memory");   // O, the references and the sums have been read
    }
  }

  __syncthreads();
  ptx::cluster_arrive();   // neither CTA leaves while the other may still arrive on its barriers or read its operands
  ptx::cluster_wait();
  if (warp == 0) ptx::tmem_dealloc_pair(tmem_base, 512);
  if (tid == 0 && *abort_flag && p.status) atomicExch(p.status, 1);
}

// Joins the partials of the items that a bin boundary cut, and finishes them as the drain above would (division by
// the sum, gate, rounding).  Block (bin - 1, 32 features, CTA of the item): the block of the bin in which an item's second
// piece lies does the item, the others leave.  Thread = (row, 16 features): the partials are read 512 bytes a warp, the output in
// whole 32-byte sectors.
template <bool BF16, bool SINGLE>
__global__ void __launch_bounds__(256) flash_merge_kernel(const __grid_constant__ FlashParams p) {
  constexpr int CTAS = SINGLE ? 1 : 2;
  const int bin = (int)blockIdx.x + 1, rank = (int)blockIdx.z;
  const uint32_t at = p.bin_start[bin], before = p.bin_start[bin - 1];
  const int it = (int)(at >> 16);
  if ((at & 0xFFFFu) == 0 || ((before >> 16) == (uint32_t)it && (before & 0xFFFFu) != 0)) return;
  int last = bin;   // bins bin .. last start inside the item
  while (last + 1 < p.n_bins && (int)(p.bin_start[last + 1] >> 16) == it) ++last;
  const int row = threadIdx.x & (FB_M - 1), f16 = (int)blockIdx.y * 2 + (threadIdx.x >> 7);
  int head, m0;
  if constexpr (SINGLE) {
    head = it % p.Hq;
    m0 = ((p.S + FB_M - 1) / FB_M - 1 - it / p.Hq) * FB_M;
  } else {
    flash_item_at(flash_items(p.S, p.Hq, p.pair_heads), it, p.pair_heads, rank, head, m0);
  }
  const int qi = m0 + row;
  if (qi >= p.S) return;
  float m = -INFINITY;
#pragma unroll 8
  for (int b = bin - 1; b <= last; ++b) m = fmaxf(m, __ldg(&p.part_ml[(int64_t)(part_slot(b, b >= bin) * CTAS + rank) * FB_M + row].x));
  float l = 0.f;
  float4 o[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) o[c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int b = bin - 1; b <= last; ++b) {   // in the order of the keys
    const int slot = part_slot(b, b >= bin) * CTAS + rank;
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

// How the items are dealt out.  Costs are in tiles (pairs: 128 keys, 1.3 to 1.6 us each on a B200; single CTAs: 64 keys, 0.9
// to 1.05 us): a segment costs its tiles and `seg` for its Q load, first scores and drain; cutting costs `cut` (partials
// out, merge launch, partials in), and the stretches must be kSaving percent shorter than the pair or CTA with the most whole
// items works.  That much, because tiles
// take longer when every SM streams K and V at once, and because a cut saves time and not energy: back to back, under
// the power cap, the SMs that idle behind whole items leave the others a higher clock.  Stretches of less than
// `share` are not worth SMs of their own.  Measured (16 query / 2 KV heads, bf16, gated; tokens over past, us, one
// pair per item against equal stretches, 5 / 600 in a row):
//   64 over 3,000 46.5 / 45.5 -> 29.3 / 28.7; 64 over 30,000 361 / 360 -> 68 / 64; 300 over 2,000 39.1 / 37.2 -> 31.9 / 30.7;
//   500 over 30,000 369 / 369 -> 204 / 217; 1,200 over 4,000 126 / 123 -> 104 / 97; 1,200 over 30,000 746 / 747 -> 484 / 540;
//   1,700 over 30,000 770 / 839 -> 678 / 767; 1,900 over 30,000 778 / 864 -> 730 / 825;
// below the line 2,048 over 30,720 803 / 908 -> 800 / 907; 3,000 over 8,000 382 / 413 -> 376 / 415; 5,000 over 8,000
//   685 / 752 -> 672 / 763; 1,728 over 4,000 141 / 135 -> 138 / 134; 704 over 2,000 46.9 / 44.5 -> 47.8 / 45.3; 1,024 over
//   12,000 176 / 173 -> 179 / 184; 700 over 1,365 39.5 / 36.9 -> 45.5 / 43.1; 1,000 over 1,000 37.5 / 36.0 -> 47.9 / 45.2;
//   3,000 over 0 88 / 83 -> 124 / 121.
// A cut changes the results in the last bits (P is rounded to 16 bits against each segment's own reference; the error
// against float64 stays the same, 2.31e-3 relative in bf16 on either side).  The partials take up to 39 MB (296 slots).
struct FlashCosts {
  int seg, cut, share;
};
constexpr FlashCosts kPairCosts = {2, 10, 6}, kSingleCosts = {4, 16, 12};
constexpr int kSaving = 15;

// Fills p.n_bins and p.bin_start for pairs (ctas = 2) or single CTAs (n_bins = 0: an item each) and returns the bytes of
// partials that the plan needs; *cost = how long it takes, in tiles.
static int64_t flash_plan(FlashParams& p, int ctas, int sms, bool may_cut, int64_t* cost) {
  p.n_bins = 0;
  const FlashCosts c = ctas == 1 ? kSingleCosts : kPairCosts;
  int workers = sms / ctas;
  if (workers > kMaxBins) workers = kMaxBins;
  if (workers < 1) workers = 1;
  const FlashItems f = ctas == 1 ? FlashItems{(p.S + FB_M - 1) / FB_M, p.Hq} : flash_items(p.S, p.Hq, p.pair_heads);
  const int64_t items = (int64_t)f.n_qt * f.per_qt;
  auto tiles = [&](int qt) {
    return ctas == 1 ? flash_tiles<64>(qt, FB_M, p.S, p.Skv) : flash_tiles<FB_N>(qt, p.pair_heads ? FB_M : 2 * FB_M, p.S, p.Skv);
  };
  int64_t total = 0;
  for (int qt = 0; qt < f.n_qt; ++qt) total += (int64_t)(tiles(qt) + c.seg) * f.per_qt;
  *cost = total / workers;
  if (items > 8 * workers) return 0;   // more than eight rounds of items even out by themselves
  // One pair or CTA per item: the hardware hands the next item to the SMs that are done first.  Dealt back and forth over
  // the workers, longest first, that ends with the largest of these sums.
  int load[kMaxBins] = {0}, longest = 0, k = 0, step = 1;
  for (int qt = f.n_qt - 1; qt >= 0; --qt) {
    const int x = tiles(qt) + c.seg;
    for (int h = 0; h < f.per_qt; ++h) {
      load[k] += x;
      if (load[k] > longest) longest = load[k];
      k += step;
      if (k == workers || k < 0) {
        step = -step;
        k += step;
      }
    }
  }
  *cost = longest;
  const int bins = (int)(total / c.share < workers ? total / c.share : workers);
  // (bin_start holds 16 bits of tile)
  if (!may_cut || sms < ctas || tiles(f.n_qt - 1) > 0xFFFF || bins < 2 ||
      100 * (int64_t)longest <= (100 + kSaving) * (total / bins) + 100 * c.cut)
    return 0;
  // Equal stretches of the items' costs.  A piece of fewer than `seg` tiles is not worth a segment: the boundary
  // moves to the item's edge.
  uint32_t* start = p.bin_start;
  int n = 0, qt = f.n_qt - 1, h = 0, nt = tiles(qt);
  int64_t c0 = 0;     // where item (qt, h) starts
  uint32_t item = 0;
  start[n++] = 0;
  for (int b = 1; b < bins; ++b) {
    const int64_t x = total * b / bins;
    while (x >= c0 + nt + c.seg) {
      c0 += nt + c.seg;
      ++item;
      if (++h == f.per_qt) {
        h = 0;
        nt = tiles(--qt);
      }
    }
    const int64_t j = x - c0 - c.seg / 2;
    const uint32_t at = j < c.seg ? item << 16 : j > nt - c.seg ? (item + 1) << 16 : item << 16 | (uint32_t)j;
    if (at > start[n - 1] && at < (uint32_t)items << 16) start[n++] = at;
  }
  start[n] = (uint32_t)items << 16;
  p.n_bins = n;
  *cost = total / bins + c.cut;
  return (int64_t)2 * ctas * n * FB_M * (FB_D * 4 + 8);
}

// Pairs of CTAs or single ones?  Two heads of one KV head share a pair; heads that cannot be paired so give it 256 rows at a
// time, half of them empty in a sequence of up to 128.  By the two plans' times: 0.95 us per cost of a single CTA against 1.45 us
// per cost of a pair and 2 us for its later start.  Over 356 shapes, 1/1 to 128/128 heads, 2 to 2,048 tokens over a past of 0 to
// 30,000, that choice is 0.3 % behind the better of the two on average, and 1.17 times where 64 heads of keys and values bound
// both (128 tokens over 4,000).  us, single against pairs: 16/2 heads, 2 tokens 8.2, 9.8, 128 tokens 10.0, 10.4,
// 300 tokens 12.1, 12.9, 200 over 500 17.6, 17.2, 700 over 1,000 32.8, 29.6; 96/96 heads, 64 tokens 8.9, 19.8, 2,048 tokens 325,
// 253; 48/16 heads, 300 over 1,000 28.3, 47.6, 1,000 over 1,000 93.4, 85.6.  Heads that pair up and more than 512 tokens were
// never better off on single CTAs.
// Fills p as flash_plan does; *ctas = what the choice is.
static int64_t flash_choose(FlashParams& p, bool may_cut, int* ctas) {
  p.pair_heads = (p.Hq / p.Hkv) % 2 == 0 ? 1 : 0;
  const int sms = sm_count();
  int64_t pair_cost, single_cost;
  const int64_t pair_bytes = flash_plan(p, 2, sms, may_cut, &pair_cost);
  *ctas = 2;
  if (p.pair_heads && p.S > 4 * FB_M) return pair_bytes;
  FlashParams single = p;
  const int64_t single_bytes = flash_plan(single, 1, sms, may_cut, &single_cost);
  if (95 * single_cost >= 145 * pair_cost + 200) return pair_bytes;
  p = single;
  *ctas = 1;
  return single_bytes;
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
  p.S = a->S; p.Skv = a->Skv; p.Hq = a->Hq; p.Hkv = a->Hkv;
  int ctas;
  return flash_choose(p, true, &ctas);
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
  FlashParams p{};
  p.S = a->S; p.Skv = a->Skv; p.Hq = a->Hq; p.Hkv = a->Hkv;
  // the partials of cut items need the workspace; without it every item is one pair's, or one CTA's
  const bool ws_ok = a->workspace && (reinterpret_cast<uintptr_t>(a->workspace) & 15) == 0;
  int ctas;
  const int64_t need = flash_choose(p, ws_ok, &ctas);
  if (need > 0 && a->workspace_bytes < need) (void)flash_choose(p, false, &ctas);
  // a CTA's share of a K and a V tile
  const uint32_t k_box = ctas == 1 ? 64u : (uint32_t)FB_N / 2, v_box = ctas == 1 ? 64u : (uint32_t)FB_N;
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
    uint32_t box[3] = {64, k_hin ? 1u : k_box, k_hin ? k_box : 1u};
    rc = make_tensor_map(&tk, dt, 3, a->k, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != MXB_OK) return rc;
  }
  const bool v_hin = a->v_stride_h < a->v_stride_s;
  {
    uint64_t dims[3] = {(uint64_t)a->D, (uint64_t)(v_hin ? a->Hkv : a->Skv), (uint64_t)(v_hin ? a->Skv : a->Hkv)};
    uint64_t str[2] = {(uint64_t)(v_hin ? a->v_stride_h : a->v_stride_s) * 2,
                       (uint64_t)(v_hin ? a->v_stride_s : a->v_stride_h) * 2};
    uint32_t box[3] = {64, v_hin ? 1u : v_box, v_hin ? v_box : 1u};
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
  p.g_head_inner = g_hin ? 1 : 0; p.o_head_inner = o_hin ? 1 : 0; p.tma_drain = tma_drain ? 1 : 0;
  p.v_head_inner = v_hin ? 1 : 0;
  p.gate = a->gate; p.g_ss = a->gate_stride_s; p.g_sh = a->gate_stride_h;
  p.out = a->out; p.o_ss = a->out_stride_s; p.o_sh = a->out_stride_h;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.status = a->status;
  p.q_head_inner = q_hin ? 1 : 0;
  p.k_head_inner = k_hin ? 1 : 0;
  p.part_o = reinterpret_cast<float4*>(a->workspace);
  p.part_ml = reinterpret_cast<float2*>(p.part_o + (int64_t)2 * ctas * p.n_bins * (FB_D / 4) * FB_M);
  const FlashItems items = flash_items(p.S, p.Hq, p.pair_heads);
  const int64_t whole = ctas == 1 ? ceil_div((int64_t)p.S, (int64_t)FB_M) * p.Hq : (int64_t)items.n_qt * items.per_qt;
  const unsigned grid = (unsigned)(ctas * (p.n_bins > 0 ? p.n_bins : whole));
  const bool bf16 = a->dtype == MXB_BF16;
  if (ctas == 1) {
    rc = launch_flash_single(tq, tk, tv, tg, to, p, bf16, grid, st);
    if (rc != MXB_OK) return rc;
  } else {
    constexpr int smem = FlashSmem::total + 1024;
    auto* kernel = bf16 ? (p.n_bins > 0 ? flash_prefill_kernel<true, true> : flash_prefill_kernel<true, false>)
                        : (p.n_bins > 0 ? flash_prefill_kernel<false, true> : flash_prefill_kernel<false, false>);
    MXB_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kernel<<<grid, 384, smem, st>>>(tq, tk, tv, tg, to, p);
    note_launch();
  }
  if (p.n_bins > 1) {
    auto* merge = ctas == 1 ? (bf16 ? flash_merge_kernel<true, true> : flash_merge_kernel<false, true>)
                            : (bf16 ? flash_merge_kernel<true, false> : flash_merge_kernel<false, false>);
    merge<<<dim3((unsigned)(p.n_bins - 1), FB_D / 32, (unsigned)ctas), 256, 0, st>>>(p);
    note_launch();
  }
  MXB_CUDA_OK(cudaGetLastError());
  return MXB_OK;
}
