// The flash prefill (flash_prefill.cu) with one CTA per item instead of a pair: 128 query rows of one query head over
// 64-key tiles.  A tile takes 1,750 to 1,890 cycles here, bound by shared memory (operands 6 KB per MMA of 32 tensor cycles,
// arrivals, P in and out), where a pair takes 2,680 for two of them; but an item needs one SM, starts 1.5 us earlier and has
// no second CTA to leave empty.  So it is the better one for sequences of a tile or two, and where the query heads do not
// pair up and half of a pair's rows, or of a second wave of pairs, would be empty; flash_choose (flash_prefill.cu) says
// where, with both sides measured.
//
// Items are dealt out in the same two ways: one CTA per item, or one CTA per SM with an equal stretch of the concatenated
// tiles of all items, whose cut items flash_merge_kernel joins.
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
#include "flash_common.cuh"

namespace mxb {

constexpr int SB_N = 64;

struct SingleSmem {
  static constexpr int q_off = 0;                       // 4 slabs x [128 x 128 B]
  static constexpr int k_off = q_off + 4 * 16384;       // 2 stages x 4 slabs x [64 x 128 B]
  static constexpr int v_off = k_off + 2 * 32768;       // 2 stages x 4 slabs x [64 keys x 128 B]
  static constexpr int p_off = v_off + 2 * 32768;       // 2 buffers x [128 x 128 B]
  static constexpr int bar_off = p_off + 2 * 16384;
  static constexpr int rowmax_off = bar_off + 256;      // [2 tiles][2 halves][128 rows] bf16 (1 KB); reused for the row sums
  static constexpr int total = rowmax_off + 1024;
};

template <bool BF16, bool BINS>
__global__ void __launch_bounds__(384, 1) flash_single_kernel(const __grid_constant__ CUtensorMap tm_q,
                                                               const __grid_constant__ CUtensorMap tm_k,
                                                               const __grid_constant__ CUtensorMap tm_vt,
                                                               const __grid_constant__ CUtensorMap tm_g,
                                                               const __grid_constant__ CUtensorMap tm_o,
                                                               const __grid_constant__ FlashParams p) {
  using L = SingleSmem;
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
    g.nt = flash_tiles<SB_N>(qt, FB_M, p.S, p.Skv);
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
            ptx::tma_load_3d(k_s + s * 32768 + kb * 8192, &tm_k, &k_full[s], kb * 64, p.k_head_inner ? g.kvh : j * SB_N,
                             p.k_head_inner ? j * SB_N : g.kvh);
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
      const uint32_t idesc_s = ptx::idesc_f16(fmt, fmt, FB_M, SB_N, 0, 0);
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
          const uint32_t d = tmem_base + (uint32_t)(s * 2 * SB_N + half * SB_N);
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
          ptx::tma_load_3d(v_s + s * 32768 + kb * 8192, &tm_vt, &v_full[s], kb * 64, p.v_head_inner ? vg.kvh : vj * SB_N,
                           p.v_head_inner ? vj * SB_N : vg.kvh);
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
          const uint32_t sa = tmem_base + lane_off + (uint32_t)(s * 2 * SB_N + half * 32);
          ptx::tmem_ld32(sa, sv);
          ptx::tmem_ld32(sa + SB_N, sb);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 32; ++c) sv[c] = __float_as_uint(__uint_as_float(sv[c]) + __uint_as_float(sb[c]));
        }
        ptx::tc_fence_before_sync();
        ptx::mbar_arrive(&s_free[s]);
        const int key0 = i * SB_N + half * 32;
        const bool need_mask = i * SB_N + SB_N - 1 > m0 + past;  // tile reaches past the first row's diagonal
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
          grow = tmax > m_used + kGrow;
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

int launch_flash_single(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tg,
                        const CUtensorMap& to, const FlashParams& p, bool bf16, unsigned ctas, cudaStream_t st) {
  constexpr int smem = SingleSmem::total + 1024;
  auto* kernel = bf16 ? (p.n_bins > 0 ? flash_single_kernel<true, true> : flash_single_kernel<true, false>)
                      : (p.n_bins > 0 ? flash_single_kernel<false, true> : flash_single_kernel<false, false>);
  MXB_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  kernel<<<ctas, 384, smem, st>>>(tq, tk, tv, tg, to, p);
  note_launch();
  MXB_CUDA_OK(cudaGetLastError());
  return MXB_OK;
}

}  // namespace mxb
