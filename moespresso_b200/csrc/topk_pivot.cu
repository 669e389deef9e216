// Exact top-k of fp32 score rows of up to 2^21 scores: rows of up to 16,384 scores in registers, longer ones through a
// sampled pivot that lets one pass over the row throw nearly all of it away.
//
// topk_direct_kernel (rows of at most kDirectMax scores): one CTA, up to 16 keys per thread in registers.  One histogram
// of 2,048 equal bins over the row's range without outliers and a direct ranking of what is left in the threshold bin;
// rows that this does not resolve go by the key's bits (11 + 11 + 10).  Bins of values and not of key bits, because
// ordinary scores have some twenty values of the top 11 bits: the atomics of a warp then meet in a few words, and the
// threshold bin always needs a second level.
//
// topk_pivot_kernel (longer rows):
//   1. a strided sample of the row (4,096 to 32,768 scores, a histogram of the keys below its largest) gives a
//      pivot that about 1.1 to 2 k of the row's keys reach: the sample rank of k plus five standard deviations;
//   2. one streaming pass compares every score with the pivot (as floats, a vote per 32 scores) and leaves a bitmap,
//      which is expanded into the list of candidate positions in ascending order; their keys are fetched again;
//   3. the threshold is the k-th largest key of the list: one 2,048-bin histogram over [pivot, largest key], whose
//      threshold bin holds a handful of keys that are ranked against each other directly.
//   Ties: if more keys than the list holds would reach the pivot and the sampled ones in its bin are one score, the pass
//   leaves two bitmaps, larger and equal.  Either the threshold is that score and the bitmaps are emitted as they are, or
//   it lies above and the larger ones are the candidates.
//   The sample only steers: if fewer than k keys reach the pivot, or more than the list holds after all (rows whose
//   large scores hide between the sampled positions), the CTAs fall back to an 11 + 11 + 10-bit radix select that
//   streams the row (592 rows of 32,768: 116 us; a row of 131,072: 46).
//   A row belongs to one CTA or to a thread-block cluster, each CTA with a contiguous part of it.  The CTAs of a
//   cluster read the same sample (same pivot, nothing exchanged); after one cluster barrier every CTA copies all
//   lists' keys (12 KB through distributed shared memory) and finds the threshold for itself, so the second barrier
//   only keeps the lists alive until the last reader is done.
//
// Both emit in order: votes on (key > threshold) and (key == threshold) over the keys in ascending position, prefix
// counts of the votes' words, and a selected id's slot is (above before it) + min(equal before it, need): ids ascend
// and ties go to the lowest id without a sort.
//
// Bound: few rows, the chain of barriers and L2 round trips; many rows, instruction issue (6 warp instructions per 32
// scores of the pass, three times as much for sample, list and threshold) and barriers.  Against the radix select over
// whole rows before it, which spent a shared-memory atomic per score and digit: 592 rows of 32,768 scores, k = 2,048:
// 77 -> 33 us; 32 rows of 131,072: 20.1 -> 14.6; one row of 1,048,576: 63 -> 18.3; one of 2,500, k = 512: 7.8 -> 5.6
// (key bits) -> 4.2 (bins of values, 1,024 threads); 4,096: 6.0 -> 4.4; 333 of 5,003: 13.7 -> 11.9; 1,184 of 8,192: 37.5 -> 34.1.
// Scores rounded to integers (ties at the threshold), radix select / fallback alone / with the two bitmaps: 592 rows of
// 32,768 79 / 116 / 43 us, 160 of 16,384 32 / 38 / 15, 32 of 131,072 21.5 / 44 / 12, one of 131,072 16 / 46 / 9.5; one row
// of 1,048,576 equal scores 2,584 / 98 / 20.5.
#include <cooperative_groups.h>
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "ptx_sm100.cuh"
#include "topk_common.cuh"

namespace cg = cooperative_groups;

namespace mxb {

constexpr int kDirectKeys = 16;          // keys per thread of the direct kernel
constexpr int kDirectMax = 1024 * kDirectKeys;
constexpr int kPSmall = 64;              // keys of the threshold bin that are ranked directly
constexpr int kPPartMax = 131072;        // scores per CTA (two bitmaps of 16 KB)
constexpr int kPMaxCluster = 16;
constexpr int kPListMax = 14336;         // list entries: three arrays of 56 KB beside the bitmaps and histograms
constexpr float kMaxScore = 3.402823466e38f;   // larger ones, infinities and NaN are never selected

struct TopkPivotParams {
  const float* scores;
  int64_t row_stride;
  const int64_t* row_start;
  const int32_t* row_count;
  int32_t* out_ids;
  int64_t n;
  int32_t k;
  int32_t cap;          // list entries, a multiple of 32
  int32_t part;         // scores per CTA of the longest row, a multiple of 1,024
};

__device__ __forceinline__ float key_float(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? key ^ 0x80000000u : ~key);
}

// The row of this CTA or cluster: its length and first score.
__device__ __forceinline__ const float* row_scores(const TopkPivotParams& p, int row, int64_t* n) {
  int64_t c = p.row_count ? (int64_t)p.row_count[row] : p.n;
  *n = c < 0 ? 0 : (c > p.n ? p.n : c);
  return p.scores + (p.row_start ? p.row_start[row] : (int64_t)row * p.row_stride);
}

// Shared scalars of the threshold search.
struct TopkShared {
  uint32_t sums[2][32];   // of consecutive scans, in turn
  uint32_t thr[4], small_n, T, need, largest, smallest;
  uint32_t small_keys[kPSmall];
};

// Exclusive scan of one value per thread with a single barrier: every warp adds up the warps before it for itself.
// `sums` [NT / 32] must not be in use by a scan that another warp may still be reading.
template <int NT>
__device__ __forceinline__ uint32_t scan_threads(uint32_t v, uint32_t* sums, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  const uint32_t w = lane < NT / 32 ? sums[lane] : 0u;
  *total = __reduce_add_sync(0xffffffffu, w);
  return __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u) + incl - v;
}

// The bin of a 2,048-bin histogram, counted from the top, where the running count reaches min(k, total).
// out: {that minimum, bin, count above the bin, count of the bin}; the last three are set if the minimum is not 0.
template <int NT>
__device__ __forceinline__ void threshold_bin(const uint32_t* hist, uint32_t k, uint32_t* sums, uint32_t* out) {
  constexpr int PER = kBigBins / NT;
  const int top = kBigBins - 1 - (int)threadIdx.x * PER;
  uint32_t loc[PER], c = 0, all;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    loc[j] = hist[top - j];
    c += loc[j];
  }
  uint32_t run = scan_threads<NT>(c, sums, &all);
  const uint32_t ke = min(k, all);
  if (threadIdx.x == 0) out[0] = ke;
  if (run < ke && run + c >= ke) {
    bool found = false;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (!found && run + loc[j] >= ke) {
        out[1] = (uint32_t)(top - j);
        out[2] = run;
        out[3] = loc[j];
        found = true;
      }
      run += loc[j];
    }
  }
  __syncthreads();
}

// Ranks the `cnt` <= kPSmall keys in small_keys against each other: the want-th largest is the threshold.
__device__ __forceinline__ void rank_small(TopkShared* s, uint32_t cnt, uint32_t want) {
  const int tid = threadIdx.x;
  if (tid < (int)cnt) {
    const uint32_t mine = s->small_keys[tid];
    uint32_t g = 0, e = 0;
    for (uint32_t j = 0; j < cnt; ++j) {
      const uint32_t o = s->small_keys[j];
      g += o > mine;
      e += o == mine;
    }
    if (g < want && want <= g + e) {   // equal keys agree on both values
      s->T = mine;
      s->need = want - g;
    }
  }
}

// --------------------------------------------------------------------------
// rows of at most 16 keys per thread
// --------------------------------------------------------------------------
template <int NT, int KEYS, int CTAS>
__global__ void __launch_bounds__(NT, CTAS) topk_direct_kernel(TopkPivotParams p) {
  constexpr int kWords = NT / 32 * KEYS;
  // rows of more than 8,192 scores go by the key's bits: 2,048 bins of values hold too many of their keys to pay
  constexpr bool kValueBins = NT * KEYS <= 8192;
  __shared__ uint32_t hist_a[kBigBins], hist_b[kBigBins];
  __shared__ uint32_t w_gt[kWords], w_eq[kWords], w_at[kWords];
  __shared__ uint32_t w_max[32], w_min[32];
  __shared__ TopkShared s;
  ptx::grid_chain();   // (the attention may set up on idle SMs; it waits for this grid before it reads ids)
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int64_t n64;
  const float* src = ptx::behind_wait(row_scores(p, row, &n64));
  const int n = (int)n64;
  int32_t* out = p.out_ids + (int64_t)row * p.k;

  uint32_t key[KEYS];
#pragma unroll
  for (int u = 0; u < KEYS; ++u) {
    key[u] = 0xFF800000u;   // -inf
    if (u * NT + tid < n) key[u] = __float_as_uint(__ldg(src + u * NT + tid));
  }
  if constexpr (kValueBins)
    for (int i = tid; i < kBigBins; i += NT) hist_a[i] = 0;
  if (tid == 0) {
    s.small_n = s.largest = 0;
    s.smallest = 0xffffffffu;
    s.thr[0] = s.thr[1] = s.thr[2] = s.thr[3] = 0;
  }
  uint32_t top = 0, low = 0xffffffffu;
#pragma unroll
  for (int u = 0; u < KEYS; ++u) {
    key[u] = score_key_full(__uint_as_float(key[u]));
    top = max(top, key[u]);
    if (key[u]) low = min(low, key[u]);
  }
  if constexpr (kValueBins) {
    top = __reduce_max_sync(0xffffffffu, top);
    low = __reduce_min_sync(0xffffffffu, low);
    if (lane == 0) {
      w_max[warp] = top;
      w_min[warp] = low;
    }
    __syncthreads();
  }
  // ---- 2,048 equal bins over the range of the row without its outliers: from the second smallest of the warps' smallest
  // scores to the second largest of their largest, what lies beyond goes to the outer bins (subtraction, product and
  // clamps are monotone, so bins are in the order of the keys).  The threshold bin holds a few keys of an ordinary row.
  uint32_t hi = 0, lo = 0;
  if constexpr (kValueBins) {
    top = lane < NT / 32 ? w_max[lane] : 0u;
    low = lane < NT / 32 ? w_min[lane] : 0xffffffffu;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t h = __reduce_max_sync(0xffffffffu, top), l = __reduce_min_sync(0xffffffffu, low);
      if (h) hi = h;
      if (l != 0xffffffffu) lo = l;
      if (top == h) top = 0;
      if (low == l) low = 0xffffffffu;
    }
  }
  const float x_lo = key_float(lo), scale = 2048.f / (key_float(hi) - x_lo);
  const bool spread = kValueBins && hi > lo && lo != 0 && scale > 0.f && scale <= kMaxScore;   // not without a range that float can hold
  auto bin_of = [&](uint32_t k) { return (int)fminf(fmaxf((key_float(k) - x_lo) * scale, 0.f), (float)(kBigBins - 1)); };
  // Do all keys that `in` picks have one value (ties)?  Then that is the threshold.
  auto one_value = [&](auto in, uint32_t need_of) -> bool {
    uint32_t least = 0xffffffffu, most = 0;
#pragma unroll
    for (int u = 0; u < KEYS; ++u) {
      if (in(key[u])) {
        least = min(least, key[u]);
        most = max(most, key[u]);
      }
    }
    least = __reduce_min_sync(0xffffffffu, least);
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0 && most) {
      atomicMin(&s.smallest, least);
      atomicMax(&s.largest, most);
    }
    __syncthreads();
    const bool one = s.smallest == s.largest;
    if (one && tid == 0) {
      s.T = s.largest;
      s.need = need_of;
    }
    return one;
  };
  uint32_t k_eff, want;
  bool found = false;
  // Scores that crowd into few bins (a long tail, a handful of values) find their threshold's bin too full and go by the
  // key's bits after all.  Seen from a score per thread, when one in 16 shares the bin of its warp's first: of scores that
  // spread evenly 1 in 32 does, the first itself.  Without the look such rows took up to 1.5 times as long as by the bits
  // alone: exp(4 x), k = 512, us by the bits, without the look, with it: 333 rows of 4,096 8.9, 12.3, 9.3; 148 of 8,192 7.2, 8.9,
  // 7.0.  Normal scores pay 0.1 us for it.  (A threshold among tens of keys of one bin that is not seen so still costs that
  // much: the median of exp(1.5 x).  Its bin in 2,048 bins of its own took as long as the bits.)
  const int first = bin_of(key[0]), of_warp = __shfl_sync(0xffffffffu, first, 0);
  const bool crowded = kValueBins && __syncthreads_count(key[0] && first == of_warp) * 16 > min(n, NT);
  if (spread && !crowded) {
#pragma unroll
    for (int u = 0; u < KEYS; ++u)
      if (key[u]) atomicAdd(&hist_a[bin_of(key[u])], 1u);
    __syncthreads();
    threshold_bin<NT>(hist_a, (uint32_t)p.k, s.sums[0], s.thr);
    const int bin = (int)s.thr[1];
    const uint32_t cnt = s.thr[3];
    k_eff = s.thr[0];
    want = k_eff - s.thr[2];
    if (cnt <= (uint32_t)kPSmall) {
#pragma unroll
      for (int u = 0; u < KEYS; ++u)
        if (key[u] && bin_of(key[u]) == bin) s.small_keys[atomicAdd(&s.small_n, 1u)] = key[u];
      __syncthreads();
      rank_small(&s, cnt, want);
      found = true;
    } else {
      found = one_value([&](uint32_t k) { return k && bin_of(k) == bin; }, want);
    }
  }
  if (!found) {
    // ---- rows whose scores crowd into one bin, long ones, one value only: 11 + 11 + 10 key bits
    if constexpr (kValueBins) __syncthreads();   // (the counters below have been read)
    for (int i = tid; i < kBigBins; i += NT) hist_a[i] = hist_b[i] = 0;
    if (tid == 0) {
      s.small_n = s.largest = s.thr[0] = s.thr[1] = s.thr[2] = s.thr[3] = 0;
      s.smallest = 0xffffffffu;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < KEYS; ++u)
      if (key[u]) atomicAdd(&hist_a[key[u] >> 21], 1u);
    __syncthreads();
    threshold_bin<NT>(hist_a, (uint32_t)p.k, s.sums[0], s.thr);
    const uint32_t bin = s.thr[1];
    k_eff = s.thr[0];
    want = k_eff - s.thr[2];
    if (k_eff == 0) {   // no finite score
      for (int i = tid; i < p.k; i += NT) out[i] = -1;
      return;
    }
#pragma unroll
    for (int u = 0; u < KEYS; ++u)
      if ((key[u] >> 21) == bin && key[u]) atomicAdd(&hist_b[(key[u] >> 10) & 2047u], 1u);
    __syncthreads();
    for (int i = tid; i < 1024; i += NT) hist_a[i] = 0;   // read for the last time before the barrier
    threshold_bin<NT>(hist_b, want, s.sums[1], s.thr);
    const uint32_t head = (bin << 11) | s.thr[1], cnt = s.thr[3];   // the top 22 bits of the threshold
    want -= s.thr[2];
    if (cnt <= (uint32_t)kPSmall) {
#pragma unroll
      for (int u = 0; u < KEYS; ++u)
        if ((key[u] >> 10) == head && key[u]) s.small_keys[atomicAdd(&s.small_n, 1u)] = key[u];
      __syncthreads();
      rank_small(&s, cnt, want);
    } else if (!one_value([&](uint32_t k) { return k && (k >> 10) == head; }, want)) {
#pragma unroll
      for (int u = 0; u < KEYS; ++u)
        if ((key[u] >> 10) == head && key[u]) atomicAdd(&hist_a[key[u] & 1023u], 1u);
      for (int i = 1024 + tid; i < kBigBins; i += NT) hist_a[i] = 0;
      __syncthreads();
      threshold_bin<NT>(hist_a, want, s.sums[0], s.thr);
      if (tid == 0) {
        s.T = (head << 10) | s.thr[1];
        s.need = want - s.thr[2];
      }
    }
  }
  for (int i = tid + (int)k_eff; i < p.k; i += NT) out[i] = -1;
  __syncthreads();
  const uint32_t thr = s.T, need = s.need;

  // ---- ordered emission: word u * (NT / 32) + warp votes on positions u * NT + 32 * warp + (0 .. 31)
#pragma unroll
  for (int u = 0; u < KEYS; ++u) {
    const uint32_t gt = __ballot_sync(0xffffffffu, key[u] > thr), eq = __ballot_sync(0xffffffffu, key[u] == thr);
    if (lane == 0) {
      w_gt[u * (NT / 32) + warp] = gt;
      w_eq[u * (NT / 32) + warp] = eq;
    }
  }
  __syncthreads();
  {
    uint32_t c = 0;   // low half: above, high half: equal (a row has fewer than 2^16 keys)
    if (tid < kWords) c = (uint32_t)__popc(w_gt[tid]) | ((uint32_t)__popc(w_eq[tid]) << 16);
    uint32_t all;
    const uint32_t at = scan_threads<NT>(c, s.sums[1], &all);
    if (tid < kWords) w_at[tid] = at;
  }
  __syncthreads();
  const uint32_t below = (1u << lane) - 1u;
#pragma unroll
  for (int u = 0; u < KEYS; ++u) {
    if (key[u] >= thr) {   // thr > 0
      const int w = u * (NT / 32) + warp;
      const uint32_t g = (w_at[w] & 0xffffu) + __popc(w_gt[w] & below), q = (w_at[w] >> 16) + __popc(w_eq[w] & below);
      if (key[u] > thr || q < need) out[g + min(q, need)] = u * NT + tid;
    }
  }
}

// --------------------------------------------------------------------------
// longer rows
// --------------------------------------------------------------------------
// CLUSTER: several CTAs per row.  NT threads: 1,024 for a cluster's CTAs, which have an SM each, 512 (three CTAs per SM)
// for many rows.  SAMPLES: float4 groups of the sample per thread.
template <bool CLUSTER, int NT, int SAMPLES>
__global__ void __launch_bounds__(NT, NT == 512 ? 3 : 1) topk_pivot_kernel(TopkPivotParams p) {
  extern __shared__ uint32_t dyn[];
  __shared__ TopkShared s;
  __shared__ uint32_t s_sum[2], s_top, s_tie[2];
  __shared__ uint32_t cl_count[kPMaxCluster], cl_gt[kPMaxCluster], cl_eq[kPMaxCluster];

  ptx::grid_chain();   // as above
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = CLUSTER ? (int)cluster.num_blocks() : 1;
  const int rank = CLUSTER ? (int)cluster.block_rank() : 0;
  const int row = CLUSTER ? (int)(blockIdx.x / (unsigned)cs) : (int)blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  uint32_t* hist_a = dyn;                        // [kBigBins]
  uint32_t* hist_b = hist_a + kBigBins;          // [kBigBins]
  uint32_t* lpos = hist_b + kBigBins;            // [cap] this CTA's candidates: positions within the part, ascending
  uint32_t* lkey = lpos + p.cap;                 // [cap] their keys
  uint32_t* keys = CLUSTER ? lkey + p.cap : lkey;   // [cap] the keys of all candidates of the row
  const int max_words = p.part / 32;
  uint32_t* bm_gt = (CLUSTER ? keys : lkey) + p.cap;   // [max_words]; the pass's bitmap
  uint32_t* bm_eq = bm_gt + max_words;                  // [max_words]; with a tie, and in the fallback
  uint32_t* w_gt = hist_a;                       // [cap / 32] each, once the threshold is known
  uint32_t* w_eq = hist_a + 512;
  uint32_t* w_at = hist_b;

  int64_t n;
  const float* src = ptx::behind_wait(row_scores(p, row, &n));
  // this CTA's scores: equal parts of the row's own length, which may be far below the longest of a ragged batch
  const int64_t share = cs > 1 ? round_up(ceil_div(n, (int64_t)cs), (int64_t)1024) : (int64_t)p.part;
  const int64_t lo = min((int64_t)rank * share, n);
  const int len = (int)min(share, n - lo);
  const int words = (int)round_up(len, 1024) / 32;
  int32_t* out = p.out_ids + (int64_t)row * p.k;
  if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

  // ---- sample: a pivot that a little more than k keys reach.  Whole 16-byte groups of the row, evenly spaced; the
  // loads are on their way while the histograms are cleared.
  constexpr uint32_t kTotal = SAMPLES * NT;
  const int skip = (int)((16 - (reinterpret_cast<uintptr_t>(src) & 15)) & 15) >> 2;
  const float4* grp = reinterpret_cast<const float4*>(src + skip);
  const uint32_t full = (uint32_t)((n > skip ? n - skip : 0) >> 2);
  const bool sampled = n > p.cap;   // shorter rows of a ragged batch: every finite score fits the list
  auto sample = [&](int j) { return __ldg(grp + ((uint32_t)j * NT + tid) * full / kTotal); };   // below 2^13 * 2^19
  constexpr int kHeld = SAMPLES <= 2 ? SAMPLES : 1;   // longer samples are read again from L1 / L2
  float4 held[kHeld];
  if (SAMPLES <= 2 && sampled) {
#pragma unroll
    for (int j = 0; j < kHeld; ++j) held[j] = sample(j);
  }
  for (int i = tid; i < 2 * kBigBins; i += NT) hist_a[i] = 0;
  if (tid == 0) {
    s.small_n = 0;
    s.thr[0] = s.thr[1] = s.thr[2] = s.thr[3] = 0;
    s.largest = s_top = 0;
    s_sum[0] = s_sum[1] = 0;
    s_tie[0] = 0xffffffffu;
    s_tie[1] = 0;
  }
  __syncthreads();
  uint32_t pivot = 1;   // the smallest key of a finite score
  bool tie = false;     // many scores equal to the pivot: the threshold may well be among them
  if (sampled) {
    const float kr = (float)p.k * (float)(4 * kTotal) / (float)n;
    const uint32_t target = (uint32_t)(kr + 5.f * sqrtf(kr) + 4.f);
    auto each = [&](auto&& f) {
#pragma unroll 4
      for (int j = 0; j < SAMPLES; ++j) {
        float4 x;
        if constexpr (SAMPLES <= 2) x = held[j];
        else x = sample(j);
        f(score_key_full(x.x));
        f(score_key_full(x.y));
        f(score_key_full(x.z));
        f(score_key_full(x.w));
      }
    };
    uint32_t top = 0;
    each([&](uint32_t key) { top = max(top, key); });
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) atomicMax(&s_top, top);
    __syncthreads();
    top = s_top;
    // The bins cover the 2^24 keys below the largest sample, two octaves of scores: the wanted rank is nearly always
    // among them, the other samples (most) cost no atomic, and these few spread over fine bins.
    each([&](uint32_t key) {
      const uint32_t d = (top - key) >> 13;
      if (d < (uint32_t)kBigBins && key) atomicAdd(&hist_a[kBigBins - 1 - d], 1u);
    });
    __syncthreads();
    threshold_bin<NT>(hist_a, target, s.sums[0], s.thr);
    uint32_t width = 0, reach = s.thr[2] + s.thr[3];   // keys of the bin at the wanted rank, from the pivot on; samples reaching it
    if (s.thr[0] == target) {
      width = 1u << 13;
      const uint32_t below = (kBigBins - s.thr[1]) << 13;   // the bin holds the keys above top - below
      pivot = top > below ? top - below + 1 : 1u;
    } else {
      // deeper down: two levels over the whole range of keys
      for (int i = tid; i < kBigBins; i += NT) hist_a[i] = 0;
      __syncthreads();
      each([&](uint32_t key) { if (key) atomicAdd(&hist_a[key >> 21], 1u); });
      __syncthreads();
      threshold_bin<NT>(hist_a, target, s.sums[1], s.thr);
      if (s.thr[0] == target) {   // otherwise fewer finite samples than wanted: everything is a candidate
        const uint32_t bin = s.thr[1], want = target - s.thr[2];
        each([&](uint32_t key) { if (key && (key >> 21) == bin) atomicAdd(&hist_b[(key >> 10) & 2047u], 1u); });
        __syncthreads();
        threshold_bin<NT>(hist_b, want, s.sums[0], s.thr);
        pivot = max((bin << 21) | (s.thr[1] << 10), 1u);
        width = 1u << 10;
        reach = target - want + s.thr[2] + s.thr[3];
      }
    }
    // clearly more than wanted, so perhaps more than the list holds: is it one score that so many keys have?
    if (__builtin_expect(width && (float)reach > (float)target + 1.5f * sqrtf((float)target), 0)) {
      uint32_t least = 0xffffffffu, most = 0;
      each([&](uint32_t key) {
        if (key - pivot < width && key) {
          least = min(least, key);
          most = max(most, key);
        }
      });
      least = __reduce_min_sync(0xffffffffu, least);
      most = __reduce_max_sync(0xffffffffu, most);
      if (lane == 0 && most) {
        atomicMin(&s_tie[0], least);
        atomicMax(&s_tie[1], most);
      }
      __syncthreads();
      tie = s_tie[0] == s_tie[1];
      if (tie) pivot = s_tie[0];
    }
  }

  // ---- the pass: a bit per score, set if it reaches the pivot; with a tie, one if it is larger and one if it is equal
  auto pass = [&](auto with_tie) {
    constexpr bool TIE = decltype(with_tie)::value;
    const float pf = pivot <= 0x00800000u ? -kMaxScore : key_float(pivot);   // (smaller keys are no finite score's)
    for (int w0 = warp * 32; w0 < words; w0 += (NT / 32) * 32) {   // 32 words = 1,024 scores per warp
      uint32_t mine = 0, equal = 0;
      auto vote = [&](int u, float x) {
        const uint32_t m = __ballot_sync(0xffffffffu, (TIE ? x > pf : x >= pf) && x <= kMaxScore);
        if (lane == u) mine = m;
        if constexpr (TIE) {
          const uint32_t e = __ballot_sync(0xffffffffu, x == pf);
          if (lane == u) equal = e;
        }
      };
      const float* at = src + lo + 32 * w0 + lane;
      if (32 * w0 + 1024 <= len) {
        constexpr int FLIGHT = NT == 512 ? 16 : 32;   // loads in flight per thread, as the registers allow
#pragma unroll
        for (int h = 0; h < 32 / FLIGHT; ++h) {
          float x[FLIGHT];
#pragma unroll
          for (int u = 0; u < FLIGHT; ++u) x[u] = __ldg(at + 32 * (FLIGHT * h + u));
#pragma unroll
          for (int u = 0; u < FLIGHT; ++u) vote(FLIGHT * h + u, x[u]);
        }
      } else {
        for (int u = 0; u < 32; ++u) {
          const bool in = 32 * (w0 + u) + lane < len;
          vote(u, in ? __ldg(at + 32 * u) : -INFINITY);
        }
      }
      bm_gt[w0 + lane] = mine;
      if constexpr (TIE) bm_eq[w0 + lane] = equal;
    }
  };
  if (__builtin_expect(!tie, 1)) pass(std::false_type{});
  else pass(std::true_type{});
  __syncthreads();
  const int per = (words + NT - 1) / NT;
  const int w_lo = min(tid * per, words), w_hi = min(w_lo + per, words);
  // ---- ordered emission from the two bitmaps: this CTA's ids among the row's, gt_run above and eq_run equal before them
  auto emit_bitmaps = [&](uint32_t gt_run, uint32_t eq_run, uint32_t need) {
    uint32_t c_gt = 0, c_eq = 0;
    for (int w = w_lo; w < w_hi; ++w) {
      c_gt += __popc(bm_gt[w]);
      c_eq += __popc(bm_eq[w]);
    }
    uint32_t all;
    uint32_t g_at = gt_run + scan_threads<NT>(c_gt, s.sums[0], &all);
    uint32_t e_at = eq_run + scan_threads<NT>(c_eq, s.sums[1], &all);
    for (int w = w_lo; w < w_hi; ++w) {
      const uint32_t gt = bm_gt[w];
      uint32_t m = gt | bm_eq[w];
      while (m) {
        const int bit = __ffs(m) - 1;
        m &= m - 1;
        const int32_t id = (int32_t)(lo + 32 * w + bit);
        if ((gt >> bit) & 1u) {
          out[g_at + min(e_at, need)] = id;
          ++g_at;
        } else {
          if (e_at < need) out[g_at + e_at] = id;
          ++e_at;
          if (e_at >= need) m &= gt;   // (the other ties of the word are not selected)
        }
      }
    }
  };
  if (__builtin_expect(tie, 0)) {
    uint32_t g = 0, e = 0;
    for (int w = w_lo; w < w_hi; ++w) {
      g += __popc(bm_gt[w]);
      e += __popc(bm_eq[w]);
    }
    g = __reduce_add_sync(0xffffffffu, g);
    e = __reduce_add_sync(0xffffffffu, e);
    if (lane == 0 && g) atomicAdd(&s_sum[0], g);
    if (lane == 0 && e) atomicAdd(&s_sum[1], e);
    __syncthreads();
    uint32_t G = s_sum[0], E = s_sum[1], gt_run = 0, eq_run = 0;
    if constexpr (CLUSTER) {
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // as below
      if (tid < cs) {
        *cluster.map_shared_rank(&cl_count[rank], tid) = G;
        *cluster.map_shared_rank(&cl_eq[rank], tid) = E;
      }
      cluster.sync();
      G = E = 0;
      for (int q = 0; q < cs; ++q) {
        if (q < rank) {
          gt_run += cl_count[q];
          eq_run += cl_eq[q];
        }
        G += cl_count[q];
        E += cl_eq[q];
      }
    }
    if (G < (uint32_t)p.k && (uint32_t)p.k <= G + E) {   // the threshold
      emit_bitmaps(gt_run, eq_run, (uint32_t)p.k - G);
      return;
    }
    if (G >= (uint32_t)p.k) ++pivot;   // it lies above, among the scores marked as larger
    __syncthreads();
    if (tid == 0) s_sum[0] = s_sum[1] = 0;
  }
  // ---- bitmap -> ascending positions
  uint32_t own;   // candidates of this CTA
  {
    uint32_t c = 0;
    for (int w = w_lo; w < w_hi; ++w) c += __popc(bm_gt[w]);
    uint32_t at = scan_threads<NT>(c, s.sums[1], &own);
    for (int w = w_lo; w < w_hi; ++w) {
      uint32_t m = bm_gt[w];
      while (m) {
        const int bit = __ffs(m) - 1;
        m &= m - 1;
        if (at < (uint32_t)p.cap) lpos[at] = 32 * w + bit;
        ++at;
      }
    }
  }
  for (int i = tid; i < 2 * kBigBins; i += NT) hist_a[i] = 0;
  __syncthreads();
  uint32_t largest = 0;
  const uint32_t listed_n = min(own, (uint32_t)p.cap);
  for (uint32_t i0 = 0; i0 < listed_n; i0 += 4 * NT) {   // four fetches in flight per thread
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t i = i0 + u * NT + tid;
      x[u] = i < listed_n ? __ldg(src + lo + lpos[i]) : -INFINITY;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t i = i0 + u * NT + tid;
      const uint32_t key = score_key_full(x[u]);
      if (i < listed_n) lkey[i] = key;
      largest = max(largest, key);
    }
  }
  largest = __reduce_max_sync(0xffffffffu, largest);
  if (lane == 0 && largest) atomicMax(&s.largest, largest);
  __syncthreads();
  largest = s.largest;

  // ---- all candidates of the row in one place
  uint32_t C = own, before = 0;   // before: candidates of the CTAs ahead of this one
  bool fits = C <= (uint32_t)p.cap;
  if constexpr (CLUSTER) {
    // every CTA of the cluster is running: its shared memory may be written
    if (!tie) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (tid < cs) {
      *cluster.map_shared_rank(&cl_count[rank], tid) = C;
      *cluster.map_shared_rank(&cl_gt[rank], tid) = largest;   // (the slot is free until the fallback)
    }
    cluster.sync();
    C = 0;
    for (int q = 0; q < cs; ++q) {
      if (q < rank) before += cl_count[q];
      C += cl_count[q];
      largest = max(largest, cl_gt[q]);
    }
    fits = C <= (uint32_t)p.cap;
    if (fits) {   // (NT / 32) / cs warps copy a CTA's list (cs is a power of two)
      const int q = warp & (cs - 1);
      uint32_t off = 0;
      for (int i = 0; i < q; ++i) off += cl_count[i];
      const uint32_t cnt = cl_count[q];
      const uint32_t* from = cluster.map_shared_rank(lkey, q);
      const uint32_t step = 32 * ((NT / 32) / cs);
#pragma unroll 4
      for (uint32_t i = (warp / cs) * 32 + lane; i < cnt; i += step) keys[off + i] = from[i];
    }
  }
  const bool listed = fits && (pivot == 1u || C >= (uint32_t)p.k);
  // done with the other CTAs' lists (the wait comes before this CTA gives up its own)
  if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  auto lists_released = [] {
    if constexpr (CLUSTER) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  __syncthreads();   // `keys` is complete
  uint32_t k_eff, thr = 0, need = 0;
  if (listed) {
    k_eff = min((uint32_t)p.k, C);
    if (rank == 0)
      for (int i = tid + (int)k_eff; i < p.k; i += NT) out[i] = -1;
    if (k_eff == 0) {
      lists_released();
      return;
    }
    uint32_t base = pivot, want = k_eff;
    int bits = 32 - __clz(largest - pivot);   // 0 when every candidate is the pivot
    uint32_t* hist = hist_a;
    while (true) {
      const int shift = bits > 11 ? bits - 11 : 0;
      for (uint32_t i = tid; i < C; i += NT) {
        const uint32_t d = keys[i] - base;   // keys below base wrap round to the top
        if (bits == 32 || (d >> bits) == 0) atomicAdd(&hist[d >> shift], 1u);
      }
      __syncthreads();
      threshold_bin<NT>(hist, want, s.sums[0], s.thr);
      base += s.thr[1] << shift;
      want -= s.thr[2];
      const uint32_t cnt = s.thr[3];
      bits = shift;
      if (bits == 0) {
        thr = base;
        need = want;
        break;
      }
      if (cnt <= (uint32_t)kPSmall) {
        for (uint32_t i = tid; i < C; i += NT) {
          const uint32_t key = keys[i];
          if (((key - base) >> bits) == 0) s.small_keys[atomicAdd(&s.small_n, 1u)] = key;
        }
        __syncthreads();
        rank_small(&s, cnt, want);
        __syncthreads();
        thr = s.T;
        need = s.need;
        break;
      }
      if (hist == hist_b) {   // third digit: the first histogram once more
        for (int i = tid; i < kBigBins; i += NT) hist_a[i] = 0;
        hist = hist_a;
      } else {
        hist = hist_b;
      }
      __syncthreads();
    }
    // ---- ordered emission over the list: word w votes on entries 32 w .. 32 w + 31
    uint32_t gt_run = 0, eq_run = 0;
    if constexpr (CLUSTER) {
      uint32_t g = 0, e = 0;
      for (uint32_t i = tid; i < before; i += NT) {
        g += keys[i] > thr;
        e += keys[i] == thr;
      }
      g = __reduce_add_sync(0xffffffffu, g);
      e = __reduce_add_sync(0xffffffffu, e);
      if (lane == 0 && g) atomicAdd(&s_sum[0], g);
      if (lane == 0 && e) atomicAdd(&s_sum[1], e);
    }
    __syncthreads();   // the histograms have been read for the last time
    const int lwords = (int)((own + 31) / 32);
    for (int w = warp; w < lwords; w += (NT / 32)) {
      const uint32_t i = 32 * w + lane;
      const uint32_t key = i < own ? lkey[i] : 0u;
      const uint32_t gt = __ballot_sync(0xffffffffu, key > thr), eq = __ballot_sync(0xffffffffu, key == thr);
      if (lane == 0) {
        w_gt[w] = gt;
        w_eq[w] = eq;
      }
    }
    __syncthreads();
    if constexpr (CLUSTER) {
      gt_run = s_sum[0];
      eq_run = s_sum[1];
    }
    {
      uint32_t c = 0;   // low half: above, high half: equal (the list has fewer than 2^16 entries)
      if (tid < lwords) c = (uint32_t)__popc(w_gt[tid]) | ((uint32_t)__popc(w_eq[tid]) << 16);
      uint32_t all;
      const uint32_t at = scan_threads<NT>(c, s.sums[1], &all);
      if (tid < lwords) w_at[tid] = at;
    }
    __syncthreads();
    const uint32_t below = (1u << lane) - 1u;
    for (int w = warp; w < lwords; w += (NT / 32)) {
      const uint32_t gt = w_gt[w], eq = w_eq[w], at = w_at[w];
      const bool is_gt = (gt >> lane) & 1u, is_eq = (eq >> lane) & 1u;
      const uint32_t g = gt_run + (at & 0xffffu) + __popc(gt & below), q = eq_run + (at >> 16) + __popc(eq & below);
      if (is_gt || (is_eq && q < need)) out[g + min(q, need)] = (int32_t)(lo + lpos[32 * w + lane]);
    }
    lists_released();
    return;
  }

  // ---- fallback: radix select that streams the part once per digit; the CTAs of a cluster add up their histograms
  lists_released();
  uint32_t prefix = 0, mask = 0, want = 0, gt_run = 0, eq_run = 0;
  k_eff = 0;
  for (int d = 0; d < 3; ++d) {
    const int shift = d == 0 ? 21 : (d == 1 ? 10 : 0);
    const uint32_t bins = d == 2 ? 1023u : 2047u;
    __syncthreads();
    for (int i = tid; i < kBigBins; i += NT) hist_a[i] = 0;
    __syncthreads();
    for (int i = tid; i < len; i += NT) {
      const uint32_t key = score_key_full(__ldg(src + lo + i));
      if (key && (key & mask) == prefix) atomicAdd(&hist_a[(key >> shift) & bins], 1u);
    }
    __syncthreads();
    uint32_t* total = hist_a;
    if constexpr (CLUSTER) {
      cluster.sync();
      total = hist_b;
      for (int i = tid; i < kBigBins; i += NT) {
        uint32_t t = 0;
        for (int q = 0; q < cs; ++q) t += *cluster.map_shared_rank(&hist_a[i], q);
        total[i] = t;
      }
      cluster.sync();
    }
    threshold_bin<NT>(total, d == 0 ? (uint32_t)p.k : want, s.sums[0], s.thr);
    if (d == 0) want = k_eff = s.thr[0];
    if (k_eff == 0) break;
    prefix |= s.thr[1] << shift;
    mask |= bins << shift;
    want -= s.thr[2];
  }
  thr = prefix;
  need = want;
  if (k_eff > 0) {
    uint32_t g_n = 0, e_n = 0;
    for (int w = warp; w < words; w += (NT / 32)) {
      const int i = 32 * w + lane;
      const uint32_t key = i < len ? score_key_full(__ldg(src + lo + i)) : 0u;
      const uint32_t gt = __ballot_sync(0xffffffffu, key > thr), eq = __ballot_sync(0xffffffffu, key == thr);
      if (lane == 0) {
        bm_gt[w] = gt;
        bm_eq[w] = eq;
      }
      g_n += __popc(gt);
      e_n += __popc(eq);
    }
    if constexpr (CLUSTER) {
      if (lane == 0 && g_n) atomicAdd(&s_sum[0], g_n);
      if (lane == 0 && e_n) atomicAdd(&s_sum[1], e_n);
      __syncthreads();
      if (tid < cs) {
        *cluster.map_shared_rank(&cl_gt[rank], tid) = s_sum[0];
        *cluster.map_shared_rank(&cl_eq[rank], tid) = s_sum[1];
      }
    }
  }
  if constexpr (CLUSTER) {
    cluster.sync();   // last remote access; every CTA of the cluster takes the fallback together
    if (k_eff > 0)
      for (int q = 0; q < rank; ++q) {
        gt_run += cl_gt[q];
        eq_run += cl_eq[q];
      }
  }
  if (rank == 0)
    for (int i = tid + (int)k_eff; i < p.k; i += NT) out[i] = -1;
  if (k_eff == 0) return;
  __syncthreads();
  emit_bitmaps(gt_run, eq_run, need);
}

// Which rows go to the direct kernel: all that 512 threads hold, and up to twice that while each row's 1,024-thread CTA
// has an SM to itself (148 rows of 16,384: 10.4 us; 592 rows: 38, against 29 through the pivot).
static bool topk_direct(int32_t rows, int64_t n) {
  return n <= 512 * kDirectKeys || (n <= kDirectMax && rows <= sm_count());
}

// CTAs per row, 0 = these kernels do not apply
int topk_pivot_size(int32_t rows, int64_t n) {
  if (n > (int64_t)kPMaxCluster * kPPartMax) return 0;
  if (topk_direct(rows, n)) return 1;
  int cs = 1;
  // A cluster's CTAs need an SM each, all in one GPC: 32 clusters of four, 16 of eight and a handful of sixteen are
  // resident at once.  Within that, halving the parts pays down to 4,096 scores per CTA (32 rows of 131,072, CTAs per row
  // 4 / 8: 14.6 / 17.7 us; 8 rows, 8 / 16: 13.5 / 24.6; 1 row, 8 / 16: 13.1 / 12.8; 1 row of 1,048,576, 8 / 16: 47 / 18;
  // 148 rows of 32,768, 1 / 2: 14.4 / 16.9).
  while (cs < kPMaxCluster && n >= (int64_t)cs * 8192 && (int64_t)rows * cs * 2 <= 128 && (cs < 8 || rows <= 4)) cs *= 2;
  while (cs < kPMaxCluster && n > (int64_t)cs * kPPartMax) cs *= 2;
  return cs;
}

template <bool CLUSTER, int NT, int SAMPLES>
static int launch_pivot(const TopkPivotParams& p, int rows, int cs, cudaStream_t st) {
  auto kern = topk_pivot_kernel<CLUSTER, NT, SAMPLES>;
  if (cs > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    (void)cudaGetLastError();
    return MXB_ERR_UNSUPPORTED;
  }
  const size_t smem = ((size_t)2 * kBigBins + (size_t)p.cap * (CLUSTER ? 3 : 2) + (size_t)2 * (p.part / 32)) * 4;
  MXB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((int64_t)rows * cs));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)cs;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CLUSTER ? 2 : 1;
  if (cs > 8) {   // sixteen SMs of one GPC are not there on every device or SM set
    int resident = 0;
    if (cudaOccupancyMaxActiveClusters(&resident, kern, &cfg) != cudaSuccess || resident < 1) {
      (void)cudaGetLastError();
      return MXB_ERR_UNSUPPORTED;
    }
  }
  MXB_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, p));
  note_launch();
  return MXB_OK;
}

// MXB_ERR_UNSUPPORTED: no room for clusters of that size, nothing was launched
static int launch_topk_clusters(const mxb_topk_args* a, int cs, cudaStream_t st) {
  TopkPivotParams p{};
  p.scores = a->scores; p.row_stride = a->row_stride; p.row_start = a->row_start; p.row_count = a->row_count;
  p.out_ids = a->out_ids; p.n = a->n; p.k = a->k;
  if (topk_direct(a->rows, a->n)) {
    const unsigned rows = (unsigned)a->rows;
    // Every row has an SM to itself: all the threads there are, few keys each (148 rows of 4,096: 6.6 -> 5.0 us).  More
    // rows: as many CTAs per SM as the registers of 16 keys allow (333 rows of 5,003 need one wave, not two).
    if (a->rows <= sm_count()) {
      MXB_CUDA_OK(launch_early(a->n <= 1024 * 4   ? topk_direct_kernel<1024, 4, 1>
                               : a->n <= 1024 * 8 ? topk_direct_kernel<1024, 8, 1>
                                                  : topk_direct_kernel<1024, kDirectKeys, 1>,
                               dim3(rows), 1024, 0, st, p));
    } else if (a->n <= 256 * kDirectKeys) {
      MXB_CUDA_OK(launch_early(topk_direct_kernel<256, kDirectKeys, 6>, dim3(rows), 256, 0, st, p));
    } else {
      MXB_CUDA_OK(launch_early(topk_direct_kernel<512, kDirectKeys, 3>, dim3(rows), 512, 0, st, p));
    }
    note_launch();
    return MXB_OK;
  }
  p.part = (int32_t)round_up(ceil_div(a->n, (int64_t)cs), (int64_t)1024);
  // The pivot lets through m = (r k + 5 sqrt(r k) + 4) / r keys at sampling rate r, with a standard deviation of
  // sqrt(m / r); the list holds five of these more.  The smallest sample whose list stays short will do: a cluster
  // reads it once per CTA.
  const int nt = cs > 1 ? 1024 : 512;
  int samples = cs > 1 ? 1 : 2;
  double m = 0, sd = 0;
  while (true) {
    const double r = 4.0 * samples * nt / (double)a->n, kr = r * a->k;
    m = (kr + 5 * sqrt(kr) + 4) / r;
    sd = sqrt(m / r);
    if (m + 5 * sd <= 2.0 * a->k + 6144 || samples == 8) break;
    samples = samples == 1 ? 2 : 8;
  }
  p.cap = (int32_t)round_up((int64_t)fmin(m + 5 * sd, (double)a->n), 32);
  if (p.cap < kBigBins) p.cap = kBigBins;
  if (p.cap > kPListMax) p.cap = kPListMax;
  switch (cs > 1 ? samples : -samples) {
    case 1: return launch_pivot<true, 1024, 1>(p, a->rows, cs, st);
    case 2: return launch_pivot<true, 1024, 2>(p, a->rows, cs, st);
    case 8: return launch_pivot<true, 1024, 8>(p, a->rows, cs, st);
    case -2: return launch_pivot<false, 512, 2>(p, a->rows, cs, st);
    case -8: return launch_pivot<false, 512, 8>(p, a->rows, cs, st);
  }
  return fail(MXB_ERR_INVALID, "topk: no kernel for %d samples", samples);
}

// MXB_ERR_UNSUPPORTED: the row needs clusters of a size that the device has no room for
int launch_topk_pivot(const mxb_topk_args* a, int cs, cudaStream_t st) {
  int rc = launch_topk_clusters(a, cs, st);
  if (rc == MXB_ERR_UNSUPPORTED && cs > 8 && a->n <= (int64_t)8 * kPPartMax) rc = launch_topk_clusters(a, 8, st);
  return rc;
}

}  // namespace mxb
