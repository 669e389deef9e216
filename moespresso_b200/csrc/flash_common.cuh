// What the two kernels of the flash prefill share: parameters, the numbering of the work, exponentials.
#pragma once

#include "common.cuh"
#include "ptx_sm100.cuh"

namespace mxb {

constexpr int FB_M = 128, FB_D = 256;
constexpr int kMaxBins = 160;
#ifndef MXB_FLASH_POLY
#define MXB_FLASH_POLY 1
#endif
constexpr int kPolyOf8 = MXB_FLASH_POLY;   // of every eight exponentials, this many (0 .. 4) run on the FMA pipe

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
  int32_t pair_heads;  // a pair's query tiles: the same rows of two heads (one KV head), or 256 rows of one head
  int32_t* status;
  // Stretches of tiles, one per pair of CTAs or CTA (n_bins = 0: an item each).  Bin i covers the tiles from bin_start[i]
  // up to bin_start[i + 1], both (item << 16 | tile of the item).
  float4* part_o;      // [2 n_bins CTAs][64 groups of 4 features][128 rows]
  float2* part_ml;     // [2 n_bins CTAs][128 rows]: reference maximum (log2 units), sum
  int32_t n_bins;
  uint32_t bin_start[kMaxBins + 1];
};

// An item: 128 query rows in each CTA of a pair, or 128 rows of one head for a single CTA.  Items are numbered longest first.
struct FlashItems {
  int n_qt, per_qt;   // query tiles (of 128 or 256 rows) and items of one
};
__host__ __device__ inline FlashItems flash_items(int S, int Hq, int pair_heads) {
  FlashItems f;
  f.n_qt = pair_heads ? (S + FB_M - 1) / FB_M : (S + 2 * FB_M - 1) / (2 * FB_M);
  f.per_qt = pair_heads ? Hq / 2 : Hq;
  return f;
}
// Where CTA `rank` of the pair that works on item `it` stands.
__host__ __device__ inline void flash_item_at(const FlashItems& f, int it, int pair_heads, int rank, int& head, int& m0) {
  const int qt = f.n_qt - 1 - it / f.per_qt, x = it % f.per_qt;
  head = pair_heads ? 2 * x + rank : x;
  m0 = pair_heads ? qt * FB_M : (2 * qt + rank) * FB_M;
}
// tiles of N keys that the rows of query tile qt see
template <int N>
__host__ __device__ inline int flash_tiles(int qt, int rows, int S, int Skv) {
  const int64_t end = (int64_t)qt * rows + rows + (Skv - S);
  return (int)(((end < Skv ? end : (int64_t)Skv) + N - 1) / N);
}
// where a cut item's segment leaves its partial: a bin holds at most one segment that starts inside an item, and
// one that starts an item and does not finish it
__device__ __forceinline__ int part_slot(int bin, bool starts_inside) { return 2 * bin + (starts_inside ? 0 : 1); }
// The reference maximum a cut segment starts from: finite, so that a row that sees none of the segment's first tile
// (the rows above the diagonal) gets weights of 0 and not of exp(-inf + inf).
constexpr float kNoMax = -3e38f;
constexpr float kGrow = 8.f;   // the reference moves when a logit exceeds it by this many powers of two

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
__device__ __forceinline__ float fast_ex2(float x) {   // 2^x, x <= kGrow here; -inf -> 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^x on the FMA pipe for x <= ~8: round-to-nearest split x = n + f with the 1.5 * 2^23 trick, a cubic for 2^f on
// [-0.5, 0.5] (relative error 7.5e-5, below the rounding of a 16-bit P), n added into the exponent field.  One in
// eight of a tile's exponentials goes this way.  (The special-function unit's 16 results per clock per SM no longer bound
// the kernel: 0 / 1 / 2 / 3 in eight 433 / 437 / 439 / 447 us at 8,192 tokens.)  Inputs below -126 (masked keys) give 2^-126 instead of 0.
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

// flash_single.cu: the kernel of one CTA per item, on the tensor maps of 64-key K and V tiles
int launch_flash_single(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tg,
                        const CUtensorMap& to, const FlashParams& p, bool bf16, unsigned ctas, cudaStream_t st);

}  // namespace mxb
