// Cache-row formats either side of the attention path.
//
//  * fp8_kv_rows_kernel — DeepSeek-V4's E4M3FN round trip of the non-rotary prefix of 512-wide
//    compressed-KV rows: dims [0, 448) in blocks of 64, block scale
//    exp(ceil(log(max(amax, 1e-4) / 448) / ln 2) * ln 2) in float32 steps, values clipped to
//    [-448, 448], snapped to the nearest of the 127 non-negative E4M3FN magnitudes (ties to the LOWER
//    one), sign restored (NaN -> 0), multiplied back; dims [448, 512) pass through.  One warp per row,
//    lane l holds dims [16l, 16l + 16), the layout and operation order of the reference's kernel
//    (src/moespresso/runtime/deepseek_v4/decode_attention_kernel.py:149-176, 536-560).  The nearest
//    magnitude is found arithmetically (grid step of the value's binade, ceil(t - 1/2)), which selects
//    the same table entry as the reference's first-wins scan of the table.
//  * quant_i8_rows_kernel — the per-token int8 quantiser that produces the int8 + fp16-scale cache the
//    sparse decode kernels read: scale = fp16(amax / 127) (rounded up when the rounding would let a
//    value exceed 127), q = clamp(rint(x / scale), -127, 127).  No counterpart in the reference.
//    quant_i8_rows_vec_kernel is the form for rows of whole 16-byte pieces, quant_i8_rows_kernel takes any row.
#include "decode_rows.cuh"

namespace mxb {

template <bool REPLAY>
__global__ void __launch_bounds__(128) fp8_kv_rows_kernel(const float* __restrict__ x, float* __restrict__ out,
                                                          int64_t n_rows) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= n_rows) return;
  const float4* src = reinterpret_cast<const float4*>(x + row * 512 + 16 * lane);
  float4* dst = reinterpret_cast<float4*>(out + row * 512 + 16 * lane);
  float xv[16];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 v = src[j];
    xv[4 * j] = v.x; xv[4 * j + 1] = v.y; xv[4 * j + 2] = v.z; xv[4 * j + 3] = v.w;
  }
  fp8_kv_row<REPLAY>(xv, lane);   // lanes 28 .. 31 hold the rotary tail and store their input back
#pragma unroll
  for (int j = 0; j < 4; ++j) dst[j] = make_float4(xv[4 * j], xv[4 * j + 1], xv[4 * j + 2], xv[4 * j + 3]);
}

// fp16 scale of a row whose largest magnitude is amax
__device__ __forceinline__ __half i8_row_scale(float amax) {
  __half hs = __float2half_rn(amax / 127.0f);
  if (__half2float(hs) * 127.0f < amax) hs = __ushort_as_half((unsigned short)(__half_as_ushort(hs) + 1));  // next fp16 up
  if (__half2float(hs) == 0.0f) hs = __ushort_as_half((unsigned short)1);   // all-zero row: any scale will do
  return hs;
}
__device__ __forceinline__ int8_t i8_quant_exact(float x, float s) {
  return (int8_t)fminf(fmaxf(rintf(x / s), -127.0f), 127.0f);
}

template <int XT>
__global__ void __launch_bounds__(128) quant_i8_rows_kernel(const void* __restrict__ x, int8_t* __restrict__ q,
                                                            __half* __restrict__ scales, int64_t n_rows, int width) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= n_rows) return;
  float amax = 0.0f;
  for (int i = lane; i < width; i += 32) amax = fmaxf(amax, fabsf(load_elem<XT>(x, row * width + i)));
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
  const __half hs = i8_row_scale(amax);
  const float s = __half2float(hs);
  for (int i = lane; i < width; i += 32) q[row * width + i] = i8_quant_exact(load_elem<XT>(x, row * width + i), s);
  if (lane == 0) scales[row] = hs;
}

// max(|a|, |b|, |c|), NaN if one of them is
__device__ __forceinline__ float max3_nan_abs(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// One warp per row at a time, the row in registers as NV 16-byte pieces per lane (a piece beyond the row reads as
// zeros), the next row on its way.  Bound: HBM (row in, int8 row out), with instruction issue close behind: the elements
// are read once, and no element is divided.  x * (1 / s) differs from x / s by a few units in the last place, so both
// round to the same integer unless the product lies within 1e-4 of a half-integer (|product| <= 127, a relative error of
// 2^-23 is below 2e-5); a lane that holds such an element, or a NaN or an infinity, redoes its piece with the division.
// The multiply-adds are packed in pairs.  40,001 rows of 576 bf16 values: 30.2 -> 14.2 us (2.3 -> 4.9 TB/s); the scalar
// form spends 20 instructions on each division and reads every element twice, one row per warp without the look-ahead
// and the pairs took 17.0 us.
template <int XT, int NV>
__global__ void __launch_bounds__(256) quant_i8_rows_vec_kernel(const uint4* __restrict__ x, int8_t* __restrict__ q,
                                                                __half* __restrict__ scales, int64_t n_rows, int width) {
  constexpr int EPV = XT == MXB_F32 ? 4 : 8;   // elements per piece
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * 8;
  int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int pieces = width / EPV;
  uint4 next[NV];
  auto fetch = [&](int64_t r) {
#pragma unroll
    for (int v = 0; v < NV; ++v)
      next[v] = r < n_rows && 32 * v + lane < pieces ? __ldcs(x + r * pieces + 32 * v + lane) : make_uint4(0, 0, 0, 0);
  };
  fetch(row);
  for (; row < n_rows; row += step) {   // the same trip count for the lanes of a warp
    float f[NV][EPV];
    float amax = 0.0f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      unpack16<XT>(next[v], f[v]);
#pragma unroll
      for (int e = 0; e < EPV; e += 2) amax = fmaxf(fmaxf(amax, fabsf(f[v][e])), fabsf(f[v][e + 1]));
    }
    fetch(row + step);
    // magnitudes order like their bits
    amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
    const __half hs = i8_row_scale(amax);
    const float s = __half2float(hs), inv = __frcp_rn(s);
    const float2 inv2 = make_float2(inv, inv);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (32 * v + lane < pieces) {
        uint32_t b[EPV];
        float off = 0.0f;   // largest distance from the rounded integer; NaN if one is
#pragma unroll
        for (int e = 0; e < EPV; e += 2) {
          const float2 x2 = make_float2(f[v][e], f[v][e + 1]);
          // 1.5 * 2^23: the rounded integer sits in the low mantissa bits of the sum
          const float2 m = __ffma2_rn(x2, inv2, make_float2(12582912.0f, 12582912.0f));
          const float2 r = __fadd2_rn(m, make_float2(-12582912.0f, -12582912.0f));
          const float2 d = __ffma2_rn(x2, inv2, make_float2(-r.x, -r.y));
          off = max3_nan_abs(off, d.x, d.y);
          b[e] = __float_as_uint(m.x);
          b[e + 1] = __float_as_uint(m.y);
        }
        if (!(off < 0.4999f)) {
#pragma unroll
          for (int e = 0; e < EPV; ++e) b[e] = (uint8_t)i8_quant_exact(f[v][e], s);
        }
        uint32_t w[EPV / 4];
#pragma unroll
        for (int i = 0; i < EPV / 4; ++i)
          w[i] = __byte_perm(__byte_perm(b[4 * i], b[4 * i + 1], 0x0040), __byte_perm(b[4 * i + 2], b[4 * i + 3], 0x0040), 0x5410);
        int8_t* dst = q + row * width + (32 * v + lane) * EPV;
        if constexpr (EPV == 8) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
        else *reinterpret_cast<uint32_t*>(dst) = w[0];
      }
    }
    if (lane == 0) scales[row] = hs;
  }
}

}  // namespace mxb

using namespace mxb;

extern "C" int mxb_fp8_kv_rows(const mxb_fp8_kv_rows_args* a, void* stream) {
  MXB_REQUIRE(a != nullptr, MXB_ERR_INVALID, "fp8 rows: null args");
  MXB_REQUIRE(a->width == 512, MXB_ERR_INVALID, "fp8 rows expect 512-wide rows");
  MXB_REQUIRE(a->n_rows > 0, MXB_ERR_INVALID, "fp8 rows expect at least one row");
  MXB_REQUIRE(a->x && a->out, MXB_ERR_INVALID, "fp8 rows: null tensor");
  MXB_REQUIRE(a->mode == MXB_FP8KV_SERVED || a->mode == MXB_FP8KV_REPLAY, MXB_ERR_INVALID, "fp8 rows: unknown mode");
  MXB_REQUIRE(((reinterpret_cast<uintptr_t>(a->x) | reinterpret_cast<uintptr_t>(a->out)) & 15) == 0, MXB_ERR_INVALID,
              "fp8 rows must be 16-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->mode == MXB_FP8KV_REPLAY)
    fp8_kv_rows_kernel<true><<<(unsigned)ceil_div(a->n_rows, 4), 128, 0, st>>>(a->x, a->out, a->n_rows);
  else
    fp8_kv_rows_kernel<false><<<(unsigned)ceil_div(a->n_rows, 4), 128, 0, st>>>(a->x, a->out, a->n_rows);
  note_launch();
  MXB_CUDA_OK(cudaGetLastError());
  return MXB_OK;
}

extern "C" int mxb_quantize_kv_int8(const mxb_quantize_kv_int8_args* a, void* stream) {
  MXB_REQUIRE(a != nullptr, MXB_ERR_INVALID, "int8 quantiser: null args");
  MXB_REQUIRE(a->n_rows > 0 && a->width > 0, MXB_ERR_INVALID, "int8 quantiser expects at least one row and column");
  MXB_REQUIRE(a->x && a->q && a->scales, MXB_ERR_INVALID, "int8 quantiser: null tensor");
  MXB_REQUIRE(a->x_dtype == MXB_F32 || a->x_dtype == MXB_F16 || a->x_dtype == MXB_BF16, MXB_ERR_INVALID,
              "int8 quantiser rows must be float32, float16, or bfloat16");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  MXB_REQUIRE(ceil_div(a->n_rows, 4) <= 0x7FFFFFFFll, MXB_ERR_INVALID, "int8 quantiser: too many rows");
  const unsigned grid = (unsigned)ceil_div(a->n_rows, 4);
  __half* sc = reinterpret_cast<__half*>(a->scales);
  // whole 16-byte pieces on 16-byte boundaries, at most eight per lane
  const int epv = a->x_dtype == MXB_F32 ? 4 : 8;
  const int nv = a->width % epv == 0 ? (int)ceil_div(a->width / epv, 32) : 99;
  if (nv <= 8 && (reinterpret_cast<uintptr_t>(a->x) & 15) == 0 && (reinterpret_cast<uintptr_t>(a->q) & 7) == 0) {
    const uint4* xv = reinterpret_cast<const uint4*>(a->x);
    // one resident wave (three CTAs of 256 threads per SM by registers) whose warps fetch a row ahead
    const int64_t most = 3 * (int64_t)sm_count();
    const unsigned vgrid = (unsigned)(ceil_div(a->n_rows, 8) < most ? ceil_div(a->n_rows, 8) : most);
#define MXB_QVEC(XT)                                                                                             \
  if (nv <= 3) quant_i8_rows_vec_kernel<XT, 3><<<vgrid, 256, 0, st>>>(xv, a->q, sc, a->n_rows, a->width);        \
  else if (nv <= 5) quant_i8_rows_vec_kernel<XT, 5><<<vgrid, 256, 0, st>>>(xv, a->q, sc, a->n_rows, a->width);   \
  else quant_i8_rows_vec_kernel<XT, 8><<<vgrid, 256, 0, st>>>(xv, a->q, sc, a->n_rows, a->width)
    if (a->x_dtype == MXB_F32) { MXB_QVEC(MXB_F32); }
    else if (a->x_dtype == MXB_F16) { MXB_QVEC(MXB_F16); }
    else { MXB_QVEC(MXB_BF16); }
#undef MXB_QVEC
  } else if (a->x_dtype == MXB_F32) {
    quant_i8_rows_kernel<MXB_F32><<<grid, 128, 0, st>>>(a->x, a->q, sc, a->n_rows, a->width);
  } else if (a->x_dtype == MXB_F16) {
    quant_i8_rows_kernel<MXB_F16><<<grid, 128, 0, st>>>(a->x, a->q, sc, a->n_rows, a->width);
  } else {
    quant_i8_rows_kernel<MXB_BF16><<<grid, 128, 0, st>>>(a->x, a->q, sc, a->n_rows, a->width);
  }
  note_launch();
  MXB_CUDA_OK(cudaGetLastError());
  return MXB_OK;
}

// ---------------------------------------------------------------------------------------------
// Partial rotary embedding of the last `rope_dim` channels of every row (interleaved pairs), forward or
// inverse: the seam either side of the attention call
// (src/moespresso/runtime/deepseek_v4/attention.py:114-156; in-kernel forms
//  src/moespresso/runtime/deepseek_v4/decode_attention_kernel.py:398-422, 504-521).
// Row r sits at sequence index r % seq_len (the sequence axis is the second-to-last).  Angles are
// position * inverse frequency in float64, as in the NumPy definition; the result is rounded once to
// the row type.  Leading channels are copied.
// ---------------------------------------------------------------------------------------------
namespace mxb {

template <int XT>
__global__ void __launch_bounds__(128) rope_tail_kernel(const void* __restrict__ x, void* __restrict__ out,
                                                        const int64_t* __restrict__ positions,
                                                        const double* __restrict__ inv_freq, int64_t n_rows,
                                                        int seq_len, int width, int rope_dim, int inverse,
                                                        int half_chain) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= n_rows) return;
  const int64_t base = row * width;
  const int lead = width - rope_dim;
  if (x != out)
    for (int i = lane; i < lead; i += 32) store_elem<XT>(out, base + i, load_elem<XT>(x, base + i));
  const double pos = (double)positions[row % seq_len];
  if constexpr (XT == MXB_F16) {
    if (half_chain) {
      const int64_t ipos = positions[row % seq_len];
      const __half* xh = reinterpret_cast<const __half*>(x) + base + lead;
      __half* oh = reinterpret_cast<__half*>(out) + base + lead;
      for (int pr = lane; pr < rope_dim / 2; pr += 32)
        rope_half_pair(xh[2 * pr], xh[2 * pr + 1], ipos, (float)inv_freq[pr], inverse != 0, oh[2 * pr], oh[2 * pr + 1]);
      return;
    }
  }
  for (int pr = lane; pr < rope_dim / 2; pr += 32) {
    double s, c;
    sincos(pos * inv_freq[pr], &s, &c);
    if (inverse) s = -s;
    const double x0 = (double)load_elem<XT>(x, base + lead + 2 * pr);
    const double x1 = (double)load_elem<XT>(x, base + lead + 2 * pr + 1);
    store_elem_f64<XT>(out, base + lead + 2 * pr, x0 * c - x1 * s);
    store_elem_f64<XT>(out, base + lead + 2 * pr + 1, x0 * s + x1 * c);
  }
}

}  // namespace mxb

extern "C" int mxb_rope_tail(const mxb_rope_tail_args* a, void* stream) {
  MXB_REQUIRE(a != nullptr, MXB_ERR_INVALID, "rope: null args");
  MXB_REQUIRE(a->n_rows > 0 && a->seq_len > 0 && a->n_rows % a->seq_len == 0, MXB_ERR_INVALID,
              "x must have at least sequence and feature dimensions");
  MXB_REQUIRE(a->rope_dim > 0 && a->rope_dim % 2 == 0, MXB_ERR_INVALID, "rope_dim must be a positive even integer");
  MXB_REQUIRE(a->width >= a->rope_dim, MXB_ERR_INVALID, "rope_dim cannot exceed the feature dimension");
  MXB_REQUIRE(a->x && a->out && a->positions && a->inv_freq, MXB_ERR_INVALID, "rope: null tensor");
  MXB_REQUIRE(a->x_dtype == MXB_F32 || a->x_dtype == MXB_F16 || a->x_dtype == MXB_BF16, MXB_ERR_INVALID,
              "rope rows must be float32, float16, or bfloat16");
  MXB_REQUIRE(!a->half_chain || a->x_dtype == MXB_F16, MXB_ERR_INVALID, "the float16 rope chain takes float16 rows");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)ceil_div(a->n_rows, 4);
#define MXB_ROPE(XT)                                                                                          \
  rope_tail_kernel<XT><<<grid, 128, 0, st>>>(a->x, a->out, a->positions, a->inv_freq, a->n_rows, a->seq_len, \
                                             a->width, a->rope_dim, a->inverse, a->half_chain)
  if (a->x_dtype == MXB_F32) MXB_ROPE(MXB_F32);
  else if (a->x_dtype == MXB_F16) MXB_ROPE(MXB_F16);
  else MXB_ROPE(MXB_BF16);
#undef MXB_ROPE
  note_launch();
  MXB_CUDA_OK(cudaGetLastError());
  return MXB_OK;
}
