// Row operations of the DeepSeek-V4 decode chain, one warp per row: shared by the streaming kernels (indexer_qat.cu,
// kv_formats.cu) and by the fused decode operators (decode_fused.cu).  Layouts and operation orders are described there.
#pragma once

#include "common.cuh"

namespace mxb {

__device__ __forceinline__ float lattice_snap(float n) {
  // nearest of the eight e2m1 magnitudes; the first (lower) value wins a tie
  const float values[8] = {0.0f, 0.5f, 1.0f, 1.5f, 2.0f, 3.0f, 4.0f, 6.0f};
  const float absn = fabsf(n);
  float best = fabsf(__fsub_rn(absn, values[0]));
  float dq = values[0];
#pragma unroll
  for (int k = 1; k < 8; ++k) {
    const float d = fabsf(__fsub_rn(absn, values[k]));
    if (d < best) {
      best = d;
      dq = values[k];
    }
  }
  return n < 0.0f ? -dq : dq;
}

// QAT of a 128-wide row: lane l holds elements 4 l .. 4 l + 3 of the input and of the result.
__device__ __forceinline__ void indexer_qat_row(const float (&v)[4], int lane, float (&o)[4]) {
  // strides 1 and 2 inside the lane
  const float a0 = __fadd_rn(v[0], v[1]), a1 = __fsub_rn(v[0], v[1]);
  const float a2 = __fadd_rn(v[2], v[3]), a3 = __fsub_rn(v[2], v[3]);
  float x[4] = {__fadd_rn(a0, a2), __fadd_rn(a1, a3), __fsub_rn(a0, a2), __fsub_rn(a1, a3)};
  // strides 4 .. 64 pair lanes
#pragma unroll
  for (int m = 1; m <= 16; m <<= 1) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float other = __shfl_xor_sync(0xffffffffu, x[j], m);
      x[j] = (lane & m) ? __fsub_rn(other, x[j]) : __fadd_rn(x[j], other);
    }
  }
  const float kHadamardScale = 0.08838834764831845f;
#pragma unroll
  for (int j = 0; j < 4; ++j) x[j] = __fmul_rn(x[j], kHadamardScale);

  // e2m1 round trip over groups of 32 elements = 8 lanes
  // the maximum skips NaN elements (fmax), as the reference kernel's does; a group of nothing but NaN keeps NaN
  float amax = fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3])));
#pragma unroll
  for (int m = 1; m <= 4; m <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
  const float kAmaxFloor = 7.052966104933725e-38f;
  if (!isnan(amax) && !(amax > kAmaxFloor)) amax = kAmaxFloor;
  const float kLn2 = 0.6931471805599453f;           // ln 2 rounded to float32, as the float32 chain sees it
  const float ratio = __fdiv_rn(amax, 6.0f);
  const float lg = (float)log((double)ratio);        // correctly rounded float32 log
  const float log2_scale = __fdiv_rn(lg, kLn2);
  const float arg = __fmul_rn(ceilf(log2_scale), kLn2);
  const float scale = (float)exp((double)arg);       // correctly rounded float32 exp

#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float n = __fdiv_rn(x[j], scale);
    n = (isnan(n) || n > -6.0f) ? n : -6.0f;
    n = (isnan(n) || n < 6.0f) ? n : 6.0f;
    o[j] = __fmul_rn(lattice_snap(n), scale);
  }
}

__device__ __forceinline__ float e4m3_nearest_lower_tie(float absn) {
  // absn in [0, 448]
  float step;
  if (absn < 0.015625f) {
    step = 0.001953125f;   // subnormal spacing 2^-9
  } else {
    const int e = (int)((__float_as_uint(absn) >> 23) & 0xff) - 127;   // floor(log2(absn)), -6 .. 8
    step = __uint_as_float((uint32_t)(e - 3 + 127) << 23);
  }
  const float t = __fdiv_rn(absn, step);             // exact: step is a power of two
  return __fmul_rn(fabsf(ceilf(__fsub_rn(t, 0.5f))), step);  // exact; a tie (t = k + 1/2) goes to k; fabsf: ceil(-0.3) = -0
}

// nearest E4M3FN magnitude with ties to the even code: within a binade the code's parity is the parity of the
// grid multiple, so this is round-half-even on t
__device__ __forceinline__ float e4m3_nearest_even_tie(float absn) {
  float step;
  if (absn < 0.015625f) {
    step = 0.001953125f;
  } else {
    const int e = (int)((__float_as_uint(absn) >> 23) & 0xff) - 127;
    step = __uint_as_float((uint32_t)(e - 3 + 127) << 23);
  }
  return __fmul_rn(rintf(__fdiv_rn(absn, step)), step);
}

// E4M3FN round trip of a 512-wide row in place: lane l holds dims 16 l .. 16 l + 15.
// REPLAY = false: the served transcription; true: the reference's NumPy replay form (exact power-of-two scale,
// ties to the even code)
template <bool REPLAY>
__device__ __forceinline__ void fp8_kv_row(float (&xv)[16], int lane) {
  // lanes 28 .. 31 hold the rotary tail: they take part in the shuffles and store their input back
  float amax = 0.0f;   // the maximum skips NaN elements (fmax), as the reference kernel's does
#pragma unroll
  for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(xv[j]));
#pragma unroll
  for (int m = 1; m <= 2; m <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
  if (lane < 28) {
    if (!(amax > 1.0e-4f)) amax = 1.0e-4f;
    float scale;
    if (REPLAY) {
      int e;
      const double m = frexp((double)amax / 448.0, &e);   // amax / 448 = m * 2^e, m in [0.5, 1)
      scale = ldexpf(1.0f, m == 0.5 ? e - 1 : e);         // 2^ceil(log2(amax / 448)), exactly
    } else {
      const float kLn2 = 0.6931471805599453f;
      const float lg = (float)log((double)__fdiv_rn(amax, 448.0f));   // correctly rounded float32 log
      const float arg = __fmul_rn(ceilf(__fdiv_rn(lg, kLn2)), kLn2);
      scale = (float)exp((double)arg);                                // correctly rounded float32 exp
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float n = __fdiv_rn(xv[j], scale);
      n = (isnan(n) || n > -448.0f) ? n : -448.0f;
      n = (isnan(n) || n < 448.0f) ? n : 448.0f;
      const float qv = isnan(n) ? 0.0f : (REPLAY ? e4m3_nearest_even_tie(fabsf(n)) : e4m3_nearest_lower_tie(fabsf(n)));
      const float sign = n < 0.0f ? -1.0f : (n > 0.0f ? 1.0f : 0.0f);
      xv[j] = __fmul_rn(__fmul_rn(sign, qv), scale);
    }
  }
}

// One rotary pair in the fused decode kernels' float16 form: float32 angle, cos / sin rounded to float16, every product
// and sum rounded to float16 (src/moespresso/runtime/deepseek_v4/decode_attention_kernel.py:120-147, 398-422)
__device__ __forceinline__ void rope_half_pair(__half x0, __half x1, int64_t pos, float inv_freq, bool inverse, __half& y0,
                                               __half& y1) {
  const float theta = __fmul_rn((float)pos, inv_freq);
  const __half c = __float2half_rn((float)cos((double)theta));
  __half s = __float2half_rn((float)sin((double)theta));
  if (inverse) s = __hneg(s);
  // the _rn forms are never contracted into a fused multiply-add: every product is rounded on its own
  const __half m0 = __hmul_rn(x0, c), m1 = __hmul_rn(x1, s), m2 = __hmul_rn(x0, s), m3 = __hmul_rn(x1, c);
  y0 = __hsub_rn(m0, m1);
  y1 = __hadd_rn(m2, m3);
}

}  // namespace mxb
