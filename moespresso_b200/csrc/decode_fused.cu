// The fused decode operators of one ratio-4 DeepSeek-V4 token (batch 1), each as one call of the library:
//   mxb_fused_decode_prep   QAT of the indexer query, scores over the pool, exact top-k, and the KV row
//   mxb_fused_decode_sdpa   rope on q, attention over the window and the selected rows, inverse rope
// (src/moespresso/runtime/deepseek_v4/decode_attention_kernel.py:669-786).  A token is all latency: the arithmetic of
// the small kernels is nothing, so what counts is how many of them there are.  decode_prep_kernel does everything that
// precedes the score scan and decode_sdpa_prep_kernel everything that precedes the attention, whatever the row type;
// the scan, the selection and the attention are the package's kernels.  At 2,500 rows a token takes 26.5 us: seven kernels, each
// launched while the one before it runs (the attention of a few tokens needs no merge kernel); as some twenty single operators
// it took 378 us, 104 of them in kernels.
#include "decode_rows.cuh"
#include "ptx_sm100.cuh"

namespace mxb {

constexpr int kRowDim = 512, kRopeDim = 64, kIdxDim = 128;

struct TokenParams {     // int32 or int64 [position, write index]
  const void* p;
  int32_t wide;
  __device__ __forceinline__ int64_t at(int i) const {
    return wide ? reinterpret_cast<const int64_t*>(p)[i] : (int64_t)reinterpret_cast<const int32_t*>(p)[i];
  }
};

// Rotates the last 64 channels of a row, a pair per lane; the other channels stay where they are.
__device__ __forceinline__ void rope_row(__half* dst, const __half* src, int64_t pos, const float* inv_freq, bool inverse,
                                         int lane) {
  const int i = kRowDim - kRopeDim + 2 * lane;
  __half y0, y1;
  rope_half_pair(src[i], src[i + 1], pos, inv_freq[lane], inverse, y0, y1);
  dst[i] = y0;
  dst[i + 1] = y1;
}

struct DecodePrepParams {
  const void* q;          // [H, 128]
  const float* weights;   // [H]
  const __half* kv_row;   // [512]
  const float* inv_freq;  // [32]
  TokenParams token;
  float scale;
  int32_t H;
  float* q_qat;           // [H, 128]
  float* w_scaled;        // [H]
  __half* row;            // [512]
};

// Warp w: QAT of head w; warp H: E4M3FN round trip of dims [0, 448) of the KV row; warp H + 1: rope of its other 64, a
// pair per lane (cos and sin are the longest chain here); warp H + 2: the score scale folded into the head weights.
template <int QT>
__global__ void __launch_bounds__(128) decode_prep_kernel(DecodePrepParams p) {
  const int lane = threadIdx.x & 31, w = (int)blockIdx.x * 4 + (threadIdx.x >> 5);
  ptx::grid_chain();
  if (w < p.H) {
    float v[4], o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = load_elem<QT>(p.q, (int64_t)w * kIdxDim + 4 * lane + j);
    indexer_qat_row(v, lane, o);
    *reinterpret_cast<float4*>(p.q_qat + w * kIdxDim + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
  } else if (w == p.H) {
    float xv[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) xv[j] = __half2float(p.kv_row[16 * lane + j]);
    fp8_kv_row<false>(xv, lane);
    if (lane < 28) {
#pragma unroll
      for (int j = 0; j < 16; ++j) p.row[16 * lane + j] = __float2half_rn(xv[j]);
    }
  } else if (w == p.H + 1) {
    rope_row(p.row, p.kv_row, p.token.at(0), p.inv_freq, false, lane);
  } else if (w == p.H + 2) {
    for (int h = lane; h < p.H; h += 32) p.w_scaled[h] = __fmul_rn(p.weights[h], p.scale);
  }
}

struct SdpaPrepParams {
  const __half* q;        // [H, 512]
  const __half* window;   // [W, 512]
  const __half* row;      // [512]
  const __half* sinks;    // [H]
  const float* inv_freq;  // [32]
  TokenParams token;
  int32_t H, W;
  __half* q_roped;        // [H, 512]
  __half* keys;           // [W, 512]: the window with row `write index` replaced (by an index inside it)
  float* sinks_f;         // [H]
  int64_t* pos0;          // every window row is a key: the position of the newest is at least W - 1
};

__device__ __forceinline__ void copy_row(__half* dst, const __half* src, int lane, bool vec) {
  if (vec) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
    uint4* d = reinterpret_cast<uint4*>(dst);
    const uint4 a = s[lane], b = s[lane + 32];
    d[lane] = a;
    d[lane + 32] = b;
  } else {
    for (int i = lane; i < kRowDim; i += 32) dst[i] = src[i];
  }
}

// Warp w: head w of q, then row w - H of the window; warp H + W: the sinks and the position.
__global__ void __launch_bounds__(128) decode_sdpa_prep_kernel(SdpaPrepParams p) {
  const int lane = threadIdx.x & 31, w = (int)blockIdx.x * 4 + (threadIdx.x >> 5);
  const bool vec = ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.window) |
                     reinterpret_cast<uintptr_t>(p.row)) & 15) == 0;
  ptx::grid_chain();
  if (w < p.H) {
    const __half* src = p.q + (int64_t)w * kRowDim;
    __half* dst = p.q_roped + (int64_t)w * kRowDim;
    copy_row(dst, src, lane, vec);
    __syncwarp();
    rope_row(dst, src, p.token.at(0), p.inv_freq, false, lane);
  } else if (w < p.H + p.W) {
    const int r = w - p.H;
    copy_row(p.keys + (int64_t)r * kRowDim, p.token.at(1) == r ? p.row : p.window + (int64_t)r * kRowDim, lane, vec);
  } else if (w == p.H + p.W) {
    for (int h = lane; h < p.H; h += 32) p.sinks_f[h] = __half2float(p.sinks[h]);
    if (lane == 0) {
      const int64_t pos = p.token.at(0);
      p.pos0[0] = pos > p.W - 1 ? pos : p.W - 1;
    }
  }
}

__global__ void __launch_bounds__(128) decode_unrope_kernel(__half* out, const float* inv_freq, TokenParams token, int H) {
  const int lane = threadIdx.x & 31, w = (int)blockIdx.x * 4 + (threadIdx.x >> 5);
  ptx::grid_chain();
  if (w < H) rope_row(out + (int64_t)w * kRowDim, out + (int64_t)w * kRowDim, token.at(0), inv_freq, true, lane);
}

// pieces of one workspace, each 256-byte aligned
struct Carver {
  uint8_t* base;
  int64_t used = 0;
  void* take(int64_t bytes) {
    void* p = base ? base + used : nullptr;
    used += round_up(bytes, 256);
    return p;
  }
};

}  // namespace mxb

using namespace mxb;

static int prep_check(const mxb_fused_decode_prep_args* a) {
  MXB_REQUIRE(a != nullptr, MXB_ERR_INVALID, "fused decode prep: null args");
  MXB_REQUIRE(a->n_heads >= 1 && a->n_heads <= 64, MXB_ERR_INVALID, "q_idx must carry between 1 and 64 heads");
  MXB_REQUIRE(a->topk > 0 && a->topk < a->n_rows, MXB_ERR_INVALID, "topk must be positive and smaller than n_rows");
  MXB_REQUIRE(a->q_dtype == MXB_F32 || a->q_dtype == MXB_F16 || a->q_dtype == MXB_BF16, MXB_ERR_INVALID,
              "q_idx must be float32, float16, or bfloat16");
  return MXB_OK;
}

extern "C" int64_t mxb_fused_decode_prep_workspace_bytes(const mxb_fused_decode_prep_args* a) {
  if (prep_check(a) != MXB_OK) return 0;
  Carver ws{nullptr};
  ws.take((int64_t)a->n_heads * kIdxDim * 4);
  ws.take((int64_t)a->n_heads * 4);
  ws.take(mxb_topk_workspace_bytes(1, a->n_rows, a->topk));
  return ws.used;
}

extern "C" int mxb_fused_decode_prep(const mxb_fused_decode_prep_args* a, void* stream) {
  int rc = prep_check(a);
  if (rc != MXB_OK) return rc;
  MXB_REQUIRE(a->q_idx && a->pooled_qat && a->weights && a->kv_row && a->inv_freq && a->params && a->sel && a->row && a->scores,
              MXB_ERR_INVALID, "fused decode prep: null tensor");
  const int64_t need = mxb_fused_decode_prep_workspace_bytes(a);
  MXB_REQUIRE(a->workspace && a->workspace_bytes >= need && (reinterpret_cast<uintptr_t>(a->workspace) & 255) == 0,
              MXB_ERR_WORKSPACE, "fused decode prep: 256-byte aligned workspace of %lld bytes required", (long long)need);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  Carver ws{reinterpret_cast<uint8_t*>(a->workspace)};
  DecodePrepParams p{};
  p.q = a->q_idx; p.weights = a->weights; p.kv_row = reinterpret_cast<const __half*>(a->kv_row);
  p.inv_freq = a->inv_freq; p.token = {a->params, a->params_int64}; p.scale = a->scale; p.H = a->n_heads;
  p.q_qat = reinterpret_cast<float*>(ws.take((int64_t)a->n_heads * kIdxDim * 4));
  p.w_scaled = reinterpret_cast<float*>(ws.take((int64_t)a->n_heads * 4));
  p.row = reinterpret_cast<__half*>(a->row);
  const int64_t topk_bytes = mxb_topk_workspace_bytes(1, a->n_rows, a->topk);
  void* topk_ws = ws.take(topk_bytes);
  const unsigned grid = (unsigned)ceil_div(a->n_heads + 3, 4);
  auto* prep = a->q_dtype == MXB_F32   ? decode_prep_kernel<MXB_F32>
               : a->q_dtype == MXB_F16 ? decode_prep_kernel<MXB_F16>
                                       : decode_prep_kernel<MXB_BF16>;
  MXB_CUDA_OK(launch_early(prep, dim3(grid), 128, 0, st, p));
  note_launch();

  mxb_indexer_scores_args s{};
  s.q = p.q_qat; s.q_dtype = MXB_F32;
  s.q_stride_b = (int64_t)a->n_heads * kIdxDim; s.q_stride_h = kIdxDim; s.q_stride_t = kIdxDim;
  s.keys = a->pooled_qat; s.key_dtype = MXB_F32; s.weights = p.w_scaled; s.scores = a->scores;
  s.score_stride_b = a->n_rows; s.score_stride_t = a->n_rows;
  s.B = 1; s.T = 1; s.H = a->n_heads; s.D = kIdxDim; s.n_rows = a->n_rows; s.rows_total = a->n_rows;
  s.flags = MXB_INDEXER_EXACT_FP32;
  rc = mxb_indexer_scores(&s, stream);
  if (rc != MXB_OK) return rc;

  mxb_topk_args t{};
  t.scores = a->scores; t.row_stride = a->n_rows; t.out_ids = a->sel; t.rows = 1; t.n = a->n_rows; t.k = a->topk;
  t.workspace = topk_bytes > 0 ? topk_ws : nullptr; t.workspace_bytes = topk_bytes;
  return mxb_topk_select(&t, stream);
}

// the attention call behind the prepared operands
static mxb_sparse_attn_args sdpa_attention(const mxb_fused_decode_sdpa_args* a) {
  mxb_sparse_attn_args s{};
  s.q_dtype = MXB_F16;
  s.q_stride_b = (int64_t)a->n_heads * kRowDim; s.q_stride_h = kRowDim; s.q_stride_t = kRowDim;
  s.comp_kv = a->pooled; s.kv_dtype = MXB_F16; s.n_comp = a->n_rows;
  s.raw_cap = a->window_rows;
  s.topk = a->sel; s.k = a->topk;
  s.out = a->out; s.out_dtype = MXB_F16;
  s.out_stride_b = (int64_t)a->n_heads * kRowDim; s.out_stride_h = kRowDim; s.out_stride_t = kRowDim;
  s.B = 1; s.T = 1; s.H = a->n_heads; s.Dqk = kRowDim; s.Dv = kRowDim; s.scale = a->scale;
  return s;
}

extern "C" int64_t mxb_fused_decode_sdpa_workspace_bytes(const mxb_fused_decode_sdpa_args* a) {
  if (!a || a->n_heads < 1 || a->window_rows < 0) return 0;
  const mxb_sparse_attn_args s = sdpa_attention(a);
  Carver ws{nullptr};
  ws.take((int64_t)a->n_heads * kRowDim * 2);
  ws.take((int64_t)a->window_rows * kRowDim * 2);
  ws.take((int64_t)a->n_heads * 4);
  ws.take(8);
  ws.take(mxb_sparse_attn_workspace_bytes(&s));
  return ws.used;
}

extern "C" int mxb_fused_decode_sdpa(const mxb_fused_decode_sdpa_args* a, void* stream) {
  MXB_REQUIRE(a != nullptr, MXB_ERR_INVALID, "fused decode sdpa: null args");
  MXB_REQUIRE(a->n_heads >= 1 && a->window_rows >= 0 && a->topk >= 0 && a->n_rows >= 0, MXB_ERR_INVALID,
              "fused decode sdpa: sizes must not be negative, and q must carry at least one head");
  MXB_REQUIRE(a->q && a->row && a->sinks && a->inv_freq && a->params && a->out && (a->window_rows == 0 || a->window),
              MXB_ERR_INVALID, "fused decode sdpa: null tensor");
  const int64_t need = mxb_fused_decode_sdpa_workspace_bytes(a);
  MXB_REQUIRE(a->workspace && a->workspace_bytes >= need && (reinterpret_cast<uintptr_t>(a->workspace) & 255) == 0,
              MXB_ERR_WORKSPACE, "fused decode sdpa: 256-byte aligned workspace of %lld bytes required", (long long)need);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  mxb_sparse_attn_args s = sdpa_attention(a);
  Carver ws{reinterpret_cast<uint8_t*>(a->workspace)};
  SdpaPrepParams p{};
  p.q = reinterpret_cast<const __half*>(a->q); p.window = reinterpret_cast<const __half*>(a->window);
  p.row = reinterpret_cast<const __half*>(a->row); p.sinks = reinterpret_cast<const __half*>(a->sinks);
  p.inv_freq = a->inv_freq; p.token = {a->params, a->params_int64}; p.H = a->n_heads; p.W = a->window_rows;
  p.q_roped = reinterpret_cast<__half*>(ws.take((int64_t)a->n_heads * kRowDim * 2));
  p.keys = reinterpret_cast<__half*>(ws.take((int64_t)a->window_rows * kRowDim * 2));
  p.sinks_f = reinterpret_cast<float*>(ws.take((int64_t)a->n_heads * 4));
  p.pos0 = reinterpret_cast<int64_t*>(ws.take(8));
  const int64_t attn_bytes = mxb_sparse_attn_workspace_bytes(&s);
  s.workspace = ws.take(attn_bytes);
  s.workspace_bytes = attn_bytes;
  MXB_CUDA_OK(launch_early(decode_sdpa_prep_kernel, dim3((unsigned)ceil_div((int64_t)a->n_heads + a->window_rows + 1, 4)), 128, 0,
                           st, p));
  note_launch();
  s.q = p.q_roped;
  s.raw_kv = a->window_rows > 0 ? p.keys : nullptr;
  s.sinks = p.sinks_f;
  s.pos0_dev = p.pos0;
  int rc = mxb_sparse_attn(&s, stream);
  if (rc != MXB_OK) return rc;
  MXB_CUDA_OK(launch_early(decode_unrope_kernel, dim3((unsigned)ceil_div(a->n_heads, 4)), 128, 0, st,
                           reinterpret_cast<__half*>(a->out), a->inv_freq, p.token, a->n_heads));
  note_launch();
  return MXB_OK;
}
