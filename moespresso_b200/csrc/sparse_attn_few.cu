// Indexed mixed (sparse) attention for a few tokens: a latency problem, not a throughput one.
//
// One token's list of 512 to 2,048 rows is 0.15 to 0.3 GFLOP and 0.3 to 2.4 MB, and the tensor-core kernel for many
// tokens (sparse_attn_tc.cu: all 64 heads and at least two 64-row units per CTA) spends 17 to 23 us on it with 12 to 16
// CTAs: a serial chain of set-up, list scan, gather, 36 logit MMAs at M = 64, softmax, rescale, P V and the merge of 128 KB
// of partials per split.  Here a token is cut finer, by heads as well as by rows: CTA = (token, 16 heads, 64 to 256 list
// rows), the row splits of a head group form one thread-block cluster (up to 16 CTAs), and nothing is pipelined because
// nothing repeats:
//
//   q once into shared memory (int8 rows: scaled, two heads per warp) and from there into every warp's registers, before
//   the selection is waited for (eight warps loading the fragments from global memory took 4,000 cycles, int8 7,700)
//   list ids -> rows; every warp fetches its own eight rows of every 64 (16-byte asynchronous copies) and multiplies them
//   as soon as they are there:  S[16 heads x 8 rows] = Q . K^T
//   softmax over the CTA's rows with their exact maximum
//   O[16 heads x 64 features per warp] = P . V
//   (m, l) to every CTA of the cluster and O, unweighted, to the CTA that owns the features; one cluster barrier;
//   the owner weights and adds the splits in split order, the sink joining once, and writes the output.
//
// The contractions are warp-level MMAs (m16n8k16, fp32 accumulation): with 16 heads, 64 rows and one pass, the operands
// are used once, an MMA's result is needed at once, and a tcgen05.mma of this size would be a round trip through
// shared-memory descriptors, TMEM and two barriers for 0.5 us of arithmetic.  The rows of a head group are fetched by four
// CTAs instead of one; they come from L2 and the SMs would idle otherwise.
//
// The operand registers hold features under a permutation that both sides share: inside a 64-feature block lane t of a quad
// takes 16 consecutive features, four MMA steps of four, so that a lane's operands of a whole block are 32 (int8: 16)
// consecutive bytes of a row.
//
// int8 rows: bytes become fp16 integers exactly (0x6400 | u = 1024 + u).  q is scaled per head by a power of two so that its
// largest element lies in [2^14, 2^15), or by 2^126 if it is below 2^-112: a 16-bit q is then an fp16 number exactly, but for
// elements below 2^-28 of the largest.  The row's scale is folded into the logit and into P, as in the kernel for many tokens:
// the references follow logit + log2(scale), the denominator takes the rounded weights divided by the scale.
//
// What bounds it: latency, front to back (launch, list, rows, two contractions of one pass, cluster barrier, output); a
// further 64 rows per CTA cost 2 us.  Both sides measured: at the rule in launch_sparse_few.
#include "common.cuh"
#include "ptx_sm100.cuh"
#include "sparse_attn.cuh"

namespace mxb {

constexpr int kFewHeads = 16;     // heads of a CTA (M of the MMAs)
constexpr int kFewThreads = 256;
constexpr int kFewDv = 512;       // eight warps of 64 features
constexpr int kFewMaxSplits = 16; // CTAs of a cluster
constexpr int kFewBlk = 32;       // features that one CTA of the cluster owns at a time
constexpr int kFewBlkBytes = kFewHeads * kFewBlk * 4;

// List rows that a CTA can hold at most.
__host__ __device__ constexpr int few_max_rows(int eb) { return eb == 1 ? 256 : 128; }

struct FewLayout {
  int row_pitch;    // bytes of a staged row: an odd multiple of 16, so that eight rows cover all banks
  int s_pitch;      // floats of a head's logits; its 16-bit weights are written over them
  int q_off;        // the 16 heads as operands: where partials arrive later
  int s_off, row_off, scale_off, recv_off, ml_off, fac_off, misc_off, total;
};
__host__ __device__ inline FewLayout few_layout(int Dqk, int eb, int rows, int splits) {
  FewLayout L;
  L.row_pitch = Dqk * eb + 16;
  L.s_pitch = rows + 4;
  L.s_off = rows * L.row_pitch;
  L.row_off = L.s_off + kFewHeads * L.s_pitch * 4;
  L.scale_off = L.row_off + rows * 8;
  L.recv_off = L.scale_off + (eb == 1 ? rows * 12 : 0);
  L.q_off = L.recv_off;
  L.ml_off = L.recv_off + (kFewDv / kFewBlk + splits - 1) / splits * splits * kFewBlkBytes;
  L.fac_off = L.ml_off + splits * kFewHeads * 8;
  L.misc_off = L.fac_off + splits * kFewHeads * 4;
  L.total = L.misc_off + 80;
  return L;
}

struct FewParams {
  SparseParams s;
  int32_t groups;   // of 16 heads
  int32_t rows;     // list entries of a CTA
  int32_t out_dtype, q_dtype;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  if constexpr (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float a, float b) {
  if constexpr (BF16) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}
// bytes (lo, hi) of x (already biased by 128) -> the two int8 values as fp16, exactly
template <int SEL>
__device__ __forceinline__ uint32_t i8_pair_f16(uint32_t x) {
  const uint32_t u = __byte_perm(x, 0x64646464u, SEL);
  const __half2 bias = __half2half2(__ushort_as_half((unsigned short)0x6480));   // 1024 + 128
  const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&u), bias);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float few_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// What token (b, t) sees, and entry e_lo + threadIdx.x of its list (raw window rows, then the selected rows) for the threads
// below R: the address of the row or null, int8 rows also the scale.  *keff becomes the number of selected entries before
// the walk ends (p.k on entry); returns the number of raw rows.  The list is all that the selection right before the launch
// writes: it is waited for here.
template <int ROW_BYTES, bool I8>
__device__ __forceinline__ int few_list(const SparseParams& p, int b, int t, const int32_t* ids, int e_lo, int R, int* keff,
                                        const uint8_t*& row, float& rs) {
  const int tid = threadIdx.x;
  const int64_t pos_b = p.pos0_dev ? p.pos0_dev[b] : p.pos0;
  const int64_t qpos = pos_b + t, last_pos = pos_b + p.T - 1;
  const int64_t count = p.comp_row_count ? (int64_t)p.comp_row_count[b] : p.n_comp;
  const int64_t cbase = p.comp_row_start ? p.comp_row_start[b] : (int64_t)b * p.n_comp;
  int64_t visible = count;
  if (p.ratio > 0) {
    visible = (qpos + 1) / p.ratio;
    if (visible > count) visible = count;
  }
  int64_t first_raw_pos = 0, first = 0;
  int n_raw = 0;
  if (p.raw_cap > 0) {
    first_raw_pos = last_pos + 1 - p.raw_cap;
    const int64_t window_first = (p.window != 0 && qpos + 1 > p.window) ? qpos + 1 - p.window : 0;
    first = first_raw_pos > window_first ? first_raw_pos : window_first;
    if (first < 0) first = 0;
    const int64_t last = qpos < last_pos ? qpos : last_pos;
    n_raw = last >= first ? (int)(last - first + 1) : 0;
  }
  if (p.after_select) ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();
  // whether the list ends before this CTA's rows is known only after the scan, but a row inside the visible range may be
  // looked at either way
  row = nullptr;
  rs = 1.f;
  if (tid < R) {
    const int e = e_lo + tid;
    int64_t r = -1;
    bool raw = false;
    if (e < n_raw) {
      r = (int64_t)b * p.raw_cap + ((int64_t)p.raw_start + (first + e - first_raw_pos)) % p.raw_cap;
      raw = true;
    } else if (e - n_raw < p.k) {
      const int32_t id = ids[e - n_raw];
      if (id >= 0 && (int64_t)id < visible) r = cbase + id;
    }
    if (r >= 0) {
      row = reinterpret_cast<const uint8_t*>(raw ? p.raw_kv : p.comp_kv) + r * ROW_BYTES;
      // (a zero scale, i.e. an all-zero row, still counts in the denominator: it is taken as fp16's smallest number)
      if (I8) rs = fmaxf(__half2float(raw ? p.raw_scales[r] : p.comp_scales[r]), 5.9604645e-8f);
    }
  }
  int mine = p.k;   // first list entry that ends the walk
  for (int j0 = tid; j0 < p.k; j0 += 8 * kFewThreads) {   // eight ids in flight
    int32_t v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = j0 + u * kFewThreads < p.k ? ids[j0 + u * kFewThreads] : -1;
#pragma unroll
    for (int u = 7; u >= 0; --u)
      if ((int64_t)v[u] >= visible && j0 + u * kFewThreads < mine) mine = j0 + u * kFewThreads;
  }
  if (mine < p.k) atomicMin(keff, mine);
  return n_raw;
}

// One split's share of its head, lane r of a half warp = split r: exp(m - m*) over the denominator of the whole token, the
// sink joining once, and m*, the denominator themselves (partial output: no sink, not divided).  LOG2: m and sink in log2
// units; otherwise in natural ones, which float32 tables keep (a product with log2(e) would round a large m).
template <bool LOG2>
__device__ __forceinline__ float few_weight(float2 ml, float sink2, bool partial, float& m2, float& den) {
  m2 = ml.x;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) m2 = fmaxf(m2, __shfl_xor_sync(0xffffffffu, m2, o));
  m2 = fmaxf(m2, sink2);
  auto e = [](float x) { return LOG2 ? exp2f(x) : expf(x); };
  const float w = ml.x == -INFINITY ? 0.f : e(ml.x - m2);
  den = ml.y * w;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);   // the same order on every run
  den += sink2 == -INFINITY ? 0.f : e(sink2 - m2);
  return w * (partial ? 1.f : den > 0.f ? 1.f / den : 0.f);
}

// NB: 64-feature blocks of a row (Dqk / 64).
template <int KVT, int NB>
__global__ void __launch_bounds__(kFewThreads, 1) sparse_attn_few_kernel(const __grid_constant__ FewParams fp) {
  constexpr bool I8 = KVT == MXB_I8, BF16 = KVT == MXB_BF16;
  constexpr int EB = I8 ? 1 : 2;
  constexpr int kChunks = NB * 64 * EB / 16;   // 16-byte pieces of a row
  constexpr int kMaxTiles = few_max_rows(EB) / 64;
  const SparseParams& p = fp.s;
  extern __shared__ __align__(16) uint8_t smem[];
  const int C = p.nsplit, R = fp.rows;
  const FewLayout L = few_layout(NB * 64, EB, R, C);
  float* s_s = reinterpret_cast<float*>(smem + L.s_off);
  const uint8_t** row_s = reinterpret_cast<const uint8_t**>(smem + L.row_off);   // [R] address of the row, or null
  float* scale_s = reinterpret_cast<float*>(smem + L.scale_off);                 // int8 rows, [R] each: scale,
  float* lscale_s = scale_s + R;                                                 //   its log2,
  float* iscale_s = lscale_s + R;                                                //   and its inverse
  const float* recv = reinterpret_cast<const float*>(smem + L.recv_off);
  float2* ml_s = reinterpret_cast<float2*>(smem + L.ml_off);
  float* fac_s = reinterpret_cast<float*>(smem + L.fac_off);
  int* keff_s = reinterpret_cast<int*>(smem + L.misc_off);
  float* qmul_s = reinterpret_cast<float*>(smem + L.misc_off + 16);   // [16] int8 rows: undoes the power of two that q was scaled by

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int split = (int)(blockIdx.x % (unsigned)C);
  const int unit = (int)(blockIdx.x / (unsigned)C);
  const int bt = unit / fp.groups, h0 = (unit - bt * fp.groups) * kFewHeads;
  const int b = bt / p.T, t = bt - b * p.T;
  if (!p.after_select) ptx::grid_dependency_wait();   // behind a selection q and all else but the list are complete
  const void* q_in = ptx::behind_wait(p.q);
  if (tid == 0) *keff_s = p.k;

  // ---- q: every warp turns two heads into operands in shared memory, then all warps read the fragments of all 16
  {
    constexpr int kQPitch = NB * 128 + 16;   // an odd multiple of 16 bytes
    uint8_t* q_s = smem + L.q_off;
    const bool vec = fp.q_dtype != MXB_F32 && ((reinterpret_cast<uintptr_t>(q_in) & 15) == 0) && p.q_sb % 8 == 0 &&
                     p.q_sh % 8 == 0 && p.q_st % 8 == 0;
    auto two = [&](uint32_t x) -> float2 {
      if (fp.q_dtype == MXB_BF16) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x));
      return __half22float2(*reinterpret_cast<const __half2*>(&x));
    };
    uint32_t w[2][3][4];   // [head][piece of eight features][pair]
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int h = h0 + 2 * warp + hh;
      const int64_t base = (int64_t)b * p.q_sb + (int64_t)h * p.q_sh + (int64_t)t * p.q_st;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int ck = c * 32 + lane;
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        if (h < p.H && ck < NB * 8) {
          if (vec) {
            x = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(q_in) + base) + ck);
          } else {
            uint32_t e4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int64_t at = base + 8 * ck + 2 * e;
              if (fp.q_dtype == MXB_F32) {
                e4[e] = pack16<BF16>(reinterpret_cast<const float*>(q_in)[at], reinterpret_cast<const float*>(q_in)[at + 1]);
              } else {
                const uint16_t* src = reinterpret_cast<const uint16_t*>(q_in) + at;
                e4[e] = (uint32_t)src[0] | ((uint32_t)src[1] << 16);
              }
            }
            x = make_uint4(e4[0], e4[1], e4[2], e4[3]);
          }
        }
        w[hh][c][0] = x.x; w[hh][c][1] = x.y; w[hh][c][2] = x.z; w[hh][c][3] = x.w;
      }
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      if constexpr (I8) {
        float amax = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 v = two(w[hh][c][e]);
            amax = fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y)));
          }
        amax = warp_max(amax);
        const int ex = (int)(__float_as_uint(amax) >> 23) - 127;   // floor(log2(max)); zeros and denormals: -127
        const int sh = min(14 - ex, 126);   // at least -114; 2^126 brings any 16-bit q to where fp16 holds all its bits
        const float up = __uint_as_float((uint32_t)(127 + sh) << 23);
        if (lane == 0) qmul_s[2 * warp + hh] = __uint_as_float((uint32_t)(127 - sh) << 23);
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 v = two(w[hh][c][e]);
            w[hh][c][e] = pack16<false>(v.x * up, v.y * up);
          }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int ck = c * 32 + lane;
        if (ck < NB * 8)
          *reinterpret_cast<uint4*>(q_s + (2 * warp + hh) * kQPitch + ck * 16) =
              make_uint4(w[hh][c][0], w[hh][c][1], w[hh][c][2], w[hh][c][3]);
      }
    }
  }
  __syncthreads();   // (the list's end is initialised, too)
  uint32_t qf[NB][4][4];        // fragments: [block][step][A registers]
  float q_mul[2] = {1.f, 1.f};
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const uint8_t* qrow = smem + L.q_off + (g + 8 * hh) * (NB * 128 + 16) + 32 * t4;
    if constexpr (I8) q_mul[hh] = qmul_s[g + 8 * hh];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const uint4 x = *reinterpret_cast<const uint4*>(qrow + i * 128), y = *reinterpret_cast<const uint4*>(qrow + i * 128 + 16);
      qf[i][0][hh] = x.x; qf[i][0][2 + hh] = x.y;
      qf[i][1][hh] = x.z; qf[i][1][2 + hh] = x.w;
      qf[i][2][hh] = y.x; qf[i][2][2 + hh] = y.y;
      qf[i][3][hh] = y.z; qf[i][3][2 + hh] = y.w;
    }
  }
  // (0) Every CTA of the cluster has started and has read its q out of the place where partials arrive: waited for before
  // the first remote store.
  ptx::cluster_arrive();

  const int e_lo = split * R;
  const int32_t* ids = p.topk + (int64_t)bt * p.k;
  int n_raw;
  {
    const uint8_t* row;
    float rs;
    n_raw = few_list<NB * 64 * EB, I8>(p, b, t, ids, e_lo, R, keff_s, row, rs);
    if (tid < R) {
      row_s[tid] = row;
      if constexpr (I8) {
        scale_s[tid] = rs;
        lscale_s[tid] = log2f(rs);
        iscale_s[tid] = __frcp_rn(rs);
      }
    }
  }
  __syncthreads();
  const int e_end = n_raw + *keff_s;   // entries of the list

  // ---- every warp fetches its own rows: row tile i holds rows 64 i + 8 warp .. + 7
  const int tiles = R >> 6;
  const uint32_t row0 = ptx::smem_u32(smem);
  const int live = e_end - e_lo;   // entries before the list's end
  auto row_ok = [&](int r) { return row_s[r] != nullptr && r < live; };
  for (int i = 0; i < tiles; ++i) {
    int rr = lane / kChunks, ck = lane % kChunks;   // (a row is 32 to 72 pieces)
#pragma unroll
    for (int c0 = 0; c0 < 8 * kChunks; c0 += 32) {
      const int r = i * 64 + warp * 8 + rr;
      const uint32_t dst = row0 + (uint32_t)(r * L.row_pitch + ck * 16);
      const uint8_t* row = r < live ? row_s[r] : nullptr;
      const int at = ck * 16;
      ck += 32;
      if (ck >= kChunks) {
        ck -= kChunks;
        ++rr;
      }
      if (row) {
        cp_async16(dst, row + at);
      } else {
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0u) : "memory");   // zeros: 0 weight x 0
      }
    }
    cp_async_commit();
  }

  // ---- S = Q K^T for the warp's rows
  const float scale_log2 = p.scale * 1.4426950408889634f;
  for (int i = 0; i < tiles; ++i) {
    if (i + 1 == tiles) cp_async_wait<0>();
    else if (i + 2 == tiles) cp_async_wait<1>();
    else if (i + 3 == tiles) cp_async_wait<2>();
    else cp_async_wait<3>();
    __syncwarp();
    const int rt = i * 64 + warp * 8;
    const uint8_t* krow = smem + (size_t)(rt + g) * L.row_pitch + 16 * EB * t4;
    float acc[4][4];
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[s][e] = 0.f;
#pragma unroll
    for (int blk = 0; blk < NB; ++blk) {
      uint32_t kf[8];
      if constexpr (I8) {
        const uint4 x = *reinterpret_cast<const uint4*>(krow + blk * 64);
        const uint32_t xs[4] = {x.x ^ 0x80808080u, x.y ^ 0x80808080u, x.z ^ 0x80808080u, x.w ^ 0x80808080u};
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          kf[2 * s] = i8_pair_f16<0x4140>(xs[s]);
          kf[2 * s + 1] = i8_pair_f16<0x4342>(xs[s]);
        }
      } else {
        const uint4 x = *reinterpret_cast<const uint4*>(krow + blk * 128), y = *reinterpret_cast<const uint4*>(krow + blk * 128 + 16);
        kf[0] = x.x; kf[1] = x.y; kf[2] = x.z; kf[3] = x.w;
        kf[4] = y.x; kf[5] = y.y; kf[6] = y.z; kf[7] = y.w;
      }
#pragma unroll
      for (int s = 0; s < 4; ++s)   // four accumulators: an MMA waits for the one four before it
        mma_16816<BF16>(acc[s], qf[blk][s][0], qf[blk][s][1], qf[blk][s][2], qf[blk][s][3], kf[2 * s], kf[2 * s + 1]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = rt + 2 * t4 + (e & 1), h = g + 8 * (e >> 1);
      float x = (acc[0][e] + acc[1][e]) + (acc[2][e] + acc[3][e]);
      if constexpr (I8) {
        x = fmaf(x, scale_log2 * q_mul[e >> 1] * scale_s[r], lscale_s[r]);
      } else {
        x *= scale_log2;
      }
      s_s[h * L.s_pitch + r] = row_ok(r) ? x : -INFINITY;
    }
  }
  __syncthreads();

  // ---- softmax: a warp takes two heads; the 16-bit weights go over the logits they came from
  float2 my_ml = make_float2(-INFINITY, 0.f);   // lane 0 / 1: of head 2 warp / 2 warp + 1
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    float* srow = s_s + (2 * warp + hh) * L.s_pitch;
    float x[2 * kMaxTiles];   // rows 2 lane, 2 lane + 1 of each 64
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < kMaxTiles; ++i) {
      float2 v = make_float2(-INFINITY, -INFINITY);
      if (i < tiles) v = *reinterpret_cast<const float2*>(srow + i * 64 + 2 * lane);
      x[2 * i] = v.x;
      x[2 * i + 1] = v.y;
      m = fmaxf(m, fmaxf(v.x, v.y));
    }
    m = warp_max(m);
    __syncwarp();
    float l = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxTiles; ++i) {
      if (i >= tiles) break;
      const float a = x[2 * i] == -INFINITY ? 0.f : few_exp2(x[2 * i] - m);
      const float c = x[2 * i + 1] == -INFINITY ? 0.f : few_exp2(x[2 * i + 1] - m);
      const uint32_t w = pack16<BF16>(a, c);
      reinterpret_cast<uint32_t*>(srow)[i * 32 + lane] = w;
      float2 back;   // the weights as the operand holds them
      if constexpr (BF16) back = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
      else back = __half22float2(*reinterpret_cast<const __half2*>(&w));
      if constexpr (I8) {
        const float2 inv = *reinterpret_cast<const float2*>(iscale_s + i * 64 + 2 * lane);
        l = fmaf(back.x, inv.x, l);
        l = fmaf(back.y, inv.y, l);
      } else {
        l += back.x + back.y;
      }
    }
    l = warp_sum(l);
    if (lane == hh) my_ml = make_float2(m, l);
  }
  __syncthreads();

  // ---- O = P V: a warp's 64 features, all rows
  float o[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
  const uint32_t p0 = ptx::smem_u32(s_s) + (uint32_t)((lane & 15) * L.s_pitch * 4 + (lane >> 4) * 16);
  for (int ks = 0; ks < R / 16; ++ks) {
    uint32_t a[4];
    ldsm_x4(p0 + (uint32_t)(ks * 32), a);
    if constexpr (I8) {
      // lane (g, t4): n-tile j of a 32-feature block holds feature 4 g + j, rows 2 t4, + 1 (b0) and + 8, + 9 (b1)
      const uint8_t* v = smem + (size_t)(ks * 16 + 2 * t4) * L.row_pitch + warp * 64 + 4 * g;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(v + q * 32) ^ 0x80808080u;
        const uint32_t w1 = *reinterpret_cast<const uint32_t*>(v + q * 32 + L.row_pitch) ^ 0x80808080u;
        const uint32_t w2 = *reinterpret_cast<const uint32_t*>(v + q * 32 + 8 * L.row_pitch) ^ 0x80808080u;
        const uint32_t w3 = *reinterpret_cast<const uint32_t*>(v + q * 32 + 9 * L.row_pitch) ^ 0x80808080u;
        const uint32_t x01 = __byte_perm(w0, w1, 0x5140), x23 = __byte_perm(w0, w1, 0x7362);
        const uint32_t y01 = __byte_perm(w2, w3, 0x5140), y23 = __byte_perm(w2, w3, 0x7362);
        mma_16816<false>(o[4 * q], a[0], a[1], a[2], a[3], i8_pair_f16<0x4140>(x01), i8_pair_f16<0x4140>(y01));
        mma_16816<false>(o[4 * q + 1], a[0], a[1], a[2], a[3], i8_pair_f16<0x4342>(x01), i8_pair_f16<0x4342>(y01));
        mma_16816<false>(o[4 * q + 2], a[0], a[1], a[2], a[3], i8_pair_f16<0x4140>(x23), i8_pair_f16<0x4140>(y23));
        mma_16816<false>(o[4 * q + 3], a[0], a[1], a[2], a[3], i8_pair_f16<0x4342>(x23), i8_pair_f16<0x4342>(y23));
      }
    } else {
      // matrices of eight rows x eight features: rows 0-7 / 8-15 of the step, two n-tiles at a time
      const uint32_t v = row0 + (uint32_t)((ks * 16 + (lane & 15)) * L.row_pitch + warp * 128 + (lane >> 4) * 16);
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        uint32_t bv[4];
        ldsm_x4_trans(v + (uint32_t)(j * 16), bv);
        mma_16816<BF16>(o[j], a[0], a[1], a[2], a[3], bv[0], bv[1]);
        mma_16816<BF16>(o[j + 1], a[0], a[1], a[2], a[3], bv[2], bv[3]);
      }
    }
  }

  // ---- partials to their owners: block x of 32 features belongs to CTA x % C
  ptx::cluster_wait();   // (0)
  {
    const uint32_t recv0 = ptx::smem_u32(recv);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int blk = 2 * warp + q;
      const uint32_t dst = ptx::cluster_map(recv0 + (uint32_t)(((blk / C) * C + split) * kFewBlkBytes + lane * 16), (uint32_t)(blk % C));
#pragma unroll
      for (int j = 0; j < 4; ++j)
        ptx::st_cluster_v4(dst + (uint32_t)(j * 512), o[4 * q + j][0], o[4 * q + j][1], o[4 * q + j][2], o[4 * q + j][3]);
    }
    const uint32_t ml0 = ptx::smem_u32(ml_s + split * kFewHeads + 2 * warp);
    const float m0 = __shfl_sync(0xffffffffu, my_ml.x, lane & 1), l0 = __shfl_sync(0xffffffffu, my_ml.y, lane & 1);
    if (lane < 2 * C) {   // lane i: head i & 1 of this warp to CTA i / 2 (at most 16)
      const uint32_t dst = ptx::cluster_map(ml0 + (uint32_t)((lane & 1) * 8), (uint32_t)(lane >> 1));
      ptx::st_cluster_f32(dst, m0);
      ptx::st_cluster_f32(dst + 4, l0);
    }
  }
  __syncwarp();
  ptx::cluster_arrive();   // (1) everything has arrived; nothing remote is touched after this
  ptx::cluster_wait();

  // ---- weights: exp2(m - m*) over the denominator of the whole token, the sink joining once
  {   // half a warp per head, a lane per split
    const int hl = 2 * warp + (lane >> 4), r = lane & 15, h = h0 + hl;
    const bool partial = p.partial_ml != nullptr;   // un-normalised output and (m, l): the sink joins in the caller's merge
    const float sink2 = (p.sinks && h < p.H && !partial) ? p.sinks[h] * 1.4426950408889634f : -INFINITY;
    const float2 v = r < C ? ml_s[r * kFewHeads + hl] : make_float2(-INFINITY, 0.f);
    float m2, den;
    const float f = few_weight<true>(v, sink2, partial, m2, den);
    if (partial && split == 0 && r == 0 && h < p.H)
      *reinterpret_cast<float2*>(p.partial_ml + ((int64_t)bt * p.H + h) * 2) = make_float2(m2 * 0.6931471805599453f, den);
    if (r < C) fac_s[r * kFewHeads + hl] = f;
  }
  __syncthreads();
  const int64_t ob = (int64_t)b * p.o_sb + (int64_t)t * p.o_st;
  for (int x = tid; ; x += kFewThreads) {   // item: (block, n-tile, lane) as its MMA left it
    const int slot = x >> 7, blk = slot * C + split;
    if (blk >= kFewDv / kFewBlk) break;
    const int j = (x >> 5) & 3;
    const float4* src = reinterpret_cast<const float4*>(recv) + (size_t)slot * C * 128 + (x & 127);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int r = 0; r < C; ++r) {
      const float4 v = src[(size_t)r * 128];
      const float f0 = fac_s[r * kFewHeads + g], f1 = fac_s[r * kFewHeads + g + 8];
      acc.x = fmaf(v.x, f0, acc.x); acc.y = fmaf(v.y, f0, acc.y);
      acc.z = fmaf(v.z, f1, acc.z); acc.w = fmaf(v.w, f1, acc.w);
    }
    const float v4[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int n = 2 * t4 + (e & 1);   // column of the n-tile
      const int d = blk * kFewBlk + (I8 ? 4 * n + j : 8 * j + n), h = h0 + g + 8 * (e >> 1);
      if (h < p.H) {
        const int64_t at = ob + (int64_t)h * p.o_sh + d;
        if (fp.out_dtype == MXB_F32) store_elem<MXB_F32>(p.out, at, v4[e]);
        else if (fp.out_dtype == MXB_F16) store_elem<MXB_F16>(p.out, at, v4[e]);
        else store_elem<MXB_BF16>(p.out, at, v4[e]);
      }
    }
  }
}

// float32 tables and queries: the same cut with HG heads and up to 64 rows per CTA, on the FMA pipe.  Bound by latency and by
// shared-memory reads (a row once for HG heads).  The kernel of sparse_attn.cu walks 32-row tiles with eight heads a CTA, a
// chain of staging, dots, softmax and values per tile, and leaves partials to a merge kernel: k = 512, 64 heads of 576, 20.6
// and 5 us, a float32 decode step over 4,096 rows 33.1 us; with this kernel 18.8.  Relative error
// against float64 2.3e-7 (the other kernel 2.9e-7 to 3.7e-7).
template <int HG>
struct FewF32Layout {
  static constexpr int kRows = 64, kHP = (HG + 3) / 4 * 4;
  int pitch;        // floats of a staged row: + 16 bytes, so that eight rows cover all banks
  int q_off, part_off, p_off, row_off, recv_off, ml_off, fac_off, misc_off, total;
  __host__ __device__ FewF32Layout(int Dqk, int splits) {
    pitch = Dqk + 4;
    q_off = kRows * pitch * 4;
    part_off = q_off + HG * Dqk * 4;
    p_off = part_off + 4 * HG * kRows * 4;
    row_off = p_off + kRows * kHP * 4;
    recv_off = row_off + kRows * 8;
    ml_off = recv_off + (kFewDv / kFewBlk + splits - 1) / splits * splits * HG * kFewBlk * 4;
    fac_off = ml_off + splits * HG * 8;
    misc_off = (fac_off + splits * HG * 4 + 15) / 16 * 16;
    total = misc_off + 16;
  }
};

template <int NB, int HG>
__global__ void __launch_bounds__(kFewThreads, 1) sparse_attn_few_f32_kernel(const __grid_constant__ FewParams fp) {
  using Lay = FewF32Layout<HG>;
  constexpr int R = Lay::kRows, HP = Lay::kHP, D = NB * 64;
  constexpr int kChunks = D / 4;   // 16-byte pieces of a row
  const SparseParams& p = fp.s;
  extern __shared__ __align__(16) uint8_t smem[];
  const int C = p.nsplit;
  const Lay L(D, C);
  const float* rows_s = reinterpret_cast<const float*>(smem);
  float* q_s = reinterpret_cast<float*>(smem + L.q_off);         // [HG][D]
  float* part_s = reinterpret_cast<float*>(smem + L.part_off);   // [4 feature quarters][HG][R]
  float* p_s = reinterpret_cast<float*>(smem + L.p_off);         // [R][HP]
  const uint8_t** row_s = reinterpret_cast<const uint8_t**>(smem + L.row_off);
  const float* recv = reinterpret_cast<const float*>(smem + L.recv_off);   // [slot][split][HG][32]
  float2* ml_s = reinterpret_cast<float2*>(smem + L.ml_off);     // [split][HG]
  float* fac_s = reinterpret_cast<float*>(smem + L.fac_off);     // [split][HG]
  int* keff_s = reinterpret_cast<int*>(smem + L.misc_off);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int split = (int)(blockIdx.x % (unsigned)C);
  const int unit = (int)(blockIdx.x / (unsigned)C);
  const int bt = unit / fp.groups, h0 = (unit - bt * fp.groups) * HG;
  const int b = bt / p.T, t = bt - b * p.T;
  if (!p.after_select) ptx::grid_dependency_wait();   // behind a selection q and all else but the list are complete
  const float* q_in = reinterpret_cast<const float*>(ptx::behind_wait(p.q));
  ptx::cluster_arrive();   // (0) every CTA of the cluster has started: waited for before the first remote store
  if (tid == 0) *keff_s = p.k;
  {
    const int64_t qbase = (int64_t)b * p.q_sb + (int64_t)t * p.q_st;
#pragma unroll 4
    for (int i = tid; i < HG * D; i += kFewThreads) {
      const int hl = i / D, h = h0 + hl;
      q_s[i] = h < p.H ? q_in[qbase + (int64_t)h * p.q_sh + (i - hl * D)] : 0.f;
    }
  }
  __syncthreads();   // the list's end is initialised
  const int e_lo = split * R;
  const uint8_t* my_row;
  float unused;
  const int n_raw = few_list<D * 4, false>(p, b, t, p.topk + (int64_t)bt * p.k, e_lo, R, keff_s, my_row, unused);
  if (tid < R) row_s[tid] = my_row;
  __syncthreads();
  const int live = n_raw + *keff_s - e_lo;   // entries before the list's end

  // ---- a warp fetches eight rows
  {
    const uint32_t row0 = ptx::smem_u32(smem);
    int rr = 0, ck = lane;
#pragma unroll 12
    for (int c0 = 0; c0 < 8 * kChunks; c0 += 32) {
      const int r = warp * 8 + rr;
      const uint32_t dst = row0 + (uint32_t)(r * L.pitch * 4 + ck * 16);
      const uint8_t* row = r < live ? row_s[r] : nullptr;
      const int at = ck * 16;
      ck += 32;
      if (ck >= kChunks) {
        ck -= kChunks;
        ++rr;
      }
      if (row) cp_async16(dst, row + at);
      else asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0u) : "memory");
    }
    cp_async_commit();
    cp_async_wait<0>();
  }
  __syncthreads();

  // ---- S: thread = (row, quarter of the features), all heads
  {
    const int r = (warp & 1) * 32 + lane, quarter = warp >> 1;
    constexpr int N4 = D / 16;   // float4 of a quarter
    const float4* kr = reinterpret_cast<const float4*>(rows_s + r * L.pitch) + quarter * N4;
    const float4* qr = reinterpret_cast<const float4*>(q_s) + quarter * N4;
    float2 acc[HG];   // even and odd features
#pragma unroll
    for (int h = 0; h < HG; ++h) acc[h] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int c = 0; c < N4; ++c) {
      const float4 k4 = kr[c];
#pragma unroll
      for (int h = 0; h < HG; ++h) {
        const float4 x = qr[h * (D / 4) + c];
        acc[h] = __ffma2_rn(make_float2(x.x, x.y), make_float2(k4.x, k4.y), acc[h]);
        acc[h] = __ffma2_rn(make_float2(x.z, x.w), make_float2(k4.z, k4.w), acc[h]);
      }
    }
#pragma unroll
    for (int h = 0; h < HG; ++h) part_s[(quarter * HG + h) * R + r] = acc[h].x + acc[h].y;
  }
  __syncthreads();

  // ---- softmax: a warp takes heads warp, warp + 8; (m, l) go to every CTA of the cluster
  ptx::cluster_wait();   // (0)
  for (int h = warp; h < HG; h += 8) {
    float x[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = i * 32 + lane;
      const float dot = (part_s[h * R + r] + part_s[(HG + h) * R + r]) + (part_s[(2 * HG + h) * R + r] + part_s[(3 * HG + h) * R + r]);
      x[i] = row_s[r] != nullptr && r < live ? dot * p.scale : -INFINITY;
    }
    const float m = warp_max(fmaxf(x[0], x[1]));
    float l = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float w = x[i] == -INFINITY ? 0.f : expf(x[i] - m);
      p_s[(i * 32 + lane) * HP + h] = w;
      l += w;
    }
    l = warp_sum(l);
    if (lane < C) {
      const uint32_t dst = ptx::cluster_map(ptx::smem_u32(ml_s + split * HG + h), (uint32_t)lane);
      ptx::st_cluster_f32(dst, m);
      ptx::st_cluster_f32(dst + 4, l);
    }
  }
  __syncthreads();

  // ---- O: thread = two features, all heads
  float2 o[HG];
#pragma unroll
  for (int h = 0; h < HG; ++h) o[h] = make_float2(0.f, 0.f);
  const int n_rows = min(R, max(live, 0));   // (the rows behind them weigh nothing)
#pragma unroll 4
  for (int r = 0; r < n_rows; ++r) {
    const float2 v = *reinterpret_cast<const float2*>(rows_s + r * L.pitch + 2 * tid);
    float w[HP];
#pragma unroll
    for (int i = 0; i < HP; i += 4) *reinterpret_cast<float4*>(&w[i]) = *reinterpret_cast<const float4*>(p_s + r * HP + i);
#pragma unroll
    for (int h = 0; h < HG; ++h) o[h] = __ffma2_rn(make_float2(w[h], w[h]), v, o[h]);
  }
  {
    const int blk = tid >> 4;   // block of 32 features, of CTA blk % C
    const uint32_t dst = ptx::cluster_map(
        ptx::smem_u32(recv + (size_t)((blk / C) * C + split) * HG * kFewBlk + ((2 * tid) & (kFewBlk - 1))), (uint32_t)(blk % C));
#pragma unroll
    for (int h = 0; h < HG; ++h)
      asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(dst + (uint32_t)(h * kFewBlk * 4)), "f"(o[h].x), "f"(o[h].y)
                   : "memory");
  }
  __syncwarp();
  ptx::cluster_arrive();   // (1) everything has arrived; nothing remote is touched after this
  ptx::cluster_wait();
  for (int h1 = 2 * warp; h1 < HG; h1 += 16) {   // (the same trips for both halves of a warp)
    const int hl = h1 + (lane >> 4), r = lane & 15, h = h0 + hl;
    const bool partial = p.partial_ml != nullptr, on = hl < HG;
    const float sink = (p.sinks && on && h < p.H && !partial) ? p.sinks[h] : -INFINITY;
    const float2 v = on && r < C ? ml_s[r * HG + hl] : make_float2(-INFINITY, 0.f);
    float m2, den;
    const float f = few_weight<false>(v, sink, partial, m2, den);
    if (partial && on && split == 0 && r == 0 && h < p.H)
      *reinterpret_cast<float2*>(p.partial_ml + ((int64_t)bt * p.H + h) * 2) = make_float2(m2, den);
    if (on && r < C) fac_s[r * HG + hl] = f;
  }
  __syncthreads();
  const int64_t ob = (int64_t)b * p.o_sb + (int64_t)t * p.o_st;
  for (int x = tid;; x += kFewThreads) {   // item: (slot, head, feature of the block)
    const int slot = x / (HG * kFewBlk), i = x - slot * (HG * kFewBlk), blk = slot * C + split;
    if (blk >= kFewDv / kFewBlk) break;
    const int hl = i / kFewBlk, h = h0 + hl;
    const float* src = recv + (size_t)slot * C * HG * kFewBlk + i;
    float acc = 0.f;
#pragma unroll 4
    for (int r = 0; r < C; ++r) acc = fmaf(src[(size_t)r * HG * kFewBlk], fac_s[r * HG + hl], acc);
    if (h < p.H) {
      const int64_t at = ob + (int64_t)h * p.o_sh + blk * kFewBlk + (i & (kFewBlk - 1));
      if (fp.out_dtype == MXB_F32) store_elem<MXB_F32>(p.out, at, acc);
      else if (fp.out_dtype == MXB_F16) store_elem<MXB_F16>(p.out, at, acc);
      else store_elem<MXB_BF16>(p.out, at, acc);
    }
  }
}

// Which calls come here: splits left to the library, 512 values of 512 or 576 features.  int8 rows need a
// 16-bit q (a float32 one would be rounded to 11 bits; the other kernel keeps 15).
static bool sparse_few_eligible(const SparseParams& p, int kv_dtype, int q_dtype) {
  if (p.H < 1) return false;
  return p.may_split && p.Dv == kFewDv && (p.Dqk == 512 || p.Dqk == 576) && p.H <= 64 &&
         !(kv_dtype == MXB_I8 && q_dtype == MXB_F32);
}

// MXB_ERR_UNSUPPORTED: the clusters are not all resident at once, nothing was launched.  `cached`: how many are, 0 = not asked
// yet (one per kernel, device, shared memory and cluster size).
static int launch_few_kernel(void (*kern)(FewParams), const FewParams& fp, int smem, int clusters, int* cached, cudaStream_t st) {
  const int C = fp.s.nsplit;
  MXB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
  if (C > 8) MXB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * C));
  cfg.blockDim = dim3(kFewThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // (the kernel waits, see grid_chain)
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int resident = cached ? *cached : 0;
  if (resident == 0) {
    if (cudaOccupancyMaxActiveClusters(&resident, kern, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      resident = -1;
    }
    if (resident == 0) resident = -1;
    if (cached) *cached = resident;
  }
  if (resident < clusters) return MXB_ERR_UNSUPPORTED;
  cfg.numAttrs = 2;
  MXB_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, fp));
  note_launch();
  return MXB_OK;
}

template <int KVT, int NB>
static int launch_few_typed(const FewParams& fp, int smem, int clusters, cudaStream_t st) {
  static int resident[16][3][kFewMaxSplits + 1];   // rows 64, 128, 256
  int dev = 0;
  MXB_CUDA_OK(cudaGetDevice(&dev));
  int* cached = dev >= 0 && dev < 16 ? &resident[dev][fp.rows >> 7][fp.s.nsplit] : nullptr;
  return launch_few_kernel(sparse_attn_few_kernel<KVT, NB>, fp, smem, clusters, cached, st);
}

template <int NB, int HG>
static int launch_few_f32(FewParams fp, cudaStream_t st) {
  static int resident[16][kFewMaxSplits + 1];
  int dev = 0;
  MXB_CUDA_OK(cudaGetDevice(&dev));
  int* cached = dev >= 0 && dev < 16 ? &resident[dev][fp.s.nsplit] : nullptr;
  fp.groups = (fp.s.H + HG - 1) / HG;
  const int64_t clusters = (int64_t)fp.s.B * fp.s.T * fp.groups;
  const int smem = FewF32Layout<HG>(NB * 64, fp.s.nsplit).total;
  if (clusters * fp.s.nsplit > sm_count() || smem > 227 * 1024) return MXB_ERR_UNSUPPORTED;
  return launch_few_kernel(sparse_attn_few_f32_kernel<NB, HG>, fp, smem, (int)clusters, cached, st);
}

static int launch_few(const FewParams& fp, int kv_dtype, int smem, int clusters, cudaStream_t st) {
#define MXB_FEW(KT, NBLK) \
  if (kv_dtype == KT && fp.s.Dqk == 64 * NBLK) return launch_few_typed<KT, NBLK>(fp, smem, clusters, st);
  MXB_FEW(MXB_F16, 8)
  MXB_FEW(MXB_F16, 9)
  MXB_FEW(MXB_BF16, 8)
  MXB_FEW(MXB_BF16, 9)
  MXB_FEW(MXB_I8, 8)
  MXB_FEW(MXB_I8, 9)
#undef MXB_FEW
  return MXB_ERR_UNSUPPORTED;
}

// MXB_ERR_UNSUPPORTED: nothing was launched, the call is the other kernel's.
int launch_sparse_few(const SparseParams& p, int kv_dtype, int q_dtype, int out_dtype, cudaStream_t st) {
  if (!sparse_few_eligible(p, kv_dtype, q_dtype)) return MXB_ERR_UNSUPPORTED;
  const int eb = kv_dtype == MXB_I8 ? 1 : 2;
  const int raw = p.window > 0 && p.window < p.raw_cap ? p.window : p.raw_cap;   // raw rows of a token at most
  const int64_t entries = (int64_t)p.k + raw;
  FewParams fp;
  fp.s = p;
  fp.groups = (p.H + kFewHeads - 1) / kFewHeads;
  fp.out_dtype = out_dtype;
  fp.q_dtype = q_dtype;
  if (kv_dtype == MXB_F32) {
    // The fewest heads per CTA whose clusters are all resident at once (16 of eight CTAs are not, 13 are; 7 of sixteen).
    if (q_dtype != MXB_F32 || entries < 1 || entries > 64 * kFewMaxSplits) return MXB_ERR_UNSUPPORTED;
    fp.rows = 64;
    fp.s.nsplit = (int)ceil_div(entries, (int64_t)64);
    int rc = MXB_ERR_UNSUPPORTED;
#define MXB_FEW32(HG) \
  if (rc == MXB_ERR_UNSUPPORTED) rc = p.Dqk == 576 ? launch_few_f32<9, HG>(fp, st) : launch_few_f32<8, HG>(fp, st);
    MXB_FEW32(4) MXB_FEW32(5) MXB_FEW32(10)
#undef MXB_FEW32
    return rc;
  }
  const int64_t clusters = (int64_t)p.B * p.T * fp.groups;
  // The fewest rows per CTA whose clusters are all resident at once; a second wave of them would take as long as the kernel
  // for many tokens.  us per launch, 64 heads of 576 features, that kernel -> this one (rows per CTA):
  //   bf16  k = 512: 1 token 18.4 -> 8.5 (64), 8 18.6 -> 10.5 (128), from 9 on the other's;
  //         k = 2,048: 1 token 21.6 -> 10.8 (128), from 2 on the other's
  //   int8  k = 512: 1 token 23.2 -> 9.4 (64), 8 24.1 -> 11.4 (128), 12 24.1 -> 15.5 (256);
  //         k = 2,048: 1 token 27.2 -> 11.6 (128), 3 27.3 -> 14.8 (256), from 4 on the other's
  for (int rows = 64; rows <= few_max_rows(eb); rows *= 2) {
    const int64_t splits = ceil_div(entries, rows);
    if (splits < 1 || splits > kFewMaxSplits || clusters * splits > sm_count()) continue;
    const int smem = few_layout(p.Dqk, eb, rows, (int)splits).total;
    if (smem > 227 * 1024) continue;
    fp.rows = rows;
    fp.s.nsplit = (int)splits;
    const int rc = launch_few(fp, kv_dtype, smem, (int)clusters, st);
    if (rc != MXB_ERR_UNSUPPORTED) return rc;
  }
  return MXB_ERR_UNSUPPORTED;
}

}  // namespace mxb
