// CUDA-core (SIMT) flex-attention kernels: forward, dQ and dK/dV with f32 arithmetic throughout.
//
// They serve the float32 dtype (tcgen05 has no fp32 MMA; the f32 tolerance of 2e-3 on gradients rules
// out tf32) and any head_dim in {32, 64, 128}, and they are the on-GPU cross-check for the tensor-core
// kernels.  Tile skipping follows the same mask map as the tensor-core kernels.
//
// A CTA owns a tile of rows (queries in fwd/dq, keys in dkv) and walks the opposite side 64 positions at a time; both
// sides sit in shared memory as f32 and every contraction is register-blocked: thread (ty, tx) of NT / 16 x 16 computes RM rows
// x 4 columns of the scores and RM rows x D / 16 columns of the outputs.  What bounds it is shared memory (RM = 4: 8
// 16-byte reads per 64 FMAs, 53 % of the data pipe and 43 % of the FMA pipe busy at [16,16,256,64]); one warp per row with
// the rows read from global memory, as before, was bound by those uncoalesced reads (1.3 TFLOP/s at every size).
//   * enough 64-row tiles for every SM: RM = 4, one group of 256 threads per CTA.  [4,16,512,128] causal softcap forward +
//     dq + dkv 849 us, 17.8 TFLOP/s.
//   * fewer: 16-row tiles (four times the CTAs), and several groups of threads per CTA that take every G-th step and add up
//     their partial results at the end, because the chain of steps is what such a launch waits for.  A group is 128 threads of
//     two rows each: with 256 of one row the reads of the opposite side (9 accesses of the data pipe per 16 FMAs, now 10 per 32)
//     took the time, with 64 of four rows a step is too long a chain where there are few.  Forward, dq and dkv of a pass, us,
//     256 / 128 / 64 threads: [1,4,512,64] causal 78 / 58 / 65, [3,8,208,128] 271 / 195 / 215, [1,2,2048,128] causal 736 / 517 / 550,
//     [9,12,64,128] 105 / 93 / 136, [1,4,128,32] causal 20.8 / 20.8 / 29.
#include "sched.cuh"
#include "sm100.cuh"

namespace flexattn {
namespace {

__device__ __forceinline__ void from_f(float* p, float x) { *p = x; }
__device__ __forceinline__ void from_f(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }

constexpr int kCols = 64;       // opposite-side positions per step

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int NT>
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(NT) : "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Rows [r0, r0 + n) of a row-major [*, D] array as f32 into shared memory with row stride D + 4 floats (16-byte reads of
// 16 consecutive rows then fall on different banks); rows at or past `limit` become zero.  f32 goes through cp.async
// (the caller commits and waits), bf16 through registers.
template <int D>
__device__ __forceinline__ void load_rows(float* dst, const float* __restrict__ src, int r0, int n, int limit, int tid,
                                          int threads) {
  constexpr int kPer = D / 4;
  for (int c = tid; c < n * kPer; c += threads) {
    const int r = c / kPer, d = (c % kPer) * 4;
    const bool in = r0 + r < limit;
    const float* g = in ? src + (size_t)(r0 + r) * D + d : src;
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst + r * (D + 4) + d);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(g), "r"(in ? 16 : 0) : "memory");
  }
}
template <int D>
__device__ __forceinline__ void load_rows(float* dst, const __nv_bfloat16* __restrict__ src, int r0, int n, int limit,
                                          int tid, int threads) {
  constexpr int kPer = D / 8;
  for (int c = tid; c < n * kPer; c += threads) {
    const int r = c / kPer, d = (c % kPer) * 8;
    uint4 raw = make_uint4(0u, 0u, 0u, 0u);
    if (r0 + r < limit) raw = __ldg(reinterpret_cast<const uint4*>(src + (size_t)(r0 + r) * D + d));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
    const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
    const float2 e = __bfloat1622float2(h[2]), f = __bfloat1622float2(h[3]);
    float4* o = reinterpret_cast<float4*>(dst + r * (D + 4) + d);
    o[0] = make_float4(a.x, a.y, b.x, b.y);
    o[1] = make_float4(e.x, e.y, f.x, f.y);
  }
}

// acc[r][c] = <row ty * RM + r of A, row tx + 16 c of B> over D, both in shared memory.
template <int D, int RM>
__device__ __forceinline__ void mm_abt(float (&acc)[RM][4], const float* sA, const float* sB, int ty, int tx) {
  const float* a0 = sA + ty * RM * (D + 4);
  const float* b0 = sB + tx * (D + 4);
#pragma unroll
  for (int r = 0; r < RM; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
#pragma unroll 4
  for (int d = 0; d < D; d += 4) {
    float4 b[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(b0 + c * 16 * (D + 4) + d);
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const float4 a = *reinterpret_cast<const float4*>(a0 + r * (D + 4) + d);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        acc[r][c] = fmaf(a.x, b[c].x, acc[r][c]);
        acc[r][c] = fmaf(a.y, b[c].y, acc[r][c]);
        acc[r][c] = fmaf(a.z, b[c].z, acc[r][c]);
        acc[r][c] = fmaf(a.w, b[c].w, acc[r][c]);
      }
    }
  }
}

// The D / 16 columns of an output row that thread column tx owns.
template <int D>
__device__ __forceinline__ int out_col(int tx, int n) {
  return D == 32 ? tx * 2 + n : (n >> 2) * 64 + tx * 4 + (n & 3);
}
// acc[r][n] += sum over 64 positions j of P[ty * RM + r][j] * B[j][out_col(n)].
template <int D, int RM>
__device__ __forceinline__ void mm_pb(float (&acc)[RM][D / 16], const float* sP, const float* sB, int ty, int tx) {
  const float* p0 = sP + ty * RM * (kCols + 4);
#pragma unroll 2
  for (int j = 0; j < kCols; j += 4) {
    float4 p[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) p[r] = *reinterpret_cast<const float4*>(p0 + r * (kCols + 4) + j);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float b[D / 16];
      const float* br = sB + (j + u) * (D + 4);
      if constexpr (D == 32) {
        const float2 v = *reinterpret_cast<const float2*>(br + tx * 2);
        b[0] = v.x; b[1] = v.y;
      } else {
#pragma unroll
        for (int n = 0; n < D / 16; n += 4) {
          const float4 v = *reinterpret_cast<const float4*>(br + out_col<D>(tx, n));
          b[n] = v.x; b[n + 1] = v.y; b[n + 2] = v.z; b[n + 3] = v.w;
        }
      }
#pragma unroll
      for (int r = 0; r < RM; ++r) {
        const float pr = u == 0 ? p[r].x : u == 1 ? p[r].y : u == 2 ? p[r].z : p[r].w;
#pragma unroll
        for (int n = 0; n < D / 16; ++n) acc[r][n] = fmaf(pr, b[n], acc[r][n]);
      }
    }
  }
}
template <typename T, int D>
__device__ __forceinline__ void store_row(T* row, const float (&acc)[D / 16], float scale, int tx) {
#pragma unroll
  for (int n = 0; n < D / 16; ++n) from_f(row + out_col<D>(tx, n), acc[n] * scale);
}

__device__ __forceinline__ bool keep_rt(int kind, int i, int j, int window, int stride, int di, int dj) {
  switch (kind) {
    case FLEXATTN_MASK_CAUSAL: return mask_keep<FLEXATTN_MASK_CAUSAL>(i, j, window, stride, di, dj);
    case FLEXATTN_MASK_SLIDING_WINDOW: return mask_keep<FLEXATTN_MASK_SLIDING_WINDOW>(i, j, window, stride, di, dj);
    case FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL:
      return mask_keep<FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL>(i, j, window, stride, di, dj);
    case FLEXATTN_MASK_DOCUMENT: return mask_keep<FLEXATTN_MASK_DOCUMENT>(i, j, window, stride, di, dj);
    case FLEXATTN_MASK_S2: return mask_keep<FLEXATTN_MASK_S2>(i, j, window, stride, di, dj);
    default: return true;
  }
}
__device__ __forceinline__ float score_rt(int kind, float s, int i, int j, float slope, float cap, float inv_cap) {
  switch (kind) {
    case FLEXATTN_SCORE_ALIBI: return score_fwd<FLEXATTN_SCORE_ALIBI>(s, i, j, slope, cap, inv_cap);
    case FLEXATTN_SCORE_SOFTCAP: return score_fwd<FLEXATTN_SCORE_SOFTCAP>(s, i, j, slope, cap, inv_cap);
    default: return s;
  }
}
__device__ __forceinline__ float dsig_rt(int kind, float s, float inv_cap) {
  return kind == FLEXATTN_SCORE_SOFTCAP ? score_dsig<FLEXATTN_SCORE_SOFTCAP>(s, inv_cap) : 1.0f;
}

// Rows of a tile.
template <int RM, int NT>
constexpr int kRowsOf = NT / 16 * RM;
// Shared memory of a CTA: `row_tiles` tiles [rows][D + 4] of its own rows, and per group two tiles [64][D + 4] of the
// opposite side and one of weights [rows][68].
template <int D, int RM, int G, int NT>
constexpr size_t simt_smem(int row_tiles) {
  return sizeof(float) * ((size_t)row_tiles * kRowsOf<RM, NT> * (D + 4) + (size_t)G * (2 * kCols * (D + 4) + kRowsOf<RM, NT> * (kCols + 4)));
}

// Which (slice, tile) a CTA works on: the last tiles of every slice first (under a causal mask they are the longest).
struct SimtTile {
  int bh, b, h, first;  // first row of the tile
};
template <int BM>
__device__ __forceinline__ SimtTile simt_tile(const DevParams& P, int n_tiles, bool last_first) {
  const int slices = P.batch * P.heads;
  const int t = (int)(blockIdx.x / (unsigned)slices);
  SimtTile s;
  s.bh = (int)(blockIdx.x % (unsigned)slices);
  s.b = s.bh / P.heads;
  s.h = s.bh % P.heads;
  s.first = (last_first ? n_tiles - 1 - t : t) * BM;
  return s;
}
__device__ __forceinline__ bool mask_is_causal(int kind) {  // no key after its query
  return kind == FLEXATTN_MASK_CAUSAL || kind == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL || kind == FLEXATTN_MASK_DOCUMENT ||
         kind == FLEXATTN_MASK_S2;
}
__device__ __forceinline__ bool mask_is_window(int kind) {  // no key `window` or more before its query
  return kind == FLEXATTN_MASK_SLIDING_WINDOW || kind == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL;
}
// Keys [kbeg, kend) a tile of query rows [i0, i0 + BM) reads: the 128-wide tiles of the mask map, narrowed to the rows at
// hand.  The window's lower end only where every row keeps its own diagonal key: what a row without any key returns
// (undefined) then stays what the map's tiles give.
template <int BM>
__device__ __forceinline__ void key_range(const DevParams& P, const int4& rm, int mask, int i0, int& kbeg, int& kend) {
  kbeg = rm.x * kTile;
  kend = min(rm.y * kTile, P.seq_k);
  if (mask_is_causal(mask)) kend = min(kend, i0 + BM);
  if (mask_is_window(mask) && i0 + BM <= P.seq_k && i0 >= P.window) kbeg = max(kbeg, i0 - P.window + 1);
}

// Adds the accumulators of all groups into group 0's (true there); `work`: the group's own two tiles, no longer read.
// Called by every thread of the CTA.
template <int D, int RM, int G, int NT>
__device__ __forceinline__ bool sum_groups(float (&acc)[RM][D / 16], float* work, int group, int tid) {
  constexpr int kStride = 2 * kCols * (D + 4) + kRowsOf<RM, NT> * (kCols + 4);
  static_assert(RM * (D / 16) * NT <= 2 * kCols * (D + 4), "a group's partial results fit its two tiles");
  __syncthreads();  // earlier readers of `work` are done
#pragma unroll
  for (int r = 0; r < RM; ++r)
#pragma unroll
    for (int n = 0; n < D / 16; ++n) work[(r * (D / 16) + n) * NT + tid] = acc[r][n];
  __syncthreads();
  if (group > 0) return false;
#pragma unroll
  for (int g = 1; g < G; ++g)
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int n = 0; n < D / 16; ++n) acc[r][n] += work[g * kStride + (r * (D / 16) + n) * NT + tid];
  return true;
}

template <typename T, int D, int RM, int G, int NT>
__global__ void __launch_bounds__(NT * G, G == 1 && D <= 64 ? 2 : 1) simt_fwd_kernel(DevParams P, int score, int mask, int n_tiles) {
  constexpr int BM = kRowsOf<RM, NT>, LD = D + 4, LP = kCols + 4;
  extern __shared__ float4 smem_f4[];
  const int group = G > 1 ? (int)threadIdx.x / NT : 0, tid = (int)threadIdx.x - group * NT;
  const int ty = tid >> 4, tx = tid & 15;
  float* sQ = reinterpret_cast<float*>(smem_f4);
  float* sK = sQ + BM * LD + group * (2 * kCols * LD + BM * LP);
  float* sV = sK + kCols * LD;
  float* sP = sV + kCols * LD;
  const SimtTile t = simt_tile<BM>(P, n_tiles, true);
  const int i0 = t.first;
  const T* q = static_cast<const T*>(P.q) + (size_t)t.bh * P.seq_q * D;
  const T* k = static_cast<const T*>(P.k) + (size_t)t.bh * P.seq_k * D;
  const T* v = static_cast<const T*>(P.v) + (size_t)t.bh * P.seq_k * D;
  const int4 rm = P.row_map[(size_t)(P.map_rows > 1 ? t.b : 0) * P.n_qt + i0 / kTile];
  int kbeg, kend;
  key_range<BM>(P, rm, mask, i0, kbeg, kend);
  const int* doc = P.doc_ids ? P.doc_ids + (size_t)t.b * P.doc_stride : nullptr;
  const float slope = P.alibi_slopes ? P.alibi_slopes[t.h] : 0.f;
  const float inv_cap = P.cap != 0.f ? 1.f / P.cap : 0.f;
  float m[RM], l[RM], acc[RM][D / 16];
  int di[RM];
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int i = i0 + ty * RM + r;
    m[r] = kMasked;
    l[r] = 0.f;
    di[r] = (doc && i < P.seq_q) ? doc[i] : 0;
#pragma unroll
    for (int n = 0; n < D / 16; ++n) acc[r][n] = 0.f;
  }
  kbeg += group * kCols;  // the groups take every G-th step
  load_rows<D>(sQ, q, i0, BM, P.seq_q, threadIdx.x, NT * G);
  if (kbeg < kend) load_rows<D>(sK, k, kbeg, kCols, kend, tid, NT);
  cp_commit();
  if (kbeg < kend) load_rows<D>(sV, v, kbeg, kCols, kend, tid, NT);
  cp_commit();
  if constexpr (G > 1) {
    cp_wait<1>();
    __syncthreads();  // Q comes from every group
  }
  for (int j0 = kbeg; j0 < kend; j0 += G * kCols) {
    const bool full = j0 >= rm.z * kTile && j0 + kCols <= rm.w * kTile;  // every pair of the tile is kept
    cp_wait<1>();
    group_sync<NT>(group);  // Q and K of this step have landed
    float s[RM][4];
    mm_abt<D, RM>(s, sQ, sK, ty, tx);
    group_sync<NT>(group);  // K has been read: the next one is loaded during the softmax and P V
    if (j0 + G * kCols < kend) load_rows<D>(sK, k, j0 + G * kCols, kCols, kend, tid, NT);
    cp_commit();
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int i = i0 + ty * RM + r;
      float x[4], mx = kMasked;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int j = j0 + tx + 16 * c;
        x[c] = kMasked;
        if (j < kend && (full || keep_rt(mask, i, j, P.window, P.stride, di[r], doc ? doc[j] : 0)))
          x[c] = score_rt(score, s[r][c] * P.sm_scale, i, j, slope, P.cap, inv_cap) +
                 ((P.ab && i < P.seq_q) ? P.ab[((size_t)t.bh * P.seq_q + i) * P.seq_k + j] : 0.f);
        mx = fmaxf(mx, x[c]);
      }
#pragma unroll
      for (int sft = 8; sft > 0; sft >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, sft));
      const float m_new = fmaxf(m[r], mx);
      const float alpha = __expf(m[r] - m_new);
      float ps = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float p = j0 + tx + 16 * c < kend ? __expf(x[c] - m_new) : 0.f;
        sP[(ty * RM + r) * LP + tx + 16 * c] = p;
        ps += p;
      }
#pragma unroll
      for (int sft = 8; sft > 0; sft >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, sft);
      l[r] = l[r] * alpha + ps;
      m[r] = m_new;
#pragma unroll
      for (int n = 0; n < D / 16; ++n) acc[r][n] *= alpha;
    }
    cp_wait<1>();
    group_sync<NT>(group);  // P is in place, V has landed
    mm_pb<D, RM>(acc, sP, sV, ty, tx);
    group_sync<NT>(group);  // V and P have been read
    if (j0 + G * kCols < kend) load_rows<D>(sV, v, j0 + G * kCols, kCols, kend, tid, NT);
    cp_commit();
  }
  cp_wait<0>();
  if constexpr (G > 1) {
    // merge the groups' partial softmaxes: each leaves (m, l, acc) of its threads in its own K / V tiles
    constexpr int kVals = RM * (2 + D / 16);
    static_assert(kVals * NT <= 2 * kCols * LD, "a group's partial results fit its K and V tiles");
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      float* w = sK + r * (2 + D / 16) * NT + tid;
      w[0] = m[r];
      w[NT] = l[r];
#pragma unroll
      for (int n = 0; n < D / 16; ++n) w[(2 + n) * NT] = acc[r][n];
    }
    __syncthreads();
    if (group > 0) return;
    for (int g = 1; g < G; ++g) {
      const float* w = sK + g * (2 * kCols * LD + BM * LP) + tid;
#pragma unroll
      for (int r = 0; r < RM; ++r, w += (2 + D / 16) * NT) {
        const float m_new = fmaxf(m[r], w[0]);
        const float a = __expf(m[r] - m_new), b = __expf(w[0] - m_new);
        l[r] = l[r] * a + w[NT] * b;
        m[r] = m_new;
#pragma unroll
        for (int n = 0; n < D / 16; ++n) acc[r][n] = acc[r][n] * a + w[(2 + n) * NT] * b;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int i = i0 + ty * RM + r;
    if (i >= P.seq_q) continue;
    const size_t row = (size_t)t.bh * P.seq_q + i;
    store_row<T, D>(static_cast<T*>(P.o) + row * D, acc[r], l[r] > 0.f ? 1.f / l[r] : 0.f, tx);
    if (tx == 0) { P.l[row] = l[r]; P.m[row] = m[r]; }
  }
}

template <typename T, int D, int RM, int G, int NT>
__global__ void __launch_bounds__(NT * G, G == 1 && D <= 64 ? 2 : 1) simt_dq_kernel(DevParams P, int score, int mask, int n_tiles) {
  constexpr int BM = kRowsOf<RM, NT>, LD = D + 4, LP = kCols + 4;
  extern __shared__ float4 smem_f4[];
  const int group = G > 1 ? (int)threadIdx.x / NT : 0, tid = (int)threadIdx.x - group * NT;
  const int ty = tid >> 4, tx = tid & 15;
  float* sQ = reinterpret_cast<float*>(smem_f4);
  float* sDO = sQ + BM * LD;
  float* sK = sDO + BM * LD + group * (2 * kCols * LD + BM * LP);
  float* sV = sK + kCols * LD;
  float* sP = sV + kCols * LD;
  const SimtTile t = simt_tile<BM>(P, n_tiles, true);
  const int i0 = t.first;
  const T* q = static_cast<const T*>(P.q) + (size_t)t.bh * P.seq_q * D;
  const T* dO = static_cast<const T*>(P.d_o) + (size_t)t.bh * P.seq_q * D;
  const T* k = static_cast<const T*>(P.k) + (size_t)t.bh * P.seq_k * D;
  const T* v = static_cast<const T*>(P.v) + (size_t)t.bh * P.seq_k * D;
  const int4 rm = P.row_map[(size_t)(P.map_rows > 1 ? t.b : 0) * P.n_qt + i0 / kTile];
  int kbeg, kend;
  key_range<BM>(P, rm, mask, i0, kbeg, kend);
  const int* doc = P.doc_ids ? P.doc_ids + (size_t)t.b * P.doc_stride : nullptr;
  const float slope = P.alibi_slopes ? P.alibi_slopes[t.h] : 0.f;
  const float inv_cap = P.cap != 0.f ? 1.f / P.cap : 0.f;
  float m[RM], inv_l[RM], delta[RM], acc[RM][D / 16];
  int di[RM];
  const int kfirst = kbeg + group * kCols;  // the groups take every G-th step
  load_rows<D>(sQ, q, i0, BM, P.seq_q, threadIdx.x, NT * G);
  load_rows<D>(sDO, dO, i0, BM, P.seq_q, threadIdx.x, NT * G);
  if (kfirst < kend) {
    load_rows<D>(sK, k, kfirst, kCols, kend, tid, NT);
    load_rows<D>(sV, v, kfirst, kCols, kend, tid, NT);
  }
  cp_commit();
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int i = i0 + ty * RM + r;
    const bool in = i < P.seq_q;
    const size_t row = (size_t)t.bh * P.seq_q + i;
    const float l = in ? P.l[row] : 0.f;
    m[r] = in ? P.m[row] : 0.f;
    inv_l[r] = l > 0.f ? 1.f / l : 0.f;
    delta[r] = in ? P.delta[row] : 0.f;
    di[r] = (doc && in) ? doc[i] : 0;
#pragma unroll
    for (int n = 0; n < D / 16; ++n) acc[r][n] = 0.f;
    if (P.dab && in && group == 0) {  // the bias gradient is dense: zero outside the keys this row visits
      float* dab_row = P.dab + row * P.seq_k;
      for (int j = tx; j < kbeg; j += 16) dab_row[j] = 0.f;
      for (int j = max(kend, 0) + tx; j < P.seq_k; j += 16) dab_row[j] = 0.f;
    }
  }
  if constexpr (G > 1) {
    cp_wait<0>();
    __syncthreads();  // Q and dO come from every group
  }
  for (int j0 = kfirst; j0 < kend; j0 += G * kCols) {
    const bool full = j0 >= rm.z * kTile && j0 + kCols <= rm.w * kTile;
    cp_wait<0>();
    group_sync<NT>(group);
    float s[RM][4], dp[RM][4];
    mm_abt<D, RM>(s, sQ, sK, ty, tx);
    mm_abt<D, RM>(dp, sDO, sV, ty, tx);
    group_sync<NT>(group);  // V has been read (K is needed once more)
    if (j0 + G * kCols < kend) load_rows<D>(sV, v, j0 + G * kCols, kCols, kend, tid, NT);
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int i = i0 + ty * RM + r;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int j = j0 + tx + 16 * c;
        float ds = 0.f, dt = 0.f;  // dt: gradient of the logit after the score function (what the bias sees)
        const size_t at = ((size_t)t.bh * P.seq_q + i) * P.seq_k + j;
        if (i < P.seq_q && j < kend && (full || keep_rt(mask, i, j, P.window, P.stride, di[r], doc ? doc[j] : 0))) {
          const float sc = s[r][c] * P.sm_scale;
          const float x = score_rt(score, sc, i, j, slope, P.cap, inv_cap) + (P.ab ? P.ab[at] : 0.f);
          dt = __expf(x - m[r]) * inv_l[r] * (dp[r][c] - delta[r]);
          ds = dt * dsig_rt(score, sc, inv_cap) * P.sm_scale;
        }
        if (P.dab && i < P.seq_q && j < kend) P.dab[at] = dt;
        sP[(ty * RM + r) * LP + tx + 16 * c] = ds;
      }
    }
    group_sync<NT>(group);
    mm_pb<D, RM>(acc, sP, sK, ty, tx);
    group_sync<NT>(group);
    if (j0 + G * kCols < kend) load_rows<D>(sK, k, j0 + G * kCols, kCols, kend, tid, NT);
    cp_commit();
  }
  cp_wait<0>();
  if constexpr (G > 1) {
    if (!sum_groups<D, RM, G, NT>(acc, sK, group, tid)) return;
  }
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int i = i0 + ty * RM + r;
    if (i < P.seq_q) store_row<T, D>(static_cast<T*>(P.dq) + ((size_t)t.bh * P.seq_q + i) * D, acc[r], 1.f, tx);
  }
}

template <typename T, int D, int RM, int G, int NT>
__global__ void __launch_bounds__(NT * G, G == 1 && D <= 64 ? 2 : 1) simt_dkv_kernel(DevParams P, int score, int mask, int n_tiles) {
  constexpr int BM = kRowsOf<RM, NT>, LD = D + 4, LP = kCols + 4;
  extern __shared__ float4 smem_f4[];
  const int group = G > 1 ? (int)threadIdx.x / NT : 0, tid = (int)threadIdx.x - group * NT;
  const int ty = tid >> 4, tx = tid & 15;
  float* sK = reinterpret_cast<float*>(smem_f4);
  float* sV = sK + BM * LD;
  float* sQ = sV + BM * LD + group * (2 * kCols * LD + BM * LP);
  float* sDO = sQ + kCols * LD;
  float* sP = sDO + kCols * LD;  // P^T, then dS^T
  const SimtTile t = simt_tile<BM>(P, n_tiles, false);  // early keys see the most queries under a causal mask
  const int k0 = t.first;
  const T* k = static_cast<const T*>(P.k) + (size_t)t.bh * P.seq_k * D;
  const T* v = static_cast<const T*>(P.v) + (size_t)t.bh * P.seq_k * D;
  const T* q = static_cast<const T*>(P.q) + (size_t)t.bh * P.seq_q * D;
  const T* dO = static_cast<const T*>(P.d_o) + (size_t)t.bh * P.seq_q * D;
  const float* lrow = P.l + (size_t)t.bh * P.seq_q;
  const float* mrow = P.m + (size_t)t.bh * P.seq_q;
  const float* drow = P.delta + (size_t)t.bh * P.seq_q;
  const int4 cm = P.col_map[(size_t)(P.map_rows > 1 ? t.b : 0) * P.n_kt + k0 / kTile];
  // queries [qbeg, qend) these keys see: the map's tiles, narrowed to the keys at hand (masked pairs add nothing)
  int qbeg = cm.x * kTile, qend = min(cm.y * kTile, P.seq_q);
  if (mask_is_causal(mask)) qbeg = max(qbeg, k0);
  if (mask_is_window(mask) && P.window < P.seq_q) qend = min(qend, k0 + BM - 1 + P.window);
  const int* doc = P.doc_ids ? P.doc_ids + (size_t)t.b * P.doc_stride : nullptr;
  const float slope = P.alibi_slopes ? P.alibi_slopes[t.h] : 0.f;
  const float inv_cap = P.cap != 0.f ? 1.f / P.cap : 0.f;
  float acc_k[RM][D / 16], acc_v[RM][D / 16];
  int dj[RM];
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int j = k0 + ty * RM + r;
    dj[r] = (doc && j < P.seq_k) ? doc[j] : 0;
#pragma unroll
    for (int n = 0; n < D / 16; ++n) { acc_k[r][n] = 0.f; acc_v[r][n] = 0.f; }
  }
  qbeg += group * kCols;  // the groups take every G-th step
  load_rows<D>(sK, k, k0, BM, P.seq_k, threadIdx.x, NT * G);
  load_rows<D>(sV, v, k0, BM, P.seq_k, threadIdx.x, NT * G);
  if (qbeg < qend) {
    load_rows<D>(sQ, q, qbeg, kCols, qend, tid, NT);
    load_rows<D>(sDO, dO, qbeg, kCols, qend, tid, NT);
  }
  cp_commit();
  if constexpr (G > 1) {
    cp_wait<0>();
    __syncthreads();  // K and V come from every group
  }
  for (int i0 = qbeg; i0 < qend; i0 += G * kCols) {
    const bool full = i0 >= cm.z * kTile && i0 + kCols <= cm.w * kTile;
    float mi[4], inv_l[4], de[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + tx + 16 * c;
      const float l = i < qend ? lrow[i] : 0.f;
      mi[c] = i < qend ? mrow[i] : 0.f;
      inv_l[c] = l > 0.f ? 1.f / l : 0.f;
      de[c] = i < qend ? drow[i] : 0.f;
    }
    cp_wait<0>();
    group_sync<NT>(group);
    float s[RM][4], dp[RM][4];
    mm_abt<D, RM>(s, sK, sQ, ty, tx);
    mm_abt<D, RM>(dp, sV, sDO, ty, tx);
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int j = k0 + ty * RM + r;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = i0 + tx + 16 * c;
        float p = 0.f, ds = 0.f;
        if (j < P.seq_k && i < qend && (full || keep_rt(mask, i, j, P.window, P.stride, doc ? doc[i] : 0, dj[r]))) {
          const float sc = s[r][c] * P.sm_scale;
          const float x = score_rt(score, sc, i, j, slope, P.cap, inv_cap) +
                          (P.ab ? P.ab[((size_t)t.bh * P.seq_q + i) * P.seq_k + j] : 0.f);
          p = __expf(x - mi[c]) * inv_l[c];
          ds = p * (dp[r][c] - de[c]) * dsig_rt(score, sc, inv_cap) * P.sm_scale;
        }
        sP[(ty * RM + r) * LP + tx + 16 * c] = p;
        dp[r][c] = ds;
      }
    }
    group_sync<NT>(group);
    mm_pb<D, RM>(acc_v, sP, sDO, ty, tx);
    group_sync<NT>(group);  // dO and P have been read: the next dO is loaded during dS^T Q
    if (i0 + G * kCols < qend) load_rows<D>(sDO, dO, i0 + G * kCols, kCols, qend, tid, NT);
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) sP[(ty * RM + r) * LP + tx + 16 * c] = dp[r][c];
    group_sync<NT>(group);
    mm_pb<D, RM>(acc_k, sP, sQ, ty, tx);
    group_sync<NT>(group);
    if (i0 + G * kCols < qend) load_rows<D>(sQ, q, i0 + G * kCols, kCols, qend, tid, NT);
    cp_commit();
  }
  cp_wait<0>();
  if constexpr (G > 1) {
    if (!sum_groups<D, RM, G, NT>(acc_k, sQ, group, tid)) {
      sum_groups<D, RM, G, NT>(acc_v, sQ, group, tid);
      return;
    }
    sum_groups<D, RM, G, NT>(acc_v, sQ, group, tid);
  }
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int j = k0 + ty * RM + r;
    if (j >= P.seq_k) continue;
    const size_t row = (size_t)t.bh * P.seq_k + j;
    store_row<T, D>(static_cast<T*>(P.dk) + row * D, acc_k[r], 1.f, tx);
    store_row<T, D>(static_cast<T*>(P.dv) + row * D, acc_v[r], 1.f, tx);
  }
}

using SimtKernel = void (*)(DevParams, int, int, int);

// One form of a kernel: 64-row tiles and one group, or 16-row tiles and several groups.
struct SimtChoice {
  SimtKernel kernel;
  size_t smem;
  int threads;
  SmemAttrOnce* once;
};
cudaError_t simt_launch(cudaStream_t st, const DevParams& d, int score, int mask, int rows, const SimtChoice& big,
                        const SimtChoice& small) {
  const long long slices = (long long)d.batch * d.heads;
  const int sms = sm_count();
  if (sms <= 0) return cudaErrorInvalidDevice;
  // The line, us of forward and backward with the small form and the big one: 128 such tiles [4,8,200,64] causal 87 (the big
  // one would leave SMs idle), 180 [5,12,153,64] causal 121 and 98, 243 [9,3,555,32] 222 and 181, 256 [2,64,112,64] 177 and 111.
  const bool use_big = (rows + 63) / 64 * slices >= sms;
  const SimtChoice& c = use_big ? big : small;
  const int bm = use_big ? 64 : 16;
  const int n_tiles = (rows + bm - 1) / bm;
  if (n_tiles * slices > 0x7fffffffLL) return cudaErrorInvalidValue;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(c.kernel), (int)c.smem, c.once) != FLEXATTN_OK) return cudaErrorInvalidValue;
  c.kernel<<<(unsigned)(n_tiles * slices), c.threads, c.smem, st>>>(d, score, mask, n_tiles);
  return cudaGetLastError();
}

// KERNEL with ROW_TILES tiles of its own rows, for T and D.  Groups of the small form: as many as shared memory holds.
#define FLEXATTN_SIMT_CASE(KERNEL, T, DD, ROW_TILES)                                                                \
  do {                                                                                                             \
    constexpr int kG = DD == 128 ? 2 : 4;                                                                          \
    static SmemAttrOnce big_once{}, small_once{};                                                                  \
    return simt_launch(st, d, score, mask, rows,                                                                   \
                       SimtChoice{KERNEL<T, DD, 4, 1, 256>, simt_smem<DD, 4, 1, 256>(ROW_TILES), 256, &big_once},  \
                       SimtChoice{KERNEL<T, DD, 2, kG, 128>, simt_smem<DD, 2, kG, 128>(ROW_TILES), 128 * kG, &small_once}); \
  } while (0)
#define FLEXATTN_SIMT_DISPATCH(KERNEL, ROW_TILES)                                              \
  do {                                                                                                             \
    if (dtype == FLEXATTN_BF16) {                                                                                  \
      if (d.head_dim == 32) FLEXATTN_SIMT_CASE(KERNEL, __nv_bfloat16, 32, ROW_TILES);          \
      if (d.head_dim == 64) FLEXATTN_SIMT_CASE(KERNEL, __nv_bfloat16, 64, ROW_TILES);          \
      if (d.head_dim == 128) FLEXATTN_SIMT_CASE(KERNEL, __nv_bfloat16, 128, ROW_TILES);        \
    } else {                                                                                                       \
      if (d.head_dim == 32) FLEXATTN_SIMT_CASE(KERNEL, float, 32, ROW_TILES);                  \
      if (d.head_dim == 64) FLEXATTN_SIMT_CASE(KERNEL, float, 64, ROW_TILES);                  \
      if (d.head_dim == 128) FLEXATTN_SIMT_CASE(KERNEL, float, 128, ROW_TILES);                \
    }                                                                                                              \
    return cudaErrorInvalidValue;                                                                                  \
  } while (0)

}  // namespace

cudaError_t launch_simt_fwd(cudaStream_t st, const DevParams& d, int dtype, int score, int mask) {
  const int rows = d.seq_q;
  FLEXATTN_SIMT_DISPATCH(simt_fwd_kernel, 1);
}
cudaError_t launch_simt_dq(cudaStream_t st, const DevParams& d, int dtype, int score, int mask) {
  const int rows = d.seq_q;
  FLEXATTN_SIMT_DISPATCH(simt_dq_kernel, 2);
}
cudaError_t launch_simt_dkv(cudaStream_t st, const DevParams& d, int dtype, int score, int mask) {
  const int rows = d.seq_k;
  FLEXATTN_SIMT_DISPATCH(simt_dkv_kernel, 2);
}

}  // namespace flexattn
