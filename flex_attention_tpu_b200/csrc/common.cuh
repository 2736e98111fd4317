// Internal definitions shared by every translation unit of libflexattn.so.
#pragma once
#ifdef FLEXATTN_JIT
// Run-time compilation (NVRTC) of a tensor-core kernel around a user score function: no host headers exist there,
// so the handful of types the device code needs are spelled out.
typedef signed char int8_t;
typedef unsigned char uint8_t;
typedef unsigned short uint16_t;
typedef int int32_t;
typedef unsigned int uint32_t;
typedef long long int64_t;
typedef unsigned long long uint64_t;
typedef unsigned long long uintptr_t;
struct alignas(64) CUtensorMap_st {
  unsigned long long opaque[16];
};
typedef CUtensorMap_st CUtensorMap;
#else
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#endif

#include "../../include/flexattn.h"

namespace flexattn {

constexpr int kTile = FLEXATTN_TILE;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
// Finite stand-in for -inf (log2 domain in the tensor-core kernels, natural units in the SIMT ones):
// a row whose keys so far are all masked keeps m == kMasked, its garbage weights exp(0) == 1 are
// wiped by alpha == exp(kMasked - m_new) == 0 as soon as a kept key arrives.  The reference kernels use
// -0.7 * FLT_MAX for the same reason (flex_attention_kernel.py:288).
constexpr float kMasked = -1.0e30f;

// ---------------------------------------------------------------------------------------------
// Mask map (lives in the caller's workspace).
// ---------------------------------------------------------------------------------------------
struct MapHeader {
  int32_t magic, mask_kind, window, stride;
  int32_t seq_q, seq_k, n_qt, n_kt;
  int32_t rows;  // batch for document masks, else 1
  int32_t pad[7];
};
constexpr int32_t kMapMagic = 0x464c5841;  // "FLXA"

struct MapLayout {
  int n_qt, n_kt, rows, n_t;
  size_t off_row, off_col, off_doc, off_order, off_order_rm, off_order_pair, off_run_lo, off_run_hi, off_sorted, bytes;
};

__host__ __device__ inline MapLayout map_layout(int batch, int seq_q, int seq_k, int mask_kind) {
  MapLayout L;
  L.n_qt = (seq_q + kTile - 1) / kTile;
  L.n_kt = (seq_k + kTile - 1) / kTile;
  L.n_t = L.n_qt > L.n_kt ? L.n_qt : L.n_kt;
  L.rows = (mask_kind == FLEXATTN_MASK_DOCUMENT) ? batch : 1;
  L.off_row = sizeof(MapHeader);
  L.off_col = L.off_row + sizeof(int4) * (size_t)L.rows * L.n_qt;
  L.off_doc = L.off_col + sizeof(int4) * (size_t)L.rows * L.n_kt;
  size_t doc = (mask_kind == FLEXATTN_MASK_DOCUMENT) ? sizeof(int2) * (size_t)batch * L.n_t : 0;
  // q tiles of every map row ordered by their number of kv tiles, largest first (work order of the persistent
  // forward kernel)
  L.off_order = (L.off_doc + doc + 15) & ~(size_t)15;
  // ... and the row-map entries in that order (so that walking the order needs no dependent load)
  L.off_order_rm = (L.off_order + sizeof(int32_t) * (size_t)L.rows * L.n_qt + 15) & ~(size_t)15;
  // document masks: first / one-past-last position of the run of equal ids every position sits in, and one flag per
  // batch row saying that its ids never decrease (then equal ids are contiguous and a row's kept keys are one
  // interval, so the kernels mask partial tiles from these two numbers instead of comparing ids per element)
  const size_t len = (size_t)(seq_q > seq_k ? seq_q : seq_k);
  const size_t runs = (mask_kind == FLEXATTN_MASK_DOCUMENT) ? sizeof(int32_t) * (size_t)batch * len : 0;
  L.off_run_lo = (L.off_order_rm + sizeof(int4) * (size_t)L.rows * L.n_qt + 15) & ~(size_t)15;
  L.off_run_hi = (L.off_run_lo + runs + 15) & ~(size_t)15;
  L.off_sorted = (L.off_run_hi + runs + 15) & ~(size_t)15;
  // the pairs of adjacent q tiles in such an order as well (work order of the two-query-tile forward kernel); behind the rest,
  // at most a 17th of it (4 bytes a pair, 68 and more a q tile of a document row)
  L.off_order_pair = (L.off_sorted + (runs ? sizeof(int32_t) * (size_t)batch : 0) + 255) & ~(size_t)255;
  L.bytes = (L.off_order_pair + sizeof(int32_t) * (size_t)L.rows * ((L.n_qt + 1) / 2) + 255) & ~(size_t)255;
  return L;
}

// Device-side view of a problem: what the kernels need, already resolved by the host.
struct DevParams {
  const void* q;
  const void* k;
  const void* v;
  void* o;
  const void* d_o;
  void* dq;
  void* dk;
  void* dv;
  float* l;
  float* m;
  float* delta;
  const int32_t* doc_ids;
  const float* alibi_slopes;
  const float* ab;  // optional dense bias [B,H,Sq,Sk]
  float* dab;       // optional bias gradient, written by the dQ kernels
  const int4* row_map;  // [rows][n_qt]
  const int4* col_map;  // [rows][n_kt]
  const int32_t* order;  // [rows][n_qt]: q tiles by decreasing number of kv tiles
  const int4* order_rm;  // [rows][n_qt]: row_map entry of order[i]
  const int32_t* order_pair;  // [rows][(n_qt + 1) / 2]: pairs of q tiles (2 p, 2 p + 1) by decreasing number of kv tiles
  const int32_t* run_lo;      // document masks: [batch][doc_stride] first position of each position's run of equal ids
  const int32_t* run_hi;      // ... one past its last position
  const int32_t* doc_sorted;  // ... [batch] 1 when the row's ids never decrease (runs are whole documents)
  int32_t* status;
  int batch, heads, seq_q, seq_k, head_dim;
  int n_qt, n_kt, map_rows, doc_stride;
  int window, stride;
  float sm_scale, cap;
  int kv_splits;   // split forward: CTAs a query tile's kv tiles are dealt to (1, 2, 4 or 8)
  int user_score;  // handle of a run-time compiled score function (host side only)
  int n_st;        // kMaskS2Gather: tiles of the keys on the stride grid; 0: the call is not gathered
};

// ---------------------------------------------------------------------------------------------
// S2, gathered.  A query keeps its local window and, before it, the keys on the stride grid: walked as one causal range that is every
// tile below the diagonal for 128 / stride keys in each.  The gathered form splits the kept pairs in two, both plain intervals:
//   window tiles    the causal sliding window; tile kt holds keys 128 kt ..
//   strided tiles   tile t holds the keys (128 t + c) * stride, c < 128, fetched as such by TMA (a tensor map whose row pitch is
//                   `stride` rows); a query i keeps those with (128 t + c) * stride <= i - window
// A query tile's kv tiles are numbered as ONE range [x, end): from z on they are window tiles (the number is kt), below it strided
// ones (t = number - x).  Ranges follow from the sizes: the gathered kernels read no map.  [2,16,4096,64], 512 keys, stride 64: 16.5 tiles a
// query tile become 6.
// ---------------------------------------------------------------------------------------------
constexpr int kMaskS2Gather = FLEXATTN_MASK_S2 + 1;  // inside the kernels only
__host__ __device__ inline int s2_keys(int seq_k, int stride) { return (seq_k - 1) / stride + 1; }
__host__ __device__ inline int4 s2_row(int qt, int seq_q, int seq_k, int window, int stride) {  // {x, end, z, 0}
  const int i0 = qt * kTile, i1 = (seq_q - i0 < kTile ? seq_q : i0 + kTile) - 1;
  const int last = i1 < seq_k - 1 ? i1 : seq_k - 1, n = s2_keys(seq_k, stride) - 1;
  const int w1 = last / kTile + 1;
  int w0 = window <= i0 ? (i0 - window + 1) / kTile : 0;
  if (window <= i0 && i0 - window + 1 > seq_k - 1) w0 = w1;
  int strided = 0;
  if (i1 >= window) {
    const int k = (i1 - window) / stride;
    strided = (k < n ? k : n) / kTile + 1;
  }
  return make_int4(w0 - strided, w1, w0, 0);
}
// Query tiles of kv tile `v` (strided ones behind the n_kt window tiles): {first, end, first fully kept, end of those}
__host__ __device__ inline int4 s2_col(int v, int seq_q, int seq_k, int n_qt, int n_kt, int window, int stride) {
  const int whole = seq_q / kTile;  // query tiles without rows past the end
  int4 r = make_int4(0, 0, 0, 0);
  if (v < n_kt) {
    const int j0 = v * kTile, j1 = (seq_k - j0 < kTile ? seq_k : j0 + kTile) - 1;
    if (j0 >= seq_q) return r;
    r.x = v;
    r.y = window < seq_q - j1 ? (j1 + window - 1) / kTile + 1 : n_qt;
    r.z = v + 1;
    r.w = window < kTile ? 0 : window < seq_q ? (window - kTile + j0) / kTile + 1 : n_qt;
  } else {
    const long long k0 = (long long)(v - n_kt) * kTile, first = k0 * stride + window, all = (k0 + kTile - 1) * stride + window;
    if (first >= seq_q) return r;
    r.x = (int)(first / kTile);
    r.y = n_qt;
    r.z = all < seq_q ? (int)((all + kTile - 1) / kTile) : n_qt;
    r.w = n_qt;
  }
  if (r.w > whole) r.w = whole;
  if (r.w < r.z) r.z = r.w = r.x;
  return r;
}

// ---------------------------------------------------------------------------------------------
// Compile-time mask functors.  True = keep.  di/dj are the document ids of positions i/j (only read
// by the document mask).
// ---------------------------------------------------------------------------------------------
template <int MK>
__device__ __forceinline__ bool mask_keep(int i, int j, int window, int stride, int di, int dj) {
  if constexpr (MK == FLEXATTN_MASK_NONE) {
    return true;
  } else if constexpr (MK == FLEXATTN_MASK_CAUSAL) {
    return i >= j;
  } else if constexpr (MK == FLEXATTN_MASK_SLIDING_WINDOW) {
    return (i - j) < window;
  } else if constexpr (MK == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL) {
    return (unsigned)(i - j) < (unsigned)window;
  } else if constexpr (MK == FLEXATTN_MASK_DOCUMENT) {
    return (i >= j) && (di == dj);
  } else {  // S2
    return ((unsigned)(i - j) < (unsigned)window) || ((i >= j) && (j % stride == 0));
  }
}

// For the mask kinds whose kept keys of a query row (and kept queries of a key row) form ONE interval, a partial tile
// evaluates the mask once per row and 32 columns as a bitmap (range_bits32 of the row's interval, shifted to the
// group's first column) instead of once per element.  Document masks are intervals when the ids of the batch row never
// decrease.  An S2 row is an interval plus the keys on the stride grid below it, which is a bitmap as well: the grid
// is ONE pattern shifted to the group's first multiple (the remainder of a key index by the run-time stride, 30
// instructions, is taken once per 32 columns; per element it made S2 ten times slower than the dense causal mask).
template <int MK>
constexpr bool kMaskIsBits = MK == FLEXATTN_MASK_NONE || MK == FLEXATTN_MASK_CAUSAL || MK == FLEXATTN_MASK_SLIDING_WINDOW ||
                             MK == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL || MK == FLEXATTN_MASK_S2 || MK == kMaskS2Gather;
__device__ __forceinline__ uint32_t range_bits32(int lo, int hi) {  // bits [lo, hi) of a word, clipped to [0, 32)
  lo = lo > 0 ? lo : 0;
  hi = hi < 32 ? hi : 32;
  if (hi <= lo) return 0u;
  return (hi == 32 ? 0xffffffffu : ((1u << hi) - 1u)) & ~((1u << lo) - 1u);
}
// Kept keys [klo, khi) of query row i (the sequence end included); for S2 its local window, the strided keys come on top
// (keep_bits32).
template <int MK>
__device__ __forceinline__ void row_key_interval(int i, int seq_k, int window, int& klo, int& khi) {
  const bool lower = MK == FLEXATTN_MASK_SLIDING_WINDOW || MK == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL ||
                     MK == FLEXATTN_MASK_S2;  // j > i - window
  const bool upper = MK == FLEXATTN_MASK_CAUSAL || MK == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL || MK == FLEXATTN_MASK_S2;  // j <= i
  klo = lower && window <= i ? i - window + 1 : 0;  // (never near INT_MIN, where klo - j would wrap around)
  khi = upper ? (i + 1 < seq_k ? i + 1 : seq_k) : seq_k;
}
// S2: the stride grid's bits inside 32 columns when the first of them is on the grid (bit 0, stride, 2 stride ...).
__device__ __forceinline__ uint32_t stride_pattern32(int stride) {
  uint32_t pat = 1u;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int sh = stride << s;  // doubling: 2, 4, 8, 16, 32 multiples
    if (stride < 32 && sh < 32) pat |= pat << sh;
  }
  return pat;
}
// Kept columns of the 32 keys j .. j+31 for a query row with the interval [klo, khi).
template <int MK>
__device__ __forceinline__ uint32_t keep_bits32(int j, int klo, int khi, int stride, uint32_t pattern) {
  uint32_t bits = range_bits32(klo - j, khi - j);
  if constexpr (MK == FLEXATTN_MASK_S2) {
    const int r = j % stride, first = r == 0 ? 0 : stride - r;  // first multiple of the stride at or after j
    if (first < 32) bits |= (pattern << first) & range_bits32(0, khi - j);
  }
  return bits;
}
// Kept queries [qlo, qhi) of key row j: always an interval (an S2 key on the stride grid is seen by every later query).
template <int MK>
__device__ __forceinline__ void row_query_interval(int j, int seq_q, int window, int stride, int& qlo, int& qhi) {
  const bool lower = MK == FLEXATTN_MASK_CAUSAL || MK == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL || MK == FLEXATTN_MASK_S2;  // i >= j
  const bool upper = MK == FLEXATTN_MASK_SLIDING_WINDOW || MK == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL ||
                     (MK == FLEXATTN_MASK_S2 && j % stride != 0);  // i < j + window
  qlo = lower ? j : 0;
  qhi = upper && window < seq_q - j ? j + window : seq_q;  // (no sum that a huge window could overflow)
}
// A document mask over ids that never decrease is an interval as well: query row i keeps the keys [run_lo(i), i],
// key row j the queries [j, run_hi(j)), with run_lo / run_hi from the mask map.

// Compile-time score functors on the scaled score s = sm_scale * <q,k>, natural units.
// score_fwd returns t = score_mod(s) + bias(i, j); score_dsig returns d score_mod / d s.
template <int SK>
__device__ __forceinline__ float score_fwd(float s, int i, int j, float slope, float cap, float inv_cap) {
  if constexpr (SK == FLEXATTN_SCORE_ALIBI) {
    return s - slope * (float)(i - j);
  } else if constexpr (SK == FLEXATTN_SCORE_SOFTCAP) {
    return cap * tanhf(s * inv_cap);
  } else {
    return s;
  }
}
template <int SK>
__device__ __forceinline__ float score_dsig(float s, float inv_cap) {
  if constexpr (SK == FLEXATTN_SCORE_SOFTCAP) {
    float th = tanhf(s * inv_cap);
    return 1.0f - th * th;
  } else {
    return 1.0f;
  }
}

__device__ __forceinline__ void report_status(int32_t* status, int code, int kernel_id, int detail) {
  if (status != nullptr) {
    if (atomicCAS(status, 0, code) == 0) {
      status[1] = kernel_id;
      status[2] = (int)(blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z));
      status[3] = detail;
    }
  }
}
__device__ __forceinline__ void report_timeout(int32_t* status, int kernel_id, int detail) {
  report_status(status, (int)FLEXATTN_ERR_TIMEOUT, kernel_id, detail);
}

// Bounds-checked build (-DFLEXATTN_DEBUG, libflexattn_debug.so): every direct global-memory access of the
// tensor-core kernels (everything that does not go through a TMA tensor map, which clips by itself) is guarded.
// An index outside its array is recorded as {FLEXATTN_ERR_DEBUG_BOUNDS, kernel id, block, site} in the status
// words and the access is skipped, so a wrong index shows up as a status instead of a memory fault.  In the
// ordinary build the check is the constant `true` and disappears.
#ifdef FLEXATTN_DEBUG
constexpr bool kDebugChecks = true;
#else
constexpr bool kDebugChecks = false;
#endif
__device__ __forceinline__ bool dbg_in_bounds(long long idx, long long limit, int32_t* status, int kernel_id, int site) {
  if constexpr (!kDebugChecks) {
    return true;
  } else {
    if (idx >= 0 && idx < limit) return true;
    report_status(status, (int)FLEXATTN_ERR_DEBUG_BOUNDS, kernel_id, site);
    return false;
  }
}
#define FLEXATTN_DBG_OK(idx, limit, kernel_id, site) \
  ::flexattn::dbg_in_bounds((long long)(idx), (long long)(limit), P.status, (kernel_id), (site))

#ifndef FLEXATTN_JIT
// Whether an S2 call is gathered: where that leaves enough fewer tiles a query tile than every tile below the diagonal (a gathered
// one costs up to 1.2 of a dense one: its mask is never skipped in the window, and the two-query-tile forward has no such form).
inline bool s2_gathers(const FlexAttnParams& p) {
  if (p.mask_kind != FLEXATTN_MASK_S2 || p.ab != nullptr || p.score_kind == FLEXATTN_SCORE_USER || p.stride < 2 || p.window <= 0) return false;
  const double n = ((p.seq_q < p.seq_k ? p.seq_q : p.seq_k) + kTile - 1) / kTile;
  return 1.2 * ((double)p.window / kTile + 2 + n / (2.0 * p.stride)) < 0.5 * (n + 1);
}
// Host-side validation of a forward call, shared by flexattn_fwd and flexattn_fwd_noalloc (api.cu).
int validate_fwd_args(const FlexAttnParams* p, bool* tc);

// Registers per thread the kernels that hand them round among their warpgroups have to be launched with
constexpr int kPairLaunchRegs = 168, kSplitLaunchRegs = 168, kFusedLaunchRegs = 128;

// Bounds-checked build: whether FLEXATTN_HOST_FAULT in the environment names `what`, a fault that the host code is to see as if it
// had happened (tests): "registers", the kernels that hand registers round were compiled for too few of them; "strided_map", the encoder
// refuses the tensor maps of gathered S2.
#ifdef FLEXATTN_DEBUG
bool host_fault(const char* what);
#else
inline bool host_fault(const char*) { return false; }
#endif

// ---------------------------------------------------------------------------------------------
// Launchers implemented by the kernel translation units; each returns a cudaError_t.
// ---------------------------------------------------------------------------------------------
cudaError_t launch_mask_map(cudaStream_t st, const FlexAttnParams& p);
cudaError_t launch_delta(cudaStream_t st, const FlexAttnParams& p);
cudaError_t launch_simt_fwd(cudaStream_t st, const DevParams& d, int dtype, int score, int mask);
cudaError_t launch_simt_dq(cudaStream_t st, const DevParams& d, int dtype, int score, int mask);
cudaError_t launch_simt_dkv(cudaStream_t st, const DevParams& d, int dtype, int score, int mask);
// tensor-core (tcgen05) kernels: bf16, D in {64,128}
int launch_sm100_fwd_pipe(cudaStream_t st, const DevParams& d, int score, int mask);  // persistent, three score tiles in flight
// Two query tiles per CTA, one row per thread; few query tiles, a cluster each.  FLEXATTN_ERR_UNSUPPORTED_BACKEND (of the first around a
// user score function also FLEXATTN_ERR_JIT_COMPILE): this build of it cannot run, nothing was launched, the persistent one serves the call.
int launch_sm100_fwd_pair(cudaStream_t st, const DevParams& d, int score, int mask);
int launch_sm100_fwd_split(cudaStream_t st, const DevParams& d, int score, int mask);
bool fwd_pair_pays(const FlexAttnParams& p, int sms);  // whether the first of them serves a call rather than the persistent one (fwd_choice.cu)
int split_clusters_at_once(int c);  // clusters of c CTAs of that kernel the device holds at a time; 0: unknown
int launch_sm100_dq(cudaStream_t st, const DevParams& d, int score, int mask);
int launch_sm100_dkv(cudaStream_t st, const DevParams& d, int score, int mask);
// delta, dQ, dK and dV in one pass over the tile pairs; no dense bias.  scratch: bwd_fused_scratch_bytes
int launch_sm100_bwd_fused(cudaStream_t st, const DevParams& d, int score, int mask, void* scratch);
size_t bwd_fused_scratch_bytes(const FlexAttnParams& p);
double bwd_fused_slack(const FlexAttnParams& p, int sms);  // query tiles a CTA walks per kv tile of its slice in flight
// ... with a dense bias (d.ab) and / or its gradient (d.dab, dQ only)
int launch_sm100_fwd_pipe_bias(cudaStream_t st, const DevParams& d, int score, int mask);
int launch_sm100_dq_bias(cudaStream_t st, const DevParams& d, int score, int mask);
int launch_sm100_dkv_bias(cudaStream_t st, const DevParams& d, int score, int mask);

// Launch of a kernel compiled at run time around a user score function (jit.cu).  which: 0 forward, 1 dQ, 2 dK/dV, each
// also in a form for a dense bias, 3 forward of two query tiles, 4 fused backward;
// args: the kernel's parameters as for cuLaunchKernel.  Returns a FlexAttnStatus.
constexpr int kJitForward = 0, kJitForwardPair = 3;
int jit_launch(int which, bool bias, int handle, int head_dim, int mask, unsigned grid_x, unsigned grid_y, unsigned threads,
               size_t smem_bytes, cudaStream_t st, void** args);
// Which of two kernels that can both serve a call around a user score function does: the first, but under capture, where nothing can
// be loaded, the second if only that one is there.
int jit_first_or_loaded(int first, int second, int handle, int head_dim, int mask, cudaStream_t st);
// Compiles and loads the fused backward for a user score function where that is still to do.  FLEXATTN_ERR_JIT_COMPILE: it
// cannot serve the call (nothing has been launched), the separate kernels may.
int jit_fused_ready(int handle, int head_dim, int mask, size_t smem_bytes, cudaStream_t st);
#endif  // !FLEXATTN_JIT

}  // namespace flexattn

// user_score(s, b, h, i, j) and user_dscore(...): identity here; a run-time compilation substitutes the user's
// expressions for this header.
#include "user_score.cuh"
