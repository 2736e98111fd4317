// The C ABI of libflexattn.so: argument validation, backend choice and dispatch.  No allocation, no
// host synchronisation (except flexattn_read_mask_map, a test/tool helper).  The only state that outlives a
// call is per device: the abort word of the tensor-core kernels (set by a device-side time-out, cleared by
// flexattn_reset_abort) and the caches of device attributes and symbol addresses next to it.
#include <stdlib.h>
#include <string.h>

#include <algorithm>

#include <nvtx3/nvToolsExt.h>

#include "common.cuh"
#include "sched.cuh"

namespace flexattn {
namespace {


bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// NVTX range around the host side of an entry point (validation, tensor-map encoding, launch): shows up in ncu /
// Nsight timelines and costs nothing when no tool is attached (header-only NVTX resolves to a no-op then).
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

int validate_common(const FlexAttnParams* p) {
  if (p == nullptr) return FLEXATTN_ERR_NULL_POINTER;
  if (p->batch <= 0 || p->heads <= 0 || p->seq_q <= 0 || p->seq_k <= 0) return FLEXATTN_ERR_BAD_SHAPE;
  if ((long long)p->batch * p->heads > 0x7fffffffLL / 2) return FLEXATTN_ERR_BAD_SHAPE;
  if (p->dtype != FLEXATTN_BF16 && p->dtype != FLEXATTN_F32) return FLEXATTN_ERR_UNSUPPORTED_DTYPE;
  if (p->head_dim != 32 && p->head_dim != 64 && p->head_dim != 128) return FLEXATTN_ERR_UNSUPPORTED_HEAD_DIM;
  if (p->score_kind < FLEXATTN_SCORE_NONE || p->score_kind > FLEXATTN_SCORE_USER) return FLEXATTN_ERR_UNSUPPORTED_MOD;
  if (p->mask_kind < FLEXATTN_MASK_NONE || p->mask_kind > FLEXATTN_MASK_S2) return FLEXATTN_ERR_UNSUPPORTED_MOD;
  if (p->backend < FLEXATTN_BACKEND_AUTO || p->backend > FLEXATTN_BACKEND_TCGEN05) return FLEXATTN_ERR_UNSUPPORTED_BACKEND;
  return FLEXATTN_OK;
}

int validate_window(const FlexAttnParams* p) {
  const int mk = p->mask_kind;
  if ((mk == FLEXATTN_MASK_SLIDING_WINDOW || mk == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL || mk == FLEXATTN_MASK_S2) &&
      p->window <= 0)
    return FLEXATTN_ERR_UNSUPPORTED_MOD;
  if (mk == FLEXATTN_MASK_S2 && p->stride <= 0) return FLEXATTN_ERR_UNSUPPORTED_MOD;
  return FLEXATTN_OK;
}

int validate_mods(const FlexAttnParams* p) {
  const int mk = p->mask_kind, e = validate_window(p);
  if (e) return e;
  if (mk == FLEXATTN_MASK_DOCUMENT && p->doc_ids == nullptr) return FLEXATTN_ERR_NULL_POINTER;
  if (p->score_kind == FLEXATTN_SCORE_ALIBI && p->alibi_slopes == nullptr) return FLEXATTN_ERR_NULL_POINTER;
  if (p->score_kind == FLEXATTN_SCORE_SOFTCAP && !(p->softcap > 0.f)) return FLEXATTN_ERR_UNSUPPORTED_MOD;
  if (p->score_kind == FLEXATTN_SCORE_USER && p->user_score <= 0) return FLEXATTN_ERR_UNSUPPORTED_MOD;
  return FLEXATTN_OK;
}

int validate_workspace(const FlexAttnParams* p) {
  if (p->workspace == nullptr) return FLEXATTN_ERR_NULL_POINTER;
  if (!aligned16(p->workspace)) return FLEXATTN_ERR_MISALIGNED;
  MapLayout L = map_layout(p->batch, p->seq_q, p->seq_k, p->mask_kind);
  if (p->workspace_bytes < L.bytes) return FLEXATTN_ERR_WORKSPACE_TOO_SMALL;
  return FLEXATTN_OK;
}

// true when the tensor-core kernels serve this problem
bool use_tcgen05(const FlexAttnParams* p, int* err) {
  // the tensor-core kernels take bf16 and D in {64, 128}
  const bool capable = p->dtype == FLEXATTN_BF16 && (p->head_dim == 64 || p->head_dim == 128);
  *err = FLEXATTN_OK;
  // a user score function exists only as a run-time compiled tensor-core kernel
  if (p->score_kind == FLEXATTN_SCORE_USER && (!capable || p->backend == FLEXATTN_BACKEND_SIMT)) {
    *err = FLEXATTN_ERR_UNSUPPORTED_BACKEND;
    return false;
  }
  if (p->backend == FLEXATTN_BACKEND_SIMT) return false;
  if (p->backend == FLEXATTN_BACKEND_TCGEN05 && !capable) *err = FLEXATTN_ERR_UNSUPPORTED_BACKEND;
  return capable;
}

DevParams make_dev(const FlexAttnParams* p) {
  DevParams d{};
  MapLayout L = map_layout(p->batch, p->seq_q, p->seq_k, p->mask_kind);
  char* ws = static_cast<char*>(p->workspace);
  d.q = p->q; d.k = p->k; d.v = p->v; d.o = p->o; d.d_o = p->d_o;
  d.dq = p->dq; d.dk = p->dk; d.dv = p->dv;
  d.l = p->l; d.m = p->m; d.delta = p->delta;
  d.doc_ids = p->mask_kind == FLEXATTN_MASK_DOCUMENT ? p->doc_ids : nullptr;
  d.alibi_slopes = p->score_kind == FLEXATTN_SCORE_ALIBI ? p->alibi_slopes : nullptr;
  d.ab = p->ab;
  d.dab = p->dab;
  d.row_map = reinterpret_cast<const int4*>(ws + L.off_row);
  d.col_map = reinterpret_cast<const int4*>(ws + L.off_col);
  d.order = reinterpret_cast<const int32_t*>(ws + L.off_order);
  d.order_rm = reinterpret_cast<const int4*>(ws + L.off_order_rm);
  d.order_pair = reinterpret_cast<const int32_t*>(ws + L.off_order_pair);
  if (p->mask_kind == FLEXATTN_MASK_DOCUMENT) {
    d.run_lo = reinterpret_cast<const int32_t*>(ws + L.off_run_lo);
    d.run_hi = reinterpret_cast<const int32_t*>(ws + L.off_run_hi);
    d.doc_sorted = reinterpret_cast<const int32_t*>(ws + L.off_sorted);
  }
  d.status = p->status;
  d.batch = p->batch; d.heads = p->heads; d.seq_q = p->seq_q; d.seq_k = p->seq_k; d.head_dim = p->head_dim;
  d.n_qt = L.n_qt; d.n_kt = L.n_kt; d.map_rows = L.rows;
  d.doc_stride = p->seq_q > p->seq_k ? p->seq_q : p->seq_k;
  d.window = p->window; d.stride = p->stride > 0 ? p->stride : 1;
  d.sm_scale = p->sm_scale; d.cap = p->score_kind == FLEXATTN_SCORE_SOFTCAP ? p->softcap : 0.f;
  d.user_score = p->score_kind == FLEXATTN_SCORE_USER ? p->user_score : 0;
  return d;
}

// for the kernels that have a gathered form of S2, where s2_gathers
void gather_s2(DevParams* d) {
  if (d->stride > d->seq_k) d->stride = d->seq_k;  // (key 0 is on every grid; a tensor map's pitch is bounded)
  d->n_st = (s2_keys(d->seq_k, d->stride) + kTile - 1) / kTile;
}

#define FLEXATTN_REQUIRE(ptr)                                     \
  do {                                                            \
    if ((ptr) == nullptr) return FLEXATTN_ERR_NULL_POINTER;       \
    if (!aligned16(ptr)) return FLEXATTN_ERR_MISALIGNED;          \
  } while (0)

int prologue(const FlexAttnParams* p) {
  int e = validate_common(p);
  if (e) return e;
  e = validate_mods(p);
  if (e) return e;
  return validate_workspace(p);
}

}  // namespace

// Everything flexattn_fwd checks before it launches (shapes, kinds, workspace, pointers, backend).  tc: whether
// the tensor-core kernel serves the call.
int validate_fwd_args(const FlexAttnParams* p, bool* tc) {
  int e = prologue(p);
  if (e) return e;
  FLEXATTN_REQUIRE(p->q); FLEXATTN_REQUIRE(p->k); FLEXATTN_REQUIRE(p->v); FLEXATTN_REQUIRE(p->o);
  FLEXATTN_REQUIRE(p->l); FLEXATTN_REQUIRE(p->m);
  *tc = use_tcgen05(p, &e);
  return e;
}

}  // namespace flexattn

using namespace flexattn;

extern "C" {

int flexattn_abi_version(void) { return FLEXATTN_ABI_VERSION; }

const char* flexattn_status_string(int status) {
  switch (status) {
    case FLEXATTN_OK: return "ok";
    case FLEXATTN_ERR_NULL_POINTER: return "null pointer";
    case FLEXATTN_ERR_BAD_SHAPE: return "bad shape";
    case FLEXATTN_ERR_UNSUPPORTED_DTYPE: return "unsupported dtype";
    case FLEXATTN_ERR_UNSUPPORTED_HEAD_DIM: return "unsupported head_dim (32, 64 or 128)";
    case FLEXATTN_ERR_MISALIGNED: return "pointer not 16-byte aligned";
    case FLEXATTN_ERR_WORKSPACE_TOO_SMALL: return "workspace too small";
    case FLEXATTN_ERR_UNSUPPORTED_MOD: return "unsupported or ill-formed score_mod / mask";
    case FLEXATTN_ERR_CUDA: return "CUDA error at launch";
    case FLEXATTN_ERR_TIMEOUT: return "device-side wait timed out";
    case FLEXATTN_ERR_UNSUPPORTED_BACKEND: return "backend cannot serve this dtype / head_dim";
    case FLEXATTN_ERR_NOALLOC_LIMIT:
      return "mask map larger than the fixed scratch array of the no-allocation entry point (1 MiB)";
    case FLEXATTN_ERR_JIT_UNAVAILABLE: return "run-time compiler (libnvrtc) or driver module loader not available";
    case FLEXATTN_ERR_JIT_COMPILE: return "the user score function did not compile (see flexattn_user_score_log)";
    case FLEXATTN_ERR_DEBUG_BOUNDS: return "bounds-checked build: an out-of-range global-memory access was skipped";
    default: return "unknown status";
  }
}

size_t flexattn_workspace_bytes(const FlexAttnParams* p) {
  if (validate_common(p) != FLEXATTN_OK) return 0;
  return map_layout(p->batch, p->seq_q, p->seq_k, p->mask_kind).bytes;
}

int flexattn_build_mask_map(void* stream, const FlexAttnParams* p) {
  NvtxRange nvtx("flexattn_build_mask_map");
  int e = prologue(p);
  if (e) return e;
  if (p->mask_kind == FLEXATTN_MASK_DOCUMENT && (reinterpret_cast<uintptr_t>(p->doc_ids) & 3u)) return FLEXATTN_ERR_MISALIGNED;
  return launch_mask_map(static_cast<cudaStream_t>(stream), *p) == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}

namespace {
// kv tiles an average query tile visits, from the mask kind alone (a document mask depends on the data: 0, never split)
int mean_kv_tiles(const FlexAttnParams* p) {
  const int n_kt = (p->seq_k + FLEXATTN_TILE - 1) / FLEXATTN_TILE;
  const int in_window = p->window / FLEXATTN_TILE + 1;
  switch (p->mask_kind) {
    case FLEXATTN_MASK_NONE: return n_kt;
    case FLEXATTN_MASK_CAUSAL: return (n_kt + 1) / 2;
    case FLEXATTN_MASK_SLIDING_WINDOW: return n_kt < in_window ? n_kt : (n_kt + in_window) / 2;  // window back, all ahead
    case FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL: return n_kt < in_window ? n_kt : in_window;
    case FLEXATTN_MASK_S2: return (n_kt + 1) / 2;  // strided columns keep every tile below the diagonal alive
    default: return 0;
  }
}
constexpr int kSplitMinTiles = 12;  // kv tiles a query tile sees from which its split over CTAs pays
int forced_fwd_kernel() {  // 0: choose by shape, 1: two-query-tile kernel, 2: persistent kernel, 3: split kernel
  static const int choice = [] {
    const char* e = getenv("FLEXATTN_FWD_KERNEL");
    if (e == nullptr) return 0;
    if (strcmp(e, "pair") == 0) return 1;
    if (strcmp(e, "pipe") == 0) return 2;
    if (strcmp(e, "split") == 0) return 3;
    return 0;
  }();
  return choice;
}
// CTAs per query tile of the split kernel (fwd_split_sm100.cu); 0: another kernel.  It takes rows of kSplitMinTiles kv tiles
// where a query tile gets at least two CTAs, or where its only tile has no more than 32 rows (the other warps then skip
// their part).  Against the persistent kernel: 64 slices x 1 row x 8191 keys 108 (two-query-tile kernel) -> 47 us, 74 x 4096
// 39 -> 31, 256 x 6 rows x 8663 (D = 64) 146 -> 127, one causal slice of 4096 39 -> 20; with one CTA per tile and full
// tiles the persistent kernel's overlap of items wins (144 x 100 rows x 3000 39 us against 48), and with shorter rows
// ([16,64,1] x 1024 keys 85 against 109).
int kv_splits(const FlexAttnParams* p) {
  if (p->ab != nullptr || p->score_kind == FLEXATTN_SCORE_USER) return 0;
  const int sms = sm_count(), tiles = mean_kv_tiles(p);
  const long long n_qt = (p->seq_q + FLEXATTN_TILE - 1) / FLEXATTN_TILE, items = n_qt * p->batch * p->heads;
  if (sms <= 0 || tiles < kSplitMinTiles || items > 0x7fffffff / 8) return 0;
  // as many CTAs as run at once (a second wave of clusters costs what the split gains), with four kv tiles or more each
  int c = 1;
  while (c < 8 && tiles >= 8 * c && items <= split_clusters_at_once(2 * c)) c *= 2;
  return c > 1 || p->seq_q <= 32 ? c : 0;
}
// Whether S2 that would be gathered goes to the split kernel, in its dense form: where that takes the rows of a few query tiles apart
// so far that one of its streams has less than a quarter of the longest gathered row.  One slice of 4096, D = 64, us gathered / split: 64 keys
// and stride 2 25.4 / 20.3, 512 and 3 21.9 / 20.4, 64 and 3 20.1 / 20.3, 512 and 4 19.2 / 20.5; 5000 (two CTAs a query tile) 64 and 2 29.4 / 35.3.
bool split_beats_gathered_s2(const FlexAttnParams* p) {
  const int c = kv_splits(p), n = (std::min(p->seq_q, p->seq_k) + FLEXATTN_TILE - 1) / FLEXATTN_TILE;
  return c > 0 && (double)p->window / FLEXATTN_TILE + 2 + (double)n / p->stride > 4.0 * n / (2 * c);
}
}  // namespace

int flexattn_fwd(void* stream, const FlexAttnParams* p) {
  NvtxRange nvtx("flexattn_fwd");
  bool tc = false;
  const int e = validate_fwd_args(p, &tc);
  if (e) return e;
  DevParams d = make_dev(p);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (tc) {
    // Three tensor-core forward kernels: the two-query-tile one (fwd_pair_sm100.cu: one row per thread, K/V shared by two
    // tiles, pairs dealt out as CTAs get on; the fastest where there are enough of them), the persistent one (fwd_pipe_sm100.cu:
    // query tiles one by one, for fewer items, a dense bias and gathered S2) and the split one (fwd_split_sm100.cu: a cluster per
    // query tile, best for few query tiles against many keys).  FLEXATTN_FWD_KERNEL=pair, =pipe or =split in the environment
    // forces one where it can run (read once per process).
    const bool pair_can = p->ab == nullptr;
    const int forced = forced_fwd_kernel();
    if (forced == 0 && s2_gathers(*p) && !split_beats_gathered_s2(p)) {  // (few tiles a query tile: the persistent kernel)
      DevParams g = d;
      gather_s2(&g);
      const int r = launch_sm100_fwd_pipe(st, g, p->score_kind, p->mask_kind);
      if (r != FLEXATTN_ERR_UNSUPPORTED_BACKEND) return r;  // (its tensor maps were refused, nothing launched: the dense form)
    }
    if (forced == 0 || forced == 3) {
      d.kv_splits = kv_splits(p);
      if (forced == 3 && d.kv_splits == 0 && pair_can && p->score_kind != FLEXATTN_SCORE_USER &&
          p->mask_kind != FLEXATTN_MASK_DOCUMENT)
        d.kv_splits = 1;
      if (d.kv_splits > 0) {
        const int r = launch_sm100_fwd_split(st, d, p->score_kind, p->mask_kind);
        if (r != FLEXATTN_ERR_UNSUPPORTED_BACKEND) return r;
      }
    }
    bool pair = pair_can && (forced == 1 || (forced == 0 && fwd_pair_pays(*p, sm_count())));
    if (pair_can && forced == 0 && p->score_kind == FLEXATTN_SCORE_USER)
      pair = jit_first_or_loaded(pair ? kJitForwardPair : kJitForward, pair ? kJitForward : kJitForwardPair, p->user_score, p->head_dim,
                                 p->mask_kind, st) == kJitForwardPair;
    if (pair) {
      const int r = launch_sm100_fwd_pair(st, d, p->score_kind, p->mask_kind);
      if (r != FLEXATTN_ERR_UNSUPPORTED_BACKEND && r != FLEXATTN_ERR_JIT_COMPILE) return r;
    }
    if (d.ab != nullptr) return launch_sm100_fwd_pipe_bias(st, d, p->score_kind, p->mask_kind);
    return launch_sm100_fwd_pipe(st, d, p->score_kind, p->mask_kind);
  }
  return launch_simt_fwd(st, d, p->dtype, p->score_kind, p->mask_kind) == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}

int flexattn_bwd_preprocess(void* stream, const FlexAttnParams* p) {
  NvtxRange nvtx("flexattn_bwd_preprocess");
  int e = validate_common(p);
  if (e) return e;
  FLEXATTN_REQUIRE(p->o); FLEXATTN_REQUIRE(p->d_o); FLEXATTN_REQUIRE(p->delta);
  return launch_delta(static_cast<cudaStream_t>(stream), *p) == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}

namespace {
int launch_dq(cudaStream_t st, const FlexAttnParams* p, bool tc) {
  const DevParams d = make_dev(p);
  if (tc && (d.ab != nullptr || d.dab != nullptr)) return launch_sm100_dq_bias(st, d, p->score_kind, p->mask_kind);
  if (tc) return launch_sm100_dq(st, d, p->score_kind, p->mask_kind);
  return launch_simt_dq(st, d, p->dtype, p->score_kind, p->mask_kind) == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}
int launch_dkv(cudaStream_t st, const FlexAttnParams* p, bool tc) {
  const DevParams d = make_dev(p);
  if (tc && d.ab != nullptr) return launch_sm100_dkv_bias(st, d, p->score_kind, p->mask_kind);
  if (tc) return launch_sm100_dkv(st, d, p->score_kind, p->mask_kind);
  return launch_simt_dkv(st, d, p->dtype, p->score_kind, p->mask_kind) == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}
// `to` waits for what has been enqueued on `from` so far.
int order_after(cudaStream_t to, cudaStream_t from, cudaEvent_t ev) {
  return cudaEventRecord(ev, from) == cudaSuccess && cudaStreamWaitEvent(to, ev, 0) == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}
}  // namespace

int flexattn_bwd_dq(void* stream, const FlexAttnParams* p) {
  NvtxRange nvtx("flexattn_bwd_dq");
  int e = prologue(p);
  if (e) return e;
  FLEXATTN_REQUIRE(p->q); FLEXATTN_REQUIRE(p->k); FLEXATTN_REQUIRE(p->v); FLEXATTN_REQUIRE(p->d_o);
  FLEXATTN_REQUIRE(p->l); FLEXATTN_REQUIRE(p->m); FLEXATTN_REQUIRE(p->delta); FLEXATTN_REQUIRE(p->dq);
  const bool tc = use_tcgen05(p, &e);
  if (e) return e;
  return launch_dq(static_cast<cudaStream_t>(stream), p, tc);
}

int flexattn_bwd_dkv(void* stream, const FlexAttnParams* p) {
  NvtxRange nvtx("flexattn_bwd_dkv");
  int e = prologue(p);
  if (e) return e;
  FLEXATTN_REQUIRE(p->q); FLEXATTN_REQUIRE(p->k); FLEXATTN_REQUIRE(p->v); FLEXATTN_REQUIRE(p->d_o);
  FLEXATTN_REQUIRE(p->l); FLEXATTN_REQUIRE(p->m); FLEXATTN_REQUIRE(p->delta);
  FLEXATTN_REQUIRE(p->dk); FLEXATTN_REQUIRE(p->dv);
  const bool tc = use_tcgen05(p, &e);
  if (e) return e;
  return launch_dkv(static_cast<cudaStream_t>(stream), p, tc);
}

int flexattn_bwd(void* stream, void* side_stream, const FlexAttnParams* p) {
  NvtxRange nvtx("flexattn_bwd");
  int e = prologue(p);
  if (e) return e;
  FLEXATTN_REQUIRE(p->q); FLEXATTN_REQUIRE(p->k); FLEXATTN_REQUIRE(p->v); FLEXATTN_REQUIRE(p->o); FLEXATTN_REQUIRE(p->d_o);
  FLEXATTN_REQUIRE(p->l); FLEXATTN_REQUIRE(p->m); FLEXATTN_REQUIRE(p->delta);
  FLEXATTN_REQUIRE(p->dq); FLEXATTN_REQUIRE(p->dk); FLEXATTN_REQUIRE(p->dv);
  const bool tc = use_tcgen05(p, &e);
  if (e) return e;
  cudaStream_t st = static_cast<cudaStream_t>(stream), side = static_cast<cudaStream_t>(side_stream);
  if (launch_delta(st, *p) != cudaSuccess) return FLEXATTN_ERR_CUDA;
  if (side == st) {
    e = launch_dkv(st, p, tc);
    return e ? e : launch_dq(st, p, tc);
  }
  // an event of this call's own: a shared one could be recorded by another thread between the record and the wait
  cudaEvent_t ev = nullptr;
  if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return FLEXATTN_ERR_CUDA;
  e = order_after(side, st, ev);
  if (e == FLEXATTN_OK) {
    e = launch_dkv(side, p, tc);
    const int e_dq = launch_dq(st, p, tc);
    const int e_join = order_after(st, side, ev);  // also after a failed launch: the caller frees by `stream` alone
    if (e == FLEXATTN_OK) e = e_dq ? e_dq : e_join;
  }
  cudaEventDestroy(ev);  // (given back once the recorded work is done)
  return e;
}

namespace {
int forced_bwd_kernel() {  // 0: choose by shape, 1: fused, 2: separate kernels
  static const int choice = [] {
    const char* e = getenv("FLEXATTN_BWD_KERNEL");
    if (e == nullptr) return 0;
    return strcmp(e, "fused") == 0 ? 1 : strcmp(e, "split") == 0 ? 2 : 0;
  }();
  return choice;
}
bool fused_can(const FlexAttnParams* p) {
  int e = FLEXATTN_OK;
  return use_tcgen05(p, &e) && e == FLEXATTN_OK && p->ab == nullptr && p->dab == nullptr;
}
// Whether the fused backward serves the call.  It does 5 contractions of a tile pair and its exponentials once where dQ and dK/dV
// do 7 and twice, but the parts of a query tile are added one after the other: a kv tile has to stay some 2.4 tiles behind the
// one before it in its slice.  `slack`, the query tiles a CTA walks per kv tile of the slice that is in flight, says whether
// there is room for that.  Times in us, fused / separate, on 148 SMs, calls one after the other on a stream (replayed from a
// graph, where dQ starts before dK/dV, the separate ones are up to a tenth slower; the lines are drawn by the mean of both);
// slices x queries x keys.
// D = 64, where the exponentials weigh most:
//   no mask     slack 2.6: 24 x 2048 127 / 159, 192 x 256 31 / 44; 1.7: 16 x 2048 128 / 111, 32 x 1024 x 8192 398 / 383;
//               0.1: 16 x 128 x 8192 211 / 87.  Chains of few parts need less: 64 x 512 40 / 45, 48 x 512 37 / 37
//   causal, S2  24 x 1024 43 / 43, 28 x 1000 43 / 48; 16 x 2048 88 / 82, 16 x 1536 65 / 54, 18 x 1152 52 / 41
//   windows and documents, 16 slices on: 16 x 1280 25 / 30 and 33 / 36
//   softcap and user functions (more per pair, the same chain): 16 x 2048 unmasked 131 / 148, 32 x 720 53 / 56;
//               32 x 237 x 8081 303 / 185
// D = 128, where its shared-memory traffic (dQ on its way out) takes most of the gain:
//   no mask     128 x 1024 240 / 269, 12 x 8192 1159 / 1260, 160 x 512 x 64 53 / 61, 96 x 256 38 / 40; 16 x 8192 1735 / 1661,
//               64 x 1024 147 / 130, 6 x 15360 1983 / 1897, 32 x 2048 x 8192 976 / 870, 8 x 32768 15154 / 11871,
//               96 x 1024 x 384 107 / 95
//   causal, S2  128 x 8192 6371 / 7090, 24 x 8192 1290 / 1357, 96 x 256 31 / 33, 64 x 512 43 / 44; 64 x 873 90 / 86,
//               16 x 16384 3453 / 3259, 9 x 16384 2100 / 1927, 64 x 1024 x 512 81 / 74, 192 x 12544 x 384 2217 / 1968
//   windows and documents: 128 x 2048 documents 349 / 406, 48 x 4096 with 1024 keys 375 / 404; 16 x 2048 with 256 keys 49 / 46
//   softcap     16 x 2048 causal 103 / 113, 40 x 512 38 / 39, 64 x 512 unmasked 57 / 63; 16 x 1536 causal 82 / 74,
//               24 x 1024 unmasked 86 / 74, 64 x 14683 x 492 causal 1307 / 1205
//   a window open ahead: 256 x 528 207 / 240; 128 x 4096 2154 / 2013
//   user functions: none (16 x 2048 causal 112 / 109, unmasked 169 / 155, 64 x 1024 131 / 122; 64 x 4096 1075 / 1073, 1822 / 1905)
// Either: 72 x 445 x 18173 causal 192 / 304, 64 x 256 x 8960 with 267 keys 66 / 113 (most kv tiles see no query);
//         16 x 496 x 1206 causal 33 / 29, 24 x 264 x 4885 45 / 41
bool fused_pays(const FlexAttnParams* p) {
  const int forced = forced_bwd_kernel();
  if (forced) return forced == 1;
  const long long slices = (long long)p->batch * p->heads, sms = sm_count();
  if (sms <= 0 || slices < 1) return false;
  const long long n_qt = (p->seq_q + FLEXATTN_TILE - 1) / FLEXATTN_TILE, n_kt = (p->seq_k + FLEXATTN_TILE - 1) / FLEXATTN_TILE;
  const int mask = p->mask_kind;
  const bool common_start = mask == FLEXATTN_MASK_NONE || mask == FLEXATTN_MASK_SLIDING_WINDOW;  // every kv tile begins at query 0
  const bool long_rows = mask == FLEXATTN_MASK_CAUSAL || mask == FLEXATTN_MASK_S2;  // ... along the diagonal, all to the last query
  const bool scored = p->score_kind == FLEXATTN_SCORE_SOFTCAP || p->score_kind == FLEXATTN_SCORE_USER;
  const long long items = slices * (common_start || n_kt < n_qt ? n_kt : n_qt);  // kv tiles that see a query
  // many kv tiles that see no query: the fused kernel only stores their zeros
  if (!common_start && n_kt >= 3 * n_qt && slices >= 16 && slices * n_kt >= 7 * sms)
    return p->head_dim == 64 || p->score_kind != FLEXATTN_SCORE_USER;
  // S2, gathered: the separate kernels walk every tile below the diagonal.  The fused one takes as long as its longest strided tile's
  // row of query tiles, which they match while they fit the chip at once: slices x queries, 128 keys, stride 32: 8 x 3000 (D = 64)
  // 58 / 79, 16 x 1500 37 / 52, 16 x 2000 (D = 128) 61 / 86, 16 x 8000 255 / 841; 4 x 5000 113 / 97, 8 x 2000 55 / 41, 16 x 1100 39 / 35.
  // Every other key on the grid makes as many strided tiles as window tiles, and all of them see the last query tiles, one after the
  // other; long rows of few slices wait alike at D = 128 (64 keys): stride 2 3 x 8192 (D = 64) 194 / 155, 8 x 3200 86 / 85, 4 x 8192 201 / 223;
  // stride 4 at D = 128 2 x 12000 241 / 226, 3 x 8192 174 / 166, 6 x 4096 104 / 105.
  if (s2_gathers(*p)) return 5 * items >= (p->stride == 2 || (p->head_dim == 128 && slices < 4) ? 8 : 6) * sms;
  if (items < sms) return false;
  const double slack = bwd_fused_slack(*p, (int)sms);
  if (p->head_dim == 64) {
    if (slices < 16) return false;
    if (common_start && scored) return slack >= 1.1;
    if (common_start) return slack >= 2 || slices >= sms || (slack >= 1.25 && slices >= 8 * n_kt);
    return !long_rows || slices >= 24 || slack >= (scored ? 1.25 : 1.8);
  }
  if (p->score_kind == FLEXATTN_SCORE_USER) return false;
  const bool few = items < 5 * sms;
  if (scored) {
    if (slices < 16 || (n_qt > 2 * n_kt && few && slices < sms)) return false;
    if (common_start) return slack >= 1.7 || slices >= sms;
    return mask == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL || slices >= 40 || 5 * items >= 8 * sms;
  }
  if (mask == FLEXATTN_MASK_SLIDING_WINDOW) return slices >= sms && n_qt <= 8;
  if (slices >= sms && (slack >= 2.1 || n_qt <= 32)) return true;
  if (n_qt > n_kt && few && (common_start || long_rows)) return false;
  if (common_start) return (slack >= (slices >= 24 ? 2.2 : 2.4) && 2 * items >= 5 * sms) || (slices >= 96 && n_kt <= 2);
  if (slices >= (long_rows && n_qt > 4 ? 96 : 64)) return true;
  return 2 * items >= 9 * sms && (long_rows ? slices >= 24 && slack >= 2.2 : slices >= 16);
}
}  // namespace

size_t flexattn_bwd_scratch_bytes(const FlexAttnParams* p) {
  // (asked before the pointers are bound, so not all of `prologue`; the numbers below divide by the window)
  if (validate_common(p) != FLEXATTN_OK || validate_window(p) != FLEXATTN_OK || !fused_can(p) || !fused_pays(p)) return 0;
  return bwd_fused_scratch_bytes(*p);
}

int flexattn_bwd_fused(void* stream, const FlexAttnParams* p, void* scratch, size_t scratch_bytes) {
  NvtxRange nvtx("flexattn_bwd_fused");
  int e = prologue(p);
  if (e) return e;
  FLEXATTN_REQUIRE(p->q); FLEXATTN_REQUIRE(p->k); FLEXATTN_REQUIRE(p->v); FLEXATTN_REQUIRE(p->o); FLEXATTN_REQUIRE(p->d_o);
  FLEXATTN_REQUIRE(p->l); FLEXATTN_REQUIRE(p->m); FLEXATTN_REQUIRE(p->delta);
  FLEXATTN_REQUIRE(p->dq); FLEXATTN_REQUIRE(p->dk); FLEXATTN_REQUIRE(p->dv); FLEXATTN_REQUIRE(scratch);
  if (!fused_can(p)) return FLEXATTN_ERR_UNSUPPORTED_BACKEND;
  DevParams d = make_dev(p);
  if (s2_gathers(*p)) gather_s2(&d);
  if (scratch_bytes < bwd_fused_scratch_bytes(*p)) return FLEXATTN_ERR_WORKSPACE_TOO_SMALL;
  return launch_sm100_bwd_fused(static_cast<cudaStream_t>(stream), d, p->score_kind, p->mask_kind, scratch);
}

int flexattn_read_mask_map(void* stream, const FlexAttnParams* p, int which, int b, int index, int32_t out[4]) {
  int e = prologue(p);
  if (e) return e;
  if (out == nullptr) return FLEXATTN_ERR_NULL_POINTER;
  MapLayout L = map_layout(p->batch, p->seq_q, p->seq_k, p->mask_kind);
  const int n = which ? L.n_kt : L.n_qt;
  if (b < 0 || b >= L.rows || index < 0 || index >= n || (which != 0 && which != 1)) return FLEXATTN_ERR_BAD_SHAPE;
  const char* src = static_cast<const char*>(p->workspace) + (which ? L.off_col : L.off_row) +
                    sizeof(int4) * ((size_t)b * n + index);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemcpyAsync(out, src, sizeof(int4), cudaMemcpyDeviceToHost, st) != cudaSuccess) return FLEXATTN_ERR_CUDA;
  return cudaStreamSynchronize(st) == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}

}  // extern "C"
