// The whole backward in one pass over the tile pairs on the 5th-generation tensor cores (sm_100a): five contractions
// per pair where the separate dQ and dK/dV kernels (bwd_dq_sm100.cu, bwd_dkv_sm100.cu; the reference's two Pallas
// kernels, flex_attention_dq_bwd.py:282-385 and flex_attention_dkv_kernel.py:177-280) take seven, and the exponentials
// of a pair once instead of twice.
//
//   S^T  = K Q^T, dP^T = V dO^T      thread = key row, columns = query positions
//   P^T, dS^T                        bf16 over S^T / dP^T in tensor memory; dS^T also as a shared-memory tile
//   dV += P^T dO ; dK += dS^T Q      A from tensor memory
//   dQ_part = dS K                   A = the dS^T tile read M-major, B = K read MN-major
//
// A work item is a 128-row kv tile of one slice; dK and dV stay in tensor memory over its query tiles, dQ_part is added
// to an f32 scratch in L2 with bulk reductions.  dq is stored by the CTA with the last part of a query tile,
// which takes the sum back, or by a small kernel at the end (fused_plan says which).  Tensor memory is full at D = 128
// (S, dP, dK, dV = 512 columns): dQ_part takes the dP columns, whose dS^T the dK MMA has read by then (MMAs of one thread
// execute in issue order), and dP of the next tile follows once the drain warps hold dQ_part in registers.  Issue order:
//
//   ... dV(n) S(n+1) dK(n) dQ(n) dP(n+1) dV(n+1) S(n+2) ...      (D = 64: dP(n+1) before dQ(n), which has its own columns)
//
// Results repeat bit for bit: the parts of a query tile are added in ONE order, kv tiles from the last one down.  A flag
// per query tile says which kv tile has been added last; the turn warp waits for the predecessor's.  Items are taken in
// list order from a ticket counter and wait only for items earlier in the list, which are running or done, so somebody
// always gets on; under a causal mask the kv tiles of a slice walk along the diagonal one step apart, and the waits are
// over before they begin.  Slices are taken in groups whose Q, dO and scratch fit L2, and the scratch is a ring of a few
// groups' slices: the first part of a query tile waits until the tile's last user in the ring is done.
//
// Persistent: one CTA of 16 warps per SM.  0-7 element-wise (two warpgroups, 64 query columns each), 8-11 drain,
// 12 MMA issue, 13 loads, 14 turn, 15 publishes flags.
#include "sched.cuh"
#include "sm100.cuh"

namespace flexattn {
namespace FLEXATTN_TU_NAMESPACE {

constexpr int kThreads = 512;
constexpr int kDrainWarp = 8, kMmaWarp = 12, kTmaWarp = 13, kTurnWarp = 14;  // 15: flags
constexpr int kRegsEw = 152, kRegsDrain = 152, kRegsRest = 56;  // 2 * 152 + 152 + 56 = 4 * 128: what the launch holds
constexpr int kItemRing = 4;
constexpr int kFusedId = 7;  // kernel id in the status words
constexpr int kAllAdded = 0x40000000;
constexpr uint32_t kSlotBytes = 4096;  // 32 columns of a drain warp's 32 rows; two slots per warp

struct FusedArgs {
  float* dq_acc;   // [ring][n_qt][128 * D] (S2, gathered: [chains of a launch][n_qt]...): element (32 w + lane, 4 c + k) of a tile at ((w * D / 4 + c) * 32 + lane) * 4 + k
  float* stats;    // [slices][n_qt][2][128]: -(m log2e + log2 l) pre-scaled for pack_bf16_trunc, delta
  int32_t* flags;  // [slices * chains][n_qt]: n_kt - (kv tile added last), 0: none, kAllAdded
  int32_t* ticket;
  int slice0, slices;  // slices of this launch (of batch * heads)
  int group, ring;     // how many of them form a group, and how many the scratch holds
  int store_dq;        // the last part of a query tile stores dq; otherwise it is added like the others
  int chains;          // sums per query tile: 2 for S2, gathered (window tiles, strided tiles: chain = 2 * slice + strided), else 1
  float* s2_dkv;       // ... f32 dK (unscaled) and dV of the keys on the stride grid, from their window tile and their strided one:
                       // [slices][keys on the grid][2: window, strided][2: dK, dV][D]
};

// Query tiles of kv tile `kt`: {first, end, first fully kept, end of those}
template <int MK>
__device__ __forceinline__ int4 col_entry(const DevParams& P, int b, int kt) {
  if constexpr (MK == kMaskS2Gather) return s2_col(kt, P.seq_q, P.seq_k, P.n_qt, P.n_kt, P.window, P.stride);
  return __ldg(&P.col_map[(size_t)(P.map_rows > 1 ? b : 0) * P.n_kt + kt]);
}

struct FusedSmem {
  uint64_t bar_k[2], bar_v[2], bar_kfree[2], bar_vfree[2], bar_q[2], bar_do[2], bar_qfree[2], bar_dofree[2];
  uint64_t bar_s, bar_dp, bar_p, bar_ds, bar_dq, bar_drained, bar_accfree, bar_stage[2], bar_stagefree[2];
  uint64_t bar_turn[2], bar_turnfree[2], bar_red[2], bar_back[4][2], bar_item[kItemRing], bar_itemfree[kItemRing];
  uint32_t tmem_base;
  alignas(16) int4 item_a[kItemRing];  // {slice of this launch (-1: no more), kv tile, first q tile, end q tile}
  alignas(16) int2 item_b[kItemRing];  // {first fully kept q tile, end of the fully kept run}
  alignas(16) int4 turn[2];            // {slice (-1: no more), query tile, 1: first part, 2: last part (or both), flag value}
  alignas(16) float stats[2][2][kTile];
};

// what the score functions see besides the score
struct FusedScoreCtx {
  float sm_scale, c2, slope2, capl2, csc;
  int b, h, j;
};

__device__ __forceinline__ void load_cols32(float (&dst)[32], const float* __restrict__ src) {
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    const float4 t = *reinterpret_cast<const float4*>(src + c);
    dst[c] = t.x;
    dst[c + 1] = t.y;
    dst[c + 2] = t.z;
    dst[c + 3] = t.w;
  }
}

// 32 query columns from i_first on: raw S^T in s, out p * dsigma (what dS^T needs) in s and packed bf16 P^T.
// nl: the columns' statistics; keep: kept columns of this key row (partial tiles).
template <int SK, bool kPartial>
__device__ __forceinline__ void fused_p32(uint32_t (&s)[32], uint32_t (&pk)[16], const float (&nl)[32], uint32_t keep,
                                          int i_first, const FusedScoreCtx& x) {
  if constexpr (SK == FLEXATTN_SCORE_SOFTCAP || SK == FLEXATTN_SCORE_USER) {
#pragma unroll
    for (int c = 0; c < 32; c += 2) {
      float pv[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int cc = c + u;
        float arg, dsig;
        if constexpr (SK == FLEXATTN_SCORE_USER) {
          const float sc = __uint_as_float(s[cc]) * x.sm_scale;
          arg = fmaf(user_score(sc, x.b, x.h, i_first + cc, x.j), kLog2e, nl[cc]);
          dsig = user_dscore(sc, x.b, x.h, i_first + cc, x.j);
        } else {
          const float th = ptx::tanh_approx(__uint_as_float(s[cc]) * x.csc);
          arg = fmaf(x.capl2, th, nl[cc]);
          dsig = fmaf(-th, th, 1.f);
        }
        float p = ptx::ex2(arg);
        float pd = p * dsig;
        if constexpr (kPartial) {  // a masked position contributes nothing, whatever the score function's derivative is there
          p = (keep >> cc) & 1u ? p : 0.f;
          pd = (keep >> cc) & 1u ? pd : 0.f;
        }
        pv[u] = p;
        s[cc] = __float_as_uint(pd);
      }
      pk[c >> 1] = ptx::pack_bf16_trunc(pv[0], pv[1]);
    }
  } else {
    const uint64_t c22 = ptx::pack2(x.c2, x.c2);
    const float abase = x.slope2 * (float)(x.j - i_first);  // ALiBi: slope * (j - i), one packed add per pair of columns
    uint64_t b2 = ptx::pack2(abase, abase - x.slope2);
    const uint64_t bstep2 = ptx::pack2(-2.f * x.slope2, -2.f * x.slope2);
#pragma unroll
    for (int c = 0; c < 32; c += 2) {
      const uint64_t sv2 = ptx::pack2(__uint_as_float(s[c]), __uint_as_float(s[c + 1]));
      const uint64_t nl2 = ptx::pack2(nl[c], nl[c + 1]);
      uint64_t arg2;
      if constexpr (SK == FLEXATTN_SCORE_ALIBI) {
        arg2 = ptx::fma2(sv2, c22, ptx::add2(b2, nl2));
        b2 = ptx::add2(b2, bstep2);
      } else {
        arg2 = ptx::fma2(sv2, c22, nl2);
      }
      float a0, a1;
      ptx::unpack2(arg2, a0, a1);
      float p0 = ptx::ex2(a0), p1 = ptx::ex2(a1);
      if constexpr (kPartial) {
        p0 = (keep >> c) & 1u ? p0 : 0.f;
        p1 = (keep >> (c + 1)) & 1u ? p1 : 0.f;
      }
      pk[c >> 1] = ptx::pack_bf16_trunc(p0, p1);
      s[c] = __float_as_uint(p0);
      s[c + 1] = __float_as_uint(p1);
    }
  }
}

// dS^T = (p dsigma) * (dP^T - delta), packed bf16
__device__ __forceinline__ void fused_ds32(const uint32_t (&pd)[32], const uint32_t (&pr)[32], uint32_t (&pk)[16],
                                           const float (&dl)[32]) {
#pragma unroll
  for (int c = 0; c < 32; c += 2) {
    float d0, d1;
    const uint64_t pd2 = ptx::pack2(__uint_as_float(pd[c]), __uint_as_float(pd[c + 1]));
    const uint64_t pr2 = ptx::pack2(__uint_as_float(pr[c]), __uint_as_float(pr[c + 1]));
    ptx::unpack2(ptx::mul2(pd2, ptx::sub2(pr2, ptx::pack2(dl[c], dl[c + 1]))), d0, d1);
    pk[c >> 1] = ptx::pack_bf16_trunc(d0, d1);
  }
}

__device__ __forceinline__ int ld_acquire(const int32_t* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int32_t* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   ptx::smem_u32(smem_dst)),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(ptx::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store(float* dst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(reinterpret_cast<uint64_t>(dst)),
               "r"(ptx::smem_u32(smem_src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_add_f32(float* dst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(
                   reinterpret_cast<uint64_t>(dst)),
               "r"(ptx::smem_u32(smem_src)), "r"(bytes)
               : "memory");
}

// kStore: whether dq is stored with the last part of a query tile (FusedArgs::store_dq), known when it is compiled: 18 KB of code that
// the other form does not carry through the instruction cache ([2,16,8192,128] with 1024 keys and ALiBi 490 -> 455 us); kAsked (the
// kernels compiled at run time, where each takes seconds): looked up.
constexpr int kAsked = 2;
template <int D, int SK, int MK, int kStore = kAsked>
__global__ void __launch_bounds__(kThreads, 1)
    fused_sm100_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                       const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                       const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_ks,
                       const __grid_constant__ CUtensorMap tm_vs, const DevParams P, const FusedArgs F, int* abort_flag) {
  constexpr int kPanels = D / 64;
  constexpr uint32_t kTileBytes = kPanels * ptx::kPanelBytes;
  // At D = 128 shared memory holds one K, V (those of the next item wait for this one's last MMAs) and one dO, whose two
  // readers dP(n), dV(n) are neighbours on the tensor core: the next one has the time of S, dK, dQ to arrive.
  constexpr int kKvStages = D == 64 ? 2 : 1, kDoStages = D == 64 ? 2 : 1;
  // dS^T(n) may be written once dQ(n-1) (one tile) or dQ(n-2) (two) has run: dP(n) was issued later, so its completion says so
  constexpr int kDsStages = D == 64 ? 2 : 1;
  constexpr uint32_t kDsBytes = 2 * ptx::kPanelBytes;
  constexpr uint32_t kStatBytes = 2 * kTile * sizeof(float);
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColS = 0, kColDP = 128, kColDK = 256, kColDV = 256 + D;
  constexpr bool kOwnDq = D == 64;  // dQ_part has columns of its own
  constexpr uint32_t kColDQ = kOwnDq ? 384 : kColDP;
  constexpr bool kDoc = MK == FLEXATTN_MASK_DOCUMENT;
  constexpr bool kGather = MK == kMaskS2Gather;  // tm_ks, tm_vs: the keys and values on the stride grid
  const int n_vt = kGather ? P.n_kt + P.n_st : P.n_kt;  // kv tiles of a slice: its window tiles, and behind them its strided ones

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = sK + kKvStages * kTileBytes;
  uint8_t* sQ = sV + kKvStages * kTileBytes;   // two stages
  uint8_t* sDO = sQ + 2 * kTileBytes;
  uint8_t* sDS = sDO + kDoStages * kTileBytes;  // dS^T: 128 keys x 128 queries; panel h belongs to warpgroup h
  uint8_t* sOut = sDS + kDsStages * kDsBytes;   // dQ_part on its way out: two slots per drain warp
  FusedSmem* sh = reinterpret_cast<FusedSmem*>(sOut + 8 * kSlotBytes);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (aborted_on_entry(abort_flag, P.status, kFusedId)) return;
  if (ptx::smem_u32(smem) & 1023u) {  // the swizzled tiles need it (no room is left to round up)
    if (tid == 0) give_up(abort_flag, P.status, kFusedId, 98);
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&sh->bar_k[s], 1);
      ptx::mbar_init(&sh->bar_v[s], 1);
      ptx::mbar_init(&sh->bar_kfree[s], 1);
      ptx::mbar_init(&sh->bar_vfree[s], 1);
      ptx::mbar_init(&sh->bar_q[s], 1);
      ptx::mbar_init(&sh->bar_do[s], 1);
      ptx::mbar_init(&sh->bar_qfree[s], 1);
      ptx::mbar_init(&sh->bar_dofree[s], 1);
      ptx::mbar_init(&sh->bar_stage[s], 4);  // the four warps of a warpgroup
      ptx::mbar_init(&sh->bar_stagefree[s], 1);
      ptx::mbar_init(&sh->bar_turn[s], 1);
      ptx::mbar_init(&sh->bar_turnfree[s], 5);  // four drain warps and the flag warp
      ptx::mbar_init(&sh->bar_red[s], 4);
      for (int w = 0; w < 4; ++w) ptx::mbar_init(&sh->bar_back[w][s], 1);
    }
    ptx::mbar_init(&sh->bar_s, 1);
    ptx::mbar_init(&sh->bar_dp, 1);
    ptx::mbar_init(&sh->bar_p, 8);
    ptx::mbar_init(&sh->bar_ds, 8);
    ptx::mbar_init(&sh->bar_dq, 1);
    ptx::mbar_init(&sh->bar_drained, 4);
    ptx::mbar_init(&sh->bar_accfree, 8);
    for (int s = 0; s < kItemRing; ++s) {
      ptx::mbar_init(&sh->bar_item[s], 1);
      ptx::mbar_init(&sh->bar_itemfree[s], 14);  // eight element-wise warps, four drain warps, MMA, turn
    }
    ptx::fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(&sh->tmem_base, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = sh->tmem_base;

  // In every role: r = index of an item of this CTA, u = index among its items with work (phases of what happens once
  // per item), T = index of a tile in the stream of all of them (stage T % 2, phase (T / 2) & 1, or phase T & 1).
  if (warp < kDrainWarp) {
    ptx::setmaxnreg_inc<kRegsEw>();
    // ------------------------------------------------------------------ element-wise warpgroups
    const int row = tid & 127, half = warp >> 2;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t colS = kColS + 64 * half, colDP = kColDP + 64 * half;
    uint8_t* panel = sDS + half * ptx::kPanelBytes;
    uint8_t* panel_row = panel + row * 128;
    FusedScoreCtx x;
    x.sm_scale = P.sm_scale;
    x.c2 = P.sm_scale * kLog2e;
    x.slope2 = 0.f;
    x.capl2 = P.cap * kLog2e;
    x.csc = (SK == FLEXATTN_SCORE_SOFTCAP) ? P.sm_scale / P.cap : 0.f;
    const long long n_doc = (long long)P.batch * P.doc_stride;
    int T = 0, u = 0, fail_at = 0;
    uint32_t panels = 0;  // stored so far
    bool ok = true;
    // one 64-column panel of this warpgroup, already written, leaves through a bulk store; the panel is free on return.
    auto store_panel = [&](const CUtensorMap* tm, int col, int kt, int bh) {
      const uint32_t phase = panels++ & 1;
      ptx::fence_proxy_async_smem();
      ptx::mbar_arrive_warp(&sh->bar_stage[half]);
      if ((warp & 3) == 0) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_stage[half], phase));
        if (ok && lane == 0) {
          ptx::tma_store_3d(tm, panel, col, kt * kTile, bh);
          ptx::tma_store_commit();
          ptx::tma_store_wait_read();
          ptx::mbar_arrive(&sh->bar_stagefree[half]);
        }
        __syncwarp();
      }
      ok = ok && __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_stagefree[half], phase));
      if (!ok) fail_at = 13;
    };
    for (int r = 0; ok; ++r) {
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_item[r % kItemRing], (r / kItemRing) & 1));
      if (!ok) { fail_at = 9; break; }
      const int4 ia = sh->item_a[r % kItemRing];
      const int2 ib = sh->item_b[r % kItemRing];
      ptx::mbar_arrive_warp(&sh->bar_itemfree[r % kItemRing]);
      if (ia.x < 0) break;
      const int bh = F.slice0 + ia.x, kt = ia.y, N = ia.w - ia.z;
      const bool strided = kGather && kt >= P.n_kt;
      const int key = (strided ? kt - P.n_kt : kt) * kTile + row, keys = strided ? s2_keys(P.seq_k, P.stride) : P.seq_k;
      const bool row_ok = key < keys;
      const int j = strided ? min(key, keys) * P.stride : key;  // this thread's key position
      x.b = bh / P.heads;
      x.h = bh - x.b * P.heads;
      x.j = j;
      if constexpr (SK == FLEXATTN_SCORE_ALIBI)
        x.slope2 = FLEXATTN_DBG_OK(x.h, P.heads, kFusedId, 701) ? __ldg(&P.alibi_slopes[x.h]) * kLog2e : 0.f;
      // the queries [qlo, qhi) this key row keeps, where the mask is an interval of them (all kinds but documents whose
      // ids come back)
      bool doc_runs = false;
      int qlo = 0, qhi = 0, dj = -2;
      const int32_t* doc = nullptr;
      if constexpr (kGather) {
        row_query_interval<FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL>(j, P.seq_q, P.window, 1, qlo, qhi);
        if (strided) {
          qlo = P.window < P.seq_q - j ? j + P.window : P.seq_q;
          qhi = P.seq_q;
        }
      } else if constexpr (!kDoc) {
        row_query_interval<MK>(j, P.seq_q, P.window, P.stride, qlo, qhi);
      }
      if constexpr (kDoc) {
        const long long at = (long long)x.b * P.doc_stride + j;
        doc = P.doc_ids + (size_t)x.b * P.doc_stride;
        doc_runs = FLEXATTN_DBG_OK(x.b, P.batch, kFusedId, 702) && P.doc_sorted[x.b] != 0;
        if (row_ok && FLEXATTN_DBG_OK(at, n_doc, kFusedId, 703)) {
          dj = doc[j];
          if (doc_runs) {
            qlo = j;
            qhi = min(P.run_hi[at], P.seq_q);
          }
        }
      }
      // A key past the end keeps nothing, and its tile counts as partial: p of such a column is exp2(-lse), which may be
      // infinite, and dQ_part would take it times the zero row of K.
      if (!row_ok) {
        doc_runs = true;
        qlo = qhi = 0;
      }
      const bool ragged = ((strided ? kt - P.n_kt : kt) + 1) * kTile > keys;
      for (int n = 0; n < N && ok; ++n, ++T) {
        const int st = T & 1, qt = ia.z + n, i0 = qt * kTile + 64 * half;
        const bool partial = ragged || !(qt >= ib.x && qt < ib.y);
        const float* nlse = sh->stats[st][0] + 64 * half;
        const float* delta = sh->stats[st][1] + 64 * half;
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_q[st], (T >> 1) & 1));  // the statistics came with Q
        if (!ok) { fail_at = 10; break; }
        float stat[32];
        load_cols32(stat, nlse);
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_s, T & 1));
        if (!ok) { fail_at = 11; break; }
        ptx::tc_fence_after();
        uint32_t p[2][32];
        ptx::tmem_ld32(lane_base + colS, p[0]);
        ptx::tmem_ld32(lane_base + colS + 32, p[1]);
        ptx::tmem_wait_ld();
        ptx::tmem_ld_acquire(p[0]);
        ptx::tmem_ld_acquire(p[1]);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t pk[16];
          const int i1 = i0 + 32 * g;
          if (g == 1) load_cols32(stat, nlse + 32);
          if (partial) {
            uint32_t keep = range_bits32(qlo - i1, qhi - i1);
            if constexpr (kDoc) {
              if (!doc_runs) {
                keep = 0u;
                for (int c = 0; c < 32; ++c) {
                  const int i = i1 + c;
                  if (i < P.seq_q && i >= j && FLEXATTN_DBG_OK((long long)x.b * P.doc_stride + i, n_doc, kFusedId, 704) &&
                      __ldg(doc + i) == dj)
                    keep |= 1u << c;
                }
              }
            }
            fused_p32<SK, true>(p[g], pk, stat, keep, i1, x);
          } else {
            fused_p32<SK, false>(p[g], pk, stat, 0u, i1, x);
          }
          // P^T over the first half of this warpgroup's S^T columns (read by now)
          ptx::tmem_st16(lane_base + colS + 16 * g, pk);
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(&sh->bar_p);

        load_cols32(stat, delta);
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_dp, T & 1));
        if (!ok) { fail_at = 12; break; }
        ptx::tc_fence_after();
        uint8_t* ds_row = panel_row + (uint32_t)(T % kDsStages) * kDsBytes;
        uint32_t pr[2][32];
        ptx::tmem_ld32(lane_base + colDP, pr[0]);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t pk[16];
          if (g == 1) load_cols32(stat, delta + 32);
          ptx::tmem_wait_ld();
          ptx::tmem_ld_acquire(pr[g]);
          if (g == 0) ptx::tmem_ld32(lane_base + colDP + 32, pr[1]);
          fused_ds32(p[g], pr[g], pk, stat);
          // columns 32.. of this warpgroup are read after the first store, which lands on 0..15
          ptx::tmem_st16(lane_base + colDP + 16 * g, pk);
#pragma unroll
          for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(ds_row + (((4 * g + c) ^ (row & 7)) << 4)) =
                make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::fence_proxy_async_smem();  // the tile is an MMA operand
        ptx::mbar_arrive_warp(&sh->bar_ds);
      }
      if (!ok) break;
      // dK * sm_scale (warpgroup 0) and dV (warpgroup 1) as bf16; the accumulators are free once they are in registers
      if (N > 0) {
        // The last dQ of the item, and with it every MMA before: K has been read.  A wait by parity must not come a phase late, and
        // how late these warps get here is not bounded; this barrier has one phase per item that uses the stage, and its next one
        // needs their P.  (bar_dq, with a phase per tile, may be one or two further on.)
        if constexpr (kDebugChecks) __nanosleep(20000);  // the bounds-checked build always gets here late
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_kfree[u % kKvStages], (u / kKvStages) & 1));
        if (!ok) { fail_at = 15; break; }
        ++u;
        ptx::tc_fence_after();
      }
      uint32_t out[D / 2];
      const float sc = half ? 1.f : P.sm_scale;
      // a key on the stride grid has two sums, which meet in s2_finish_kernel: they leave as f32
      float* s2_row = nullptr;
      if constexpr (kGather) {
        if (row_ok && (strided || j % P.stride == 0)) {
          const long long at = ((long long)ia.x * s2_keys(P.seq_k, P.stride) + j / P.stride) * 4 + 2 * strided + half;
          if (FLEXATTN_DBG_OK(at, (long long)F.slices * s2_keys(P.seq_k, P.stride) * 4, kFusedId, 715)) s2_row = F.s2_dkv + at * D;
        }
      }
#pragma unroll
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t v[32];
        if (N > 0) {
          ptx::tmem_ld32(lane_base + (half ? kColDV : kColDK) + c0, v);
          ptx::tmem_wait_ld();
          ptx::tmem_ld_acquire(v);
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = 0u;
        }
        if (kGather && s2_row != nullptr) {
#pragma unroll
          for (int c = 0; c < 32; c += 4) *reinterpret_cast<uint4*>(s2_row + c0 + c) = make_uint4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        }
#pragma unroll
        for (int c = 0; c < 32; c += 2)
          out[(c0 + c) >> 1] = ptx::pack_bf16(__uint_as_float(v[c]) * sc, __uint_as_float(v[c + 1]) * sc);
      }
      if (N > 0) {
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(&sh->bar_accfree);
      }
      if (strided) continue;
#pragma unroll
      for (int p0 = 0; p0 < kPanels; ++p0) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(panel_row + ((c ^ (row & 7)) << 4)) =
              make_uint4(out[32 * p0 + 4 * c], out[32 * p0 + 4 * c + 1], out[32 * p0 + 4 * c + 2], out[32 * p0 + 4 * c + 3]);
        if (ok) store_panel(half ? &tm_dv : &tm_dk, p0 * 64, kt, bh);
      }
    }
    if (!ok && lane == 0) give_up(abort_flag, P.status, kFusedId, fail_at);
  } else if (warp < kMmaWarp) {
    ptx::setmaxnreg_inc<kRegsDrain>();
    // ------------------------------------------------------------------ drain: dQ_part -> scratch
    // Through shared memory and the bulk engine: vector reductions straight from the registers (25 bytes per cycle and SM,
    // as fast) fill the load/store queue, behind which every shared-memory access and barrier of the other warps waits
    // (4000 cycles per tile instead of 2900).
    const int w = warp - kDrainWarp;
    const uint32_t lane_base = tmem + ((uint32_t)(w * 32) << 16);
    uint8_t* slots = sOut + 2 * w * kSlotBytes;
    int T = 0, fail_at = 0;
    bool ok = true, pending = false;
    uint32_t back_phase = 0;
    // the bulk operations of tile t have completed, the flag warp may say so: one tile later, or at the end of the item
    auto finish = [&](int t) {
      if (lane == 0) {
        ptx::tma_store_wait_all();
        asm volatile("fence.proxy.async.global;" ::: "memory");
        ptx::mbar_arrive(&sh->bar_red[t & 1]);
      }
      __syncwarp();
      pending = false;
    };
    for (int r = 0; ok; ++r) {
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_item[r % kItemRing], (r / kItemRing) & 1));
      if (!ok) { fail_at = 30; break; }
      const int4 ia = sh->item_a[r % kItemRing];
      ptx::mbar_arrive_warp(&sh->bar_itemfree[r % kItemRing]);
      if (ia.x < 0) break;
      for (int n = ia.z; n < ia.w && ok; ++n, ++T) {
        // Last parts: the sum comes back through the slots, 32 columns at a time and two on their way; the first two are asked
        // for before dQ_part is there, where the turn has come by then.
        const float* back = nullptr;
        auto fetch = [&](int c) {
          if (lane != 0) return;
          uint64_t* bar = &sh->bar_back[w][c & 1];
          ptx::mbar_arrive_expect_tx(bar, kSlotBytes);
          bulk_load(slots + (c & 1) * kSlotBytes, back + c * 1024, kSlotBytes, bar);
        };
        auto fetch_first = [&](const int4& turn) {
          if (kStore != 0 && (turn.z & 3) == 2 && back == nullptr &&
              FLEXATTN_DBG_OK((long long)turn.x * P.n_qt + turn.y, (long long)F.slices * F.chains * P.n_qt, kFusedId, 708)) {
            back = F.dq_acc + ((size_t)(turn.x % F.ring) * P.n_qt + turn.y) * kTile * D + w * 32 * D;
            if (lane == 0) ptx::tma_store_wait_read();  // what the slots held has left
            fetch(0);
            fetch(1);
          }
        };
        if (kStore != 0 && __all_sync(0xffffffffu, ptx::mbar_test_wait(&sh->bar_turn[T & 1], (T >> 1) & 1))) fetch_first(sh->turn[T & 1]);
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_dq, T & 1));
        if (!ok) { fail_at = 31; break; }
        ptx::tc_fence_after();
        uint32_t v[D / 32][32];
#pragma unroll
        for (int c = 0; c < D / 32; ++c) ptx::tmem_ld32(lane_base + kColDQ + 32 * c, v[c]);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < D / 32; ++c) ptx::tmem_ld_acquire(v[c]);
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(&sh->bar_drained);  // the columns are free
        if (pending) finish(T - 1);
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_turn[T & 1], (T >> 1) & 1));
        if (!ok) { fail_at = 32; break; }
        const int4 turn = sh->turn[T & 1];
        fetch_first(turn);
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sh->bar_turnfree[T & 1]);
        const bool first = turn.z & 1, last = kStore != 0 && (turn.z & 2);
        float* tile = F.dq_acc + ((size_t)(turn.x % F.ring) * P.n_qt + turn.y) * kTile * D + w * 32 * D;
        if (!FLEXATTN_DBG_OK((long long)turn.x * P.n_qt + turn.y, (long long)F.slices * F.chains * P.n_qt, kFusedId, 705)) {
        } else if (last) {
          uint32_t out[D / 2];
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            const float4* sum = reinterpret_cast<const float4*>(slots + (c & 1) * kSlotBytes) + lane;
            if (back != nullptr) ok = ok && __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_back[w][c & 1], back_phase));
            if (!ok) fail_at = 33;
#pragma unroll
            for (int k = 0; k < 32; k += 4) {
              const float4 a = back == nullptr ? make_float4(0.f, 0.f, 0.f, 0.f) : sum[(k >> 2) * 32];
              out[16 * c + (k >> 1)] =
                  ptx::pack_bf16((a.x + __uint_as_float(v[c][k])) * P.sm_scale, (a.y + __uint_as_float(v[c][k + 1])) * P.sm_scale);
              out[16 * c + (k >> 1) + 1] =
                  ptx::pack_bf16((a.z + __uint_as_float(v[c][k + 2])) * P.sm_scale, (a.w + __uint_as_float(v[c][k + 3])) * P.sm_scale);
            }
            __syncwarp();
            if (c + 2 < D / 32 && ok && back != nullptr) fetch(c + 2);
            if ((c & 1) && back != nullptr) back_phase ^= 1;
          }
          // dq leaves through the slots too, 64 columns in each; row by row from the registers it would fill the queue
#pragma unroll
          for (int p0 = 0; p0 < kPanels; ++p0)
#pragma unroll
            for (int c = 0; c < 8; ++c)
              *reinterpret_cast<uint4*>(slots + p0 * kSlotBytes + lane * 128 + ((c ^ (lane & 7)) << 4)) =
                  make_uint4(out[32 * p0 + 4 * c], out[32 * p0 + 4 * c + 1], out[32 * p0 + 4 * c + 2], out[32 * p0 + 4 * c + 3]);
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (ok && lane == 0 && turn.y * kTile + 32 * w < P.seq_q) {
#pragma unroll
            for (int p0 = 0; p0 < kPanels; ++p0)
              ptx::tma_store_3d(&tm_dq, slots + p0 * kSlotBytes, p0 * 64, turn.y * kTile + 32 * w, F.slice0 + turn.x);
            ptx::tma_store_commit();
          }
        } else {
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            uint8_t* slot = slots + (c & 1) * kSlotBytes;
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the slot's last one has been read
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 32; k += 4)
              *reinterpret_cast<uint4*>(slot + k * 128 + lane * 16) = make_uint4(v[c][k], v[c][k + 1], v[c][k + 2], v[c][k + 3]);
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (first) bulk_store(tile + c * 1024, slot, kSlotBytes);  // nothing to add to
              else bulk_add_f32(tile + c * 1024, slot, kSlotBytes);
              ptx::tma_store_commit();
            }
          }
        }
        pending = true;
        if (n + 1 == ia.w) finish(T);
      }
    }
    if (!ok && lane == 0) give_up(abort_flag, P.status, kFusedId, fail_at);
  } else {
    ptx::setmaxnreg_dec<kRegsRest>();
    if (warp == kTmaWarp) {
      // ---------------------------------------------------------------- loads; takes the items
      if (ptx::elect_one()) {
        bool ok = true;
        ptx::prefetch_tensormap(&tm_q);
        ptx::prefetch_tensormap(&tm_do);
        ptx::prefetch_tensormap(&tm_k);
        ptx::prefetch_tensormap(&tm_v);
        auto load_tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int row0, int bh, uint32_t extra) {
          ptx::mbar_arrive_expect_tx(bar, kTileBytes + extra);
#pragma unroll
          for (int p = 0; p < kPanels; ++p) ptx::tma_load_3d(dst + p * ptx::kPanelBytes, tm, bar, p * 64, row0, bh);
        };
        const int total = F.slices * n_vt;
        int T = 0, u = 0;
        int w = atomicAdd(F.ticket, 1);
        for (int r = 0;; ++r) {
          if (r >= kItemRing) {
            ok = ptx::mbar_wait_relaxed(&sh->bar_itemfree[r % kItemRing], (r / kItemRing - 1) & 1);
            if (!ok) break;
          }
          if (w >= total) {
            sh->item_a[r % kItemRing] = make_int4(-1, 0, 0, 0);
            ptx::mbar_arrive(&sh->bar_item[r % kItemRing]);
            break;
          }
          const int g = w / (F.group * n_vt), in_group = w - g * F.group * n_vt;
          const int width = min(F.group, F.slices - g * F.group);
          const int rank = in_group / width;
          const int slice = g * F.group + in_group - rank * width, kt = n_vt - 1 - rank;
          const int bh = F.slice0 + slice, b = bh / P.heads;
          const int4 cm = col_entry<MK>(P, b, kt);
          const bool strided = kGather && kt >= P.n_kt;
          const int kv_row = (strided ? kt - P.n_kt : kt) * kTile;
          sh->item_a[r % kItemRing] = make_int4(slice, kt, cm.x, cm.y);
          sh->item_b[r % kItemRing] = make_int2(cm.z, cm.w);
          ptx::mbar_arrive(&sh->bar_item[r % kItemRing]);
          const int N = cm.y - cm.x;
          auto load_q = [&](int n) {
            const int st = (T + n) & 1;
            if (T + n >= 2) ok = ok && ptx::mbar_wait_relaxed(&sh->bar_qfree[st], (((T + n) >> 1) - 1) & 1, 20);
            if (!ok) return;
            const bool in = FLEXATTN_DBG_OK((long long)slice * P.n_qt + cm.x + n, (long long)F.slices * P.n_qt, kFusedId, 709);
            load_tile(sQ + st * kTileBytes, &tm_q, &sh->bar_q[st], (cm.x + n) * kTile, bh, in ? kStatBytes : 0);
            if (in) bulk_load(sh->stats[st], F.stats + ((size_t)slice * P.n_qt + cm.x + n) * 2 * kTile, kStatBytes, &sh->bar_q[st]);
          };
          auto load_do = [&](int n) {
            const int st = (T + n) % kDoStages;
            if (T + n >= kDoStages)
              ok = ok && ptx::mbar_wait_relaxed(&sh->bar_dofree[st], ((T + n) / kDoStages - 1) & 1, 20);
            if (!ok) return;
            load_tile(sDO + st * kTileBytes, &tm_do, &sh->bar_do[st], (cm.x + n) * kTile, bh, 0);
          };
          if (N > 0) {
            const int ks = u % kKvStages, kph = (u / kKvStages - 1) & 1;
            load_q(0);
            // V and K of the previous item (D = 64: of the last but one) have been read
            if (u >= kKvStages) ok = ok && ptx::mbar_wait_relaxed(&sh->bar_vfree[ks], kph, 20);
            if (!ok) break;
            load_tile(sV + ks * kTileBytes, strided ? &tm_vs : &tm_v, &sh->bar_v[ks], kv_row, bh, 0);
            load_do(0);
            if (u >= kKvStages) ok = ok && ptx::mbar_wait_relaxed(&sh->bar_kfree[ks], kph, 20);
            if (!ok) break;
            load_tile(sK + ks * kTileBytes, strided ? &tm_ks : &tm_k, &sh->bar_k[ks], kv_row, bh, 0);
            for (int n = 1; n < N && ok; ++n) {
              if (kDoStages == 1) {  // dO(n) waits for dV(n-1), later than Q(n) for dK(n-2)
                load_q(n);
                load_do(n);
              } else {
                load_do(n);
                load_q(n);
              }
            }
            if (!ok) break;
            T += N;
            ++u;
          }
          w = atomicAdd(F.ticket, 1);
        }
        if (!ok) give_up(abort_flag, P.status, kFusedId, 20);
      }
    } else if (warp == kMmaWarp) {
      // ---------------------------------------------------------------- MMA issue
      if (ptx::elect_one()) {
        bool ok = true;
        int fail_at = 1;
        constexpr uint32_t idesc_s = ptx::make_idesc(128, 128, false);
        constexpr uint32_t idesc_acc = ptx::make_idesc(128, D, true);
        constexpr uint32_t idesc_dq = ptx::make_idesc(128, D, true, true);
        const uint32_t aK = ptx::smem_u32(sK), aV = ptx::smem_u32(sV), aQ = ptx::smem_u32(sQ), aDO = ptx::smem_u32(sDO);
        const uint32_t aDS = ptx::smem_u32(sDS);
        int T = 0, u = 0;
        // descriptors are rebuilt for each group of MMAs: kept across the loop they need a hundred registers
        auto kmajor = [](uint32_t a) {
          asm volatile("" : "+r"(a));
          return ptx::base_kmajor(a);
        };
        auto mnmajor = [](uint32_t a) {
          asm volatile("" : "+r"(a));
          return ptx::base_mnmajor(a);
        };
        auto wait = [&](uint64_t* bar, uint32_t par, int site) {
          if (ok && !ptx::mbar_wait(bar, par)) {
            ok = false;
            fail_at = site;
          }
        };
        auto do_off = [&](int t) { return (uint32_t)(t % kDoStages) * kTileBytes; };
        auto issue_s = [&](int t, uint32_t k_off) {  // S^T = K Q^T
          const ptx::DescBase bK = kmajor(aK + k_off), bQ = kmajor(aQ + (uint32_t)(t & 1) * kTileBytes);
          ptx::tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            ptx::mma_ss(tmem + kColS, ptx::desc_at(bK, ptx::koff_kmajor(kk)), ptx::desc_at(bQ, ptx::koff_kmajor(kk)), idesc_s, kk > 0);
          ptx::mma_commit(&sh->bar_s);
        };
        // dP^T = V dO^T of tile t; the dP columns are free of dS^T(t - 1) (issue order) and of dQ_part(t - 1) (drained)
        auto issue_dp = [&](int t, uint32_t k_off) {
          wait(&sh->bar_do[t % kDoStages], (t / kDoStages) & 1, 7);
          if (!kOwnDq && t > 0) wait(&sh->bar_drained, (t - 1) & 1, 17);
          if (!ok) return;
          const ptx::DescBase bV = kmajor(aV + k_off), bDO = kmajor(aDO + do_off(t));
          ptx::tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            ptx::mma_ss(tmem + kColDP, ptx::desc_at(bV, ptx::koff_kmajor(kk)), ptx::desc_at(bDO, ptx::koff_kmajor(kk)), idesc_s, kk > 0);
          ptx::mma_commit(&sh->bar_dp);
        };
        for (int r = 0; ok; ++r) {
          wait(&sh->bar_item[r % kItemRing], (r / kItemRing) & 1, 1);
          if (!ok) break;
          const int4 ia = sh->item_a[r % kItemRing];
          ptx::mbar_arrive(&sh->bar_itemfree[r % kItemRing]);
          if (ia.x < 0) break;
          const int N = ia.w - ia.z;
          if (N <= 0) continue;
          const int ks = u % kKvStages;
          const uint32_t kph = (u / kKvStages) & 1, k_off = (uint32_t)ks * kTileBytes;
          wait(&sh->bar_q[T & 1], (T >> 1) & 1, 2);
          wait(&sh->bar_k[ks], kph, 3);
          if (!ok) break;
          issue_s(T, k_off);
          wait(&sh->bar_v[ks], kph, 4);
          issue_dp(T, k_off);
          for (int n = 0; n < N && ok; ++n, ++T) {
            const bool more = n + 1 < N;
            wait(&sh->bar_p, T & 1, 8);
            if (n == 0 && u > 0) wait(&sh->bar_accfree, (u - 1) & 1, 16);  // dK, dV of the previous item have been read
            if (!ok) break;
            ptx::tc_fence_after();
            {  // dV += P^T dO; warpgroup w wrote query columns [64 w, 64 w + 64) at column 64 w of the S^T block
              const ptx::DescBase bDOt = mnmajor(aDO + do_off(T));
#pragma unroll
              for (int kk = 0; kk < kTile / 16; ++kk)
                ptx::mma_ts(tmem + kColDV, tmem + kColS + 64 * (kk >> 2) + (kk & 3) * 8, ptx::desc_at(bDOt, ptx::koff_mnmajor(kk)),
                            idesc_acc, n > 0 || kk > 0);
              ptx::mma_commit(&sh->bar_dofree[T % kDoStages]);
              if (!more) ptx::mma_commit(&sh->bar_vfree[ks]);
            }
            if (more) {
              wait(&sh->bar_q[(T + 1) & 1], ((T + 1) >> 1) & 1, 18);
              if (!ok) break;
              issue_s(T + 1, k_off);
            }
            wait(&sh->bar_ds, T & 1, 19);
            if (!ok) break;
            ptx::tc_fence_after();
            {  // dK += dS^T Q
              const ptx::DescBase bQt = mnmajor(aQ + (uint32_t)(T & 1) * kTileBytes);
#pragma unroll
              for (int kk = 0; kk < kTile / 16; ++kk)
                ptx::mma_ts(tmem + kColDK, tmem + kColDP + 64 * (kk >> 2) + (kk & 3) * 8, ptx::desc_at(bQt, ptx::koff_mnmajor(kk)),
                            idesc_acc, n > 0 || kk > 0);
              ptx::mma_commit(&sh->bar_qfree[T & 1]);
            }
            if (kOwnDq) {
              if (more) issue_dp(T + 1, k_off);
              if (T > 0) wait(&sh->bar_drained, (T - 1) & 1, 21);
              if (!ok) break;
              ptx::tc_fence_after();
            }
            {  // dQ_part = dS K
              const ptx::DescBase bDS = mnmajor(aDS + (uint32_t)(T % kDsStages) * kDsBytes), bKt = mnmajor(aK + k_off);
#pragma unroll
              for (int kk = 0; kk < kTile / 16; ++kk)
                ptx::mma_ss(tmem + kColDQ, ptx::desc_at(bDS, ptx::koff_mnmajor(kk)), ptx::desc_at(bKt, ptx::koff_mnmajor(kk)),
                            idesc_dq, kk > 0);
              ptx::mma_commit(&sh->bar_dq);
              if (!more) ptx::mma_commit(&sh->bar_kfree[ks]);
            }
            if (!kOwnDq && more) issue_dp(T + 1, k_off);
          }
          ++u;
        }
        if (!ok) give_up(abort_flag, P.status, kFusedId, fail_at);
      }
    } else if (warp == kTurnWarp) {
      // ---------------------------------------------------------------- whose turn it is at a query tile
      int T = 0, fail_at = 40;
      bool ok = true;
      auto publish = [&](int slice, int qt, int which, int value) {
        if (T >= 2) ok = ok && __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_turnfree[T & 1], ((T >> 1) - 1) & 1));
        if (!ok) { fail_at = 41; return; }
        if (lane == 0) {
          sh->turn[T & 1] = make_int4(slice, qt, which, value);
          ptx::mbar_arrive(&sh->bar_turn[T & 1]);
        }
        __syncwarp();
        ++T;
      };
      for (int r = 0; ok; ++r) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&sh->bar_item[r % kItemRing], (r / kItemRing) & 1));
        if (!ok) break;
        const int4 ia = sh->item_a[r % kItemRing];
        ptx::mbar_arrive_warp(&sh->bar_itemfree[r % kItemRing]);
        if (ia.x < 0) {
          publish(-1, 0, 0, 0);
          break;
        }
        const int b = (F.slice0 + ia.x) / P.heads, kt = ia.y;
        // (the strided tiles' parts are a sum of their own)
        const int strided = kGather && kt >= P.n_kt, first_kt = strided ? P.n_kt : 0, end_kt = strided ? n_vt : P.n_kt;
        const int chain = kGather ? 2 * ia.x + strided : ia.x;
        // nearest kv tile beyond this one, upwards or downwards, that sees query tile qt; -1: none
        auto nearest = [&](int qt, int step) {
          for (int j0 = kt + step; j0 >= first_kt && j0 < end_kt; j0 += 32 * step) {
            const int j = j0 + step * lane;
            bool sees = false;
            if (j >= first_kt && j < end_kt) {
              const int4 range = col_entry<MK>(P, b, j);
              sees = qt >= range.x && qt < range.y;
            }
            const unsigned any = __ballot_sync(0xffffffffu, sees);
            if (any) return j0 + step * (__ffs(any) - 1);
          }
          return -1;
        };
        for (int qt = ia.z; qt < ia.w && ok; ++qt) {
          const int pred = nearest(qt, 1);  // its part is added before this one
          const bool last = kStore != 0 && (kStore == 1 || F.store_dq) && nearest(qt, -1) < 0;
          // the first part of a tile waits for the slice that had its place in the ring before
          const int prior = pred >= 0 ? chain : chain - F.ring;
          const int want = pred >= 0 ? n_vt - pred : kAllAdded;
          if (prior >= 0) {
            const long long at = (long long)prior * P.n_qt + qt;
            if (FLEXATTN_DBG_OK(at, (long long)F.slices * F.chains * P.n_qt, kFusedId, 706) && ld_acquire(F.flags + at) < want) {
              const unsigned long long t0 = ptx::globaltimer_ns();
              int polls = 0;
              while (ok && ld_acquire(F.flags + at) < want) {
                if ((++polls & 63) == 0 && ptx::globaltimer_ns() - t0 > ptx::kWaitLimitNs) ok = false;
              }
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) { fail_at = 42; break; }
            asm volatile("fence.proxy.async.global;" ::: "memory");  // the parts are added through the async proxy
          }
          publish(chain, qt, (pred < 0 ? 1 : 0) | (last ? 2 : 0), last ? kAllAdded : n_vt - kt);
        }
      }
      if (!ok && lane == 0) give_up(abort_flag, P.status, kFusedId, fail_at);
    } else {
      // ---------------------------------------------------------------- flags: a part has been added
      bool ok = true;
      for (int T = 0; ok; ++T) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&sh->bar_turn[T & 1], (T >> 1) & 1, 40));
        if (!ok) break;
        const int4 turn = sh->turn[T & 1];
        if (turn.x < 0) break;
        ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&sh->bar_red[T & 1], (T >> 1) & 1, 20));
        if (!ok) break;
        if (lane == 0) {
          __threadfence();  // what the drain warps have added comes before the flag
          const long long at = (long long)turn.x * P.n_qt + turn.y;
          if (FLEXATTN_DBG_OK(at, (long long)F.slices * F.chains * P.n_qt, kFusedId, 707)) st_release(F.flags + at, turn.w);
          ptx::mbar_arrive(&sh->bar_turnfree[T & 1]);
        }
        __syncwarp();
      }
      if (!ok && lane == 0) give_up(abort_flag, P.status, kFusedId, 50);
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
}

#ifndef FLEXATTN_JIT
static_assert(256 * kRegsEw + 128 * kRegsDrain + 128 * kRegsRest <= kThreads * kFusedLaunchRegs, "more registers than the CTA is launched with");

// Before it: delta = rowsum(o * do) to the caller, both row statistics to the padded tiles the loads take, flags and ticket
// to zero.  Bound by HBM latency: all that a thread reads (16-byte chunks of kUnroll rows of o and do, l and m) is asked for before
// the first sum.  [16,12,512,64] 9.0 -> 7.1 us, [8,16,2048,128] 37 -> 33; four rows were no faster, and slower where the grid is
// small.  A query tile that no kv tile sees gets its zeros here.
template <int D>
__global__ void __launch_bounds__(256) prep_kernel(const DevParams P, const FusedArgs F) {
  constexpr int kUnroll = 2, kTpr = D / 8, kRows = 256 / kTpr;  // kRows * kUnroll rows of a block: all of one tile
  constexpr int kBlocksPerTile = kTile / (kRows * kUnroll);
  const long long tile = blockIdx.x / kBlocksPerTile, slice = tile / P.n_qt;
  const int qt = (int)(tile - slice * P.n_qt), row0 = (int)(blockIdx.x % kBlocksPerTile) * kRows * kUnroll + threadIdx.x / kTpr;
  const int i0 = qt * kTile + row0, chunk = threadIdx.x & (kTpr - 1);
  const long long at0 = (F.slice0 + slice) * P.seq_q + i0;
  const bool in = FLEXATTN_DBG_OK(tile, (long long)F.slices * P.n_qt, kFusedId, 711);
  uint4 a[kUnroll], b[kUnroll];
  float l[kUnroll], m[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const bool live = i0 + u * kRows < P.seq_q && FLEXATTN_DBG_OK(at0 + u * kRows, (long long)P.batch * P.heads * P.seq_q, kFusedId, 710);
    a[u] = b[u] = make_uint4(0u, 0u, 0u, 0u);
    l[u] = m[u] = 0.f;
    if (live) {
      a[u] = __ldcs(static_cast<const uint4*>(P.o) + (at0 + u * kRows) * kTpr + chunk);
      b[u] = __ldg(static_cast<const uint4*>(P.d_o) + (at0 + u * kRows) * kTpr + chunk);
      if (chunk == 0) {
        l[u] = P.l[at0 + u * kRows];
        m[u] = P.m[at0 + u * kRows];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a[u]);
    const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&b[u]);
    float acc = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 fa = __bfloat1622float2(pa[c]), fb = __bfloat1622float2(pb[c]);
      acc = fmaf(fa.x, fb.x, acc);
      acc = fmaf(fa.y, fb.y, acc);
    }
#pragma unroll
    for (int s = kTpr / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    if (chunk == 0) {
      const long long at = at0 + u * kRows;
      const int row = row0 + u * kRows;
      float nl = -1.0e30f;  // rows past the end and fully masked ones: p = 0
      if (i0 + u * kRows < P.seq_q && FLEXATTN_DBG_OK(at, (long long)P.batch * P.heads * P.seq_q, kFusedId, 710)) {
        P.delta[at] = acc;
        if (l[u] > 0.f) nl = ptx::kRoundLog2 - fmaf(m[u], kLog2e, __log2f(l[u]));
      }
      if (in) {
        float* t = F.stats + tile * 2 * kTile + row;
        t[0] = nl;
        t[kTile] = acc;
      }
    }
  }
  if (blockIdx.x % kBlocksPerTile == 0 && in) {  // the first block of a tile
    const int4* cmap = P.col_map + (size_t)(P.map_rows > 1 ? (F.slice0 + slice) / P.heads : 0) * P.n_kt;
    bool seen = F.chains > 1;  // (S2, gathered: the finishing kernel knows which sums there are)
    for (int j = threadIdx.x; j < (F.chains > 1 ? 0 : P.n_kt); j += 256) {
      const int2 range = __ldg(reinterpret_cast<const int2*>(cmap + j));
      seen = seen || (qt >= range.x && qt < range.y);
    }
    seen = __syncthreads_or(seen);
    if (threadIdx.x == 0) {
      if (F.chains > 1) F.flags[2 * slice * P.n_qt + qt] = F.flags[(2 * slice + 1) * P.n_qt + qt] = 0;
      else F.flags[tile] = seen ? 0 : kAllAdded;
      if (blockIdx.x == 0) *F.ticket = 0;
    }
    if (!seen) {
      const long long first = ((F.slice0 + slice) * P.seq_q + qt * kTile) * kTpr;
      const int n = min(kTile, P.seq_q - qt * kTile) * kTpr;
      for (int c = threadIdx.x; c < n; c += 256)
        if (FLEXATTN_DBG_OK(first + c, (long long)P.batch * P.heads * P.seq_q * kTpr, kFusedId, 712))
          static_cast<uint4*>(P.dq)[first + c] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
}

// After it, where the last part of a query tile has been added like the others: the f32 tiles become dq, times sm_scale.  A
// thread takes 16 columns of a row: the loads of a warp are 512 consecutive bytes, its stores whole 32-byte sectors.
// kGather: two sums per tile, or one of them.
template <int D, bool kGather>
__global__ void __launch_bounds__(256) finish_kernel(const DevParams P, const FusedArgs F) {
  const int tile = blockIdx.x, slice = tile / P.n_qt, qt = tile - slice * P.n_qt;
  if (!FLEXATTN_DBG_OK(tile, (long long)F.slices * P.n_qt, kFusedId, 713)) return;
  const float* src = F.dq_acc + (size_t)tile * kTile * D;
  const float* more = nullptr;
  if constexpr (kGather) {
    const int4 rm = s2_row(qt, P.seq_q, P.seq_k, P.window, P.stride);
    src = F.dq_acc + ((size_t)(2 * slice + (rm.y > rm.z ? 0 : 1)) * P.n_qt + qt) * kTile * D;
    if (rm.y > rm.z && rm.z > rm.x) more = F.dq_acc + ((size_t)(2 * slice + 1) * P.n_qt + qt) * kTile * D;
  } else if (F.flags[tile] == kAllAdded) {
    return;  // no kv tile sees it: zeroed before
  }
#pragma unroll
  for (int e = threadIdx.x; e < kTile * D / 16; e += 256) {
    const int lane = e & 31, c16 = (e >> 5) % (D / 16), w = (e >> 5) / (D / 16);
    const int i = qt * kTile + 32 * w + lane;
    uint32_t out[8];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const size_t at = ((size_t)(w * (D / 4) + 4 * c16 + c) * 32 + lane) * 4;
      float4 v = __ldcs(reinterpret_cast<const float4*>(src + at));
      if (kGather && more != nullptr) {
        const float4 t = __ldcs(reinterpret_cast<const float4*>(more + at));
        v.x += t.x;
        v.y += t.y;
        v.z += t.z;
        v.w += t.w;
      }
      out[2 * c] = ptx::pack_bf16(v.x * P.sm_scale, v.y * P.sm_scale);
      out[2 * c + 1] = ptx::pack_bf16(v.z * P.sm_scale, v.w * P.sm_scale);
    }
    if (i < P.seq_q && FLEXATTN_DBG_OK((long long)(F.slice0 + slice) * P.seq_q + i, (long long)P.batch * P.heads * P.seq_q, kFusedId, 714)) {
      uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(P.dq) + ((size_t)(F.slice0 + slice) * P.seq_q + i) * D + 16 * c16);
      dst[0] = make_uint4(out[0], out[1], out[2], out[3]);
      dst[1] = make_uint4(out[4], out[5], out[6], out[7]);
    }
  }
}

// ... and the keys on the stride grid get the sum of their two dK, dV.  A thread takes 8 columns.
template <int D>
__global__ void __launch_bounds__(256) s2_finish_kernel(const DevParams P, const FusedArgs F) {
  constexpr int kTpr = D / 8;
  const int n = s2_keys(P.seq_k, P.stride);
  const long long e = (long long)blockIdx.x * 256 + threadIdx.x, key = e / (2 * kTpr);  // of all slices of the launch
  const int which = (int)(e / kTpr) & 1, c = (int)(e % kTpr) * 8;
  if (key >= (long long)F.slices * n) return;
  const float* a = F.s2_dkv + (key * 4 + which) * D + c;
  const float4 w0 = __ldcs(reinterpret_cast<const float4*>(a)), w1 = __ldcs(reinterpret_cast<const float4*>(a + 4));
  const float4 s0 = __ldcs(reinterpret_cast<const float4*>(a + 2 * D)), s1 = __ldcs(reinterpret_cast<const float4*>(a + 2 * D + 4));
  const float sc = which ? 1.f : P.sm_scale;
  const uint4 out = make_uint4(ptx::pack_bf16((w0.x + s0.x) * sc, (w0.y + s0.y) * sc), ptx::pack_bf16((w0.z + s0.z) * sc, (w0.w + s0.w) * sc),
                               ptx::pack_bf16((w1.x + s1.x) * sc, (w1.y + s1.y) * sc), ptx::pack_bf16((w1.z + s1.z) * sc, (w1.w + s1.w) * sc));
  const long long slice = key / n, row = (F.slice0 + slice) * P.seq_k + (key - slice * n) * P.stride;
  if (FLEXATTN_DBG_OK(row, (long long)P.batch * P.heads * P.seq_k, kFusedId, 716))
    *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(which ? P.dv : P.dk) + row * D + c) = out;
}

constexpr size_t smem_bytes(int D) {
  return (size_t)(D == 64 ? 8 : 5) * (D / 64) * ptx::kPanelBytes + (D == 64 ? 4 : 2) * ptx::kPanelBytes + 8 * kSlotBytes + sizeof(FusedSmem);
}
static_assert(smem_bytes(128) <= 232448 && smem_bytes(64) <= 232448, "more shared memory than a CTA can have");

struct Maps {
  CUtensorMap q, d_o, k, v, dk, dv, dq, ks, vs;
};

// grid 0: only prepares the kernel and says whether it can be launched
template <int D, int SK, int MK, int kStore>
int launch_form(cudaStream_t st, const DevParams& d, const FusedArgs& f, const Maps& t, unsigned grid, int* af) {
  constexpr size_t smem = smem_bytes(D);
  auto kern = fused_sm100_kernel<D, SK, MK, kStore>;
  static const bool whole_file = launch_registers(reinterpret_cast<const void*>(kern)) >= kFusedLaunchRegs;
  if (!whole_file) return FLEXATTN_ERR_UNSUPPORTED_BACKEND;
  static SmemAttrOnce attr_once{};  // per kernel instantiation, per device
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), (int)smem, &attr_once) != FLEXATTN_OK) return FLEXATTN_ERR_CUDA;
  if (grid == 0) return FLEXATTN_OK;
  kern<<<grid, kThreads, smem, st>>>(t.q, t.d_o, t.k, t.v, t.dk, t.dv, t.dq, t.ks, t.vs, d, f, af);
  return cudaGetLastError() == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}

template <int D, int SK, int MK>
int launch_one(cudaStream_t st, const DevParams& d, const FusedArgs& f, const Maps& t, unsigned grid, int* af) {
  // (documents always store it, S2, gathered, never: fused_plan)
  if constexpr (MK != FLEXATTN_MASK_DOCUMENT) {
    if (MK == kMaskS2Gather || !f.store_dq) return launch_form<D, SK, MK, 0>(st, d, f, t, grid, af);
  }
  if constexpr (MK != kMaskS2Gather) return launch_form<D, SK, MK, 1>(st, d, f, t, grid, af);
  return FLEXATTN_ERR_UNSUPPORTED_MOD;
}

template <int D, int SK>
int launch_mask(cudaStream_t st, const DevParams& d, int mask, const FusedArgs& f, const Maps& t, unsigned grid, int* af) {
  switch (mask) {
    case FLEXATTN_MASK_NONE: return launch_one<D, SK, FLEXATTN_MASK_NONE>(st, d, f, t, grid, af);
    case FLEXATTN_MASK_CAUSAL: return launch_one<D, SK, FLEXATTN_MASK_CAUSAL>(st, d, f, t, grid, af);
    case FLEXATTN_MASK_SLIDING_WINDOW: return launch_one<D, SK, FLEXATTN_MASK_SLIDING_WINDOW>(st, d, f, t, grid, af);
    case FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL:
      return launch_one<D, SK, FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL>(st, d, f, t, grid, af);
    case FLEXATTN_MASK_DOCUMENT: return launch_one<D, SK, FLEXATTN_MASK_DOCUMENT>(st, d, f, t, grid, af);
    case kMaskS2Gather: return launch_one<D, SK, kMaskS2Gather>(st, d, f, t, grid, af);
    case FLEXATTN_MASK_S2: return launch_one<D, SK, FLEXATTN_MASK_S2>(st, d, f, t, grid, af);
    default: return FLEXATTN_ERR_UNSUPPORTED_MOD;
  }
}

template <int D>
int launch_score(cudaStream_t st, const DevParams& d, int score, int mask, const FusedArgs& f, const Maps& t, unsigned grid,
                 int* af) {
  switch (score) {
    case FLEXATTN_SCORE_NONE: return launch_mask<D, FLEXATTN_SCORE_NONE>(st, d, mask, f, t, grid, af);
    case FLEXATTN_SCORE_ALIBI: return launch_mask<D, FLEXATTN_SCORE_ALIBI>(st, d, mask, f, t, grid, af);
    case FLEXATTN_SCORE_SOFTCAP: return launch_mask<D, FLEXATTN_SCORE_SOFTCAP>(st, d, mask, f, t, grid, af);
    default: return FLEXATTN_ERR_UNSUPPORTED_MOD;
  }
}

// How a call is cut up.
// Group: the slices whose kv tiles are in the list side by side.  What a slice keeps live, 8 bytes per element of a query row (Q, dO,
// f32 sum; under a causal window the few rows around the diagonal), times the group has 80 MB of the 126 MB of L2.  Few slices
// mean many kv tiles of each in flight, which wait for one another's parts; many of them spill.  us of the backward with 48 MB,
// as before / 72 / 80 in groups of equal size / 92 / 160: [4,32,8192,128] causal 6244 / 5848 / 5884 / 5928 / 6618,
// [4,16,2048,128] 466 / 414 / 405 / 404 / 394, [4,16,2048,64] 297 / 243 / 241 / 243 / 236, [1,24,8192,64] 1325 / 1381 / 1327 / 1331 /
// 1425; 24 MB: 8592, 587, 321, 1604.
// store_dq: storing dq with the last part saves the finishing kernel and its pass over the sums, but costs the CTA that
// does it half a tile's time.  That is a gain where many kv tiles share the work (documents: [2,16,16384,128] 1510 -> 1436 us, with
// softcap 1565 -> 1525, the backward alone replayed from a graph); under a causal mask or none the one kv tile that every query
// tile meets last does it all, and long rows wait for it ([2,8,1920,128] causal 88 -> 99).  Short rows: [16,12,512,64] between
// 76 and 93 either way.  Windows of D = 64 store it too ([2,16,4096,64] with 128 keys 74 us, 81 with the finishing kernel), and those of
// D = 128 up to 6000 positions (us stored / finished: 16 heads a row, 3072 with 232 keys 206 / 226, 5756 74 / 75) and where the
// ring is smaller than all slices; longer ones are finished ([4,32,8192,128] with 256 keys and ALiBi 1077 -> 957, [5,8,15744,128] 853 / 755).
// Then the scratch is a ring: three groups of 48 MB, and no group has more than half of it (one is being finished while the next
// is started).  Without it the
// scratch holds every slice of a launch, and there are as many launches as keep it within 1 GiB (one slice, if need be).
struct FusedPlan {
  int launch, group, ring, store_dq;  // slices of a launch, ...
  int measure;                        // group of 48 MB: what fused_pays measures the room by, a third of the ring
  int chains;                          // sums per query tile
  size_t off_stats, off_flags, off_s2, bytes;
};
// s2_n: keys on the stride grid of an S2 call that is gathered, else 0
FusedPlan fused_plan(int slices, int seq_q, int n_qt, int n_kt, int head_dim, int mask, int window, int s2_n) {
  constexpr long long kL2Budget = 48ll << 20, kGroupBudget = 80ll << 20, kLimit = 1ll << 30;
  const int chains = s2_n > 0 ? 2 : 1;
  const long long acc = (long long)chains * n_qt * kTile * head_dim * 4, s2 = 16ll * s2_n * head_dim;
  const long long most = kLimit / (acc + s2) > 0 ? kLimit / (acc + s2) : 1;
  const bool windowed = mask == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL && window < seq_q - 2 * kTile;
  FusedPlan L;
  L.store_dq = windowed || mask == FLEXATTN_MASK_DOCUMENT || (n_kt <= 8 && s2_n == 0);
  L.launch = slices;
  if (!L.store_dq) {
    const long long launches = (slices + most - 1) / most;
    L.launch = (int)((slices + launches - 1) / launches);
  }
  long long group = kL2Budget / (8ll * (windowed ? window + 2 * kTile : seq_q) * head_dim);
  if (L.store_dq && 3 * group > most) group = most / 3;
  if (group < 1) group = 1;
  if (group > L.launch) group = L.launch;
  L.measure = (int)group;
  L.ring = L.store_dq && 3 * group < slices ? (int)(3 * group) : L.launch;
  if (windowed && head_dim == 128 && L.ring == L.launch && n_kt >= 48) L.store_dq = 0;
  long long most_at_once = kGroupBudget / (8ll * (windowed ? window + 2 * kTile : seq_q) * head_dim);
  if (L.ring < L.launch && most_at_once > L.ring / 2) most_at_once = L.ring / 2;
  if (most_at_once < 1) most_at_once = 1;
  const long long groups = (L.launch + most_at_once - 1) / most_at_once;
  L.group = (int)((L.launch + groups - 1) / groups);
  auto up = [](size_t n) { return (n + 255) & ~(size_t)255; };
  L.off_stats = up((size_t)L.ring * acc);
  L.off_flags = L.off_stats + up((size_t)L.launch * n_qt * 2 * kTile * sizeof(float));
  L.off_s2 = L.off_flags + up(((size_t)L.launch * chains * n_qt + 1) * sizeof(int32_t));
  L.bytes = L.off_s2 + up((size_t)L.launch * s2);
  L.chains = chains;
  return L;
}
#endif  // !FLEXATTN_JIT

}  // namespace FLEXATTN_TU_NAMESPACE

#ifndef FLEXATTN_JIT
namespace {
FusedPlan plan_of(const FlexAttnParams& p) {
  return fused_plan(p.batch * p.heads, p.seq_q, (p.seq_q + kTile - 1) / kTile, (p.seq_k + kTile - 1) / kTile, p.head_dim,
                    p.mask_kind, p.window, s2_gathers(p) ? s2_keys(p.seq_k, p.stride) : 0);
}
}  // namespace

size_t bwd_fused_scratch_bytes(const FlexAttnParams& p) { return plan_of(p).bytes; }

// A group of `width` slices on `sms` CTAs has sms / width kv tiles of each slice in flight.  (Measured by groups of 48 MB, with which
// the lines of fused_pays were drawn, all taken as equal.)
double bwd_fused_slack(const FlexAttnParams& p, int sms) {
  const FusedPlan L = plan_of(p);
  const double width = (double)L.launch / ((L.launch + L.measure - 1) / L.measure);
  return (p.seq_q + kTile - 1) / kTile * width / sms;
}

int launch_sm100_bwd_fused(cudaStream_t st, const DevParams& d, int score, int mask, void* scratch) {
  int* af = abort_flag_ptr();
  const int sms = sm_count();
  if (af == nullptr || sms <= 0) return FLEXATTN_ERR_CUDA;
  const int slices = d.batch * d.heads, D = d.head_dim;
  if (D != 64 && D != 128) return FLEXATTN_ERR_UNSUPPORTED_HEAD_DIM;
  const FusedPlan L = fused_plan(slices, d.seq_q, d.n_qt, d.n_kt, D, mask, d.window, d.n_st > 0 ? s2_keys(d.seq_k, d.stride) : 0);
  const int n_vt = d.n_kt + d.n_st;
  if (d.n_st > 0) mask = kMaskS2Gather;
  if ((long long)L.launch * n_vt > 0x7fffffff - 1024 || (long long)L.launch * d.n_qt > 0x7fffffff / 16) return FLEXATTN_ERR_BAD_SHAPE;
  Maps t;
  int e = make_tile_map(&t.q, d.q, slices, d.seq_q, D);
  if (!e) e = make_tile_map(&t.d_o, d.d_o, slices, d.seq_q, D);
  if (!e) e = make_tile_map(&t.k, d.k, slices, d.seq_k, D);
  if (!e) e = make_tile_map(&t.v, d.v, slices, d.seq_k, D);
  if (!e) e = make_tile_map(&t.dk, d.dk, slices, d.seq_k, D);
  if (!e) e = make_tile_map(&t.dv, d.dv, slices, d.seq_k, D);
  if (!e) e = make_tile_map(&t.dq, d.dq, slices, d.seq_q, D, 32);  // a drain warp's rows
  t.ks = t.k;
  t.vs = t.v;
  if (!e && d.n_st > 0) {
    e = make_strided_map(&t.ks, d.k, slices, d.seq_k, D, d.stride);
    if (!e) e = make_strided_map(&t.vs, d.v, slices, d.seq_k, D, d.stride);
  }
  FusedArgs probe{};
  probe.store_dq = L.store_dq;
  auto launch = [&](const FusedArgs& f, unsigned grid) {
    return D == 128 ? launch_score<128>(st, d, score, mask, f, t, grid, af) : launch_score<64>(st, d, score, mask, f, t, grid, af);
  };
  if (!e) e = score == FLEXATTN_SCORE_USER ? jit_fused_ready(d.user_score, D, mask, smem_bytes(D), st) : launch(probe, 0);
  char* base = static_cast<char*>(scratch);
  for (int s0 = 0; s0 < slices && !e; s0 += L.launch) {
    FusedArgs f;
    f.dq_acc = reinterpret_cast<float*>(base);
    f.stats = reinterpret_cast<float*>(base + L.off_stats);
    f.flags = reinterpret_cast<int32_t*>(base + L.off_flags);
    f.slice0 = s0;
    f.slices = slices - s0 < L.launch ? slices - s0 : L.launch;
    f.group = L.group;
    f.ring = L.chains * L.ring;
    f.chains = L.chains;
    f.s2_dkv = reinterpret_cast<float*>(base + L.off_s2);
    f.store_dq = L.store_dq;
    const int tiles = f.slices * d.n_qt, items = f.slices * n_vt;
    f.ticket = f.flags + tiles * L.chains;
    if (D == 128) prep_kernel<128><<<tiles * 4u, 256, 0, st>>>(d, f);
    else prep_kernel<64><<<tiles * 2u, 256, 0, st>>>(d, f);
    if (cudaGetLastError() != cudaSuccess) return FLEXATTN_ERR_CUDA;
    const unsigned grid = (unsigned)(items < sms ? items : sms);
    if (score == FLEXATTN_SCORE_USER) {
      void* args[] = {&t.q, &t.d_o, &t.k, &t.v, &t.dk, &t.dv, &t.dq, &t.ks, &t.vs, const_cast<DevParams*>(&d), &f, &af};
      e = jit_launch(4, false, d.user_score, D, mask, grid, 1, kThreads, smem_bytes(D), st, args);
    } else {
      e = launch(f, grid);
    }
    if (e || f.store_dq) continue;
    if (d.n_st > 0) {
      const unsigned blocks = (unsigned)(((long long)f.slices * s2_keys(d.seq_k, d.stride) * (D / 4) + 255) / 256);
      if (D == 128) finish_kernel<128, true><<<(unsigned)tiles, 256, 0, st>>>(d, f);
      else finish_kernel<64, true><<<(unsigned)tiles, 256, 0, st>>>(d, f);
      if (D == 128) s2_finish_kernel<128><<<blocks, 256, 0, st>>>(d, f);
      else s2_finish_kernel<64><<<blocks, 256, 0, st>>>(d, f);
    } else if (D == 128) {
      finish_kernel<128, false><<<(unsigned)tiles, 256, 0, st>>>(d, f);
    } else {
      finish_kernel<64, false><<<(unsigned)tiles, 256, 0, st>>>(d, f);
    }
    if (cudaGetLastError() != cudaSuccess) return FLEXATTN_ERR_CUDA;
  }
  return e;
}
#endif  // !FLEXATTN_JIT

}  // namespace flexattn
