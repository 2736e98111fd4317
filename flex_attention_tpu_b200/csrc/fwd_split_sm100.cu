// Forward flex attention for few query tiles against many keys (decode, short prompts of few heads), sm_100a.
//
// Same math and interface as fwd_pipe_sm100.cu (reference: flex_attention_kernel.py:196-327).  The other two forward kernels
// give a query tile to ONE CTA, which walks its kv tiles one after the other; with fewer query tiles than SMs that chain is
// the whole launch, and at one tile per slice half of the two-query-tile kernel is idle as well (one query row against 8191
// keys, 64 slices: 107 us = 2.5 TB/s; here 47 us = 5.7 TB/s, 89 % of a plain copy's rate).  Here the kv tiles of a query tile are split twice:
//   * over a CLUSTER of 1, 2, 4 or 8 CTAs, contiguous chunks;
//   * inside a CTA over two online-softmax streams, even and odd tiles of the chunk, each with a warpgroup, a score buffer
//     and an accumulator of its own (thread t owns query row t, as in fwd_pair_sm100.cu): while one stream computes
//     exponentials the tensor core works for the other.
// Every mask but documents, whose tile counts are only known on the device: the launch is sized before.
// The partial results (running maximum, sum, unnormalised O in f32) of all streams meet at the end through distributed
// shared memory: CTA r of the cluster merges every C-th row, so no workspace and no second launch are needed.
//
//   warps 0..3 / 4..7 : softmax of the even / odd tiles; a warp whose 32 rows lie past the end only keeps the barriers.
//   warp 8            : MMA issuer.  warp 9: TMA producer, K and V through rings of kStages stages (192 KB in flight: the
//                       loads are what bounds this kernel).  warps 10, 11: idle.
#include <mutex>

#include "score_row.cuh"

namespace flexattn {
namespace FLEXATTN_TU_NAMESPACE {

constexpr int kThreads = 384;
constexpr int kMmaWarp = 8, kTmaWarp = 9;
constexpr int kMaxStages = 6;
constexpr int kRegsSoftmax = 208, kRegsRest = 88;
static_assert(256 * kRegsSoftmax + 128 * kRegsRest <= kThreads * kSplitLaunchRegs, "more registers than the CTA is launched with");

struct SplitSmem {
  uint64_t bar_q, bar_k[kMaxStages], bar_v[kMaxStages], bar_kfree[kMaxStages], bar_vfree[kMaxStages], bar_s[2], bar_p[2], bar_pv[2];
  uint32_t tmem_base;
  int32_t dead;            // the abort word was set on entry
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t at_rank(uint32_t addr, uint32_t rank) {  // the same shared-memory address in another CTA
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
__device__ __forceinline__ float ld_cluster(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
template <int N>
__device__ __forceinline__ void ld_cluster(float (&v)[N], uint32_t a) {
  if constexpr (N == 4)
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(a) : "memory");
  else
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(a) : "memory");
}

template <int D, int SK, int MK>
__global__ void __launch_bounds__(kThreads, 1)
    fwd_split_sm100_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                           const __grid_constant__ CUtensorMap tm_v, const DevParams P, int* abort_flag) {
  constexpr int kPanels = D / 64;
  constexpr int kStages = D == 128 ? 3 : 6;
  constexpr uint32_t kTileBytes = kPanels * ptx::kPanelBytes;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColS = 0, kColO = 256;  // stream s: S at kColS + 128 s, O at kColO + 128 s
  // partial results, in the rings once every MMA has completed: O rows of D floats + 16 bytes (16-byte stores of
  // consecutive rows then fall on different banks), then {m_ref, m_true, l} of the 128 rows
  constexpr uint32_t kRowFloats = D + 4;
  constexpr uint32_t kPartBytes = (kTile * kRowFloats + 3 * kTile) * 4;
  static_assert(2 * kPartBytes <= 2 * kStages * kTileBytes, "the partial results fit the rings");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;
  uint8_t* sK = smem + kTileBytes;
  uint8_t* sV = sK + kStages * kTileBytes;
  SplitSmem* sh = reinterpret_cast<SplitSmem*>(sV + kStages * kTileBytes);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int C = (int)cluster_size(), rank = (int)cluster_rank();
  const int slices = P.batch * P.heads;
  const int item = (int)blockIdx.x / C;
  const int qt = P.n_qt - 1 - item / slices;  // late query tiles see the most keys under a causal mask: first
  const int bh = item % slices, b = bh / P.heads, h = bh % P.heads;
  const int4 rm = P.row_map[(size_t)(P.map_rows > 1 ? b : 0) * P.n_qt + qt];
  const int n_all = max(rm.y - rm.x, 0);
  const int lo = rm.x + (int)((long long)n_all * rank / C), hi = rm.x + (int)((long long)n_all * (rank + 1) / C);

  if (tid == 0) {
    sh->dead = aborted_on_entry(abort_flag, P.status, 6) ? 1 : 0;
    ptx::mbar_init(&sh->bar_q, 1);
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&sh->bar_k[s], 1);
      ptx::mbar_init(&sh->bar_v[s], 1);
      ptx::mbar_init(&sh->bar_kfree[s], 1);
      ptx::mbar_init(&sh->bar_vfree[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&sh->bar_s[s], 1);
      ptx::mbar_init(&sh->bar_p[s], 4);  // one arrival per warp of the stream's warpgroup
      ptx::mbar_init(&sh->bar_pv[s], 1);
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
  // a CTA that must not run stays in the cluster all the same: the others read its shared memory at the end
  const bool dead = sh->dead != 0;
  const int NT = dead ? 0 : hi - lo;

  if (warp >= 8) {
    ptx::setmaxnreg_dec<kRegsRest>();
    if (warp == kTmaWarp) {
      // ---------------------------------------------------------------- TMA producer
      if (ptx::elect_one() && NT > 0) {
        bool ok = true;
        ptx::prefetch_tensormap(&tm_q);
        ptx::prefetch_tensormap(&tm_k);
        ptx::prefetch_tensormap(&tm_v);
        ptx::mbar_arrive_expect_tx(&sh->bar_q, kTileBytes);
#pragma unroll
        for (int p = 0; p < kPanels; ++p) ptx::tma_load_3d(sQ + p * ptx::kPanelBytes, &tm_q, &sh->bar_q, p * 64, qt * kTile, bh);
        int st = 0;
        uint32_t ph = 1;  // parity of the release waited for: the previous round of the ring
        for (int T = 0; T < NT; ++T) {
          const int row0 = kv_tile_at<SK>(lo, hi, T) * kTile;
          if (T >= kStages) ok = ptx::mbar_wait_relaxed(&sh->bar_kfree[st], ph);
          if (!ok) break;
          ptx::mbar_arrive_expect_tx(&sh->bar_k[st], kTileBytes);
#pragma unroll
          for (int p = 0; p < kPanels; ++p)
            ptx::tma_load_3d(sK + st * kTileBytes + p * ptx::kPanelBytes, &tm_k, &sh->bar_k[st], p * 64, row0, bh);
          if (T >= kStages) ok = ptx::mbar_wait_relaxed(&sh->bar_vfree[st], ph);
          if (!ok) break;
          ptx::mbar_arrive_expect_tx(&sh->bar_v[st], kTileBytes);
#pragma unroll
          for (int p = 0; p < kPanels; ++p)
            ptx::tma_load_3d(sV + st * kTileBytes + p * ptx::kPanelBytes, &tm_v, &sh->bar_v[st], p * 64, row0, bh);
          if (++st == kStages) { st = 0; ph ^= 1u; }
        }
        if (!ok) give_up(abort_flag, P.status, 6, 20);
      }
    } else if (warp == kMmaWarp) {
      // ---------------------------------------------------------------- MMA issuer of both streams
      if (ptx::elect_one() && NT > 0) {
        bool ok = true;
        int fail_at = 1;
        constexpr uint32_t idesc_qk = ptx::make_idesc(128, 128, false);
        constexpr uint32_t idesc_pv = ptx::make_idesc(128, D, true);
        const ptx::DescBase bQ = ptx::base_kmajor(ptx::smem_u32(sQ));
        int qst = 0, pst = 0;
        uint32_t qph = 0, pph = 0;
        auto issue_qk = [&](int s) {  // S_s = Q K^T of the next tile
          ok = ptx::mbar_wait(&sh->bar_k[qst], qph);
          if (!ok) { fail_at = 3; return; }
          ptx::tc_fence_after();
          const ptx::DescBase bk = ptx::base_kmajor(ptx::smem_u32(sK + qst * kTileBytes));
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            ptx::mma_ss(tmem + kColS + (uint32_t)s * 128u, ptx::desc_at(bQ, ptx::koff_kmajor(kk)),
                        ptx::desc_at(bk, ptx::koff_kmajor(kk)), idesc_qk, kk > 0);
          ptx::mma_commit(&sh->bar_s[s]);
          ptx::mma_commit(&sh->bar_kfree[qst]);
          if (++qst == kStages) { qst = 0; qph ^= 1u; }
        };
        ok = ptx::mbar_wait(&sh->bar_q, 0);
        if (!ok) fail_at = 2;
        if (ok) issue_qk(0);
        if (ok && NT > 1) issue_qk(1);
        for (int T = 0; T < NT && ok; ++T) {
          const int s = T & 1;
          ok = ptx::mbar_wait(&sh->bar_v[pst], pph);
          if (!ok) { fail_at = 5; break; }
          ok = ptx::mbar_wait(&sh->bar_p[s], (T >> 1) & 1);
          if (!ok) { fail_at = 4; break; }
          ptx::tc_fence_after();
          const ptx::DescBase bv = ptx::base_mnmajor(ptx::smem_u32(sV + pst * kTileBytes));
          const uint32_t dS = tmem + kColS + (uint32_t)s * 128u;
#pragma unroll
          for (int kk = 0; kk < kTile / 16; ++kk)
            ptx::mma_ts(tmem + kColO + (uint32_t)s * 128u, dS + kk * 8, ptx::desc_at(bv, ptx::koff_mnmajor(kk)), idesc_pv,
                        (T > 1) || (kk > 0));
          if (T + 2 >= NT) ptx::mma_commit(&sh->bar_pv[s]);  // the stream's last tile
          ptx::mma_commit(&sh->bar_vfree[pst]);
          if (++pst == kStages) { pst = 0; pph ^= 1u; }
          // over the columns P V reads its A operand from: MMAs of one thread execute in issue order
          if (T + 2 < NT) issue_qk(s);
        }
        if (!ok) give_up(abort_flag, P.status, 6, fail_at);
      }
    }
    __syncwarp();
  } else {
    ptx::setmaxnreg_inc<kRegsSoftmax>();
    // ------------------------------------------------------------------ softmax: warpgroup s = stream s
    const int row = tid & 127;
    const int s = tid >> 7;
    const int i = qt * kTile + row;
    const bool warp_rows = qt * kTile + (warp & 3) * 32 < P.seq_q;  // any of this warp's rows exists
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t colS = kColS + (uint32_t)s * 128u, colO = kColO + (uint32_t)s * 128u;
    const float c2 = P.sm_scale * kLog2e;
    const float slope2 = (SK == FLEXATTN_SCORE_ALIBI && FLEXATTN_DBG_OK(h, P.heads, 6, 601)) ? P.alibi_slopes[h] * kLog2e : 0.f;
    const float capl2 = P.cap * kLog2e;
    const float csc = (SK == FLEXATTN_SCORE_SOFTCAP) ? P.sm_scale / P.cap : 0.f;
    float m_ref = kMasked, m_true = kMasked, l = 0.f;
    const ScoreCtx ctx{P.sm_scale, b, h};
    int klo = 0, khi = P.seq_k;  // the row's interval of kept keys
    const uint32_t pattern = MK == FLEXATTN_MASK_S2 ? stride_pattern32(P.stride) : 0u;
    row_key_interval<MK>(i, P.seq_k, P.window, klo, khi);
    bool ok = !dead;
    int fail_at = 0;
    const int N = (NT - s + 1) / 2;  // tiles s, s + 2, ... of the chunk
    for (int n = 0; n < N; ++n) {
      const uint32_t par = n & 1;
      const int kt = kv_tile_at<SK>(lo, hi, 2 * n + s), j0 = kt * kTile;
      const bool partial = !(kt >= rm.z && kt < rm.w);
      // a failed wait never leaves the loop early: every thread gets to the barrier behind it
      if (ok) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_s[s], par));
        if (!ok) fail_at = 10;
      }
      if (!ok) continue;
      if (!warp_rows) {  // P of rows past the end: whatever the columns hold, no other row sees it
        ptx::mbar_arrive_warp(&sh->bar_p[s]);
        continue;
      }
      ptx::tc_fence_after();
      float x[kTile];
      {
        uint32_t xr[4][32];
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) ptx::tmem_ld32(lane_base + colS + q4 * 32, xr[q4]);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          ptx::tmem_ld_acquire(xr[q4]);
#pragma unroll
          for (int c = 0; c < 32; ++c) x[q4 * 32 + c] = __uint_as_float(xr[q4][c]);
        }
      }
      // xs: factor still to be applied to x inside the exp2 argument (the plain-score fast path keeps the raw
      // scores and folds sm_scale*log2e into the FMA that also subtracts the running max)
      float tmax, xs = 1.0f;
      if (partial) {
        tmax = score_row<SK, MK, true>(x, i, j0, P.seq_k, P.window, P.stride, c2, slope2, capl2, csc, 0, nullptr, ctx, klo, khi,
                                       pattern);
      } else if constexpr (SK != FLEXATTN_SCORE_NONE) {
        tmax = score_row<SK, MK, false>(x, i, j0, P.seq_k, P.window, P.stride, c2, slope2, capl2, csc, 0, nullptr, ctx);
      } else {
        float mx[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
        for (int c = 4; c + 7 < kTile; c += 8) {
          mx[0] = ptx::max3(mx[0], x[c], x[c + 1]);
          mx[1] = ptx::max3(mx[1], x[c + 2], x[c + 3]);
          mx[2] = ptx::max3(mx[2], x[c + 4], x[c + 5]);
          mx[3] = ptx::max3(mx[3], x[c + 6], x[c + 7]);
        }
        mx[0] = ptx::max3(mx[0], x[kTile - 4], x[kTile - 3]);
        mx[1] = ptx::max3(mx[1], x[kTile - 2], x[kTile - 1]);
        tmax = ptx::max3(mx[0], mx[1], fmaxf(mx[2], mx[3])) * c2;  // c2 > 0: scaling commutes with max
        xs = c2;
      }
      m_true = fmaxf(m_true, tmax);
      const float m_cand = fmaxf(m_ref, tmax);
      if (__any_sync(0xffffffffu, (m_cand - m_ref) > kLazyRescale)) {
        const float alpha = ptx::ex2(m_ref - m_cand);
        l *= alpha;
        m_ref = m_cand;
        if (n > 0) {
          // O_s holds the tiles up to n-1: their P V completed before Q K^T of tile n was issued (same thread,
          // issue order), and S(n) has been read, so it is complete
#pragma unroll 1
          for (int c0 = 0; c0 < D; c0 += 32) {
            uint32_t r[32];
            ptx::tmem_ld32(lane_base + colO + c0, r);
            ptx::tmem_wait_ld();
            ptx::tmem_ld_acquire(r);
#pragma unroll
            for (int c = 0; c < 32; ++c) r[c] = __float_as_uint(__uint_as_float(r[c]) * alpha);
            ptx::tmem_st32(lane_base + colO + c0, r);
          }
          ptx::tmem_wait_st();
        }
      }
      {
        uint64_t ls2[2] = {0ull, 0ull};
        const float nm = ptx::kRoundLog2 - m_ref;  // pre-scaled by (1 + 2^-9) for pack_bf16_trunc
        const uint64_t xs2 = ptx::pack2(xs, xs), nm2 = ptx::pack2(nm, nm);
#pragma unroll
        for (int c0 = 0; c0 < kTile; c0 += 64) {
          uint32_t pk[32];
#pragma unroll
          for (int c = 0; c < 64; c += 2) {
            float a0, a1;
            ptx::unpack2(ptx::fma2(ptx::pack2(x[c0 + c], x[c0 + c + 1]), xs2, nm2), a0, a1);
            const float p0 = ptx::ex2(a0), p1 = ptx::ex2(a1);
            ls2[(c >> 1) & 1] = ptx::add2(ls2[(c >> 1) & 1], ptx::pack2(p0, p1));
            pk[c >> 1] = ptx::pack_bf16_trunc(p0, p1);
          }
          ptx::tmem_st32(lane_base + colS + (c0 >> 1), pk);
        }
        float s0, s1;
        ptx::unpack2(ptx::add2(ls2[0], ls2[1]), s0, s1);
        l += s0 + s1;
      }
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      ptx::mbar_arrive_warp(&sh->bar_p[s]);
    }
    if (ok && N > 0) {
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_pv[s], 0));  // committed once, after the last P V
      if (!ok) fail_at = 12;
    }
    // both streams' MMAs have completed, so every load has landed and been read: the rings hold the partial results now
    ptx::named_bar_sync(3, 256);
    if (ok && warp_rows) {
      float* part = reinterpret_cast<float*>(sK + s * kPartBytes);
      float* orow = part + row * kRowFloats;
      ptx::tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t r[32];
        if (N > 0) {
          ptx::tmem_ld32(lane_base + colO + c0, r);
          ptx::tmem_wait_ld();
          ptx::tmem_ld_acquire(r);
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) r[c] = 0u;
        }
#pragma unroll
        for (int c = 0; c < 32; c += 4) *reinterpret_cast<uint4*>(orow + c0 + c) = make_uint4(r[c], r[c + 1], r[c + 2], r[c + 3]);
      }
      float* stat = part + kTile * kRowFloats;
      stat[row] = m_ref;
      stat[kTile + row] = m_true;
      stat[2 * kTile + row] = l;
    }
    if (!ok && !dead && lane == 0) give_up(abort_flag, P.status, 6, fail_at);
  }

  ptx::tc_fence_before();
  cluster_sync();  // every CTA's partial results are in place
  if (warp < 8 && !dead) {
    // Merge: warp w of CTA r takes rows r + C w, r + C (w + 8) ...  Lane p < 2 C holds the statistics of partial p (CTA
    // p / 2, stream p & 1), every lane D / 32 columns of the output.
    constexpr int kPer = D / 32;
    const uint32_t base = ptx::smem_u32(sK);
    const int rows = min(kTile, P.seq_q - qt * kTile);
    const long long n_rows = (long long)slices * P.seq_q;
    for (int row = rank + C * warp; row < rows; row += 8 * C) {
      float m_ref = kMasked, m_true = kMasked, l = 0.f;
      if (lane < 2 * C) {
        const uint32_t a = at_rank(base + (lane & 1) * kPartBytes + (kTile * kRowFloats + row) * 4, lane >> 1);
        m_ref = ld_cluster(a);
        m_true = ld_cluster(a + kTile * 4);
        l = ld_cluster(a + 2 * kTile * 4);
      }
      float mx = m_ref, mt = m_true;
#pragma unroll
      for (int sft = 8; sft > 0; sft >>= 1) {  // at most 16 partials
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, sft));
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, sft));
      }
      mx = __shfl_sync(0xffffffffu, mx, 0);
      mt = __shfl_sync(0xffffffffu, mt, 0);
      const float w = lane < 2 * C ? ptx::ex2(m_ref - mx) : 0.f;
      float lsum = l * w;
#pragma unroll
      for (int sft = 8; sft > 0; sft >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, sft);
      lsum = __shfl_sync(0xffffffffu, lsum, 0);
      float acc[kPer];
#pragma unroll
      for (int c = 0; c < kPer; ++c) acc[c] = 0.f;
      for (int p = 0; p < 2 * C; ++p) {
        float v[kPer];
        ld_cluster(v, at_rank(base + (p & 1) * kPartBytes + (row * kRowFloats + lane * kPer) * 4, p >> 1));
        const float wp = __shfl_sync(0xffffffffu, w, p);
#pragma unroll
        for (int c = 0; c < kPer; ++c) acc[c] = fmaf(wp, v[c], acc[c]);
      }
      const float inv_l = lsum > 0.f ? ptx::kRoundUp / lsum : 0.f;  // l sums the pre-scaled probabilities
      const size_t grow = (size_t)bh * P.seq_q + qt * kTile + row;
      if (FLEXATTN_DBG_OK(grow, n_rows, 6, 604)) {
        uint32_t* out = reinterpret_cast<uint32_t*>(static_cast<uint16_t*>(P.o) + grow * D + lane * kPer);
#pragma unroll
        for (int c = 0; c < kPer; c += 2) out[c / 2] = ptx::pack_bf16(acc[c] * inv_l, acc[c + 1] * inv_l);
        if (lane == 0) {
          P.l[grow] = lsum * ptx::ex2(mx - mt) * ptx::kRoundInv;
          P.m[grow] = mt * kLn2;
        }
      }
    }
  }
  cluster_sync();  // nobody's shared memory goes away while another CTA may read it
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
}

constexpr size_t split_smem(int head_dim) {
  return (size_t)(head_dim / 64) * ptx::kPanelBytes * (1 + 2 * (head_dim == 128 ? 3 : 6)) + sizeof(SplitSmem) + 1024;
}

template <int D, int SK, int MK>
int launch_one(cudaStream_t st, const DevParams& d, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
               int* abort_flag) {
  constexpr size_t smem = split_smem(D);
  auto kern = fwd_split_sm100_kernel<D, SK, MK>;
  static const bool whole_file = launch_registers(reinterpret_cast<const void*>(kern)) >= kSplitLaunchRegs;
  if (!whole_file) return FLEXATTN_ERR_UNSUPPORTED_BACKEND;
  static SmemAttrOnce attr_once{};  // per kernel instantiation, per device
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), (int)smem, &attr_once) != FLEXATTN_OK) return FLEXATTN_ERR_CUDA;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)d.kv_splits;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(d.n_qt * d.batch * d.heads * d.kv_splits));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, tq, tk, tv, d, abort_flag) == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}

template <int D, int SK>
int launch_mask(cudaStream_t st, const DevParams& d, int mask, const CUtensorMap& tq, const CUtensorMap& tk,
                const CUtensorMap& tv, int* af) {
  switch (mask) {
    case FLEXATTN_MASK_NONE: return launch_one<D, SK, FLEXATTN_MASK_NONE>(st, d, tq, tk, tv, af);
    case FLEXATTN_MASK_CAUSAL: return launch_one<D, SK, FLEXATTN_MASK_CAUSAL>(st, d, tq, tk, tv, af);
    case FLEXATTN_MASK_SLIDING_WINDOW: return launch_one<D, SK, FLEXATTN_MASK_SLIDING_WINDOW>(st, d, tq, tk, tv, af);
    case FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL:
      return launch_one<D, SK, FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL>(st, d, tq, tk, tv, af);
    case FLEXATTN_MASK_S2: return launch_one<D, SK, FLEXATTN_MASK_S2>(st, d, tq, tk, tv, af);
    default: return FLEXATTN_ERR_UNSUPPORTED_MOD;
  }
}

template <int D>
int launch_score(cudaStream_t st, const DevParams& d, int score, int mask, const CUtensorMap& tq,
                 const CUtensorMap& tk, const CUtensorMap& tv, int* af) {
  switch (score) {
    case FLEXATTN_SCORE_NONE: return launch_mask<D, FLEXATTN_SCORE_NONE>(st, d, mask, tq, tk, tv, af);
    case FLEXATTN_SCORE_ALIBI: return launch_mask<D, FLEXATTN_SCORE_ALIBI>(st, d, mask, tq, tk, tv, af);
    case FLEXATTN_SCORE_SOFTCAP: return launch_mask<D, FLEXATTN_SCORE_SOFTCAP>(st, d, mask, tq, tk, tv, af);
    default: return FLEXATTN_ERR_UNSUPPORTED_MOD;
  }
}

}  // namespace FLEXATTN_TU_NAMESPACE

// Clusters of c = 2, 4 or 8 CTAs that run at once on the current device (asked once per device and size); 0 on error.
int split_clusters_at_once(int c) {
  static std::mutex mu;
  static int cached[kMaxDevices][9] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev][c] == 0) {
    auto kern = fwd_split_sm100_kernel<128, FLEXATTN_SCORE_NONE, FLEXATTN_MASK_NONE>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)split_smem(128)) != cudaSuccess) return 0;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)c;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(64 * c));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = split_smem(128);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      return 0;
    }
    cached[dev][c] = n;
  }
  return cached[dev][c];
}

int launch_sm100_fwd_split(cudaStream_t st, const DevParams& d, int score, int mask) {
  int* af = abort_flag_ptr();
  if (af == nullptr) return FLEXATTN_ERR_CUDA;
  CUtensorMap tq, tk, tv;
  const int slices = d.batch * d.heads;
  int e = make_tile_map(&tq, d.q, slices, d.seq_q, d.head_dim);
  if (e) return e;
  e = make_tile_map(&tk, d.k, slices, d.seq_k, d.head_dim);
  if (e) return e;
  e = make_tile_map(&tv, d.v, slices, d.seq_k, d.head_dim);
  if (e) return e;
  if (d.head_dim == 128) return launch_score<128>(st, d, score, mask, tq, tk, tv, af);
  if (d.head_dim == 64) return launch_score<64>(st, d, score, mask, tq, tk, tv, af);
  return FLEXATTN_ERR_UNSUPPORTED_HEAD_DIM;
}

}  // namespace flexattn
