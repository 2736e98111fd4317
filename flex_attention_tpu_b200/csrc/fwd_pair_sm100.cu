// Forward flex attention, two query tiles at a time (sm_100a).
//
// Same math and interface as fwd_pipe_sm100.cu (reference: flex_attention_kernel.py:196-327).  A CTA owns two
// adjacent 128-row query tiles of one (batch, head) and runs them as two independent online-softmax streams over the
// SAME K/V tiles, half a period apart: while stream A's warpgroup computes the exponentials of kv tile n, the tensor
// core runs stream B's P V and Q K^T, and the other way round.  In a stream thread t owns query row t (= TMEM lane
// t) and all 128 score columns of it, so a row maximum or sum needs no exchange between threads and there is no
// per-tile barrier between warpgroups; K and V are loaded once for both tiles.
//
//   warps 0..3 / 4..7 : softmax of stream A / B (registers raised to 208 per thread).
//   warp 8, one thread: MMA issuer of both streams: O_s += P_s V, then S_s = Q_s K_next^T over the columns P_s
//                       occupied (MMAs of one thread execute in issue order).
//   warp 9, one thread: TMA producer: Q_A, Q_B once a pair, K and V through two-stage rings; takes the pairs.
//   warps 10, 11      : idle (they complete the warpgroup whose registers are lowered to 88).
//
// Tensor memory: S_A, S_B, O_A, O_B = 4 x 128 columns.  Shared memory: Q_A, Q_B, 2 K, 2 V tiles and a 64-column staging panel of
// the output per stream (224 KB for D = 128).  Persistent over a list of pairs, heaviest first, with one CTA in the grid per pair:
// a CTA that runs takes over others that have not been launched (cluster launch control), one at a time, so the list is
// dealt out as the CTAs get on (dealt out in rounds, [2,16,4096,128] causal took 1.46 times the mean of the CTAs' work) and
// needs no counter that somebody would have to reset.  A stream's next Q is loaded while its last tile's softmax runs (its last
// Q K^T has read the old one), the first Q K^T of the next pair follows the last P V of this one, and while one stream reads its
// output out of tensor memory the other keeps the tensor core busy.
#include "sched.cuh"
#include "score_row.cuh"

namespace flexattn {
namespace FLEXATTN_TU_NAMESPACE {

constexpr int kThreads = 384;
constexpr int kMmaWarp = 8, kTmaWarp = 9;
constexpr int kItemRing = 2;
constexpr int kRegsSoftmax = 208, kRegsRest = 88;
struct PairSmem {
  uint64_t bar_q[2], bar_qfree[2], bar_k[2], bar_v[2], bar_kfree[2], bar_vfree[2], bar_s[2], bar_p[2], bar_pv[2];
  uint64_t bar_item[kItemRing], bar_itemfree[kItemRing], bar_next;
  alignas(16) uint4 next;  // who comes next (cancel_cta)
  PairItem item[kItemRing];
  uint32_t tmem_base;
  int32_t doc[2][kTile];  // per stream: document ids of the kv tile being processed
};

// The union [first, end) of the kv ranges of a pair's two query tiles (empty: first = end)
__device__ __forceinline__ void pair_union(const int4& a, const int4& b, int& first, int& end) {
  const bool any_a = a.y > a.x, any_b = b.y > b.x;
  first = any_a && any_b ? min(a.x, b.x) : (any_a ? a.x : b.x);
  end = any_a && any_b ? max(a.y, b.y) : (any_a ? a.y : (any_b ? b.y : b.x));
}

template <int D, int SK, int MK>
__global__ void __launch_bounds__(kThreads, 1)
    fwd_pair_sm100_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                          const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                          const DevParams P, int* abort_flag) {
  constexpr int kPanels = D / 64;
  constexpr uint32_t kTileBytes = kPanels * ptx::kPanelBytes;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColS = 0, kColO = 256;  // stream s: S at kColS + 128 s, O at kColO + 128 s

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                   // Q_A, Q_B
  uint8_t* sK = smem + 2 * kTileBytes;  // two stages
  uint8_t* sV = smem + 4 * kTileBytes;  // two stages
  uint8_t* sO = smem + 6 * kTileBytes;  // 64 columns of the output on their way out, per stream
  PairSmem* sh = reinterpret_cast<PairSmem*>(sO + 2 * ptx::kPanelBytes);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (aborted_on_entry(abort_flag, P.status, 5)) return;

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&sh->bar_q[s], 1);
      ptx::mbar_init(&sh->bar_qfree[s], 1);
      ptx::mbar_init(&sh->bar_k[s], 1);
      ptx::mbar_init(&sh->bar_v[s], 1);
      ptx::mbar_init(&sh->bar_kfree[s], 1);
      ptx::mbar_init(&sh->bar_vfree[s], 1);
      ptx::mbar_init(&sh->bar_s[s], 1);
      ptx::mbar_init(&sh->bar_p[s], 4);  // one arrival per warp of the stream's warpgroup
      ptx::mbar_init(&sh->bar_pv[s], 1);
    }
    for (int r = 0; r < kItemRing; ++r) {
      ptx::mbar_init(&sh->bar_item[r], 1);
      ptx::mbar_init(&sh->bar_itemfree[r], 9);  // eight softmax warps, MMA
    }
    ptx::mbar_init(&sh->bar_next, 1);
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

  // In every role: T = index of a kv tile in the stream of all this CTA's pairs (the union of a pair's two ranges; ring stage T & 1,
  // phase (T >> 1) & 1), u = index of a query tile among those of a stream that have keys, c = index of a tile among a
  // stream's own (phases u & 1, c & 1).
  if (warp >= 8) {
    ptx::setmaxnreg_dec<kRegsRest>();
    if (warp == kTmaWarp) {
      // ---------------------------------------------------------------- TMA producer
      if (ptx::elect_one()) {
        bool ok = true;
        ptx::prefetch_tensormap(&tm_q);
        ptx::prefetch_tensormap(&tm_k);
        ptx::prefetch_tensormap(&tm_v);
        int T = 0, u0 = 0, u1 = 0;
        const PairList list(P);
        int w = (int)blockIdx.x;
        for (int r = 0; ok; ++r) {
          PairItem it;
          it.bh = -1;
          if (w >= 0) it = list.fetch(w);
          if (r >= kItemRing) ok = ptx::mbar_wait_relaxed(&sh->bar_itemfree[r % kItemRing], (r / kItemRing - 1) & 1, 20);
          if (!ok) break;
          sh->item[r % kItemRing] = it;
          ptx::mbar_arrive(&sh->bar_item[r % kItemRing]);
          if (w < 0) break;
          const int4 rm0 = it.rm0, rm1 = it.rm1;
          const int bh = it.bh, pair = it.pair;
          int first, end;
          pair_union(rm0, rm1, first, end);
          auto load_tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int row) {
            ptx::mbar_arrive_expect_tx(bar, kTileBytes);
#pragma unroll
            for (int p = 0; p < kPanels; ++p) ptx::tma_load_3d(dst + p * ptx::kPanelBytes, tm, bar, p * 64, row, bh);
          };
          auto load_q = [&](int s, bool any, int& u) {
            if (!any || !ok) return;
            if (u > 0) ok = ptx::mbar_wait_relaxed(&sh->bar_qfree[s], (u - 1) & 1, 20);  // every Q K^T of the one before has completed
            if (!ok) return;
            load_tile(sQ + s * kTileBytes, &tm_q, &sh->bar_q[s], (2 * pair + s) * kTile);
            ++u;
          };
          // order of first use: Q_A, K(0), Q_B, V(0), K(1), V(1)
          for (int n = 0; n < end - first && ok; ++n, ++T) {
            const int row = kv_tile_at<SK>(first, end, n) * kTile;
            const uint32_t par = ((T - 2) >> 1) & 1;
            if (n == 0) load_q(0, rm0.y > rm0.x, u0);
            if (T >= 2) ok = ok && ptx::mbar_wait_relaxed(&sh->bar_kfree[T & 1], par, 20);  // every Q K^T of tile T-2 has completed
            if (!ok) break;
            load_tile(sK + (T & 1) * kTileBytes, &tm_k, &sh->bar_k[T & 1], row);
            if (n == 0) load_q(1, rm1.y > rm1.x, u1);
            if (T >= 2) ok = ok && ptx::mbar_wait_relaxed(&sh->bar_vfree[T & 1], par, 20);  // every P V of tile T-2 has completed
            if (!ok) break;
            load_tile(sV + (T & 1) * kTileBytes, &tm_v, &sh->bar_v[T & 1], row);
          }
          if (!ok) break;
          // The next pair, two tiles before this one ends.  (Taken a whole pair ahead, the list would be dealt out almost as in
          // rounds: [2,16,4096,128] causal 142 -> 170 us.)
          ptx::mbar_arrive_expect_tx(&sh->bar_next, 16);
          ptx::cancel_cta(&sh->next, &sh->bar_next);
          ok = ptx::mbar_wait(&sh->bar_next, r & 1);
          if (ok) w = ptx::cancelled_cta(&sh->next);
          ptx::fence_proxy_async_smem();  // (read before the next answer is written)
        }
        if (!ok) give_up(abort_flag, P.status, 5, 20);
      }
    } else if (warp == kMmaWarp) {
      // ---------------------------------------------------------------- MMA issuer of both streams.
      // An elected thread issues an MMA every 2 to 8 cycles until the queue is full (64 cycles of tensor work each); the
      // waits and commits around them still count, so it waits once per tile for K and V, not once per stream, and
      // commits "P V done" only for a query tile's last one, the only one anybody waits for.
      // (A second issuing thread, one per stream, was measured 13 % slower.)
      if (ptx::elect_one()) {
        bool ok = true;
        int fail_at = 1;
        constexpr uint32_t idesc_qk = ptx::make_idesc(128, 128, false);
        constexpr uint32_t idesc_pv = ptx::make_idesc(128, D, true);
        const ptx::DescBase bQ0 = ptx::base_kmajor(ptx::smem_u32(sQ)), bQ1 = ptx::base_kmajor(ptx::smem_u32(sQ + kTileBytes));
        const ptx::DescBase bK0 = ptx::base_kmajor(ptx::smem_u32(sK)), bK1 = ptx::base_kmajor(ptx::smem_u32(sK + kTileBytes));
        const ptx::DescBase bV0 = ptx::base_mnmajor(ptx::smem_u32(sV)), bV1 = ptx::base_mnmajor(ptx::smem_u32(sV + kTileBytes));
        uint32_t c0 = 0, c1 = 0, u0 = 0, u1 = 0;  // per stream: P V issued, query tiles begun
        int T = 0;
        // Item by item: the first Q K^T of a pair follow the last P V of the one before.  (Issued between those two, for the
        // stream that is done first, they would come no earlier than its softmax warps can use them, which read their output out
        // by then; and the next pair would have to be known while this one's P V wait, though the softmax warps reach the items
        // between, pairs without a kv tile, only after those.)
        for (int r = 0; ok; ++r) {
          ok = ptx::mbar_wait(&sh->bar_item[r % kItemRing], (r / kItemRing) & 1);
          if (!ok) { fail_at = 9; break; }
          const int4 rm0 = sh->item[r % kItemRing].rm0, rm1 = sh->item[r % kItemRing].rm1;
          const bool stop = sh->item[r % kItemRing].bh < 0;
          ptx::mbar_arrive(&sh->bar_itemfree[r % kItemRing]);
          if (stop) break;
          int first, end;
          pair_union(rm0, rm1, first, end);
          const int NT = end - first, n0 = rm0.y - rm0.x, n1 = rm1.y - rm1.x;
          if (NT <= 0) continue;
          int done0 = 0, done1 = 0;  // tiles of each stream whose P V has been issued (= tiles whose Q K^T was, minus one)
          int begun0 = 0, begun1 = 0;
          auto issue_qk = [&](int s, const ptx::DescBase& bk) {  // S_s = Q_s K^T; K has landed
            const uint32_t dS = tmem + kColS + (uint32_t)s * 128u;
            const ptx::DescBase bq = s ? bQ1 : bQ0;
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              ptx::mma_ss(dS, ptx::desc_at(bq, ptx::koff_kmajor(kk)), ptx::desc_at(bk, ptx::koff_kmajor(kk)), idesc_qk, kk > 0);
            ptx::mma_commit(&sh->bar_s[s]);
            if (++(s ? begun1 : begun0) == (s ? n1 : n0)) ptx::mma_commit(&sh->bar_qfree[s]);  // the query tile's last
          };
          auto issue_pv = [&](int s, const ptx::DescBase& bv) {  // O_s += P_s V; V has landed
            const int done = s ? done1 : done0;
            ok = ptx::mbar_wait(&sh->bar_p[s], (s ? c1 : c0) & 1);
            if (!ok) { fail_at = 4; return; }
            ptx::tc_fence_after();
            const uint32_t dS = tmem + kColS + (uint32_t)s * 128u;
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk)
              ptx::mma_ts(tmem + kColO + (uint32_t)s * 128u, dS + kk * 8, ptx::desc_at(bv, ptx::koff_mnmajor(kk)), idesc_pv,
                          (done > 0) || (kk > 0));
            if (done + 1 == (s ? n1 : n0)) ptx::mma_commit(&sh->bar_pv[s]);  // the query tile's last
            if (s) { ++done1; ++c1; } else { ++done0; ++c0; }
          };
          auto in0 = [&](int kt) { return kt >= rm0.x && kt < rm0.y; };
          auto in1 = [&](int kt) { return kt >= rm1.x && kt < rm1.y; };
          {  // first scores
            const int kt0 = kv_tile_at<SK>(first, end, 0);
            const ptx::DescBase bk = (T & 1) ? bK1 : bK0;
            if (in0(kt0)) ok = ptx::mbar_wait(&sh->bar_q[0], u0 & 1);
            if (ok) ok = ptx::mbar_wait(&sh->bar_k[T & 1], (T >> 1) & 1);
            if (!ok) { fail_at = 2; break; }
            ptx::tc_fence_after();
            if (in0(kt0)) issue_qk(0, bk);
            if (in1(kt0)) ok = ptx::mbar_wait(&sh->bar_q[1], u1 & 1);
            if (!ok) { fail_at = 2; break; }
            if (in1(kt0)) issue_qk(1, bk);
            ptx::mma_commit(&sh->bar_kfree[T & 1]);
          }
          for (int n = 0; n < NT && ok; ++n, ++T) {
            const int kt = kv_tile_at<SK>(first, end, n);
            const int kt_next = n + 1 < NT ? kv_tile_at<SK>(first, end, n + 1) : -1;
            const bool a0 = in0(kt), a1 = in1(kt);
            const bool q0 = kt_next >= 0 && in0(kt_next), q1 = kt_next >= 0 && in1(kt_next);
            const ptx::DescBase bv = (T & 1) ? bV1 : bV0, bk = (T & 1) ? bK0 : bK1;  // V(T), K(T+1)
            ok = ptx::mbar_wait(&sh->bar_v[T & 1], (T >> 1) & 1);
            if (!ok) { fail_at = 5; break; }
            if (kt_next >= 0) {
              // K(T+1) was requested a whole tile ago: waiting for it here, once, costs nothing and saves a wait
              // between the two streams
              if (q0 && begun0 == 0) ok = ptx::mbar_wait(&sh->bar_q[0], u0 & 1);  // a stream that starts late
              if (ok && q1 && begun1 == 0) ok = ptx::mbar_wait(&sh->bar_q[1], u1 & 1);
              if (ok) ok = ptx::mbar_wait(&sh->bar_k[(T + 1) & 1], ((T + 1) >> 1) & 1);
              if (!ok) { fail_at = 3; break; }
            }
            if (a0) issue_pv(0, bv);
            if (!ok) break;
            if (q0) issue_qk(0, bk);
            if (a1) issue_pv(1, bv);
            if (!ok) break;
            if (q1) issue_qk(1, bk);
            // both streams' MMAs on V(T) and K(T+1) have been issued: their completion frees the ring stages
            ptx::mma_commit(&sh->bar_vfree[T & 1]);
            if (kt_next >= 0) ptx::mma_commit(&sh->bar_kfree[(T + 1) & 1]);
          }
          u0 += n0 > 0;
          u1 += n1 > 0;
        }
        if (!ok) give_up(abort_flag, P.status, 5, fail_at);
      }
    }
  } else {
    ptx::setmaxnreg_inc<kRegsSoftmax>();
    // ------------------------------------------------------------------ softmax: warpgroup s = stream s
    const int row = tid & 127;
    const int s = tid >> 7;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t colS = kColS + (uint32_t)s * 128u, colO = kColO + (uint32_t)s * 128u;
    const float c2 = P.sm_scale * kLog2e;
    const long long n_rows = (long long)P.batch * P.heads * P.seq_q, n_doc = (long long)P.batch * P.doc_stride;
    const float capl2 = P.cap * kLog2e;
    const float csc = (SK == FLEXATTN_SCORE_SOFTCAP) ? P.sm_scale / P.cap : 0.f;
    constexpr bool kDoc = MK == FLEXATTN_MASK_DOCUMENT;
    const uint32_t pattern = MK == FLEXATTN_MASK_S2 ? stride_pattern32(P.stride) : 0u;
    bool ok = true;
    int fail_at = 0;
    uint32_t tiles = 0, items = 0;  // of this stream so far

    for (int r = 0;; ++r) {
    // the stream's warps leave together or not at all: the others would wait for good at the next named barrier
    if (!ptx::named_bar_all(1 + s, 128, ptx::mbar_wait(&sh->bar_item[r % kItemRing], (r / kItemRing) & 1))) {
      ok = false;
      fail_at = 9;
      break;
    }
    const int bh = sh->item[r % kItemRing].bh, qt = 2 * sh->item[r % kItemRing].pair + s;
    const int4 rms = s ? sh->item[r % kItemRing].rm1 : sh->item[r % kItemRing].rm0;
    ptx::mbar_arrive_warp(&sh->bar_itemfree[r % kItemRing]);
    if (bh < 0) break;
    const int b = bh / P.heads, h = bh - b * P.heads;
    const int i = qt * kTile + row;
    const int N = rms.y - rms.x;
    const float slope2 = (SK == FLEXATTN_SCORE_ALIBI && FLEXATTN_DBG_OK(h, P.heads, 5, 501)) ? P.alibi_slopes[h] * kLog2e : 0.f;
    const int32_t* doc = (MK == FLEXATTN_MASK_DOCUMENT) ? P.doc_ids + (size_t)b * P.doc_stride : nullptr;
    const int di = (MK == FLEXATTN_MASK_DOCUMENT && qt < P.n_qt && i < P.seq_q &&
                    FLEXATTN_DBG_OK((long long)b * P.doc_stride + i, n_doc, 5, 502)) ? doc[i] : 0;
    float m_ref = kMasked, m_true = kMasked, l = 0.f;
    const ScoreCtx ctx{P.sm_scale, b, h};
    // the interval [klo, khi) of keys this row keeps, where the mask has one: the interval kinds, and a document mask
    // when the ids of the batch row never decrease (then the mask map holds the start of every row's document)
    bool doc_runs = false;
    int klo = 0, khi = P.seq_k;
    if constexpr (kMaskIsBits<MK>) row_key_interval<MK>(i, P.seq_k, P.window, klo, khi);
    if constexpr (kDoc) {
      doc_runs = FLEXATTN_DBG_OK(b, P.batch, 5, 506) && P.doc_sorted[b] != 0;
      if (doc_runs && qt < P.n_qt && i < P.seq_q && FLEXATTN_DBG_OK((long long)b * P.doc_stride + i, n_doc, 5, 507)) {
        klo = P.run_lo[(size_t)b * P.doc_stride + i];
        khi = i + 1 < P.seq_k ? i + 1 : P.seq_k;
      }
    }

    for (int n = 0; n < N; ++n, ++tiles) {
      const uint32_t par = tiles & 1;
      const int kt = kv_tile_at<SK>(rms.x, rms.y, n), j0 = kt * kTile;
      const bool partial = !(kt >= rms.z && kt < rms.w);
      if (MK == FLEXATTN_MASK_DOCUMENT && partial && !doc_runs) {
        // one buffer per stream: readers of the previous partial tile are done (first barrier) before the ids of
        // this tile are written; the second barrier publishes them
        ptx::named_bar_sync(1 + s, 128);
        const int j = j0 + row;
        sh->doc[s][row] = (j < P.seq_k && FLEXATTN_DBG_OK((long long)b * P.doc_stride + j, n_doc, 5, 503)) ? doc[j] : -1;
        ptx::named_bar_sync(1 + s, 128);
      }
      // a failed wait never leaves the loop early: every thread keeps executing the same named barriers
      if (ok) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_s[s], par));
        if (!ok) fail_at = 10;
      }
      if (!ok) continue;
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
        if constexpr (kDoc) {
          if (doc_runs)
            tmax = score_row<SK, MK, true, true>(x, i, j0, P.seq_k, P.window, P.stride, c2, slope2, capl2, csc, di, sh->doc[s],
                                                 ctx, klo, khi, pattern);
          else
            tmax = score_row<SK, MK, true, false>(x, i, j0, P.seq_k, P.window, P.stride, c2, slope2, capl2, csc, di,
                                                  sh->doc[s], ctx);
        } else {
          tmax = score_row<SK, MK, true>(x, i, j0, P.seq_k, P.window, P.stride, c2, slope2, capl2, csc, di, sh->doc[s], ctx,
                                         klo, khi, pattern);
        }
      } else if constexpr (SK != FLEXATTN_SCORE_NONE) {
        tmax = score_row<SK, MK, false>(x, i, j0, P.seq_k, P.window, P.stride, c2, slope2, capl2, csc, di, sh->doc[s], ctx);
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

    // ---- epilogue of the stream
    if (qt < P.n_qt) {
      if (ok && N > 0) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&sh->bar_pv[s], items & 1));  // committed after the query tile's last P V
        if (!ok) fail_at = 12;
      }
      const float inv_l = l > 0.f ? ptx::kRoundUp / l : 0.f;  // l sums the pre-scaled probabilities
      const size_t grow = (size_t)bh * P.seq_q + i;
      if (N > 0) {
        // bf16 O / l, 32 columns at a time, through the two halves of the stream's staging panel (TMA layout, 64-byte swizzle):
        // one leaves with a bulk tensor store while the other is written; rows past seq_q are clipped by the tensor map.  The
        // first P of the next pair, which lets its first P V overwrite O, is written after this.
        uint8_t* stage = sO + s * ptx::kPanelBytes;
        if (ok) ptx::tc_fence_after();
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint8_t* part = stage + (c0 & 32) * (ptx::kPanelBytes / 64);
          if (ok) {
            uint32_t r[32];
            ptx::tmem_ld32(lane_base + colO + c0, r);
            ptx::tmem_wait_ld();
            ptx::tmem_ld_acquire(r);
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
              uint4 v4;
              v4.x = ptx::pack_bf16(__uint_as_float(r[c]) * inv_l, __uint_as_float(r[c + 1]) * inv_l);
              v4.y = ptx::pack_bf16(__uint_as_float(r[c + 2]) * inv_l, __uint_as_float(r[c + 3]) * inv_l);
              v4.z = ptx::pack_bf16(__uint_as_float(r[c + 4]) * inv_l, __uint_as_float(r[c + 5]) * inv_l);
              v4.w = ptx::pack_bf16(__uint_as_float(r[c + 6]) * inv_l, __uint_as_float(r[c + 7]) * inv_l);
              *reinterpret_cast<uint4*>(part + row * 64 + (((c >> 3) ^ ((row >> 1) & 3)) << 4)) = v4;
            }
            ptx::fence_proxy_async_smem();  // generic-proxy stores -> visible to the bulk store
          }
          // past this barrier the other half is free: the store before this one has read it
          if (row == 0) ptx::tma_store_wait_read();
          ptx::named_bar_sync(1 + s, 128);
          if (ok && row == 0) {
            ptx::tma_store_3d(&tm_o, part, c0, qt * kTile, bh);
            ptx::tma_store_commit();
          }
        }
        ptx::tc_fence_before();
        ++items;
      } else if (i < P.seq_q && FLEXATTN_DBG_OK(grow, n_rows, 5, 504)) {  // a query tile without any kv tile: zeros, written directly
        uint16_t* orow = static_cast<uint16_t*>(P.o) + grow * D;  // bf16 elements
        for (int c0 = 0; c0 < D; c0 += 8) *reinterpret_cast<uint4*>(orow + c0) = make_uint4(0u, 0u, 0u, 0u);
      }
      if (ok && i < P.seq_q && FLEXATTN_DBG_OK(grow, n_rows, 5, 505)) {
        P.l[grow] = l * ptx::ex2(m_ref - m_true) * ptx::kRoundInv;
        P.m[grow] = m_true * kLn2;
      }
    }
    }
    if (row == 0) ptx::tma_store_wait_read();  // shared memory must outlive the last store's reads
    if (!ok && lane == 0) give_up(abort_flag, P.status, 5, fail_at);
  }

  // ------------------------------------------------------------------ teardown
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
}

#ifndef FLEXATTN_JIT
static_assert(256 * kRegsSoftmax + 128 * kRegsRest <= kThreads * kPairLaunchRegs, "more registers than the CTA is launched with");
unsigned pair_grid(const DevParams& d) {  // one CTA per pair; 0: too many
  const long long pairs = (long long)((d.n_qt + 1) / 2) * d.batch * d.heads;
  return pairs > 0x7fffffff ? 0u : (unsigned)pairs;
}

template <int D, int SK, int MK>
int launch_one(cudaStream_t st, const DevParams& d, const CUtensorMap& tq, const CUtensorMap& tk,
               const CUtensorMap& tv, const CUtensorMap& to, int* abort_flag) {
  constexpr size_t need = (6 * (D / 64) + 2) * ptx::kPanelBytes + sizeof(PairSmem) + 1024;
  // 512 TMEM columns per CTA: never let two CTAs share an SM (the second would spin in tcgen05.alloc)
  constexpr size_t smem = need > 120 * 1024 ? need : 120 * 1024;
  auto kern = fwd_pair_sm100_kernel<D, SK, MK>;
  static const bool whole_file = launch_registers(reinterpret_cast<const void*>(kern)) >= kPairLaunchRegs;
  if (!whole_file) return FLEXATTN_ERR_UNSUPPORTED_BACKEND;
  static SmemAttrOnce attr_once{};  // per kernel instantiation, per device
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), (int)smem, &attr_once) != FLEXATTN_OK) return FLEXATTN_ERR_CUDA;
  const unsigned grid = pair_grid(d);
  if (grid == 0) return FLEXATTN_ERR_BAD_SHAPE;
  kern<<<grid, kThreads, smem, st>>>(tq, tk, tv, to, d, abort_flag);
  return cudaGetLastError() == cudaSuccess ? FLEXATTN_OK : FLEXATTN_ERR_CUDA;
}

template <int D, int SK>
int launch_mask(cudaStream_t st, const DevParams& d, int mask, const CUtensorMap& tq, const CUtensorMap& tk,
                const CUtensorMap& tv, const CUtensorMap& to, int* af) {
  switch (mask) {
    case FLEXATTN_MASK_NONE: return launch_one<D, SK, FLEXATTN_MASK_NONE>(st, d, tq, tk, tv, to, af);
    case FLEXATTN_MASK_CAUSAL: return launch_one<D, SK, FLEXATTN_MASK_CAUSAL>(st, d, tq, tk, tv, to, af);
    case FLEXATTN_MASK_SLIDING_WINDOW: return launch_one<D, SK, FLEXATTN_MASK_SLIDING_WINDOW>(st, d, tq, tk, tv, to, af);
    case FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL:
      return launch_one<D, SK, FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL>(st, d, tq, tk, tv, to, af);
    case FLEXATTN_MASK_DOCUMENT: return launch_one<D, SK, FLEXATTN_MASK_DOCUMENT>(st, d, tq, tk, tv, to, af);
    case FLEXATTN_MASK_S2: return launch_one<D, SK, FLEXATTN_MASK_S2>(st, d, tq, tk, tv, to, af);
    default: return FLEXATTN_ERR_UNSUPPORTED_MOD;
  }
}

template <int D>
int launch_score(cudaStream_t st, const DevParams& d, int score, int mask, const CUtensorMap& tq,
                 const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, int* af) {
  switch (score) {
    case FLEXATTN_SCORE_NONE: return launch_mask<D, FLEXATTN_SCORE_NONE>(st, d, mask, tq, tk, tv, to, af);
    case FLEXATTN_SCORE_ALIBI: return launch_mask<D, FLEXATTN_SCORE_ALIBI>(st, d, mask, tq, tk, tv, to, af);
    case FLEXATTN_SCORE_SOFTCAP: return launch_mask<D, FLEXATTN_SCORE_SOFTCAP>(st, d, mask, tq, tk, tv, to, af);
    default: return FLEXATTN_ERR_UNSUPPORTED_MOD;
  }
}

#endif  // !FLEXATTN_JIT

}  // namespace FLEXATTN_TU_NAMESPACE

#ifndef FLEXATTN_JIT
// No dense bias here; the caller keeps the persistent kernel for that.
int launch_sm100_fwd_pair(cudaStream_t st, const DevParams& d, int score, int mask) {
  int* af = abort_flag_ptr();
  if (af == nullptr) return FLEXATTN_ERR_CUDA;
  CUtensorMap tq, tk, tv, to;
  const int slices = d.batch * d.heads;
  int e = make_tile_map(&tq, d.q, slices, d.seq_q, d.head_dim);
  if (e) return e;
  e = make_tile_map(&tk, d.k, slices, d.seq_k, d.head_dim);
  if (e) return e;
  e = make_tile_map(&tv, d.v, slices, d.seq_k, d.head_dim);
  if (e) return e;
  e = make_tile_map(&to, d.o, slices, d.seq_q, d.head_dim, kTile, 32);
  if (e) return e;
  if (score == FLEXATTN_SCORE_USER) {
    // a kernel compiled at run time around the registered score function: same parameters, grid and shared memory
    const size_t need = (6 * (size_t)(d.head_dim / 64) + 2) * ptx::kPanelBytes + sizeof(PairSmem) + 1024;
    const unsigned grid = pair_grid(d);
    if (grid == 0) return FLEXATTN_ERR_BAD_SHAPE;
    void* args[] = {&tq, &tk, &tv, &to, const_cast<DevParams*>(&d), &af};
    return jit_launch(kJitForwardPair, false, d.user_score, d.head_dim, mask, grid, 1, kThreads,
                      need > 120 * 1024 ? need : 120 * 1024, st, args);
  }
  if (d.head_dim == 128) return launch_score<128>(st, d, score, mask, tq, tk, tv, to, af);
  if (d.head_dim == 64) return launch_score<64>(st, d, score, mask, tq, tk, tv, to, af);
  return FLEXATTN_ERR_UNSUPPORTED_HEAD_DIM;
}
#endif  // !FLEXATTN_JIT

}  // namespace flexattn
