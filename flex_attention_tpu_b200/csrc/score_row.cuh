// What the forward kernels share: the order of an item's kv tiles, and the scores of a 128-column tile where one thread is
// one query row.
#pragma once
#include "sm100.cuh"

namespace flexattn {
namespace FLEXATTN_TU_NAMESPACE {

constexpr float kLazyRescale = 8.0f;  // log2 units

// kv tile visited at step n of the range [first, end).  The ALiBi bias slope * (k_idx - q_idx) grows with the key
// position, so in ascending order the running row maximum of a steep head rises by more than the lazy-rescale
// threshold at EVERY tile, and each rescale waits for the previous P V and rewrites O.  Visiting the tiles from the
// last one down meets the largest bias first and rescales (almost) never; other score kinds keep ascending order.
template <int SK>
__device__ __forceinline__ int kv_tile_at(int first, int end, int n) {
  return SK == FLEXATTN_SCORE_ALIBI ? end - 1 - n : first + n;
}

// what a user score function sees besides the score and the positions
struct ScoreCtx {
  float sm_scale;
  int b, h;
  int step = 1;  // positions from one column to the next (the strided tiles of S2, gathered)
};

// x: this thread's 128 raw scores of one tile -> log2-domain logits in place; returns their maximum.
// kInterval: the row's kept keys are the interval [klo, khi) (interval mask kinds; documents over sorted ids): a
// partial tile then tests one bit per element of a bitmap built once per 32 columns.
template <int SK, int MK, bool kPartial, bool kInterval = kMaskIsBits<MK>>
__device__ __forceinline__ float score_row(float (&x)[kTile], int i, int j0, int seq_k, int window, int stride,
                                           float c2, float slope2, float capl2, float csc, int di,
                                           const int32_t* s_doc, const ScoreCtx ctx, int klo = 0, int khi = 0, uint32_t pattern = 0u) {
  float mx[4] = {kMasked, kMasked, kMasked, kMasked};
  uint32_t keep = 0u;  // kept columns of the current group of 32 (kInterval on partial tiles)
  if constexpr (SK == FLEXATTN_SCORE_SOFTCAP || SK == FLEXATTN_SCORE_USER) {
#pragma unroll
    for (int c = 0; c < kTile; ++c) {
      float t;
      if constexpr (SK == FLEXATTN_SCORE_USER) t = user_score(x[c] * ctx.sm_scale, ctx.b, ctx.h, i, j0 + c) * kLog2e;
      else t = capl2 * ptx::tanh_approx(x[c] * csc);
      if constexpr (kPartial && kInterval) {
        if ((c & 31) == 0) keep = keep_bits32<MK>(j0 + c, klo, khi, stride, pattern);
        t = (keep >> (c & 31)) & 1u ? t : kMasked;
      } else if constexpr (kPartial) {
        const int j = j0 + c;
        const int dj = (MK == FLEXATTN_MASK_DOCUMENT) ? s_doc[c] : 0;
        t = ((j < seq_k) && mask_keep<MK>(i, j, window, stride, di, dj)) ? t : kMasked;
      }
      x[c] = t;
      mx[c & 3] = fmaxf(mx[c & 3], t);
    }
  } else {
    // ALiBi: the bias of columns (c, c + 1) advances by a constant from pair to pair, one packed add.  The adds round alike, so
    // their errors grow along the row: it starts anew in the middle, as the persistent kernel's does (12 heads, 640 positions: log l
    // off by 7.0e-6 in the mean and 4.6e-5 at most when added over 128 columns, 1.5e-6 and 1.2e-5 over 64; no time).
    float abase = slope2 * (float)(j0 - i);
    uint64_t b2 = ptx::pack2(abase, abase + slope2);
    const uint64_t bstep2 = ptx::pack2(2.f * slope2, 2.f * slope2);
#pragma unroll
    for (int c = 0; c < kTile; c += 2) {
      if (SK == FLEXATTN_SCORE_ALIBI && c == kTile / 2) {
        abase = slope2 * (float)(j0 + c - i);
        b2 = ptx::pack2(abase, abase + slope2);
      }
      const uint64_t x2 = ptx::pack2(x[c], x[c + 1]);
      float t0, t1;
      if constexpr (SK == FLEXATTN_SCORE_ALIBI) {
        ptx::unpack2(ptx::fma2(x2, ptx::pack2(c2, c2), b2), t0, t1);
        b2 = ptx::add2(b2, bstep2);
      } else {
        ptx::unpack2(ptx::mul2(x2, ptx::pack2(c2, c2)), t0, t1);
      }
      if constexpr (kPartial && kInterval) {  // one bitmap per row and 32 columns instead of per-element tests
        if ((c & 31) == 0) keep = keep_bits32<MK>(j0 + c, klo, khi, stride, pattern);
        t0 = (keep >> (c & 31)) & 1u ? t0 : kMasked;
        t1 = (keep >> ((c & 31) + 1)) & 1u ? t1 : kMasked;
      } else if constexpr (kPartial) {
        const int j = j0 + c;
        const int d0 = (MK == FLEXATTN_MASK_DOCUMENT) ? s_doc[c] : 0;
        const int d1 = (MK == FLEXATTN_MASK_DOCUMENT) ? s_doc[c + 1] : 0;
        t0 = ((j < seq_k) && mask_keep<MK>(i, j, window, stride, di, d0)) ? t0 : kMasked;
        t1 = ((j + 1 < seq_k) && mask_keep<MK>(i, j + 1, window, stride, di, d1)) ? t1 : kMasked;
      }
      x[c] = t0;
      x[c + 1] = t1;
      mx[(c >> 1) & 3] = ptx::max3(mx[(c >> 1) & 3], t0, t1);
    }
  }
  return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
}

}  // namespace FLEXATTN_TU_NAMESPACE
}  // namespace flexattn
