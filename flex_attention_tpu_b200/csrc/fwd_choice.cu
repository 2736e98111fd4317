// Which of the two forward kernels that work through a list of query tiles serves a call: the persistent one (fwd_pipe_sm100.cu), whose
// CTAs are dealt single query tiles in rounds, or the two-query-tile one (fwd_pair_sm100.cu), whose CTAs take pairs as they get on.  Host only.
//
// A pair takes 0.8 to 0.95 of its two tiles' time, but it is a unit twice as long, fewer of them than CTAs leave SMs idle, and a last tile
// without a partner costs almost as much.  So the rule deals both lists out as the kernels do and compares the times of the fullest
// CTA.  The costs below are fitted (least squares of the logarithms, in us) to 2674 calls timed with either kernel on 148 SMs, graph
// replays: causal, windows, open windows, no mask, S2; 4 to 384 slices of 129 to 8192 queries, equal and unequal lengths.  The kernel it picks is
// 0.2 % slower than the faster of the two in the mean, 2 % of the calls lose more than 3 % (lines drawn by waves of pairs: 1.7 %, 15 %).
// Times in us, two-query-tile / persistent: 96 x 777 against 64 keys with 256 keys 19.9 / 15.8 (empty query tiles), 192 x 384 causal softcap 26.0 / 23.4
// (three tiles: every other pair is half empty), 32 x 2048 causal, D = 64, 36 / 42; 24 x 1024 unmasked, D = 128, 23 / 27.
#include <algorithm>
#include <cmath>
#include <functional>

#include "common.cuh"

namespace flexattn {
namespace {

struct FwdCosts {
  float tile, item;          // persistent kernel: a kv tile of a query tile, and what comes on top of a query tile's
  float both, single, pair;  // two-query-tile kernel: a kv tile that both query tiles see, one that only one of them does, on top of a pair's
};
FwdCosts fwd_costs(const FlexAttnParams& p) {
  const bool d64 = p.head_dim == 64;
  switch (p.score_kind) {
    case FLEXATTN_SCORE_NONE: return d64 ? FwdCosts{1.04f, 1.29f, 1.68f, 1.33f, 1.56f} : FwdCosts{1.09f, 1.79f, 1.87f, 1.72f, 2.04f};
    case FLEXATTN_SCORE_ALIBI: return d64 ? FwdCosts{1.15f, 1.78f, 1.83f, 1.07f, 2.38f} : FwdCosts{1.19f, 2.40f, 2.00f, 1.46f, 2.97f};
    case FLEXATTN_SCORE_SOFTCAP: return d64 ? FwdCosts{1.53f, 1.42f, 2.90f, 1.85f, 1.77f} : FwdCosts{1.57f, 1.97f, 2.88f, 2.12f, 2.69f};
    // a user function (a distance penalty, scalar code): 96 x 512 causal, D = 64, 24.1 / 21.3, which the costs of softcap took the other way
    default: return d64 ? FwdCosts{1.54f, 1.75f, 3.00f, 2.21f, 2.89f} : FwdCosts{1.63f, 2.32f, 3.19f, 2.40f, 3.57f};
  }
}

// The kv tiles [lo, hi) a query tile sees, from the mask kind and the sizes
struct Tiles {
  int lo, hi;
  int count() const { return hi - lo; }
};
Tiles kv_tiles(const FlexAttnParams& p, int n_kt, long long qt) {
  const long long i0 = qt * kTile, i1 = std::min<long long>(i0 + kTile, p.seq_q) - 1;
  const bool windowed = p.mask_kind == FLEXATTN_MASK_SLIDING_WINDOW || p.mask_kind == FLEXATTN_MASK_SLIDING_WINDOW_CAUSAL;
  const bool ahead = p.mask_kind == FLEXATTN_MASK_NONE || p.mask_kind == FLEXATTN_MASK_SLIDING_WINDOW;
  const long long lo = windowed ? std::max(0ll, i0 - p.window + 1) / kTile : 0;
  const long long hi = ahead ? n_kt : std::min<long long>(i1, p.seq_k - 1) / kTile + 1;
  return lo < hi ? Tiles{(int)lo, (int)hi} : Tiles{0, 0};
}

constexpr int kMostPairs = 8;      // waves of pairs from which the totals decide
constexpr int kMostSms = 256;
constexpr int kMostTiles = 2 * kMostPairs * kMostSms;

// The fullest CTA's time: `cost` of the n query tiles of a slice, largest first, every one `slices` times; in rounds of alternating direction
double dealt_in_rounds(const float* cost, int n, long long slices, int sms) {
  const long long total = n * slices, rest = total % sms, rounds = (total + sms - 1) / sms;
  const long long ctas[] = {0, sms - 1, sms / 2, std::max(rest - 1, 0ll), std::min<long long>(rest, sms - 1), std::max(sms - rest - 1, 0ll),
                            std::min<long long>(sms - rest, sms - 1)};
  double most = 0;
  for (const long long c : ctas) {
    double t = 0;
    for (long long r = 0; r < rounds; ++r) {
      const long long i = r * sms + (r & 1 ? sms - 1 - c : c);
      if (i < total) t += cost[i / slices];
    }
    most = std::max(most, t);
  }
  return most;
}
// ... of a list that the CTAs take one by one: CTAs that are equally far are kept as one entry of a heap
double taken_one_by_one(const float* cost, int n, long long slices, int sms) {
  struct Level {
    double t;
    long long ctas;
  };
  Level heap[kMostSms + 2];
  int size = 1;
  heap[0] = {0.0, sms};
  const auto later = [](const Level& a, const Level& b) { return a.t > b.t; };
  double most = 0;
  for (int k = 0; k < n; ++k) {
    for (long long left = slices; left > 0;) {
      std::pop_heap(heap, heap + size, later);
      Level l = heap[--size];
      while (size > 0 && heap[0].t == l.t) {
        std::pop_heap(heap, heap + size, later);
        l.ctas += heap[--size].ctas;
      }
      const long long now = std::min(left, l.ctas);
      if (l.ctas > now) {
        heap[size++] = {l.t, l.ctas - now};
        std::push_heap(heap, heap + size, later);
      }
      heap[size++] = {l.t + cost[k], now};
      std::push_heap(heap, heap + size, later);
      most = std::max(most, l.t + cost[k]);
      left -= now;
    }
  }
  return most;
}

// Documents: how long a row is only the device knows, and the two-query-tile kernel gains the more the longer the documents are.  The
// lines are by whole and partly filled waves, from 2254 calls (four distributions of document lengths from 30 to 4096, 8 to 128
// slices of 256 to 8192 queries), for the mean of those.  Two-query-tile / persistent, us: 96 x 384 with softcap 27 / 25 (three tiles); 32 x 1280
// 37.7 / 34.8 (2.2 waves of query tiles: the second's few are the shortest); 22 x 2048 (1.2 waves of pairs) of 64 to 1500 44 / 41, of 200 to
// 1000 35 / 38; 24 x 2048 (1.3) of those 45 / 42 and 36 / 40, of 512 to 4096 49 / 58; 24 x 1536 of 200 to 1000 36 / 42.  D = 128 without a
// score function, where a tile gains least: 128 x 777 66 / 62, 96 x 1024 49 / 54.
bool pair_pays_documents(const FlexAttnParams& p, int n_qt, double pairs, double items) {
  const bool plain128 = p.head_dim == 128 && (p.score_kind == FLEXATTN_SCORE_NONE || p.score_kind == FLEXATTN_SCORE_ALIBI);
  if (n_qt <= 3) return std::ceil(pairs) <= (plain128 ? 1.1 : 1.21) * pairs;  // half of the pairs or more end a row: full waves only
  if (pairs <= 0.77 || std::ceil(items) > 1.36 * items) return false;
  if (plain128) return pairs > 1.7 && (n_qt > 8 || n_qt % 2 == 0);
  return n_qt < 10 || pairs <= 1 || pairs >= (n_qt >= 32 ? 1.4 : 1.25);
}

}  // namespace

bool fwd_pair_pays(const FlexAttnParams& p, int sms) {
  const long long n_qt = (p.seq_q + kTile - 1) / kTile, slices = (long long)p.batch * p.heads;
  const int n_kt = (p.seq_k + kTile - 1) / kTile;
  const long long n_pairs = (n_qt + 1) / 2, pairs = n_pairs * slices, items = n_qt * slices;
  if (n_qt < 2 || items <= sms) return false;  // no second stream, or a CTA for every query tile
  if (p.mask_kind == FLEXATTN_MASK_DOCUMENT) return pair_pays_documents(p, (int)n_qt, (double)pairs / sms, (double)items / sms);
  const FwdCosts c = fwd_costs(p);
  const bool totals = pairs > (long long)kMostPairs * sms || sms > kMostSms;
  float tile_cost[kMostTiles], pair_cost[kMostTiles / 2];
  double tile_sum = 0, pair_sum = 0;
  for (long long q = 0; q < n_pairs; ++q) {
    const Tiles a = kv_tiles(p, n_kt, 2 * q), b = 2 * q + 1 < n_qt ? kv_tiles(p, n_kt, 2 * q + 1) : Tiles{0, 0};
    const int both = std::max(0, std::min(a.hi, b.hi) - std::max(a.lo, b.lo)), single = a.count() + b.count() - 2 * both;
    const float t0 = a.count() > 0 ? c.tile * a.count() + c.item : 0.7f * c.item, t1 = b.count() > 0 ? c.tile * b.count() + c.item : 0.7f * c.item;
    const float t = c.both * both + c.single * single + c.pair;
    if (!totals) {
      tile_cost[2 * q] = t0;
      if (2 * q + 1 < n_qt) tile_cost[2 * q + 1] = t1;
      pair_cost[q] = t;
    }
    tile_sum += t0 + (2 * q + 1 < n_qt ? t1 : 0.f);
    pair_sum += t;
  }
  if (totals) return pair_sum < tile_sum;
  std::sort(tile_cost, tile_cost + n_qt, std::greater<float>());
  std::sort(pair_cost, pair_cost + n_pairs, std::greater<float>());
  return taken_one_by_one(pair_cost, (int)n_pairs, slices, sms) < dealt_in_rounds(tile_cost, (int)n_qt, slices, sms);
}

}  // namespace flexattn
