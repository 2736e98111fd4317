// Which of the two forward kernels that work through a list of query tiles serves a call: the persistent one (fwd_pipe_sm100.cu), whose
// CTAs are dealt single query tiles in rounds, or the two-query-tile one (fwd_pair_sm100.cu), whose CTAs take pairs as they get on.  Host only.
//
// A pair takes 0.8 to 0.95 of its two tiles' time, but it is a unit twice as long, fewer of them than CTAs leave SMs idle, and a last tile
// without a partner costs almost as much.  So the rule deals both lists out in their order (sched.cuh: batch rows, groups of heads, heaviest
// first) as the kernels do and compares the fullest CTAs.  The costs below are fitted (least squares of the logarithms, in us) to 2674 calls
// timed with either kernel on 148 SMs, graph replays: causal, windows, open windows, no mask, S2; 4 to 384 slices of 129 to 8192 queries, equal
// and unequal lengths.  Over these and 734 calls drawn at random, batches of up to 16 rows among them, the kernel it picks is 0.12 % slower than the
// faster one in the mean and 1.2 % of the calls lose more than 3 % (lines drawn by waves of pairs: 1.8 %, 16 %; one sorted list of all slices: 0.5 %, 4 %).
// Times in us, two-query-tile / persistent: 192 x 384 causal softcap 26.0 / 23.4 (three tiles: every other pair is half empty), 8 x 4096 against
// 512 keys with a window of 256 15.1 / 10.6 (empty query tiles), 32 x 2048 causal, D = 64, 36 / 42; 3 rows of 24 x 1088 causal softcap 52 / 74 (the heaviest
// tiles of a row come after the lightest of the one before, which rounds do not even out).
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

// The kv tiles [lo, hi) a query tile sees, from the mask kind and the sizes (dense S2: all below the diagonal)
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

// A list: per batch row and group of heads, `cost` of the n units of a slice, heaviest first, each `width` times.  The groups are those of
// sched.cuh: as many heads as keep their K and V within 48 MB of L2, for pairs evened out.
struct List {
  const float* cost;
  int n;
  long long batch;
  int heads, group;
};
int heads_a_group(const FlexAttnParams& p, bool even) {
  const long long slice_bytes = 4ll * p.seq_k * p.head_dim;
  const int most = (int)std::max(1ll, std::min<long long>(p.heads, (48ll << 20) / slice_bytes));
  if (!even) return most;
  const int groups = (p.heads + most - 1) / most;
  return (p.heads + groups - 1) / groups;
}
template <class Unit>
void for_each_run(const List& l, Unit unit) {
  for (long long b = 0; b < l.batch; ++b)
    for (int h = 0; h < l.heads; h += l.group)
      for (int k = 0; k < l.n; ++k) unit(l.cost[k], std::min(l.group, l.heads - h));
}

constexpr int kMostSms = 256;
constexpr int kExactPairs = 4, kExactItems = 16;  // waves up to which a list is dealt out (1.4 us of host time in the median of those calls, 8 in the 99th percentile)
constexpr int kMostTiles = 2 * kExactItems * kMostSms;

// The fullest CTA's time where the list is dealt out in rounds of alternating direction
double dealt_in_rounds(const List& l, int sms) {
  float time[kMostSms] = {};
  int at = 0, step = 1;
  for_each_run(l, [&](float cost, int count) {
    for (int k = 0; k < count; ++k) {
      time[at] += cost;
      at += step;
      if (at < 0 || at == sms) {
        step = -step;
        at += step;
      }
    }
  });
  return *std::max_element(time, time + sms);
}
// ... where the CTAs take its units one by one: those that are equally far are one entry of a heap
double taken_one_by_one(const List& l, int sms) {
  struct Level {
    float t;
    int ctas;
  };
  Level heap[kMostSms + 2];
  int size = 1;
  heap[0] = {0.f, sms};
  const auto later = [](const Level& a, const Level& b) { return a.t > b.t; };
  float most = 0.f;
  for_each_run(l, [&](float cost, int left) {
    while (left > 0) {
      std::pop_heap(heap, heap + size, later);
      Level v = heap[--size];
      while (size > 0 && heap[0].t <= v.t + 1e-4f) {
        std::pop_heap(heap, heap + size, later);
        v.ctas += heap[--size].ctas;
      }
      const int now = std::min(left, v.ctas);
      if (v.ctas > now) {
        heap[size++] = {v.t, v.ctas - now};
        std::push_heap(heap, heap + size, later);
      }
      heap[size++] = {v.t + cost, now};
      std::push_heap(heap, heap + size, later);
      most = std::max(most, v.t + cost);
      left -= now;
    }
  });
  return most;
}

// Documents: how long a row is only the device knows, and the two-query-tile kernel gains the more the longer the documents are and the more
// batch rows there are, whose lists come one after the other.  The lines are by whole and partly filled waves, from 2254 calls of two rows
// (four distributions of document lengths from 30 to 4096, 8 to 128 slices of 256 to 8192 queries) and 700 drawn at random, for the mean of
// those.  Two-query-tile / persistent, us: 96 x 384 with softcap 27 / 25 (three tiles); 32 x 1280 37.7 / 34.8 (2.2 waves of query tiles: the second's
// few are the shortest); less than a wave, one row of 24 x 1472, D = 128, softcap, 55 / 43, of 16 x 2240 57 / 46, but two of 12 x 1536 36 / 42; 1.2 waves, two of
// 11 x 2048 44 / 41 with documents of 64 to 1500, 35 / 38 of 200 to 1000, seven of 2 x 2985 40 / 45; two of 12 x 2048 (1.3) 45 / 42 and 36 / 40, of 512 to
// 4096 49 / 58.  D = 128 without a score function, where a tile gains least: 128 x 777 66 / 62, 96 x 1024 49 / 54.
bool pair_pays_documents(const FlexAttnParams& p, int n_qt, double pairs, double items) {
  const bool plain128 = p.head_dim == 128 && (p.score_kind == FLEXATTN_SCORE_NONE || p.score_kind == FLEXATTN_SCORE_ALIBI);
  if (n_qt <= 3)  // half of the pairs or more end a row: full waves only
    return (pairs > 1 || p.batch > 1) && std::ceil(pairs) <= (plain128 ? 1.1 : 1.21) * pairs;
  const bool few_in_the_last = std::ceil(items) > 1.36 * items;
  if (plain128) return pairs > 1.7 && (n_qt > 8 || n_qt % 2 == 0) && !few_in_the_last;
  if (pairs <= 1) return (p.batch == 2 || p.batch == 3) && n_qt <= 24 && pairs > 0.85 && !few_in_the_last;
  if (few_in_the_last && p.batch < 4) return false;
  return pairs >= 1.25 || (pairs >= 1.1 && (p.batch >= 4 || (p.batch > 1 && n_qt < 10)));
}

}  // namespace

bool fwd_pair_pays(const FlexAttnParams& p, int sms) {
  const long long n_qt = (p.seq_q + kTile - 1) / kTile, slices = (long long)p.batch * p.heads;
  const int n_kt = (p.seq_k + kTile - 1) / kTile;
  const long long n_pairs = (n_qt + 1) / 2, pairs = n_pairs * slices, items = n_qt * slices;
  if (n_qt < 2 || items <= sms) return false;  // no second stream, or a CTA for every query tile
  if (p.mask_kind == FLEXATTN_MASK_DOCUMENT) return pair_pays_documents(p, (int)n_qt, (double)pairs / sms, (double)items / sms);
  const FwdCosts c = fwd_costs(p);
  const bool exact_pairs = pairs <= (long long)kExactPairs * sms && sms <= kMostSms, exact_items = items <= (long long)kExactItems * sms && sms <= kMostSms;
  float tile_cost[kMostTiles], pair_cost[kMostTiles / 2];
  double tile_sum = 0, pair_sum = 0;
  float pair_least = 1e30f, pair_most = 0.f;
  for (long long q = 0; q < n_pairs; ++q) {
    const bool two = 2 * q + 1 < n_qt;
    const Tiles a = kv_tiles(p, n_kt, 2 * q), b = two ? kv_tiles(p, n_kt, 2 * q + 1) : Tiles{0, 0};
    const int both = std::max(0, std::min(a.hi, b.hi) - std::max(a.lo, b.lo)), single = a.count() + b.count() - 2 * both;
    const float t0 = a.count() > 0 ? c.tile * a.count() + c.item : 0.7f * c.item, t1 = b.count() > 0 ? c.tile * b.count() + c.item : 0.7f * c.item;
    const float t = c.both * both + c.single * single + c.pair;
    if (exact_items) {
      tile_cost[2 * q] = t0;
      if (two) tile_cost[2 * q + 1] = t1;
    }
    if (exact_pairs) pair_cost[q] = t;
    tile_sum += t0 + (two ? t1 : 0.f);
    pair_sum += t;
    pair_least = std::min(pair_least, t);
    pair_most = std::max(pair_most, t);
  }
  double by_tiles = 1.07 * tile_sum * slices / sms, by_pairs;  // (dealt in rounds, long lists come out 4 to 10 % uneven)
  if (exact_items) {
    std::sort(tile_cost, tile_cost + n_qt, std::greater<float>());
    by_tiles = dealt_in_rounds({tile_cost, (int)n_qt, p.batch, p.heads, heads_a_group(p, false)}, sms);
  }
  if (exact_pairs) {
    std::sort(pair_cost, pair_cost + n_pairs, std::greater<float>());
    by_pairs = taken_one_by_one({pair_cost, (int)n_pairs, p.batch, p.heads, heads_a_group(p, true)}, sms);
  } else if (pair_most - pair_least < 1e-4f) {
    by_pairs = (double)((pairs + sms - 1) / sms) * pair_most;  // whole waves
  } else {
    by_pairs = pair_sum * slices / sms + 0.5 * pair_least;  // a long list ends within its last, lightest pairs
  }
  return by_pairs < by_tiles;
}

}  // namespace flexattn
