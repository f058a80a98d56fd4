// Launch rule of the fp32 kernels: how many CTAs (a cluster) share the streamed tiles of a stationary tile.
// Host code, no runtime calls: what fits the GPU is passed in.
#pragma once
#include "attn_common.cuh"

namespace attn {
namespace simt {

constexpr int TS = 32;                       // stationary rows per CTA
constexpr int TT = 64;                       // streamed rows per iteration
constexpr int kMaxSplit = 8;                 // CTAs per cluster (the portable maximum)
constexpr int kListed = 64;                  // stationary tiles of a head that the rule looks at, evenly spaced above: 1 us of the host

enum Kind { K_FWD = 0, K_BWD_ROW, K_BWD_COL, K_HVP_PRE, K_HVP_ROW, K_HVP_COL };

// A kernel as the rule sees it.  Times are in units of a streamed tile of the kernel itself; `weight` is that
// unit beside the query side's.  A CTA costs `cta` besides its tiles, `cta_shared` as part of a cluster (two
// barriers, the sum).
struct Work {
  float ctas, per_listed;      // stationary tiles of all heads: the CTAs without a split; how many a listed one stands for
  int n, longest;              // listed tiles, the most streamed tiles of any
  short streamed[kListed];     // streamed tiles of a stationary tile, in the grid's order
  short least[kListed];        // the fewest so far in that order
  int shares[4];               // of all listed tiles: the sum of ceil(streamed / c), c = 1, 2, 4, 8
  float weight, cta, cta_shared;
};

// The costs are fitted, together with the 1.35 of shared_tile, to the times of each kind under every split at 397 sizes
// (1 to 32 heads, 16 to 2000 rows, all masks, D = 32 to 128).  A kind with one output product has cheaper tiles, beside
// which the rest of its CTAs weighs more; the key side's tiles cost more than the query side's.
inline float shared_tile(bool narrow) { return narrow ? 1.35f : 1.f; }
constexpr float kLaunch = 0.3f, kLaunchHvp = 0.2f;      // 2 us of the host beside a tile of the backward, of the double backward
inline Work work_of(const Geometry& g, Kind kind, bool narrow) {
  const bool col = kind == K_BWD_COL || kind == K_HVP_COL, one = kind == K_FWD || kind == K_BWD_ROW;
  Work w;
  const int n = col ? g.N_kv : g.N_q, tiles = (int)(((long long)n + TS - 1) / TS);
  w.ctas = (float)tiles * g.BH;
  w.n = tiles < kListed ? tiles : kListed;
  w.per_listed = w.ctas / w.n;
  w.longest = 0;
  for (int& s : w.shares) s = 0;
  w.weight = kind == K_BWD_COL ? 1.4f : kind == K_HVP_COL ? 1.25f : 1.f;
  w.cta = narrow ? (one ? 0.9f : 0.6f) : one ? 0.45f : 0.24f;
  w.cta_shared = narrow ? (one ? 1.1f : 0.5f) : one ? 0.8f : 0.35f;
  for (int s = 0; s < w.n; ++s) {
    const int at = w.n == tiles ? s : (int)((long long)s * (tiles - 1) / (w.n - 1));
    const int i = col || g.mask_mode != 0 ? at : tiles - 1 - at;
    int lo, hi;
    const int end = n - i * TS < TS ? n : (i + 1) * TS;
    if (col) query_range_for_keys(g, i * TS, end, lo, hi);
    else key_range_for_queries(g, i * TS, end, lo, hi);
    const int k = hi > lo ? (int)(((long long)hi + TT - 1) / TT) - lo / TT : 0;
    w.streamed[s] = (short)(k < 32000 ? k : 32000);
    w.least[s] = s == 0 || w.streamed[s] < w.least[s - 1] ? w.streamed[s] : w.least[s - 1];
    if (w.streamed[s] > w.longest) w.longest = w.streamed[s];
    for (int e = 0; e < 4; ++e) w.shares[e] += (w.streamed[s] + (1 << e) - 1) >> e;
  }
  return w;
}

struct Splits { int a, b; bool together; };      // CTAs per tile of either kernel; one grid for both

// Both kernels in one grid, where they have the same split (`ctas` of both without it, `share` tiles at most of a CTA), or the
// second behind the first without waiting for it.  At D > 64, one CTA per SM, one grid takes 1 to 3 % less time in the backward
// at any size, and in the double backward up to one CTA per SM (above, 1 % less to 0.6 % more on average).  At D <= 64:
// where every CTA has an SM to itself, 2 to 4 % less.  A grid that wants more, up to two CTAs per SM, puts the CTAs of
// both kinds two to an SM before all SMs have one: backward 1.25, 1.11 and 1.08 times the time on average without
// clusters, in pairs and in fours (7 heads N200 26.6 against 18.9 us), double backward 0.98 to 1.0 in clusters.
// There a backward of CTAs of one or two tiles, 10 to 30 us, is shorter than the 50 us that the host takes for the call of
// autograd that asks for it, so the launch (1.9 us) counts; longer ones get two.
inline bool one_grid(int split_a, int split_b, bool narrow, bool second_order, float ctas, int share) {
  if (split_a != split_b) return false;
  if (!narrow || (split_a <= 2 && ctas * split_a <= kSms)) return true;
  return ctas * split_a <= 2 * kSms && (second_order ? split_a > 1 : share <= 2);
}

// A kernel whose tiles are shared by `c`, of which `slots` CTAs run at a time, each with `slow` per tile.
struct Part {
  float time, load, alone, fill;      // of the longest CTA; of all over the slots; a bound of its time by itself; CTAs over slots
  const Work* w;
  float slots, slow, cta, listed;     // listed tiles per CTA
  int log_c;
  float cta_time(int streamed) const { return w->weight * (((streamed + (1 << log_c) - 1) >> log_c) * slow + cta); }
  // the fewest tiles of the CTAs in front of position `at` of the grid, and of the one there
  int least(float at) const { const int i = (int)(at * listed); return w->least[i < w->n ? i : w->n - 1]; }
  // alone: the longest CTA, the whole load, and j + 1 CTAs one behind the other on some slot where there are more
  // than j times the slots
  void set(const Work& work, int log_split, int slots_, float slow_) {
    w = &work; log_c = log_split; slots = (float)slots_; slow = slow_;
    cta = log_c > 0 ? w->cta_shared : w->cta;
    const float ctas = w->ctas * (1 << log_c);
    listed = w->n / ctas;
    fill = ctas / slots;
    load = w->weight * (w->shares[log_c] * slow * w->per_listed + w->ctas * cta) * (1 << log_c) / slots;
    time = cta_time(w->longest);
    alone = load > time ? load : time;
    for (int j = 1; j <= 8 && j < fill; ++j) {
      const float v = (j + 1) * cta_time(least(j * slots));
      if (v > alone) alone = v;
    }
  }
};

// The splits of one kernel, or of two that share the GPU, the CTAs of `a` in front.  slots(c): the CTAs of either that run
// at a time in clusters of c (not more than zero: that form is not there).
// Bounds of the time decide: every kernel by itself (Part), the load of both, the longest CTA of `b` behind the load
// of `a` where that fills the GPU, else the first CTA of `b` that finds no slot behind the shortest one, and the host's
// time for a second launch.  All the
// clusters of a launch need not run at a time, but how many do has to be known: clusters of four and eight leave SMs
// of a GPC unused (132 and 120 CTAs run, not 148), and a split that does not fit pays for its second wave.
// Measured against a rule that divides the load by the number of SMs: 4 heads N576 D64 forward 29.8 -> 21 us (8 -> 4 CTAs
// per tile), 7 heads N576 D64 backward 98.9 -> 61 (1 -> 2), 10 heads N383 D64 double backward 168 -> 127 (1 -> 2), 2 heads
// N320 D80 forward 19.7 -> 14.1 (8 -> 4).  Over 396 sizes the rule's choice takes 0.3 to 1.5 % more time than the best
// one of each (the other rule 3 to 11 %), at worst a fifth, at tiles most of which have no work.
template <typename Slots>
inline Splits pick_splits(const Work& a, const Work* b, bool narrow, bool second_order, const Slots& slots) {
  // no split where there are more CTAs than two per SM, or shares without a tile would be the rule
  auto most = [](const Work& w) {
    int e = 0;
    while (e < 3 && w.ctas <= 2 * kSms && (2 << e) < 2 * w.longest) ++e;
    return e;
  };
  const int most_a = most(a), most_b = b != nullptr ? most(*b) : 0;
  int fits[4];
  for (int e = 0; e < 4; ++e) fits[e] = e <= most_a || e <= most_b ? slots(1 << e) : 0;
  Part parts[2][2][4];
  bool done[2][2][4] = {};
  auto part = [&](int which, int crowded, int e) -> const Part& {
    if (!done[which][crowded][e]) parts[which][crowded][e].set(which == 0 ? a : *b, e, fits[e], crowded != 0 ? shared_tile(narrow) : 1.f);
    done[which][crowded][e] = true;
    return parts[which][crowded][e];
  };
  // few CTAs first; more have to gain 3 %
  static const signed char kOrder[16][2] = {{0, 0}, {0, 1}, {1, 0}, {1, 1}, {0, 2}, {2, 0}, {1, 2}, {2, 1}, {2, 2}, {0, 3}, {3, 0}, {1, 3}, {3, 1}, {2, 3}, {3, 2}, {3, 3}};
  Splits best = {1, 1, false};
  float least = 0.f;
  for (const auto& o : kOrder) {
    const int ea = o[0], eb = o[1];
    if (ea > most_a || eb > most_b || fits[ea] <= 0 || fits[eb] <= 0) continue;
    Splits s = {1 << ea, 1 << eb, false};
    const int crowded = a.ctas * s.a + (b != nullptr ? b->ctas * s.b : 0.f) > kSms;
    const Part& x = part(0, crowded, ea);
    float t = x.alone;
    if (b != nullptr) {
      const Part& y = part(1, crowded, eb);
      const float bounds[3] = {y.alone, x.load + y.load, x.fill >= 1.f ? x.load + y.time : 0.f};
      for (float v : bounds) if (v > t) t = v;
      if (x.fill < 1.f && x.fill + y.fill > 1.f) {
        const float first = x.cta_time(a.least[a.n - 1]), same = y.cta_time(y.least((1.f - x.fill) * y.slots));
        const float v = same + (first < same ? first : same);
        if (v > t) t = v;
      }
      const int longest = a.longest > b->longest ? a.longest : b->longest;
      s.together = one_grid(s.a, s.b, narrow, second_order, a.ctas + b->ctas, (longest + s.a - 1) >> ea);
      if (!s.together) t += second_order ? kLaunchHvp : kLaunch;
    }
    if (least == 0.f || t < 0.97f * least) { best = s; least = t; }
  }
  return best;
}

}  // namespace simt
}  // namespace attn
