// Launch rule of the fp32 kernels: how many CTAs (a cluster) share the streamed tiles of a stationary tile.
// Host code, no runtime calls: what fits the GPU is passed in.
#pragma once
#include "attn_common.cuh"

namespace attn {
namespace simt {

constexpr int TS = 32;                       // stationary rows per CTA
constexpr int TT = 64;                       // streamed rows per iteration
constexpr int kMaxSplit = 8;                 // CTAs per cluster (the portable maximum)
constexpr int kListed = 2 * kSms;            // stationary tiles of a head that the rule looks at, evenly spaced

enum Kind { K_FWD = 0, K_BWD_ROW, K_BWD_COL, K_HVP_PRE, K_HVP_ROW, K_HVP_COL };

// A kernel as the rule sees it.  Times are in units of a streamed tile of the kernel itself; `weight` is that
// unit beside the query side's.  A CTA costs `cta` besides its tiles, `cta_shared` as part of a cluster (two
// barriers, the sum).
struct Work {
  float ctas;                  // stationary tiles of all heads: the CTAs without a split
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
inline Work work_of(const Geometry& g, Kind kind, bool narrow) {
  const bool col = kind == K_BWD_COL || kind == K_HVP_COL, one = kind == K_FWD || kind == K_BWD_ROW;
  Work w;
  const int n = col ? g.N_kv : g.N_q, tiles = (int)(((long long)n + TS - 1) / TS);
  w.ctas = (float)tiles * g.BH;
  w.n = tiles < kListed ? tiles : kListed;
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

// A kernel whose tiles are shared by `c`, of which `slots` CTAs run at a time, each with `slow` per tile.
struct Part {
  const Work& w;
  int c;
  float slots, slow, cta, per;      // per: CTAs of a listed tile
  float load;                       // of all CTAs, over the slots
  Part(const Work& work, int split, int slots_, float slow_) : w(work), c(split), slots((float)slots_), slow(slow_) {
    cta = c > 1 ? w.cta_shared : w.cta;
    per = w.n > 0 ? w.ctas * c / w.n : 0.f;
    load = per * w.weight * (w.shares[c == 1 ? 0 : c == 2 ? 1 : c == 4 ? 2 : 3] * slow + w.n * cta) / slots;
  }
  float fill() const { return w.ctas * c / slots; }
  float time(int streamed) const { return w.weight * ((streamed + c - 1) / c * slow + cta); }
  // the fewest tiles of the CTAs in front of position `at` of the grid, and of the one there
  int least(float at) const { const int i = (int)(at / per); return w.least[i < w.n ? i : w.n - 1]; }
  // Lower bound of the time by itself: the longest CTA, the whole load, and j + 1 CTAs one behind the other on
  // some slot where there are more than j times the slots.
  float alone() const {
    float t = time(w.longest);
    if (load > t) t = load;
    for (int j = 1; j <= 8 && j * slots < w.ctas * c; ++j) {
      const float v = (j + 1) * time(least(j * slots));
      if (v > t) t = v;
    }
    return t;
  }
};

// The splits of one kernel, or of two that share the GPU, the CTAs of `a` in front.  slots_a(c) and slots_b(c): the CTAs
// that run at a time in clusters of c (not more than zero: that form is not there).  `shared`: what a tile takes where two
// CTAs share an SM (1: they never do).
// Bounds of the time decide: every kernel by itself (Part), the load of both, the longest CTA of `b` behind the load
// of `a` where that fills the GPU, else the first CTA of `b` that finds no slot behind the shortest one.  All the
// clusters of a launch need not run at a time, but how many do has to be known: clusters of four and eight leave SMs
// of a GPC unused (132 and 120 CTAs run, not 148), and a split that does not fit pays for its second wave.
// Measured against a rule that divides the load by the number of SMs: 4 heads N576 D64 forward 29.8 -> 21 us (8 -> 4 CTAs
// per tile), 7 heads N576 D64 backward 98.9 -> 61 (1 -> 2), 10 heads N383 D64 double backward 168 -> 127 (1 -> 2), 2 heads
// N320 D80 forward 19.7 -> 14.1 (8 -> 4).  Over 396 sizes the rule's choice takes 0.3 to 1.5 % more time than the best
// one of each (the other rule 3 to 11 %), at worst a fifth, at tiles most of which have no work.
struct Splits { int a, b; };
template <typename SlotsA, typename SlotsB>
inline Splits pick_splits(const Work& a, const Work* b, float shared, SlotsA slots_a, SlotsB slots_b) {
  Splits best = {1, 1};
  float least = 0.f;
  Work none;
  none.ctas = none.weight = none.cta = none.cta_shared = 0.f;
  none.n = none.longest = none.shares[0] = 0;
  const Work& other = b != nullptr ? *b : none;
  // no split of more CTAs than two per SM
  auto most = [](const Work& w) { return w.ctas > 2 * kSms ? 1 : kMaxSplit; };
  for (int sum = 2; sum <= 2 * kMaxSplit; ++sum)            // few CTAs first; more have to gain 3 %
    for (int ca = 1; ca <= most(a) && ca < sum; ca *= 2) {
      const int cb = sum - ca;
      if (cb > most(other) || (cb & (cb - 1)) != 0) continue;
      if ((ca > 1 && ca >= 2 * a.longest) || (cb > 1 && cb >= 2 * other.longest)) continue;
      const int sa = slots_a(ca), sb = b != nullptr ? slots_b(cb) : 1;
      if (sa <= 0 || sb <= 0) continue;
      const float slow = a.ctas * ca + other.ctas * cb > kSms ? shared : 1.f;
      const Part x(a, ca, sa, slow), y(other, cb, sb, slow);
      float t = x.alone();
      if (b != nullptr && other.n > 0 && a.n > 0) {
        const float bounds[3] = {y.alone(), x.load + y.load, x.fill() >= 1.f ? x.load + y.time(other.longest) : 0.f};
        for (float v : bounds) if (v > t) t = v;
        if (x.fill() < 1.f && x.fill() + y.fill() > 1.f) {
          const int waits = y.least((1.f - x.fill()) * y.slots);
          const float first = x.time(a.least[a.n - 1]), same = y.time(waits);
          const float v = same + (first < same ? first : same);
          if (v > t) t = v;
        }
      } else if (b != nullptr && other.n > 0) {
        t = y.alone();
      }
      if (sum == 2 || t < 0.97f * least) { best = {ca, cb}; least = t; }
    }
  return best;
}

// Both kernels in one grid, where they have the same split (`ctas` of both without it), or the second behind the first
// without waiting for it.  At D > 64, one CTA per SM, one grid takes 1 to 3 % less time in the backward at any size, and in the
// double backward up to one CTA per SM (above, 1 % less to 0.6 % more on average).  At D <= 64 a grid that wants more than an SM per
// CTA puts the second kind's long CTAs beside the first's: backward 1.2 times the time at 148 to 296 CTAs (10 heads
// N320 52 against 40 us) and up to 1.1 from 120 CTAs in clusters of four, but 2 to 4 % less where every CTA has an SM;
// double backward the same without clusters, in clusters 1 to 5 % less up to two per SM.
inline bool one_grid(const Splits& s, bool narrow, bool second_order, float ctas) {
  if (s.a != s.b) return false;
  if (!narrow) return true;
  if (second_order && s.a > 1) return ctas * s.a <= 2 * kSms;
  return s.a <= 2 && ctas * s.a <= kSms;
}

}  // namespace simt
}  // namespace attn
