// The launch rule of the fp32 kernels, run without a GPU.  Prints one line per check that fails.
#include "simt_split.h"

#include <chrono>
#include <cstdio>

using namespace attn;
using namespace attn::simt;

namespace {
int failures = 0;
void check(bool ok, const char* what) { if (!ok) { printf("failed: %s\n", what); ++failures; } }

Geometry geometry(int BH, int N_q, int N_kv, int D, int window, int chunk, int mask_mode) {
  Geometry g = {};
  g.BH = BH; g.N_q = N_q; g.N_kv = N_kv; g.D = D; g.window = window; g.mask_mode = mask_mode;
  g.qi_base = chunk * N_q; g.ki_base = g.qi_base + N_q - N_kv;
  return g;
}

// CTAs of a B200 that run at a time in clusters of c, one CTA per SM and two
int slots(bool two, int c) { return c <= 2 ? (two ? 296 : 148) : c == 4 ? (two ? 284 : 132) : two ? 264 : 120; }

enum Op { FWD, BWD, HVP };
Splits rule(Op op, const Geometry& g) {
  const bool narrow = g.D <= 64;
  auto s = [&](int c) { return slots(narrow, c); };
  if (op == FWD) return pick_splits(work_of(g, K_FWD, narrow), nullptr, narrow, false, s);
  const Work a = work_of(g, op == BWD ? K_BWD_COL : K_HVP_COL, narrow), b = work_of(g, op == BWD ? K_BWD_ROW : K_HVP_ROW, narrow);
  return pick_splits(a, &b, narrow, op == HVP, s);
}

// Sizes at which a split that a model without the second wave of clusters, or without the kernel beside, takes is
// 1.2 to 1.6 times as slow as the best on a B200; `a` and `b` are those within 6 % of it.
struct Measured { Op op; int BH, N_q, N_kv, D, window, chunk, mask_mode, a, b; };
const Measured kMeasured[] = {
    {FWD, 4, 320, 320, 64, 320, 0, 0, 4, 1},    {FWD, 4, 576, 576, 64, 576, 0, 0, 4, 1},    {FWD, 5, 562, 1056, 32, 64, 1, 0, 1, 1},
    {FWD, 2, 320, 320, 80, 320, 0, 0, 4, 1},    {FWD, 2, 320, 320, 128, 320, 0, 0, 4, 1},   {FWD, 1, 1024, 1024, 128, 1024, 0, 0, 4, 1},
    {FWD, 29, 75, 75, 80, 24, 3, 0, 1, 1},      {FWD, 19, 108, 262, 128, 262, 0, 1, 1, 1},
    {BWD, 4, 576, 576, 64, 576, 0, 0, 4, 4},    {BWD, 7, 576, 576, 64, 576, 0, 0, 2, 2},    {BWD, 4, 479, 479, 64, 479, 0, 0, 4, 4},
    {BWD, 4, 320, 183, 64, 183, 3, 1, 4, 1},    {BWD, 2, 320, 320, 64, 320, 0, 0, 8, 4},    {BWD, 1, 320, 320, 80, 320, 0, 0, 8, 4},
    {BWD, 10, 128, 128, 128, 128, 0, 0, 2, 1},  {BWD, 1, 196, 1526, 128, 64, 0, 0, 4, 4},
    {HVP, 7, 576, 576, 64, 576, 0, 0, 2, 2},    {HVP, 10, 383, 383, 64, 383, 0, 0, 2, 2},   {HVP, 4, 320, 320, 64, 320, 0, 0, 4, 4},
    {HVP, 4, 576, 576, 64, 576, 0, 0, 4, 4},    {HVP, 2, 562, 165, 96, 165, 1, 0, 4, 4},    {HVP, 4, 869, 428, 112, 428, 3, 0, 2, 2},
};

void measured_sizes() {
  for (const Measured& m : kMeasured) {
    const Splits s = rule(m.op, geometry(m.BH, m.N_q, m.N_kv, m.D, m.window, m.chunk, m.mask_mode));
    char what[128];
    snprintf(what, sizeof(what), "op %d BH%d %d x %d D%d: %d and %d CTAs per tile, not %d and %d", m.op, m.BH, m.N_q, m.N_kv, m.D, m.a, m.b, s.a, s.b);
    check(s.a == m.a && s.b == m.b, what);
  }
}

void limits() {
  for (int D : {64, 128})
    for (Op op : {FWD, BWD, HVP}) {
      check(rule(op, geometry(1, 32, 64, D, 64, 0, 1)).a == 1, "one streamed tile is not shared");
      check(rule(op, geometry(64, 1024, 1024, D, 1024, 0, 0)).a == 1, "more CTAs than two per SM are not split");
      check(rule(op, geometry(1, 100, 100, D, 100, 0, 0)).a <= 4, "no more CTAs than half-empty shares");
      const Splits nothing = rule(op, geometry(2, 64, 64, D, 0, 0, 0));
      check(nothing.a == 1 && nothing.b == 1, "tiles without work are not shared");
      // a cluster size the device cannot run is not taken
      const Geometry g = geometry(1, 576, 576, D, 576, 0, 0);
      const Work a = work_of(g, K_HVP_COL, D == 64), b = work_of(g, K_HVP_ROW, D == 64);
      auto pairs = [&](int c) { return c <= 2 ? slots(D == 64, c) : c == 4 ? 0 : -1; };
      const Splits s = pick_splits(a, &b, D == 64, true, pairs);
      check(s.a == 2 && s.b == 2, "clusters of two where larger ones do not run");
    }
}

// Pairs of kernels in one grid and in two
void grids() {
  auto together = [](Op op, const Geometry& g) { return rule(op, g).together; };
  check(together(BWD, geometry(4, 128, 128, 64, 128, 0, 0)) && together(HVP, geometry(4, 100, 100, 48, 100, 0, 0)), "an SM for every CTA: one grid");
  check(!together(BWD, geometry(10, 320, 320, 64, 320, 0, 0)), "backward, 10 heads N320 D64: 52 us in one grid, 35 in two");
  check(!together(BWD, geometry(2, 383, 383, 64, 383, 0, 0)), "backward, 2 heads N383 D64: 24.7 us in one grid, 18.9 in two");
  check(together(BWD, geometry(8, 256, 256, 64, 256, 0, 0)), "CTAs of two tiles: the launch counts");
  check(!one_grid(1, 1, true, true, 160, 2) && one_grid(2, 2, true, true, 98, 2) && !one_grid(2, 2, true, true, 149, 2), "double backward: in clusters, up to two CTAs per SM");
  check(together(BWD, geometry(16, 320, 320, 128, 320, 0, 0)) && one_grid(8, 8, false, true, 40, 4), "D > 64: one grid");
  check(!one_grid(2, 1, false, false, 20, 4) && !one_grid(2, 1, true, true, 20, 1), "different splits: two launches");
  check(!rule(FWD, geometry(1, 64, 64, 64, 64, 0, 0)).together, "one kernel");
}

void long_sequences() {
  const int n = 0x7fffffff;
  const auto start = std::chrono::steady_clock::now();
  for (int window : {n >> 1, 100}) {
    const Geometry g = geometry(1, n >> 1, n >> 1, 64, window, 0, 0);
    check(rule(FWD, g).a == 1 && rule(BWD, g).a == 1, "a long sequence is not split");
  }
  check(rule(FWD, geometry(1, 64, n >> 1, 64, n >> 1, 0, 1)).a == 8, "two tiles of queries against many keys");
  check(std::chrono::steady_clock::now() - start < std::chrono::milliseconds(5), "host time of a long sequence");
}
}  // namespace

int main() {
  measured_sizes();
  limits();
  grids();
  long_sequences();
  return failures;
}
