// Host-side rules of the tensor-core launches, run without a GPU: the three runtime calls they make are
// defined here, ahead of the runtime library's.  Prints one line per check that fails.
#include "tc_common.cuh"

#include <chrono>
#include <cstdio>

namespace {
int device = 0, clusters_of[2] = {10, 5}, queries = 0;
bool failing = false;
int failures = 0;
void check(bool ok, const char* what) { if (!ok) { printf("failed: %s\n", what); ++failures; } }
}  // namespace

#ifndef __CUDA_ARCH__      // the device pass has its own
extern "C" {
cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  ++queries;
  if (failing) return cudaErrorUnknown;
  *n = clusters_of[device];
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
}
#endif

using namespace attn;
using namespace attn::tc;

static void some_kernel() {}

static void cluster_queries() {
  TileKernelState state;
  auto slots = [&] { return cluster_slots(&some_kernel, 4, 352, 200000, state); };
  failing = true;
  check(slots() <= 0, "a failed query gives no slots");
  failing = false;
  check(slots() == 40, "a failed query is made again");
  device = 1;
  check(slots() == 20, "the second device has its own number");
  device = 0;
  const int before = queries;
  check(slots() == 40 && queries == before, "a known number is not asked for again");
}

static Geometry geometry(int BH, int N_q, int N_kv, int window, int mask_mode) {
  Geometry g = {};
  g.BH = BH; g.N_q = N_q; g.N_kv = N_kv; g.D = 64; g.ki_base = N_q - N_kv; g.window = window; g.mask_mode = mask_mode;
  return g;
}

static void load_of_a_problem() {
  const Geometry g = geometry(3, 1000, 1700, 600, 0);
  for (int col = 0; col < 2; ++col) {
    const SplitLoad w = stream_load(g, col != 0, 1.f);
    const int n = col ? g.N_kv : g.N_q, tiles = (n + 127) / 128;
    int most = 0, sum = 0;
    for (int t = 0; t < tiles; ++t) {
      int first = 1 << 30, last = -1;      // streamed tiles with a visible pair, one pair at a time
      for (int a = t * 128; a < t * 128 + 128 && a < n; ++a)
        for (int b = 0; b < (col ? g.N_q : g.N_kv); ++b)
          if (col ? visible(g, b, a) : visible(g, a, b)) { first = b / 64 < first ? b / 64 : first; last = b / 64 > last ? b / 64 : last; }
      const int k = last < 0 ? 0 : last - first + 1;
      most = k > most ? k : most;
      sum += k;
    }
    check(w.units == 3.f * tiles && w.longest == most && w.mean == (float)sum / tiles, "load of a small problem, tile by tile");
  }
  // A billion rows cost no more on the host than 131072, and the load is still that of the problem
  const auto start = std::chrono::steady_clock::now();
  const Geometry huge = geometry(1, 1 << 30, 1 << 30, 1 << 30, 0), narrow = geometry(1, 1 << 30, 1 << 30, 256, 0);
  const SplitLoad w = stream_load(huge, false, 1.f), v = stream_load(narrow, true, 1.f);
  check(!two_per_sm_pays(geometry(1, 1 << 12, 1 << 30, 1 << 30, 1), false, true, 850.f, 850.f), "few tiles: one CTA per SM");
  check(std::chrono::steady_clock::now() - start < std::chrono::milliseconds(5), "host time of a long sequence");
  check(w.longest == (float)(1 << 24) && w.mean > 0.99f * (1 << 23) && w.mean < 1.01f * (1 << 23), "load of a long sequence");
  check(v.longest == 6.f && v.mean > 5.9f && v.mean <= 6.f, "load of a long sequence with a window");
}

static void bound_of_a_stream() {
  unsigned seed = 1;
  auto below = [&](int n) { seed = seed * 1664525u + 1013904223u; return (int)((seed >> 8) % (unsigned)n); };
  for (int i = 0; i < 20000; ++i) {
    Geometry g = geometry(1, 1 + below(4000), 1 + below(4000), 1 + below(4200), below(8) == 0);
    const int chunk = below(9);
    if (i == 0) g = geometry(1, 1024, 4000, 1920, 0);       // keys 1057 to 3103 of a tile of queries: 33 tiles
    g.qi_base = (i == 0 ? 8 : chunk) * g.N_q;
    g.ki_base = g.qi_base + g.N_q - g.N_kv;
    const float row = stream_load(g, false, 1.f).longest, col = stream_load(g, true, 1.f).longest;
    check((float)longest_stream(g) >= (row > col ? row : col), "bound of the streamed tiles");
    if (failures > 3) return;
  }
  check(longest_stream(geometry(1, 2048, 2048, 2048, 0)) == 32 && longest_stream(geometry(1, 2048, 2048, 1, 1)) == 32, "whole sequences");
  check(longest_stream(geometry(1, 9000, 9000, 64, 0)) == 4, "a window");
}

// Keys in front of the sequence have no query: their tiles cost next to nothing, so they change no decision.
static void keys_in_front() {
  int paying = 0;
  for (int BH = 4; BH <= 96; BH += 4)
    for (int N = 128; N <= 2304; N += 160) {
      const Geometry plain = geometry(BH, N, N, 8192, 0), front = geometry(BH, N, N + 8192, 8192, 0);
      const TwoPerSm alone = backward_two_per_sm(plain), with = backward_two_per_sm(front);
      check(with.row == alone.row && with.col == alone.col, "keys in front of the sequence, both kinds");
      const bool cols = two_per_sm_pays(plain, true, false, kColClocks, kColClocksTwo);
      check(two_per_sm_pays(front, true, false, kColClocks, kColClocksTwo) == cols, "keys in front of the sequence, the key side");
      paying += (alone.row && alone.col) + cols;
      const SplitLoad w = stream_load(front, true, 1.f), v = stream_load(plain, true, 1.f);
      check(w.busy == v.units && v.busy == v.units && w.busy_mean == v.mean && w.units == v.units + 64.f * BH, "tiles without a stream");
      if (failures > 5) return;
    }
  check(paying > 100 && paying < 600, "either answer occurs");
}

// Where both kinds have a CTA for every SM there is one answer for the two of them.  Without a mask it turns with the
// fourth round of CTAs (444 of them), or with streams of 24 tiles in all; with few long streams the longest is the bound.
static void one_answer_for_both_kinds() {
  int twos = 0, ones = 0;
  for (int BH = 4; BH <= 96; BH += 4)
    for (int N = 200; N <= 4000; N += 119)
      for (int other = 0; other < 4; ++other) {
        const Geometry g = geometry(BH, N, other == 0 ? N : N * (3 + other) / 4 + 128 * other, 4096, other != 3);
        const SplitLoad r = stream_load(g, false, 1.f), c = stream_load(g, true, 1.f);
        const TwoPerSm two = backward_two_per_sm(g);
        if (r.busy >= kSms && c.busy >= kSms) {
          check(two.row == two.col, "one answer for both kinds");
          ++(two.row ? twos : ones);
        }
        check((!two.row || r.busy >= kSms) && (!two.col || c.busy >= kSms), "two CTAs per SM need a CTA for every SM");
        if (failures > 5) return;
      }
  check(twos > 100 && ones > 100, "either answer occurs");
  auto both = [](int BH, int N_q, int N_kv, int mask_mode) { return backward_two_per_sm(geometry(BH, N_q, N_kv, N_kv, mask_mode)).row; };
  check(!both(20, 1354, 1354, 1) && !both(24, 1110, 1110, 1), "without a mask, three rounds");
  check(both(16, 1700, 1700, 1) && both(32, 866, 866, 1) && both(28, 778, 1139, 1), "without a mask, a fourth round");
  check(both(36, 768, 768, 1) && !both(18, 1500, 1400, 1), "without a mask, short streams");
  check(both(32, 1024, 1024, 0) && both(20, 2048, 2048, 0) && !both(12, 2048, 2048, 0) && !both(10, 2000, 2000, 0), "causal");
}

// Forward: equal tiles run in rounds of 148 or of 296, and long streams take longer with two CTAs per SM.
static void forward_in_rounds() {
  auto two = [](int BH, int N_q, int N_kv, int D, int window, int chunk, int mask_mode) {
    Geometry g = geometry(BH, N_q, N_kv, window, mask_mode);
    g.D = D; g.qi_base = chunk * N_q; g.ki_base = g.qi_base + N_q - N_kv;
    return forward_two_per_sm(g);
  };
  check(!two(24, 2048, 8138, 64, 6090, 5, 0) && !two(28, 1825, 7146, 48, 5321, 5, 0) && !two(20, 2048, 6165, 64, 4117, 2, 0), "long windows");
  check(!two(16, 3000, 3000, 64, 3000, 0, 1) && !two(16, 3000, 3000, 96, 3000, 0, 1) && !two(16, 3000, 3000, 128, 3000, 0, 1), "long, no mask");
  check(!two(8, 5888, 5888, 96, 5888, 0, 1) && !two(36, 1487, 6545, 96, 5058, 5, 0), "two to three rounds");
  check(!two(148, 128, 128, 64, 128, 0, 1) && !two(74, 256, 256, 64, 256, 0, 1) && two(76, 256, 256, 64, 256, 0, 1), "one round");
  check(two(64, 2048, 2048, 64, 2048, 0, 1) && two(128, 1692, 1692, 128, 1692, 0, 1), "many rounds");
  check(two(16, 2048, 2048, 128, 2048, 0, 1) && two(20, 2048, 2048, 48, 1024, 8, 0), "two rounds of short streams");
  check(two(96, 2048, 2048, 64, 2048, 0, 0) && two(64, 1024, 1024, 128, 1024, 0, 0) && two(64, 4096, 4096, 128, 4096, 0, 0), "causal");
  check(two(96, 256, 256, 64, 256, 0, 0) && two(80, 176, 176, 128, 176, 0, 0) && two(80, 174, 363, 96, 189, 5, 0), "causal, short");
  check(two(96, 12000, 12000, 64, 12000, 0, 0) && two(48, 9345, 9345, 64, 9345, 0, 0) && two(32, 16384, 16384, 128, 16384, 0, 0), "causal, many rounds");
  check(!two(16, 12488, 12488, 80, 12488, 0, 0) && !two(24, 1860, 1860, 80, 1860, 0, 0) && !two(24, 1500, 1500, 64, 1500, 0, 0), "causal, one per SM");
}

int main() {
  forward_in_rounds();
  keys_in_front();
  one_answer_for_both_kinds();
  cluster_queries();
  load_of_a_problem();
  bound_of_a_stream();
  return failures;
}
