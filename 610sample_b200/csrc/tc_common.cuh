// Definitions shared by the tensor-core kernel files: tile sizes, warp roles,
// tensor-map bundle and small device helpers.
#pragma once

#include "attn_common.cuh"
#include "tc_primitives.cuh"

#include <atomic>
#include <cooperative_groups.h>

namespace attn {
namespace tc {

constexpr int BM = 128;            // stationary rows per CTA
constexpr int BN = 64;             // streamed rows per iteration
constexpr int kMathWarps = 8;
constexpr int kMathThreads = kMathWarps * 32;
constexpr int kProducerWarp = 8;   // the MMA-issuing warps follow it
constexpr int kTmemCols = 512;
constexpr uint32_t kHalfSmem = 233472 / 2 - 1024;   // dynamic shared memory of a CTA that shares its SM with another
constexpr uint32_t kAtomBytesStat = BM * 128;   // [128 rows][64 halves], 16 KB
constexpr uint32_t kAtomBytesStrm = BN * 128;   // [ 64 rows][64 halves],  8 KB

// Kernel ids inside device status codes (the backward kernels use 18 and 19, the forward kernel
// 20, the self-test 0x6f); the values are documented with the C ABI and do not change.
enum Kind { HVP_PRE = 4, HVP_ROW = 5, HVP_COL = 6 };
enum TensorId { T_Q = 0, T_K, T_V, T_dO, T_gQ, T_gK, T_gV, T_O, T_COUNT };

// Output tensors by operation: forward {O}; backward {dQ, dK, dV}; double backward
// {g_dO, g_Q, g_K, g_V}.  Output maps have a box of 64 columns x 128 rows.
enum OutId { TO_O = 0, TO_dQ = 0, TO_dK = 1, TO_dV = 2, TO_gdO = 0, TO_gQ = 1, TO_gK = 2, TO_gV = 3, TO_COUNT = 4 };

struct TmaMaps { CUtensorMap m[T_COUNT]; CUtensorMap out[TO_COUNT]; };

template <int V> struct Int { static constexpr int value = V; };

// The issuing warps' loops with the k-steps of a head dimension: role(Int<steps>), a constant for the tile widths and the
// head dimensions of models between them, 0 (the tile width's steps, each compared with g.D / 16) for 16, 32, 48
// and 112, which would be four more copies of the loops.  A comparison costs the issuing thread about as much as the
// step it skips: a score batch of the forward took 335 clocks to issue at D = 96 as at D = 128.  First backward, two
// launches, 220 sizes of 512 to 8192 rows: 0.987, 0.979, 0.986 and 0.993 of the time at D = 64, 80, 96 and 128, where no
// step is skipped but the gaps between the steps go (0.95 to 1.026 each).  Forward, 547 sizes of 32 to 5000 rows, with V
// awaited ahead of P: 0.987, 0.994, 0.987 and 0.988 on average; at D = 80 below 8 us 1.006 (0.05 us: the loops of the third
// head dimension in line lie apart from the code before), and single sizes that change between the two modes of the tile's
// period take up to 1.065 of the time, others 0.93 (the same source compiled with the loops in another order
// moves them as far).  The double backward keeps the comparisons: with two long batches in flight the gaps let the other
// issuing warp's products in (85 us with, 90 without at B2 H16 N844 D128; D = 64 even).
template <int D, typename Role>
__device__ __forceinline__ void with_k_steps(int head_dim, Role&& role) {
  if (head_dim == D) role(Int<D / 16>{});
  else if (D == 128 && head_dim == 96) role(Int<6>{});
  else if (D == 128 && head_dim == 80) role(Int<5>{});
  else role(Int<0>{});
}

template <typename T> struct Pack;
template <> struct Pack<__nv_bfloat16> {
  static constexpr int kIsBf16 = 1;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w));
  }
};
template <> struct Pack<__half> {
  static constexpr int kIsBf16 = 0;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return __half22float2(*reinterpret_cast<__half2*>(&w));
  }
};

// Launches and the order between them.  Every tensor-core kernel is launched with programmatic
// stream serialization: its CTAs may become resident while the predecessor in the stream still
// runs, set up their barriers and tensor memory, and wait (pdl_wait) before the first access to
// global memory.  What they read may therefore be written while they are already running: it goes through
// ordinary loads, never through the read-only path (__ldg, const __restrict__), which a compiler may
// move above the wait.  Each CTA triggers its successor right after that wait.  A kernel that only has to
// come after the predecessor of its predecessor (Geometry::beside) skips the wait at its start: it
// is launched when every CTA of the predecessor has passed ITS wait, so everything before the
// predecessor is complete, and its CTAs take the SMs the predecessor's last CTAs leave idle.  Its
// last CTA waits at its end instead, so that this kernel never completes before its predecessor
// and whatever follows in the stream may rely on both.  Without the wait at its start nothing is promised
// about what an SM's L1 holds, so such a kernel reads global memory through L2 only, where every write of
// a completed kernel is: TMA, cp.async.cg, and from_l2 for the rest.  A second stream with an event fork and join does the same for 4 us more
// of host time and a launch latency on either side, and cannot be used under stream capture.
__device__ __forceinline__ void pdl_begin(const Geometry& g) { if (!g.beside) pdl_wait(); }
// A persistent kernel's last CTA may have been taken over by another one, so there every CTA waits.
__device__ __forceinline__ void pdl_end_persistent(const Geometry& g) {
  if (g.beside && threadIdx.x == 0) pdl_wait();
}
__device__ __forceinline__ void pdl_end(const Geometry& g) {
  if (g.beside && blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) pdl_wait();
}

template <typename V> __device__ __forceinline__ V from_l2(const V* p) { return __ldcg(p); }

// Opt-in to `smem` bytes of dynamic shared memory, once per kernel and device (`done`: one bit per device).
template <typename Kern>
inline cudaError_t set_smem_once(Kern kern, size_t smem, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

template <typename... P, typename... A>
inline cudaError_t launch_pdl_cluster(void (*kern)(P...), unsigned ctas, unsigned threads, size_t smem, unsigned cluster,
                                      cudaStream_t s, const A&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kern)(P...), unsigned ctas, unsigned threads, size_t smem, cudaStream_t s, const A&... args) {
  return launch_pdl_cluster(kern, ctas, threads, smem, 1, s, args...);
}

// Two kernels of one operation that do not depend on each other, dQ and dK/dV or g_Q and g_K/g_V: the CTAs of one first,
// the other's on the SMs its last CTAs leave idle.  The kernel with the longer CTAs goes first, so that the
// tail is made of short ones: the row kernel where a query sees more keys than a key is seen by queries (chunks of
// 1024 queries against a window of 8192: 128 tiles per row CTA, 16 per column CTA; backward 410 ->
// 392 us at H32 D80), else the column kernel, whose tile costs more.
inline bool row_side_first(const Geometry& g) {
  if (g.mask_mode != 0) return g.N_kv > g.N_q;
  return (g.window < g.N_kv ? g.window : g.N_kv) > (g.window < g.N_q ? g.window : g.N_q);
}

// As two launches, the second beside the first (always the double backward, the first backward where it is not one
// grid): the second one relies on the first having been launched, so it is not launched where that failed.
template <typename Row, typename Col>
inline cudaError_t side_by_side(const Geometry& g, Row row, Col col) {
  Geometry second = g;
  second.beside = 1;
  if (row_side_first(g)) {
    const cudaError_t e = row(g);
    return e == cudaSuccess ? col(second) : e;
  }
  const cudaError_t e = col(g);
  return e == cudaSuccess ? row(second) : e;
}

// ---- Splitting the streamed tiles of a stationary tile over a cluster --------------------------
// Problems with few stationary tiles (small batches, short chunks against a long window) leave SMs
// idle.  There the streamed tiles of a stationary tile are dealt out, in contiguous shares, to the
// CTAs of a cluster; each leaves its fp32 result in its own shared memory, and all of them add the
// parts through distributed shared memory, in rank order (so results are reproducible), each for its
// share of the elements.  The kernels have the split as a template parameter: with the shared form's
// epilogue in the common kernel, every launch paid a few per cent for it.

// this CTA's share of the n tiles from t0
__device__ __forceinline__ void take_share(int split, int part, int& t0, int& n) {
  const int first = n * part / split, last = n * (part + 1) / split;
  t0 += first;
  n = last - first;
}

// fp32 result tile [BM][DT] in shared memory, 16-byte chunks XORed with row % 8: a thread writes its row
template <int DT>
__device__ __forceinline__ int partial_at(int row, int chunk) { return row * DT + ((chunk ^ (row & 7)) << 2); }

template <int DT>
__device__ __forceinline__ void store_partial16(float* partial, int row, int col, const float (&f)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    *reinterpret_cast<float4*>(partial + partial_at<DT>(row, (col >> 2) + q)) = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
}

// Every thread of the cluster: the shared memory written before is readable by all its CTAs.
__device__ __forceinline__ void cluster_barrier() { cooperative_groups::this_cluster().sync(); }

// The math threads of every CTA: rows [0, rows) of the sum over the parts, weight(part, row) times
// each, post(row, column, float4) applied to it, to dst (row pitch D).
template <int DT, typename T, typename Weight, typename Post>
__device__ __forceinline__ void reduce_parts(float* partial, int split, int part, T* dst, int rows, int D, Weight weight, Post post) {
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int chunks = D >> 2;
  for (int i = part * kMathThreads + (int)threadIdx.x; i < rows * chunks; i += split * kMathThreads) {
    const int row = i / chunks, chunk = i - row * chunks;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = 0; q < split; ++q) {
      const float w = weight(q, row);
      if (!(w > 0.f)) continue;      // a part without weight is never read as a number, as in the epilogue of an unsplit tile
      const float4 x = *reinterpret_cast<const float4*>(cluster.map_shared_rank(partial, q) + partial_at<DT>(row, chunk));
      v.x = fmaf(x.x, w, v.x); v.y = fmaf(x.y, w, v.y); v.z = fmaf(x.z, w, v.z); v.w = fmaf(x.w, w, v.w);
    }
    post(row, 4 * chunk, v);
    *reinterpret_cast<uint2*>(dst + (size_t)row * D + 4 * chunk) = make_uint2(Pack<T>::pack(v.x, v.y), Pack<T>::pack(v.z, v.w));
  }
}

// Host: how many CTAs share a stationary tile.  A CTA costs kCtaClocks besides `tile_clocks` for each
// tile it visits (prologue, pipeline fill, epilogue), and split_clocks more when it shares a tile (two
// cluster barriers, the sum).  Only splits whose clusters all fit the GPU at a time are considered (a
// second wave of clusters starts late: 36 against 29 us for 96 tiles in pairs, 148 CTAs fitting),
// and only where the time of the longest CTA falls by a tenth; with another kernel beside this one, whose
// CTAs take the SMs left over, where the longer of the two falls by a quarter.
// Measured at B1 H8 D128, 256 queries against 4352 keys (16 tiles of 66): forward 34 -> 17 us with six
// parts, backward 44 -> 31, double backward 160 -> 64 us; B1 H8 N512 D64 (32 tiles of 8): no split,
// 10.5 us, with two 10.4.
constexpr float kCtaClocks = 12000.f;
constexpr int kMaxSplit = 8;
inline float split_clocks(int D) { return 3000.f + 45.f * D; }

// a kernel's stationary tiles, the most and the mean streamed tiles one of them visits, clocks per tile; how many of
// the stationary tiles visit any (keys in front of the sequence or of its windows do not), and the mean of those
struct SplitLoad { float units, longest, mean, tile_clocks, busy, busy_mean; };

template <typename Slots>
inline int pick_split(const SplitLoad& w, const SplitLoad* other, int D, Slots slots) {
  int best = 1;
  float least = 0.f;
  for (int c = 1; c <= kMaxSplit && (c == 1 || (c <= w.longest && w.units * c <= kSms)); ++c) {
    if (c > 1 && w.units * c > slots(c)) continue;
    float t = w.longest / c * w.tile_clocks + kCtaClocks + (c > 1 ? split_clocks(D) : 0.f);
    if (other != nullptr) {
      const float left = kSms - w.units * c > 1.f ? kSms - w.units * c : 1.f;
      const float theirs = (float)(int)(other->units / left + 0.999f) * (other->longest * other->tile_clocks + kCtaClocks);
      if (theirs > t) t = theirs;
    }
    if (c == 1 || t < (best > 1 ? 1.f : other != nullptr ? 0.75f : 0.9f) * least) { best = c; least = t; }
  }
  return best;
}

// From every tile where there are up to 1024 (131072 rows), from that many evenly spaced ones above: every
// launch pays for this on the host (2^30 rows: 2.9 ms for all of them, 1.5 us for 1024).
constexpr int kLoadSamples = 1024;
inline SplitLoad stream_load(const Geometry& g, bool col, float tile_clocks) {
  const int n = col ? g.N_kv : g.N_q, tiles = (n + BM - 1) / BM;
  const int samples = tiles < kLoadSamples ? tiles : kLoadSamples;
  int most = 0, busy = 0;
  long long sum = 0;
  for (int s = 0; s < samples; ++s) {
    const int i = samples == tiles ? s : (int)((long long)s * (tiles - 1) / (samples - 1));
    int lo, hi;
    if (col) query_range_for_keys(g, i * BM, (i + 1) * BM, lo, hi);
    else key_range_for_queries(g, i * BM, (i + 1) * BM, lo, hi);
    const int k = hi > lo ? (hi + BN - 1) / BN - lo / BN : 0;
    if (k > most) most = k;
    sum += k;
    busy += k > 0;
  }
  return {(float)g.BH * tiles, (float)most, samples > 0 ? (float)sum / samples : 0.f, tile_clocks,
          samples > 0 ? (float)g.BH * tiles * busy / samples : 0.f, busy > 0 ? (float)sum / busy : 0.f};
}

// What a kernel's launches keep: the devices its shared-memory opt-in has been made on, and by device
// the CTAs that run at a time in clusters of each size (0: not asked for yet).
struct TileKernelState {
  std::atomic<unsigned long long> smem_set{0}, smem_set_split{0};
  std::atomic<int> slots[64][kMaxSplit + 1] = {};
};

// CTAs of `kern` that run at a time in clusters of c on the current device `dev`; 0 where that cannot be told.
template <typename Kern>
inline int cluster_slots_on(int dev, Kern kern, int c, unsigned threads, size_t smem, TileKernelState& state) {
  std::atomic<int>& known = state.slots[dev & 63][c];
  int n = known.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)c;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (set_smem_once(kern, smem, state.smem_set_split) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, (const void*)kern, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;      // asked again by the next call
    }
    n = clusters > 0 ? clusters * c : -1;
    known.store(n, std::memory_order_relaxed);
  }
  return n;
}
template <typename Kern>
inline int cluster_slots(Kern kern, int c, unsigned threads, size_t smem, TileKernelState& state) {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess ? cluster_slots_on(dev, kern, c, threads, smem, state) : 0;
}

// Shared memory of a CTA that has its SM to itself: more than half of it, so that the 512-column tensor-memory
// allocation never waits for a co-resident CTA
inline size_t whole_sm_smem(size_t wanted) { return wanted < 122880u ? 122880u : wanted; }

// The split that a kernel's load asks for (`shared`: its form with a split).  A tile takes `tile_clocks`;
// other_clocks is the same for the other side's kernel where that runs beside this one, else 0.
template <typename... P>
inline int choose_split(void (*shared)(P...), const Geometry& g, bool col, unsigned threads, size_t smem_wanted, float tile_clocks, float other_clocks,
                        TileKernelState& state) {
  const long long units = (long long)g.BH * (((col ? g.N_kv : g.N_q) + BM - 1) / BM);
  // no split pays where half of the longest stream is cheaper than what a split costs
  if (2 * units > kSms || !((col ? g.N_q : g.N_kv) * (0.5f / BN) * tile_clocks > split_clocks(g.D))) return 1;
  const SplitLoad w = stream_load(g, col, tile_clocks);
  const bool paired = other_clocks > 0.f;
  SplitLoad other = {};
  if (paired) other = stream_load(g, !col, other_clocks);
  // of a pair, the kernel with the longer CTAs only: two kernels of clusters do not share the GPU well
  if (!(w.longest * w.tile_clocks > other.longest * other.tile_clocks)) return 1;
  return pick_split(w, paired ? &other : nullptr, g.D, [&](int c) { return cluster_slots(shared, c, threads, whole_sm_smem(smem_wanted), state); });
}

// Launch of a tensor-core kernel, one CTA per SM, with `split` CTAs per tile: `whole` where that is one, else `shared`.
template <typename... P>
inline cudaError_t launch_split(void (*whole)(P...), void (*shared)(P...), const TmaMaps& maps, Geometry g, const Tensors& t,
                                cudaStream_t s, bool col, unsigned threads, size_t smem_wanted, int split, TileKernelState& state) {
  const long long units = (long long)g.BH * (((col ? g.N_kv : g.N_q) + BM - 1) / BM);
  if (units <= 0) return cudaSuccess;
  if (units * kMaxSplit > 0x7fffffffLL) return cudaErrorInvalidValue;
  const size_t smem = whole_sm_smem(smem_wanted);
  g.split = split;
  auto kern = g.split > 1 ? shared : whole;
  const cudaError_t e = set_smem_once(kern, smem, g.split > 1 ? state.smem_set_split : state.smem_set);
  return e != cudaSuccess ? e : launch_pdl_cluster(kern, (unsigned)(units * g.split), threads, smem, (unsigned)g.split, s, maps, g, t);
}

template <typename... P>
inline cudaError_t launch_tiles(void (*whole)(P...), void (*shared)(P...), const TmaMaps& maps, const Geometry& g, const Tensors& t,
                                cudaStream_t s, bool col, unsigned threads, size_t smem_wanted, float tile_clocks, float other_clocks,
                                TileKernelState& state) {
  const int split = choose_split(shared, g, col, threads, smem_wanted, tile_clocks, other_clocks, state);
  return launch_split(whole, shared, maps, g, t, s, col, threads, smem_wanted, split, state);
}

// Upper bound of the streamed tiles of any stationary tile, of either side.
inline int longest_stream(const Geometry& g) {
  const long long n = g.N_kv > g.N_q ? g.N_kv : g.N_q, all = (n + BN - 1) / BN;
  if (g.mask_mode != 0) return (int)all;
  const long long rows = (long long)g.window + BM - 1;              // of one side that a tile of the other can see, from any row on
  const long long seen = (rows - 1 + BN - 1) / BN + 1;
  return (int)(seen < all ? seen : all);
}

// ---- Two kernels in one grid ------------------------------------------------------------------
// Two kernels of one operation that do not depend on each other, as one launch: a kernel is a type with `run`,
// which does the work of CTA `block` of its own grid.  The CTAs of the first kind are in front, so those of
// the second take the SMs that its last ones leave idle, without a launch of their own: one launch less on
// the host (2 us), no start of a second grid to wait for, nothing to wait for at its end.  dQ with dK/dV: H4, 64 queries, 256
// keys, D64 7.0 -> 5.9 us; B2 H8, 200 of 500, D96 11.0 -> 9.7; B2 H12, 777 of 1301, D80 42.2 -> 40.6; B4 H16
// N1024 D128 96.9 -> 94.7.  Kernels in clusters and kernels that take over CTAs of their grid keep a launch
// of their own, and so do long streams.
template <typename Tile>
__global__ void __launch_bounds__(Tile::kThreads, Tile::kPerSm)
tile_kernel(const __grid_constant__ TmaMaps maps, const Geometry g, const Tensors t) {
  Tile::run(maps, g, t, blockIdx.x);
}

template <typename First, typename Second>
__global__ void __launch_bounds__(First::kThreads, First::kPerSm)
pair_kernel(const __grid_constant__ TmaMaps maps, const Geometry g, const Tensors t, const unsigned first_ctas, const int second_head_group) {
  if (blockIdx.x < first_ctas) {
    First::run(maps, g, t, blockIdx.x);
  } else {
    Geometry q = g;
    q.head_group = second_head_group;
    Second::run(maps, q, t, blockIdx.x - first_ctas);
  }
}

// ---- Persistent CTAs -------------------------------------------------------------------------
// The double-backward kernels fill an SM's shared and tensor memory, so a second CTA cannot hide what a
// CTA costs besides its tiles.  There a running CTA takes over CTAs that have not been launched yet
// (cluster launch control): the producer asks for the next one while the last tiles of the current one are
// under way, announces it to the other warps, and its loads go straight on in the same ring of
// stages.  Heavy tiles come first in the grid's order, as without it.
struct WorkControl {
  alignas(16) uint32_t answer[4];
  uint64_t answered;
  uint64_t full[2], empty[2];        // two announcements, used in turn
  int unit[2];
};
constexpr int kWorkReaders = kMathWarps + 2;

__device__ __forceinline__ void work_init(WorkControl* w) {
  mbar_init(smem_u32(&w->answered), 1);
  for (int i = 0; i < 2; ++i) {
    mbar_init(smem_u32(&w->full[i]), 1);
    mbar_init(smem_u32(&w->empty[i]), kWorkReaders);
  }
}
// producer thread, once per item
__device__ __forceinline__ void work_request(WorkControl* w) {
  fence_proxy_async_smem();          // the previous answer has been read
  mbar_arrive_expect_tx(smem_u32(&w->answered), 16);
  clc_request(smem_u32(w->answer), smem_u32(&w->answered));
}
// producer thread: announcement number n, from 0; the unit, or -1 at the end
__device__ __forceinline__ bool work_announce(WorkControl* w, int n, int* unit, volatile uint32_t* abort_flag, unsigned int* status,
                                              uint32_t code) {
  if (!mbar_wait(smem_u32(&w->answered), n & 1, abort_flag, status, code)) return false;
  *unit = clc_answer(smem_u32(w->answer));
  if (!mbar_wait(smem_u32(&w->empty[n & 1]), ((n >> 1) & 1) ^ 1, abort_flag, status, code)) return false;
  w->unit[n & 1] = *unit;
  mbar_arrive(smem_u32(&w->full[n & 1]));
  return true;
}
// a whole warp of the other roles
__device__ __forceinline__ bool work_next(WorkControl* w, int n, int* unit, volatile uint32_t* abort_flag, unsigned int* status,
                                          uint32_t code) {
  const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&w->full[n & 1]), (n >> 1) & 1, abort_flag, status, code));
  // the shuffle tells the compiler that the value, and every loop bound that follows from it, is uniform
  *unit = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile int*>(&w->unit[n & 1]), 0);
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&w->empty[n & 1]));
  return ok;
}

// Equal CTAs with no other kernel to fill up with run in rounds: of 148 one to an SM, of 296 two to an SM, where a
// last round of up to 148 takes 0.8 of a whole one, half of its CTAs having an SM to themselves.  The rounds come apart as there
// are more of them.  Long streams, whose tiles take longer with two CTAs per SM, so want whole rounds: forward, D64, 24 heads
// of 2048 queries against a window of 6090 (2.6 rounds) 122 us with one per SM, 164 with two; 16 heads N3000 without mask
// 67 and 77; but 64 heads N2048 without mask (6.9 rounds) 107 and 99.
inline bool two_per_sm_pays_in_rounds(const SplitLoad& w, float tile_clocks_two) {
  if (w.busy <= kSms) return false;      // one round: 74 heads N256 D64 without mask 5.7 us, 7.0 with a group of math warps for each
  const long long n = (long long)w.busy, ones = (n - 1) / kSms, pairs = n / (2 * kSms), rest = n % (2 * kSms);
  // rounds, the last one whole, and by how much the others' coming apart makes up for that
  const float per_sm = w.busy / kSms, per_pair = per_sm / 2.f, last = rest == 0 ? 0.f : rest <= kSms ? 0.8f : 1.f;
  const float rounds = per_sm + (ones + 1 - per_sm) / (1.f + 0.1f * ones);
  const float rounds_two = per_pair + (pairs + last - per_pair) / (1.f + 0.3f * pairs);
  return rounds_two * (2.f * w.longest * tile_clocks_two + 8000.f) < rounds * (w.busy_mean * w.tile_clocks + 10000.f);
}

// Two CTAs per SM, each with half of the tensor memory and one group of math warps (the forward, and
// the first backward at D = 64, where that is enough): while one sets up, fills its pipeline or writes
// its result, the other computes.  A CTA costs kCtaClocks besides its tiles, a third of its time at 17
// tiles of 64 keys; of that 2 to 4 thousand remain.  But a CTA then takes twice as long for a tile, and a little
// more, so the longest one must not become the bound: few CTAs stay one to an SM.
// B8 H12 N2048 D64 causal: forward 117 -> 92 us; B4 H16 N1024 D128 forward 36 ->
// 25; B4 H16 N4096 D128 280 -> 253; B2 H8 N2048 D128 without mask (256 CTAs) 40 -> 36.
// Only tiles that visit any count, on either side of the rule: the first chunks of a sliding window have most of their
// keys in front of the sequence, and a CTA without a tile costs next to nothing.  First backward with 148 tiles of keys
// and fewer of queries, 640 drawn sizes: 191 go to the other form for it, which takes 0.938 of the time (0.81 to 1.17; H20, 128
// queries of 1374 keys, D64, 40 of 220 tiles of keys with a query: 10.5 -> 8.4 us).
inline bool two_per_sm_pays(const SplitLoad& w, bool alone, float tile_clocks_two) {
  if (w.busy < kSms) return false;
  auto larger = [](float x, float y) { return x > y ? x : y; };
  if (alone && w.busy_mean > 0.9f * w.longest) return two_per_sm_pays_in_rounds(w, tile_clocks_two);
  const float per_sm = w.busy / kSms;
  const float one = larger(w.longest * w.tile_clocks + kCtaClocks, per_sm * (w.busy_mean * w.tile_clocks + kCtaClocks));
  // the longest CTA of a few short ones (up to 8 tiles) that have the GPU to themselves pays less, its neighbour being done before it
  const float besides = !alone ? 9000.f : w.longest <= 8.f ? 5000.f : kCtaClocks;
  const float two = larger(2.f * w.longest * tile_clocks_two + besides, per_sm * (w.busy_mean * tile_clocks_two + (alone ? 1000.f : 4000.f)));
  return two < (alone ? 0.97f : 0.95f) * one;
}
inline bool two_per_sm_pays(const Geometry& g, bool col, bool alone, float tile_clocks, float tile_clocks_two) {
  return (long long)g.BH * (((col ? g.N_kv : g.N_q) + BM - 1) / BM) >= kSms && two_per_sm_pays(stream_load(g, col, tile_clocks), alone, tile_clocks_two);
}

// Forward: clocks of a streamed tile with one CTA (of two groups of math warps) per SM, and of each of two.  The time depends
// on the data: where rows are peaked (Q and K of twice unit variance against once) a row's reference moves more often, and the time
// with two per SM over that with one changes by 0.95 to 0.83 at D <= 64, the longer the streams the more, and by 1.04 to 1.11 at
// D > 64 up to 40 tiles, 1.0 from 80 on.  The host does not see the data, so the clocks lie between those of either kind.
// 1577 drawn sizes (90 to 16384 rows, causal, windows, no mask, D = 48 to 128), both forms timed: the form taken is 0.6 % from the faster
// one on average, 0.5 % with peaked rows; 1.5 and 1.0 % with 850 clocks in either form and no rounds of 296.  The 156 that
// change form take 0.915 and 0.949 of the time (0.74 to 1.16 and 0.72 to 1.13).
inline bool forward_two_per_sm(const Geometry& g) {
  const float past = g.D > 64 ? g.D - 64.f : 0.f;
  return two_per_sm_pays(g, false, true, 710.f + 3.2f * past, g.D > 64 ? 870.f + 1.5f * past : 770.f);
}

// First backward at D <= 64: clocks of a streamed tile of dQ and of dK/dV, with one and with two CTAs per SM
constexpr float kRowClocks = 1000.f, kRowClocksTwo = 930.f, kColClocks = 1700.f, kColClocksTwo = 1250.f;

// Both kinds, which share the GPU, with a full set of CTAs each: one answer for the two of them.  A CTA costs 8 thousand
// clocks besides its tiles, of which 4 remain where two share an SM.  Unequal CTAs fill the GPU up, so the bound is the sum
// of all, or the longest CTA, whose tiles take twice the clocks with two on its SM.  Equal CTAs (no mask) run in rounds: up
// to three rounds of 148 one per SM is faster (two take 1.02 to 1.08 of the time at 2.8 to 3 rounds), unless streams are so short
// (24 tiles of both kinds) that what a CTA costs besides them is the larger part.  A fourth round turns it: two per SM 0.955 of
// the time at H16 N1700, 0.89 at H32 N866, 0.84 at H28, 778 of 1139.  One kind with two per SM and the other with one, in two
// launches, is up to 13 % faster where the one round of the one leaves room for the other (H20, 1152 of 1408), as much slower
// elsewhere, and 1 % slower on average over the 121 sizes where each kind asked by itself took it.
inline bool both_two_per_sm_pay(const SplitLoad& r, const SplitLoad& c) {
  if (r.busy_mean > 0.9f * r.longest && c.busy_mean > 0.9f * c.longest)
    return r.busy + c.busy > 3 * kSms || (r.busy + c.busy >= 2.5f * kSms && r.busy_mean + c.busy_mean <= 24.f);
  auto larger = [](float x, float y) { return x > y ? x : y; };
  auto sum = [&](float row, float col, float besides) { return (r.busy * (r.busy_mean * row + besides) + c.busy * (c.busy_mean * col + besides)) / kSms; };
  const float one = larger(larger(r.longest * kRowClocks, c.longest * kColClocks) + 8000.f, sum(kRowClocks, kColClocks, 8000.f));
  const float two = larger(2.f * larger(r.longest * kRowClocksTwo, c.longest * kColClocksTwo) + 8000.f, sum(kRowClocksTwo, kColClocksTwo, 4000.f));
  return two < one;
}

// Whether dQ and dK/dV run two CTAs per SM at D <= 64.  With fewer CTAs than SMs on one side the other side decides by itself.
struct TwoPerSm { bool row, col; };
inline TwoPerSm backward_two_per_sm(const Geometry& g) {
  const long long rows = (long long)g.BH * ((g.N_q + BM - 1) / BM), cols = (long long)g.BH * ((g.N_kv + BM - 1) / BM);
  if (rows < kSms && cols < kSms) return {false, false};
  const SplitLoad r = stream_load(g, false, kRowClocks), c = stream_load(g, true, kColClocks);
  if (r.busy >= kSms && c.busy >= kSms) {
    const bool both = both_two_per_sm_pay(r, c);
    return {both, both};
  }
  return {two_per_sm_pays(r, false, kRowClocksTwo), two_per_sm_pays(c, false, kColClocksTwo)};
}

// more than a third of an SM's shared memory: never a third CTA that would wait for tensor memory
inline size_t half_sm_smem(size_t wanted) { return wanted < 79872u ? 79872u : wanted; }

template <typename... P>
inline cudaError_t launch_two_per_sm(void (*kern)(P...), const TmaMaps& maps, const Geometry& g, const Tensors& t, cudaStream_t s,
                                     long long ctas, unsigned threads, size_t smem_wanted, std::atomic<unsigned long long>& smem_set) {
  if (ctas > 0x7fffffffLL) return cudaErrorInvalidValue;
  const size_t smem = half_sm_smem(smem_wanted);
  const cudaError_t e = set_smem_once(kern, smem, smem_set);
  return e != cudaSuccess ? e : launch_pdl(kern, (unsigned)ctas, threads, smem, s, maps, g, t);
}

template <typename First, typename Second>
inline cudaError_t launch_pair(const TmaMaps& maps, const Geometry& g_in, const Tensors& t, cudaStream_t s, long long first_ctas, int first_group,
                               long long second_ctas, int second_group, size_t smem_wanted, std::atomic<unsigned long long>& smem_set) {
  static_assert(First::kThreads == Second::kThreads && First::kPerSm == Second::kPerSm, "one launch configuration");
  if (first_ctas + second_ctas > 0x7fffffffLL) return cudaErrorInvalidValue;
  const size_t smem = First::kPerSm == 2 ? half_sm_smem(smem_wanted) : whole_sm_smem(smem_wanted);
  Geometry g = g_in;
  g.head_group = first_group;
  const cudaError_t e = set_smem_once(pair_kernel<First, Second>, smem, smem_set);
  return e != cudaSuccess ? e : launch_pdl(pair_kernel<First, Second>, (unsigned)(first_ctas + second_ctas), (unsigned)First::kThreads, smem, s, maps, g, t,
                                           (unsigned)first_ctas, second_group);
}

// Control block of the single-tile self-test kernel (every attention kernel has its own).
struct Control {
  uint64_t stat_full;
  uint64_t acc_done;
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
};

// status codes: (kind + 1) << 8 | wait id
__device__ __forceinline__ uint32_t wait_code(int kind, int id) { return ((uint32_t)(kind + 1) << 8) | (uint32_t)id; }

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Scores of one row that are not visible, as zeros: element i is number `first` + i of the row's visible range [0, span).  A pass
// of its own for the tiles that have such elements: within the loop of the exponentials its three instructions for an
// element are executed in every tile.
template <int N>
__device__ __forceinline__ void mask_pairs(float2 (&p)[N], int first, uint32_t span) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    p[i].x = (uint32_t)(first + 2 * i) < span ? p[i].x : 0.f;
    p[i].y = (uint32_t)(first + 2 * i + 1) < span ? p[i].y : 0.f;
  }
}

// 16 packed halves (two 16-byte chunks) of operand-tile row `row`, columns
// [col0, col0+16), into a 128-byte-swizzled [128][64] tile.
__device__ __forceinline__ void store_op16(uint32_t tile, int row, int col0, const uint32_t (&v)[8]) {
  const uint32_t a0 = tile + sw128_offset(row, col0);
  const uint32_t a1 = tile + sw128_offset(row, col0 + 8);
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a0), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3])
               : "memory");
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a1), "r"(v[4]), "r"(v[5]), "r"(v[6]),
               "r"(v[7])
               : "memory");
}

__device__ __forceinline__ void load_op16(uint32_t tile, int row, int col0, uint32_t (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 2; ++q)
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[4 * q]), "=r"(v[4 * q + 1]), "=r"(v[4 * q + 2]), "=r"(v[4 * q + 3])
                 : "r"(tile + sw128_offset(row, col0 + 8 * q))
                 : "memory");
}

// Zeros in rows [row0, row0 + BM) of plane `plane` of a [planes][n_rows][D] half-precision tensor: the
// result of a CTA that has no tile to visit (keys in front of the sequence in a chunk's window,
// queries without a visible key).  It needs no barriers, tensor memory or loads.  At H12, the fourth
// chunk of 1024 queries, 9216 keys, D64, 480 of 864 column CTAs are of this kind: backward 85 -> 78,
// double backward 171 -> 165 us.
__device__ __forceinline__ void zero_rows(void* out, int plane, int row0, int n_rows, int D, int threads) {
  const int rows = min(BM, n_rows - row0);
  uint4* p = reinterpret_cast<uint4*>(static_cast<uint16_t*>(out) + ((size_t)plane * n_rows + row0) * D);
  for (int i = threadIdx.x; i < rows * D / 8; i += threads) p[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Epilogue of the tensor-core kernels.  The 256 math threads have written a [128 rows][cols]
// half-precision result tile to shared memory at `tile`, one 128-byte-swizzled 16 KB atom per 64
// columns (store_op16).  All of them call this; `leader` (one thread) then writes the tile to
// rows [row0, row0 + 128) of plane `plane` with one TMA store per atom (rows and columns beyond
// the tensor are clipped by the map) and returns once shared memory has been read.
__device__ __forceinline__ void store_tile_tma(const CUtensorMap* map, uint32_t tile, int cols, int row0, int plane,
                                               bool leader, int math_threads = kMathThreads) {
  fence_proxy_async_smem();
  named_barrier_sync(2, (uint32_t)math_threads);
  if (leader) {
    for (int a = 0; a * 64 < cols; ++a) tma_store_3d(map, tile + (uint32_t)a * kAtomBytesStat, a * 64, row0, plane);
    bulk_commit_group();
    bulk_wait_group_read_all();
  }
}

}  // namespace tc
}  // namespace attn
