// Definitions shared by the tensor-core kernel files: tile sizes, warp roles,
// tensor-map bundle and small device helpers.
#pragma once

#include "attn_common.cuh"
#include "tc_primitives.cuh"

#include <atomic>

namespace attn {
namespace tc {

constexpr int BM = 128;            // stationary rows per CTA
constexpr int BN = 64;             // streamed rows per iteration
constexpr int kMathWarps = 8;
constexpr int kMathThreads = kMathWarps * 32;
constexpr int kProducerWarp = 8;   // the MMA-issuing warps follow it
constexpr int kTmemCols = 512;
constexpr uint32_t kAtomBytesStat = BM * 128;   // [128 rows][64 halves], 16 KB
constexpr uint32_t kAtomBytesStrm = BN * 128;   // [ 64 rows][64 halves],  8 KB

// Kernel ids inside device status codes (the backward kernels use 18 and 19, the forward kernel
// 20, the self-test 0x6f); the values are documented with the C ABI and do not change.
enum Kind { HVP_PRE = 4, HVP_ROW = 5, HVP_COL = 6 };
enum TensorId { T_Q = 0, T_K, T_V, T_dO, T_gQ, T_gK, T_gV, T_COUNT };

// Launches and the order between them.  Every tensor-core kernel is launched with programmatic
// stream serialization: its CTAs may become resident while the predecessor in the stream still
// runs, set up their barriers and tensor memory, and wait (pdl_wait) before the first access to
// global memory.  Each CTA triggers its successor right after that wait.  A kernel that only has to
// come after the predecessor of its predecessor (Geometry::beside) skips the wait at its start: it
// is launched when every CTA of the predecessor has passed ITS wait, so everything before the
// predecessor is complete, and its CTAs take the SMs the predecessor's last CTAs leave idle.  Its
// last CTA waits at its end instead, so that this kernel never completes before its predecessor
// and whatever follows in the stream may rely on both.  A second stream with an event fork and join does the same for 4 us more
// of host time and a launch latency on either side, and cannot be used under stream capture.
__device__ __forceinline__ void pdl_begin(const Geometry& g) { if (!g.beside) pdl_wait(); }
__device__ __forceinline__ void pdl_end(const Geometry& g) {
  if (g.beside && blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) pdl_wait();
}

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

// Output tensors by operation: forward {O}; backward {dQ, dK, dV}; double backward
// {g_dO, g_Q, g_K, g_V}.  Output maps have a box of 64 columns x 128 rows.
enum OutId { TO_O = 0, TO_dQ = 0, TO_dK = 1, TO_dV = 2, TO_gdO = 0, TO_gQ = 1, TO_gK = 2, TO_gV = 3, TO_COUNT = 4 };

struct TmaMaps { CUtensorMap m[T_COUNT]; CUtensorMap out[TO_COUNT]; };

// Control block of the single-tile self-test kernel (every attention kernel has its own).
struct Control {
  uint64_t stat_full;
  uint64_t acc_done;
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
};

// status codes: (kind + 1) << 8 | wait id
__device__ __forceinline__ uint32_t wait_code(int kind, int id) { return ((uint32_t)(kind + 1) << 8) | (uint32_t)id; }

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

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
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


// Zeros in rows [row0, row0 + BM) of plane `plane` of a [planes][n_rows][D] half-precision tensor: the
// result of a CTA that has no tile to visit (keys in front of the sequence in a chunk's window,
// queries without a visible key).  It needs no barriers, tensor memory or loads.  At H12, the fourth
// chunk of 1024 queries, 9216 keys, D64, 480 of 864 column CTAs are of this kind: backward 85 -> 78,
// double backward 171 -> 165 us.
__device__ __forceinline__ void zero_rows(void* out, int plane, int row0, int n_rows, int D) {
  const int rows = min(BM, n_rows - row0);
  uint4* p = reinterpret_cast<uint4*>(static_cast<uint16_t*>(out) + ((size_t)plane * n_rows + row0) * D);
  for (int i = threadIdx.x; i < rows * D / 8; i += blockDim.x) p[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Epilogue of the tensor-core kernels.  The 256 math threads have written a [128 rows][cols]
// half-precision result tile to shared memory at `tile`, one 128-byte-swizzled 16 KB atom per 64
// columns (store_op16).  All of them call this; `leader` (one thread) then writes the tile to
// rows [row0, row0 + 128) of plane `plane` with one TMA store per atom (rows and columns beyond
// the tensor are clipped by the map) and returns once shared memory has been read.
__device__ __forceinline__ void store_tile_tma(const CUtensorMap* map, uint32_t tile, int cols, int row0, int plane,
                                               bool leader) {
  fence_proxy_async_smem();
  named_barrier_sync(2, kMathWarps * 32);
  if (leader) {
    for (int a = 0; a * 64 < cols; ++a) tma_store_3d(map, tile + (uint32_t)a * kAtomBytesStat, a * 64, row0, plane);
    bulk_commit_group();
    bulk_wait_group_read_all();
  }
}

}  // namespace tc
}  // namespace attn
