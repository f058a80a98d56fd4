// fp32 CUDA-core kernels for attention forward / backward / double backward.
//
// This family serves float32 inputs (where results must agree with an fp64 oracle to 1e-4) and, when
// asked for, half-precision inputs.  All arithmetic is fp32 on CUDA cores; inputs are widened when a
// tile is staged in shared memory.  Nothing here materialises more than a 32 x 64 score tile per CTA.
//
// A CTA owns 32 STATIONARY rows of one (batch, head) -- query rows in the row kinds,
// key rows in the column kinds -- and streams 64-row tiles of the other axis:
//
//   kind      stationary        streamed          produces
//   FWD       Q                 K, V              O, L (online softmax)
//   BWD_ROW   Q, dO             K, V              dQ = s dS K
//   BWD_COL   K, V              Q, dO             dV = P^T dO, dK = s dS^T Q
//   HVP_PRE   Q, dO, g_dQ       K, V, g_dK, g_dV  Dv, dot2, dot3;  g_dO = P g_dV + (P o gdS) V - dot2 o (P V)
//   HVP_ROW   Q, dO, g_dQ       K, V, g_dK, g_dV  g_Q = s (dS g_dK + g_S K)
//   HVP_COL   K, V, g_dK, g_dV  Q, dO, g_dQ       g_K = s (dS^T g_dQ + g_S^T Q), g_V = g_dp^T dO
//
// Bound by the FMA pipe and shared-memory reads together.  A float4 read of a warp takes four clocks of
// the SM's 128 bytes per clock, or two where no quad of lanes reads more than two different float4s
// (measured: 4.0 and 2.1 with 8 of 32 lanes' values different, depending on which lanes share).  So a warp is
// 4 x 8 threads with 2 x 2 of them in every quad, which halves the reads of the streamed side; rows by
// lane / 8 and columns by lane % 8 took, at D = 128, 10 to 17 % more time (B2 H8 N1024 forward 220 -> 180,
// backward 690 -> 573, double backward 1 685 -> 1 509 us), at D = 64 1 to 5 %.  A thread holds 2 x 4 scores of every
// score matrix of its kind; in the double backward at D <= 64, where four matrices share the operands it has
// read, 4 x 4 (N1024 800 against 837 us, and the smaller backward the other way round: B2 H5 N479 62
// against 65).  At D > 64 a CTA has an SM to itself, by its registers (199 to 255 per thread, 256 threads) in the forward
// and the first backward (89 to 113 KB of shared memory at D = 128), by its shared memory too in the double
// backward (185 to 193 KB); twice the warps hide the latencies.  At D <= 64 two fit by both (124 to 128 registers
// of 256 threads, 240 to 255 of 128; at most 105 KB).
// The packed f32x2 multiply-adds run along the head dimension without a move; as scalar ones they
// have a higher rate with one or two warps per scheduler, but the issue slots they take cost 4 to 70 %.
// Rows are stored without padding where D is a multiple of 32, their 16-byte chunks XOR-swizzled by the
// row, which lets two CTAs of every kind share an SM at D <= 64: one computes while the other loads.
// Loading the next tile behind the output products instead gave nothing (forward -1 to -3 %, backward +4 %).
// Small problems: the streamed tiles of a stationary tile are dealt out to a CLUSTER of 2 to 8 CTAs
// (simt_split.h), whose partial sums are added through distributed shared memory in a fixed order; results are
// bitwise reproducible either way.
#include "attn_common.cuh"
#include "attn_launch.h"
#include "simt_split.h"
#include "tc_common.cuh"

#include <cooperative_groups.h>

namespace attn {
namespace simt {

namespace cg = cooperative_groups;

constexpr int CB = 4;         // score columns per thread, 8 apart

// By kind and tile width (DC = 1: D <= 64, 2: D <= 128): score rows per thread, 4 apart, and threads per
// CTA, (8 / RA) x 2 warps over the 32 x 64 score tile.
__host__ __device__ constexpr int rows_of(int kind, int DC) { return DC == 1 && kind >= K_HVP_PRE ? 4 : 2; }
__host__ __device__ constexpr int threads_of(int kind, int DC) { return 512 / rows_of(kind, DC); }

template <int KIND> struct Spec {
  static constexpr bool kCol = KIND == K_BWD_COL || KIND == K_HVP_COL;
  static constexpr bool kHvp = KIND >= K_HVP_PRE;
  static constexpr int kNStat = KIND == K_FWD ? 1 : !kHvp ? 2 : kCol ? 4 : 3;
  static constexpr int kNStream = !kHvp ? 2 : kCol ? 3 : 4;
  static constexpr int kNAcc = KIND == K_FWD ? 1 : kHvp ? 4 : 2;       // S, dP | S, gdS, dP, gPdV
  static constexpr int kNOp = KIND == K_FWD || KIND == K_BWD_ROW ? 1 : KIND == K_HVP_COL ? 3 : 2;
  static constexpr int kNOut = kCol ? 2 : 1;
};

// Tile layout: row r at r * pitch floats; with D a multiple of 32 the pitch is D and the float4
// chunks of a row are XORed with r % 8, otherwise the pitch is D + 4.
struct Layout {
  int pitch, mask;
  __host__ __device__ __forceinline__ explicit Layout(int D) : pitch(D % 32 == 0 ? D : D + 4), mask(D % 32 == 0 ? 7 : 0) {}
  __device__ __forceinline__ int at(int row, int chunk) const { return row * pitch + ((chunk ^ (row & mask)) << 2); }
};
__device__ __forceinline__ int op_at(int row, int col) { return row * TT + ((((col >> 2) ^ (row & 7)) << 2) | (col & 3)); }

__device__ __forceinline__ void cp_async16(float* dst, const void* src, bool in) {
  const unsigned bytes = in ? 16u : 0u;       // 0: the destination is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Four consecutive elements of a half-precision row, widened.
template <typename T> __device__ __forceinline__ float4 widen4(const T* p) {
  const uint2 w = tc::from_l2(reinterpret_cast<const uint2*>(p));
  const float2 a = tc::Pack<T>::unpack(w.x), b = tc::Pack<T>::unpack(w.y);
  return make_float4(a.x, a.y, b.x, b.y);
}

// Stage `rows` rows from row0 of a [n_rows, D] matrix as fp32, zero beyond n_rows.  DC * 16 of the NT threads
// share a row.  float goes by cp.async (complete after cp_async_wait_all and a barrier).
template <int DC, int NT, typename T>
__device__ __forceinline__ void stage_tile(float* dst, const Layout& lay, const T* src, int row0, int rows, int n_rows, int D) {
  constexpr int kLanes = 16 * DC;
  const int chunk = threadIdx.x % kLanes;
  if (chunk * 4 >= D) return;
  for (int r = threadIdx.x / kLanes; r < rows; r += NT / kLanes) {
    const bool in = row0 + r < n_rows;
    const T* p = src + (size_t)(in ? row0 + r : 0) * D + chunk * 4;
    float* q = dst + lay.at(r, chunk);
    if constexpr (sizeof(T) == 4) cp_async16(q, p, in);
    else *reinterpret_cast<float4*>(q) = in ? widen4<T>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

__device__ __forceinline__ void mac(float2& acc, const float4& x, const float4& y) {
  acc = __ffma2_rn(make_float2(x.x, x.y), make_float2(y.x, y.y), acc);
  acc = __ffma2_rn(make_float2(x.z, x.w), make_float2(y.z, y.w), acc);
}

// The raw score matrices of a kind for this thread's RA x 4 elements.
template <int KIND, int RA>
__device__ __forceinline__ void scores(float* const (&stat)[4], float* const (&strm)[4], const Layout& lay, int D,
                                       int row0, int col0, float (&out)[Spec<KIND>::kNAcc][RA][CB]) {
  using SP = Spec<KIND>;
  constexpr int kScored = KIND == K_FWD ? 1 : SP::kNStream;     // the forward's V takes no part in the scores
  float2 acc[SP::kNAcc][RA][CB];
#pragma unroll
  for (int m = 0; m < SP::kNAcc; ++m)
#pragma unroll
    for (int a = 0; a < RA; ++a)
#pragma unroll
      for (int b = 0; b < CB; ++b) acc[m][a][b] = make_float2(0.f, 0.f);
#pragma unroll (RA == 4 ? 2 : 4)
  for (int k = 0; k < (D >> 2); ++k) {
    float4 x[SP::kNStat][RA];
#pragma unroll
    for (int i = 0; i < SP::kNStat; ++i)
#pragma unroll
      for (int a = 0; a < RA; ++a) x[i][a] = *reinterpret_cast<const float4*>(stat[i] + lay.at(row0 + 4 * a, k));
#pragma unroll
    for (int b = 0; b < CB; ++b) {
      float4 y[kScored];
#pragma unroll
      for (int i = 0; i < kScored; ++i) y[i] = *reinterpret_cast<const float4*>(strm[i] + lay.at(col0 + 8 * b, k));
#pragma unroll
      for (int a = 0; a < RA; ++a) {
        mac(acc[0][a][b], x[0][a], y[0]);                       // Q K^T               | K Q^T
        if constexpr (SP::kNAcc == 2) mac(acc[1][a][b], x[1][a], y[1]);      // dO V^T  | V dO^T
        if constexpr (SP::kHvp) {
          mac(acc[1][a][b], x[2][a], y[0]);                     // g_dQ K^T            | g_dK Q^T
          mac(acc[1][a][b], x[0][a], y[2]);                     // + Q g_dK^T          | + K g_dQ^T
          mac(acc[2][a][b], x[1][a], y[1]);                     // dO V^T              | V dO^T
          if constexpr (SP::kCol) mac(acc[3][a][b], x[3][a], y[1]);          //         | g_dV dO^T
          else mac(acc[3][a][b], x[1][a], y[3]);                // dO g_dV^T
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < SP::kNAcc; ++m)
#pragma unroll
    for (int a = 0; a < RA; ++a)
#pragma unroll
      for (int b = 0; b < CB; ++b) out[m][a][b] = acc[m][a][b].x + acc[m][a][b].y;
}

// out[a][c] += sum_j Op[row0 + 4a, j] * Z[j, chunk c of this thread]
template <int DC, int RA>
__device__ __forceinline__ void out_fma(const float* op, const float* Z, const Layout& lay, int row0, int chunk0, int chunks,
                                        float2 (&out)[RA][DC][2]) {
#pragma unroll (RA == 4 ? 2 : 4)
  for (int j = 0; j < TT; j += 4) {
    float o[RA][4];
#pragma unroll
    for (int a = 0; a < RA; ++a) {
      const float4 v = *reinterpret_cast<const float4*>(op + op_at(row0 + 4 * a, j));
      o[a][0] = v.x; o[a][1] = v.y; o[a][2] = v.z; o[a][3] = v.w;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 0; c < DC; ++c) {
        if (chunk0 + 16 * c < chunks) {
          const float4 z = *reinterpret_cast<const float4*>(Z + lay.at(j + u, chunk0 + 16 * c));
#pragma unroll
          for (int a = 0; a < RA; ++a) {
            const float2 oo = make_float2(o[a][u], o[a][u]);
            out[a][c][0] = __ffma2_rn(oo, make_float2(z.x, z.y), out[a][c][0]);
            out[a][c][1] = __ffma2_rn(oo, make_float2(z.z, z.w), out[a][c][1]);
          }
        }
      }
  }
}

// sum over the eight threads of a warp that share a row
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = 8; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
  for (int o = 8; o > 1; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <typename T> __device__ __forceinline__ void store4(T* p, const float4& v) {
  *reinterpret_cast<uint2*>(p) = make_uint2(tc::Pack<T>::pack(v.x, v.y), tc::Pack<T>::pack(v.z, v.w));
}
template <> __device__ __forceinline__ void store4<float>(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
template <typename T> __device__ __forceinline__ float4 load4(const T* p) { return widen4<T>(p); }
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return tc::from_l2(reinterpret_cast<const float4*>(p)); }

// shared memory in floats
template <int KIND>
__host__ __device__ constexpr int smem_floats(int D) {
  const int pitch = D % 32 == 0 ? D : D + 4;
  return (Spec<KIND>::kNStat * TS + Spec<KIND>::kNStream * TT) * pitch + Spec<KIND>::kNOp * TS * TT + 4 * TT;
}

// DC: 1 for D <= 64, 2 up to 128.
// The work of CTA `block` of a kind's grid.
template <int KIND, int DC, typename T>
__device__ __forceinline__ void simt_tile(const Geometry& g, const Tensors& t, const int split, const int block) {
  using SP = Spec<KIND>;
  constexpr int RA = rows_of(KIND, DC), NT = threads_of(KIND, DC);
  // g_dO = P g_dV + (P o gdS) V - dot2 o (P V).  In fp32 P V is the O of the call; an O of half precision has
  // been rounded, so there the kernel sums its own (bf16, g_dK offset by one: relative error 1.66e-3
  // instead of 1.92e-3; 1.66e-3 is the rounding of the result).
  constexpr bool kOwnPV = KIND == K_HVP_PRE && sizeof(T) == 2;
  constexpr int kNSums = SP::kNOut + (kOwnPV ? 1 : 0);
  extern __shared__ __align__(16) float smem[];
  const int D = g.D;
  const Layout lay(D);
  const int n_stat = SP::kCol ? g.N_kv : g.N_q, n_strm = SP::kCol ? g.N_q : g.N_kv;
  const int tiles = (n_stat + TS - 1) / TS;
  const int unit = block / split, part = block - unit * split;
  const int bh = unit % g.BH, rank = unit / g.BH;
  const int tile = (SP::kCol || g.mask_mode != 0) ? rank : tiles - 1 - rank;     // heavy tiles first
  const int r0 = tile * TS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ty = (lane & 1) | ((lane >> 4) << 1), tx = (lane >> 1) & 7, wcol = warp & 1;      // 2 x 2 in every quad of lanes
  const int row0 = (warp >> 1) * 4 * RA + ty;         // this thread's rows: row0 + 4 a
  const int col0 = wcol * 32 + tx;                    // its score columns: col0 + 8 b
  const int chunk0 = wcol * 8 + tx, chunks = D >> 2;  // its output float4s: chunk0 + 16 c

  float* stat[4];
  float* strm[4];
  float* op[3];
  float* p = smem;
  for (int i = 0; i < 4; ++i) { stat[i] = p; if (i < SP::kNStat) p += TS * lay.pitch; }
  float* const strm_base = p;
  for (int i = 0; i < 4; ++i) { strm[i] = p; if (i < SP::kNStream) p += TT * lay.pitch; }
  for (int i = 0; i < 3; ++i) { op[i] = p; if (i < SP::kNOp) p += TS * TT; }
  float* const aux = p;                               // [4][64]: scalars of the streamed queries, or row exchange

  const size_t q_off = (size_t)bh * g.N_q * D, kv_off = (size_t)bh * g.N_kv * D, row_off = (size_t)bh * g.N_q;
  const T* const Q = (const T*)t.Q + q_off;
  const T* const K = (const T*)t.K + kv_off;
  const T* const V = (const T*)t.V + kv_off;
  const T* const dO = (const T*)t.dO + q_off;
  const T* const O = (const T*)t.O + q_off;
  const T* const gQ = (const T*)t.g_dQ + q_off;
  const T* const gK = (const T*)t.g_dK + kv_off;
  const T* const gV = (const T*)t.g_dV + kv_off;
  const T* const stat_src[4] = {SP::kCol ? K : Q, SP::kCol ? V : dO, SP::kCol ? gK : gQ, gV};
  const T* const strm_src[4] = {SP::kCol ? Q : K, SP::kCol ? dO : V, SP::kCol ? gQ : gK, gV};

  int lo, hi;
  if constexpr (SP::kCol) query_range_for_keys(g, r0, r0 + TS, lo, hi);
  else key_range_for_queries(g, r0, r0 + TS, lo, hi);
  const int t_end = hi > lo ? (hi + TT - 1) / TT : 0;
  const int t_first = lo / TT + part;

  tc::pdl_begin(g);
  tc::pdl_trigger();

#pragma unroll
  for (int i = 0; i < SP::kNStat; ++i) stage_tile<DC, NT, T>(stat[i], lay, stat_src[i], r0, TS, n_stat, D);

  // ---- scalars of this thread's rows (row kinds)
  float L2[RA] = {}, Dv[RA] = {}, d2[RA] = {}, d3[RA] = {};
  if constexpr (!SP::kCol && KIND != K_FWD) {
#pragma unroll
    for (int a = 0; a < RA; ++a) {
      const int r = r0 + row0 + 4 * a;
      const bool in = r < g.N_q;
      L2[a] = in ? tc::from_l2(t.L + row_off + r) * kLog2e : INFINITY;
      if constexpr (KIND == K_HVP_ROW) {
        if (in) { Dv[a] = tc::from_l2(t.Dv + row_off + r); d2[a] = tc::from_l2(t.dot2 + row_off + r); d3[a] = tc::from_l2(t.dot3 + row_off + r); }
      }
      if constexpr (KIND == K_BWD_ROW) {      // D_i = sum_d dO * O from the stored (rounded) O
        float s = 0.f;
        if (in)
          for (int c = tx; c < chunks; c += 8) {
            const float4 x = load4(dO + (size_t)r * D + 4 * c), y = load4(O + (size_t)r * D + 4 * c);
            s += x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
          }
        Dv[a] = row_sum(s);
      }
    }
  }
  float m_run[RA], l_run[RA] = {};                           // FWD
  float aD[RA] = {}, a2[RA] = {}, aA[RA] = {}, aE[RA] = {};   // HVP_PRE
#pragma unroll
  for (int a = 0; a < RA; ++a) m_run[a] = -INFINITY;
  float2 out[kNSums][RA][DC][2];
#pragma unroll
  for (int o = 0; o < kNSums; ++o)
#pragma unroll
    for (int a = 0; a < RA; ++a)
#pragma unroll
      for (int c = 0; c < DC; ++c) out[o][a][c][0] = out[o][a][c][1] = make_float2(0.f, 0.f);

  for (int tt = t_first; tt < t_end; tt += split) {
    const int s0 = tt * TT;
    __syncthreads();                                  // the previous tile has been used
#pragma unroll
    for (int i = 0; i < SP::kNStream; ++i) stage_tile<DC, NT, T>(strm[i], lay, strm_src[i], s0, TT, n_strm, D);
    if constexpr (SP::kCol) {                         // [L2 | Dv | dot2 | dot3] of the streamed queries
      if constexpr (SP::kHvp) {
#pragma unroll
        for (int i = tid; i < 4 * TT; i += NT) {
          const int r = s0 + (i & 63), which = i >> 6;
          const float* src = which == 0 ? t.L : which == 1 ? t.Dv : which == 2 ? t.dot2 : t.dot3;
          const float v = r < g.N_q ? tc::from_l2(src + row_off + r) : 0.f;
          aux[i] = which == 0 ? (r < g.N_q ? v * kLog2e : INFINITY) : v;
        }
      } else {
        constexpr int TQ = NT / TT;                   // threads per query
        const int r = s0 + tid / TQ;
        float s = 0.f;
        if (r < g.N_q)
          for (int c = tid % TQ; c < chunks; c += TQ) {
            const float4 x = load4(dO + (size_t)r * D + 4 * c), y = load4(O + (size_t)r * D + 4 * c);
            s += x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
          }
#pragma unroll
        for (int o = TQ / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (tid % TQ == 0) {
          aux[tid / TQ] = r < g.N_q ? tc::from_l2(t.L + row_off + r) * kLog2e : INFINITY;
          aux[TT + tid / TQ] = s;
        }
      }
    }
    cp_async_wait_all();
    __syncthreads();
    float s[SP::kNAcc][RA][CB];
    scores<KIND, RA>(stat, strm, lay, D, row0, col0, s);
    const bool full = SP::kCol ? tile_fully_visible(g, s0, s0 + TT, r0, r0 + TS) : tile_fully_visible(g, r0, r0 + TS, s0, s0 + TT);
    auto sees = [&](int a, int b) {
      const int i = r0 + row0 + 4 * a, j = s0 + col0 + 8 * b;
      return full || (SP::kCol ? visible(g, j, i) : visible(g, i, j));
    };

    if constexpr (KIND == K_FWD) {
      // running maximum of a row: over this warp's 32 columns, then over the two warps of the row
#pragma unroll
      for (int a = 0; a < RA; ++a) {
        float mx = -INFINITY;
#pragma unroll
        for (int b = 0; b < CB; ++b) {
          s[0][a][b] = sees(a, b) ? s[0][a][b] * g.scale_log2e : -INFINITY;
          mx = fmaxf(mx, s[0][a][b]);
        }
        mx = row_max(mx);
        if (tx == 0) aux[wcol * TS + row0 + 4 * a] = mx;
      }
      __syncthreads();
#pragma unroll
      for (int a = 0; a < RA; ++a) {
        const float m_new = fmaxf(m_run[a], fmaxf(aux[row0 + 4 * a], aux[TS + row0 + 4 * a]));
        const float f = m_new == -INFINITY ? 1.f : exp2f(m_run[a] - m_new);
        m_run[a] = m_new;
        l_run[a] *= f;
#pragma unroll
        for (int c = 0; c < DC; ++c)
#pragma unroll
          for (int h = 0; h < 2; ++h) out[0][a][c][h] = make_float2(out[0][a][c][h].x * f, out[0][a][c][h].y * f);
#pragma unroll
        for (int b = 0; b < CB; ++b) {
          // a score that is not a number goes on to the result, also where it is all that a row sees (m_new = -inf)
          const float pr = s[0][a][b] == -INFINITY ? 0.f : exp2f(s[0][a][b] - m_new);
          l_run[a] += pr;
          op[0][op_at(row0 + 4 * a, col0 + 8 * b)] = pr;
        }
      }
    } else {
#pragma unroll
      for (int a = 0; a < RA; ++a)
#pragma unroll
        for (int b = 0; b < CB; ++b) {
          const int col = col0 + 8 * b, at = op_at(row0 + 4 * a, col);
          RowStats rs;
          if constexpr (SP::kCol) rs = RowStats{aux[col], aux[TT + col], SP::kHvp ? aux[2 * TT + col] : 0.f, SP::kHvp ? aux[3 * TT + col] : 0.f};
          else rs = RowStats{L2[a], Dv[a], d2[a], d3[a]};
          const float pr = prob(s[0][a][b], g.scale_log2e, rs.L2, sees(a, b));
          if constexpr (KIND == K_BWD_ROW) {
            op[0][at] = pr * (s[1][a][b] - rs.Dv);
          } else if constexpr (KIND == K_BWD_COL) {
            op[0][at] = pr;
            op[1][at] = pr * (s[1][a][b] - rs.Dv);
          } else if constexpr (KIND == K_HVP_PRE) {
            const float pg = pr * (s[1][a][b] * g.scale);
            aD[a] = fmaf(pr, s[2][a][b], aD[a]);
            a2[a] += pg;
            aA[a] = fmaf(pg, s[2][a][b], aA[a]);
            aE[a] = fmaf(pr, s[3][a][b], aE[a]);
            op[0][at] = pr;
            op[1][at] = pg;
          } else {
            const HvpTerms h = hvp_terms(pr, s[2][a][b], s[1][a][b], s[3][a][b], g.scale, rs);
            op[0][at] = h.dS;
            op[1][at] = h.g_S;
            if constexpr (KIND == K_HVP_COL) op[2][at] = h.g_dp;
          }
        }
    }
    __syncthreads();
    auto add = [&](int o, int which, int z) { out_fma<DC, RA>(op[which], strm[z], lay, row0, chunk0, chunks, out[o]); };
    if constexpr (KIND == K_FWD) add(0, 0, 1);                                   // O += P V
    else if constexpr (KIND == K_BWD_ROW) add(0, 0, 0);                          // dQ += dS K
    else if constexpr (KIND == K_BWD_COL) { add(0, 0, 1); add(1, 1, 0); }        // dV += P^T dO; dK += dS^T Q
    else if constexpr (KIND == K_HVP_PRE) {                                      // g_dO' += P g_dV + (P o gdS) V
      add(0, 0, 3); add(0, 1, 1);
      if constexpr (kOwnPV) add(1, 0, 1);                                        // P V
    }
    else if constexpr (KIND == K_HVP_ROW) { add(0, 0, 2); add(0, 1, 0); }        // g_Q += dS g_dK + g_S K
    else { add(0, 0, 2); add(0, 1, 0); add(1, 2, 1); }                           // g_K += dS^T g_dQ + g_S^T Q; g_V += g_dp^T dO
  }
  cp_async_wait_all();                                // a CTA without tiles has its stationary loads in flight
  __syncthreads();

  // ---- results.  Row scalars of the two column halves (and of the other CTAs of the cluster) and
  // the output tiles are combined in the order of the halves and ranks.
  cg::cluster_group cluster = cg::this_cluster();
  float* const partial = strm_base;                   // [kNSums][TS][D] of this CTA, when the cluster has several
  float* const sums = op[0];                          // [2 halves][4][TS] row sums
  if constexpr (KIND == K_FWD || KIND == K_HVP_PRE) {
#pragma unroll
    for (int a = 0; a < RA; ++a) {
      const float v0 = KIND == K_FWD ? m_run[a] : row_sum(aD[a]);
      const float v1 = row_sum(KIND == K_FWD ? l_run[a] : a2[a]);
      const float v2 = row_sum(aA[a]), v3 = row_sum(aE[a]);
      if (tx == 0) {
        float* q = sums + wcol * 4 * TS + row0 + 4 * a;
        q[0] = v0; q[TS] = v1; q[2 * TS] = v2; q[3 * TS] = v3;
      }
    }
  }
  if (split > 1) {
#pragma unroll
    for (int o = 0; o < kNSums; ++o)
#pragma unroll
      for (int a = 0; a < RA; ++a)
#pragma unroll
        for (int c = 0; c < DC; ++c)
          if (chunk0 + 16 * c < chunks)
            reinterpret_cast<float4*>(partial)[(o * TS + row0 + 4 * a) * chunks + chunk0 + 16 * c] =
                make_float4(out[o][a][c][0].x, out[o][a][c][0].y, out[o][a][c][1].x, out[o][a][c][1].y);
    cluster.sync();
  } else {
    __syncthreads();
  }
  // what a row's scalars are after all parts: fwd (max, sum) and the factor of part q; pre (Dv, dot2, dot3)
  auto row_part = [&](int q, int which, int half, int r) {
    const float* base = split > 1 ? cluster.map_shared_rank(sums, q) : sums;
    return base[half * 4 * TS + which * TS + r];
  };
  auto fwd_max = [&](int r) {
    float m = -INFINITY;
    for (int q = 0; q < split; ++q) m = fmaxf(m, row_part(q, 0, 0, r));      // both halves hold the same maximum
    return m;
  };
  auto factor = [&](int q, int r, float m) {
    const float mq = row_part(q, 0, 0, r);
    return mq == -INFINITY ? 0.f : exp2f(mq - m);
  };
  auto row_total = [&](int which, int r) {
    float v = 0.f;
    for (int q = 0; q < split; ++q) v += row_part(q, which, 0, r) + row_part(q, which, 1, r);
    return v;
  };
  if (tid < TS && part == 0 && r0 + tid < g.N_q) {
    if constexpr (KIND == K_FWD) {
      const float m = fwd_max(tid);
      float l = 0.f;
      for (int q = 0; q < split; ++q) l += (row_part(q, 1, 0, tid) + row_part(q, 1, 1, tid)) * factor(q, tid, m);
      t.out_L[row_off + r0 + tid] = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
    } else if constexpr (KIND == K_HVP_PRE) {
      const float D_ = row_total(0, tid), d2_ = row_total(1, tid), A = row_total(2, tid), E = row_total(3, tid);
      t.Dv[row_off + r0 + tid] = D_;
      t.dot2[row_off + r0 + tid] = d2_;
      t.dot3[row_off + r0 + tid] = A - 2.f * D_ * d2_ + E;
    }
  }
  // one float4 of output o, row r (within the tile), given its sum over the parts (and that of P V)
  auto finish = [&](int o, int r, int chunk, float4 v, float4 pv) {
    if (r0 + r >= n_stat) return;
    const size_t at = (size_t)(r0 + r) * D + 4 * chunk;
    float mul = 1.f;
    if constexpr (KIND == K_BWD_ROW || KIND == K_HVP_ROW) mul = g.scale;
    if constexpr (KIND == K_BWD_COL) mul = o == 1 ? g.scale : 1.f;
    if constexpr (KIND == K_HVP_COL) mul = o == 0 ? g.scale : 1.f;
    if constexpr (KIND == K_FWD) {
      const float m = fwd_max(r);
      float l = 0.f;
      for (int q = 0; q < split; ++q) l += (row_part(q, 1, 0, r) + row_part(q, 1, 1, r)) * factor(q, r, m);
      mul = l > 0.f ? 1.f / l : 0.f;
    }
    v = make_float4(v.x * mul, v.y * mul, v.z * mul, v.w * mul);
    if constexpr (KIND == K_HVP_PRE) {
      const float4 of = kOwnPV ? pv : load4(O + at);
      const float dd = row_total(1, r);
      v.x = fmaf(-dd, of.x, v.x); v.y = fmaf(-dd, of.y, v.y); v.z = fmaf(-dd, of.z, v.z); v.w = fmaf(-dd, of.w, v.w);
    }
    T* dst;
    if constexpr (KIND == K_FWD) dst = (T*)t.out_O + q_off;
    else if constexpr (KIND == K_BWD_ROW) dst = (T*)t.out_dQ + q_off;
    else if constexpr (KIND == K_BWD_COL) dst = (T*)(o == 0 ? t.out_dV : t.out_dK) + kv_off;
    else if constexpr (KIND == K_HVP_PRE) dst = (T*)t.out_g_dO + q_off;
    else if constexpr (KIND == K_HVP_ROW) dst = (T*)t.out_g_Q + q_off;
    else dst = (T*)(o == 0 ? t.out_g_K : t.out_g_V) + kv_off;
    store4<T>(dst + at, v);
  };
  if (split > 1) {
    // each CTA of the cluster finishes its share of the float4s, adding the parts in rank order
    const int total = SP::kNOut * TS * chunks;
    for (int i = part * NT + tid; i < total; i += split * NT) {
      const int row = i / chunks, chunk = i - row * chunks, r = row % TS;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f), pv = v;
      float m = 0.f;
      if constexpr (KIND == K_FWD) m = fwd_max(r);
      for (int q = 0; q < split; ++q) {
        if constexpr (kOwnPV) {
          const float4 y = reinterpret_cast<const float4*>(cluster.map_shared_rank(partial, q))[i + TS * chunks];
          pv.x += y.x; pv.y += y.y; pv.z += y.z; pv.w += y.w;
        }
        const float4 x = reinterpret_cast<const float4*>(cluster.map_shared_rank(partial, q))[i];
        const float f = KIND == K_FWD ? factor(q, r, m) : 1.f;
        v.x = fmaf(x.x, f, v.x); v.y = fmaf(x.y, f, v.y); v.z = fmaf(x.z, f, v.z); v.w = fmaf(x.w, f, v.w);
      }
      finish(row / TS, r, chunk, v, pv);
    }
    cluster.sync();                                   // nobody leaves while its shared memory is being read
  } else {
#pragma unroll
    for (int o = 0; o < SP::kNOut; ++o)
#pragma unroll
      for (int a = 0; a < RA; ++a)
#pragma unroll
        for (int c = 0; c < DC; ++c)
          if (chunk0 + 16 * c < chunks) {
            auto sum = [&](int i) { return make_float4(out[i][a][c][0].x, out[i][a][c][0].y, out[i][a][c][1].x, out[i][a][c][1].y); };
            finish(o, row0 + 4 * a, chunk0 + 16 * c, sum(o), sum(kNSums - 1));
          }
  }
  tc::pdl_end(g);
}

template <int KIND, int DC, typename T>
__global__ void __launch_bounds__(threads_of(KIND, DC), DC == 1 ? 2 : 1) attn_simt_kernel(const Geometry g, const Tensors t, const int split) {
  simt_tile<KIND, DC, T>(g, t, split, blockIdx.x);
}

// Two kinds of one operation that do not depend on each other in one grid, the CTAs of FIRST in front: one
// launch less, 1.9 us of the host.
template <int FIRST, int SECOND, int DC, typename T>
__global__ void __launch_bounds__(threads_of(FIRST, DC), DC == 1 ? 2 : 1)
attn_simt_pair_kernel(const Geometry g, const Tensors t, const int split, const int first_ctas) {
  static_assert(threads_of(FIRST, DC) == threads_of(SECOND, DC), "one launch configuration");
  if ((int)blockIdx.x < first_ctas) simt_tile<FIRST, DC, T>(g, t, split, blockIdx.x);
  else simt_tile<SECOND, DC, T>(g, t, split, blockIdx.x - first_ctas);
}

template <int KIND>
static long long units_of(const Geometry& g) { return (long long)g.BH * (((Spec<KIND>::kCol ? g.N_kv : g.N_q) + TS - 1) / TS); }

template <int KIND, int DC, typename T>
static tc::TileKernelState& state_of() {
  static tc::TileKernelState state;
  return state;
}

// the shared memory of the variant's largest D, so that one setting serves every call
template <int KIND, int DC> constexpr size_t kVariantSmem = sizeof(float) * smem_floats<KIND>(64 * DC);

// CTAs of a kind that run at a time in clusters of c on the current device, asked for once
template <int KIND, int DC, typename T>
struct Slots {
  int dev = -1;
  Slots() { if (cudaGetDevice(&dev) != cudaSuccess) dev = -1; }
  int operator()(int c) const {
    if (c == 1) return DC == 1 ? 2 * kSms : kSms;
    return dev < 0 ? 0 : tc::cluster_slots_on(dev, attn_simt_kernel<KIND, DC, T>, c, threads_of(KIND, DC), kVariantSmem<KIND, DC>, state_of<KIND, DC, T>());
  }
};

template <int KIND, int DC, typename T>
static cudaError_t launch_split(const Geometry& g, const Tensors& t, cudaStream_t stream, int split) {
  const long long units = units_of<KIND>(g);
  if (units <= 0) return cudaSuccess;
  if (units * kMaxSplit > 0x7fffffffLL) return cudaErrorInvalidValue;
  auto kern = attn_simt_kernel<KIND, DC, T>;
  const cudaError_t e = tc::set_smem_once(kern, kVariantSmem<KIND, DC>, state_of<KIND, DC, T>().smem_set_split);
  if (e != cudaSuccess) return e;
  return tc::launch_pdl_cluster(kern, (unsigned)(units * split), threads_of(KIND, DC), sizeof(float) * smem_floats<KIND>(g.D), (unsigned)split, stream,
                                g, t, split);
}

template <int KIND, int DC, typename T>
static cudaError_t launch_dc(const Geometry& g, const Tensors& t, cudaStream_t stream) {
  const Splits s = pick_splits(work_of(g, (Kind)KIND, DC == 1), nullptr, DC == 1, false, Slots<KIND, DC, T>());
  return launch_split<KIND, DC, T>(g, t, stream, s.a);
}

template <int KIND, typename T>
static cudaError_t launch_one(const Geometry& g, const Tensors& t, cudaStream_t stream) {
  return g.D <= 64 ? launch_dc<KIND, 1, T>(g, t, stream) : launch_dc<KIND, 2, T>(g, t, stream);
}

template <int FIRST, int SECOND, int DC, typename T>
static cudaError_t launch_pair_dc(const Geometry& g, const Tensors& t, cudaStream_t stream, int split) {
  constexpr auto bytes = [](int D) { return sizeof(float) * (smem_floats<FIRST>(D) > smem_floats<SECOND>(D) ? smem_floats<FIRST>(D) : smem_floats<SECOND>(D)); };
  const long long first = units_of<FIRST>(g) * split, ctas = first + units_of<SECOND>(g) * split;
  if (ctas > 0x7fffffffLL) return cudaErrorInvalidValue;
  auto kern = attn_simt_pair_kernel<FIRST, SECOND, DC, T>;
  static std::atomic<unsigned long long> smem_set{0};
  const cudaError_t e = tc::set_smem_once(kern, bytes(64 * DC), smem_set);
  if (e != cudaSuccess) return e;
  return tc::launch_pdl_cluster(kern, (unsigned)ctas, threads_of(FIRST, DC), bytes(g.D), (unsigned)split, stream, g, t, split, (int)first);
}

// Both kinds, or one of them (`which`: 1 the first, 2 the second, 3 both).  The splits are those of both together in
// either case, so that the phases of a double backward give the bits of a single call.
template <int FIRST, int SECOND, int DC, typename T>
static cudaError_t launch_two_dc(const Geometry& g, const Tensors& t, cudaStream_t stream, int* n, int which) {
  const Work first = work_of(g, (Kind)FIRST, DC == 1), second = work_of(g, (Kind)SECOND, DC == 1);
  const Splits s = pick_splits(first, &second, DC == 1, FIRST == K_HVP_COL, Slots<FIRST, DC, T>());
  if (which == 3 && s.together) {
    ++*n;
    return launch_pair_dc<FIRST, SECOND, DC, T>(g, t, stream, s.a);
  }
  cudaError_t e = cudaSuccess;
  if (which & 1) { e = launch_split<FIRST, DC, T>(g, t, stream, s.a); ++*n; }
  if (e != cudaSuccess || (which & 2) == 0) return e;
  ++*n;
  Geometry second_of = g;
  second_of.beside = which == 3;
  return launch_split<SECOND, DC, T>(second_of, t, stream, s.b);
}

template <int FIRST, int SECOND, typename T>
static cudaError_t launch_two(const Geometry& g, const Tensors& t, cudaStream_t stream, int* n, int which = 3) {
  return g.D <= 64 ? launch_two_dc<FIRST, SECOND, 1, T>(g, t, stream, n, which) : launch_two_dc<FIRST, SECOND, 2, T>(g, t, stream, n, which);
}

template <typename T>
static cudaError_t dispatch(int op, const Geometry& g, const Tensors& t, cudaStream_t s, int* n, int phases) {
  cudaError_t e = cudaSuccess;
  *n = 0;
  auto one = [&](auto kind) {
    constexpr int K = decltype(kind)::value;
    ++*n;
    return launch_one<K, T>(g, t, s);
  };
  if (op == OP_FORWARD) {
    e = one(tc::Int<K_FWD>{});
  } else if (op == OP_BACKWARD) {
    e = launch_two<K_BWD_COL, K_BWD_ROW, T>(g, t, s, n);
  } else {
    // the scalars and both row-side outputs belong to either of their masks, as the C ABI documents it
    const bool row = (phases & (HVP_PHASE_PRE | HVP_PHASE_ROW)) != 0, col = (phases & HVP_PHASE_COL) != 0;
    if (row) e = one(tc::Int<K_HVP_PRE>{});
    if (e == cudaSuccess && (row || col)) e = launch_two<K_HVP_COL, K_HVP_ROW, T>(g, t, s, n, (col ? 1 : 0) | (row ? 2 : 0));
  }
  return e;
}

}  // namespace simt

cudaError_t launch_simt(int op, int dtype, const Geometry& g, const Tensors& t, cudaStream_t s,
                        int* launches, int phases) {
  switch (dtype) {
    case 0: return simt::dispatch<__half>(op, g, t, s, launches, phases);
    case 1: return simt::dispatch<__nv_bfloat16>(op, g, t, s, launches, phases);
    default: return simt::dispatch<float>(op, g, t, s, launches, phases);
  }
}

}  // namespace attn
