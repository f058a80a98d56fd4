// Row-side kernels of the double backward (Hessian-vector product) on sm_100a.
//
// The query side of the HVP needs two [128 x D] fp32 accumulators (g_Q, g_dO).  At
// D = 128 they would fill half of tensor memory.  The work is therefore split over two
// kernels with ONE accumulator each, which leaves 128 columns for the stationary operands:
//
//   ROW_PREDO  per-row scalars Dv, dot2, dot3 (to scratch) and
//                g_dO = P g_dV + (P o gdS) V - dot2 o O
//              (g_dp = P o (gdS - dot2), and P V = O is an input, so the unknown dot2 is
//              applied in the epilogue instead of inside the loop)
//   ROW_Q      g_Q = s (dS g_dK + g_S K), given the scalars
//
// Both stream K, g_dK, V, g_dV in 64-row tiles (three TMA stages, six at D = 64) past 128 stationary
// rows of Q, dO, g_dQ.  Q and dO are copied into TENSOR MEMORY and used from there
// as the A operand of their score products (an A operand in shared memory is re-read by
// every MMA instruction: measured 48 instead of 32 clocks for an N = 64 product); g_dQ
// stays in shared memory.
// Tensor memory:  RA [0,128) = [S | gdS] = [Q K^T | Q g_dK^T + g_dQ K^T];
// RB [128,256) = [dP | gPdV] = dO [V; g_dV]^T;  OUT [256,256+D);  Q at [384,384+D/2),
// dO at [448,448+D/2) (two halves per 32-bit column).  Per tile the math warps run two
// half-steps:
//   half-step 1 reads RA:  p = exp(S - L) and either p*gdS (ROW_PREDO, accumulating dot2)
//               or a = gdS - dot2 (ROW_Q); both are kept in registers and RA is released at once;
//   half-step 2 reads RB:  ROW_PREDO accumulates Dv, A, E (dot3 = A - 2 Dv dot2 + E) and
//               writes the operands P and P o gdS over RB; ROW_Q writes dS = p (dP - Dv) and
//               g_S = p (a (dP - Dv) + gPdV - c3), c3 = dot2 Dv + dot3, over RB.
// Output products take their A operand from RB.  Two warps issue the MMAs, each batch by one
// elected lane inside a single branch: the first warp the RA products of every tile, the second
// the outputs of a tile followed by the RB products of the next (so RB is overwritten only after
// the outputs that read it).  With one issuing warp the latency of each of its waits (about 150
// clocks even when satisfied) fell on an empty tensor pipe.  At D = 64 tensor memory has room for
// a second RB region and the RB products run a tile ahead of the outputs.  The result tile leaves
// through shared memory and a TMA store, which clips rows and columns beyond the tensor.
// Where there are more tiles of queries than SMs the CTAs are persistent (tc_common.cuh) and the stages
// a ring that runs on from one tile of queries to the next: its Q and dO tiles take an entry like a
// streamed tile, and so does its result (the g_dO pass has O loaded there and subtracts in place).  What
// remains of a CTA's fixed cost is the hand-over at the end of an item: B8 H12 N2048 D64 scalar pass 204 ->
// 183 us, g_Q pass 198 -> 179; B4 H16 N1024 D128 87 -> 75 and 82 -> 78; N4096 755 -> 709 (g_Q unchanged).
// Formulas: reference csrc/flash_double_backward_v7.cu:1257-1454.
#include "attn_launch.h"
#include "tc_common.cuh"

namespace attn {
namespace tc {

enum RowMode { ROW_PREDO = 0, ROW_Q = 1 };

constexpr int kRowMmaWarp = 9;
constexpr int kRowThreads = 352;    // 8 math warps, TMA producer, two MMA issuers

constexpr int kRowMaxStages = 6;

struct RowControl {
  WorkControl work;
  uint64_t stat_full;          // g_dQ tile in shared memory
  uint64_t stat_empty;         // the RA products of an item's last tile have read it
  uint64_t stat_tmem_ready;    // Q and dO copied to tensor memory
  // a stage has two halves with their own barriers: [K, g_dK] (index 0) and [V, g_dV] (index 1)
  uint64_t stream_full[2][kRowMaxStages];
  uint64_t stream_empty[2][kRowMaxStages];
  uint64_t ra_full;
  uint64_t ra_free;
  uint64_t rb_full[2];         // per RB buffer
  uint64_t op_full[2];         // per RB buffer: operands of a tile written
  uint64_t acc_done;
  // second issuing warp -> first: the RB products of a tile are queued.  Two barriers used in
  // turn (tile parity): the first warp may fall a whole tile behind the second (it also waits for
  // the [K, g_dK] load), and a single barrier completing twice before it is looked at would show
  // the waited-for parity as pending again.
  uint64_t rb_issued[2];
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
};

static_assert(sizeof(RowControl) <= 512, "control block larger than its slot");

template <int D>
struct RowCfg {
  static constexpr int kAtoms = D / 64;
  static constexpr int kNStream = 4;    // K, g_dK, V, g_dV (pairs back to back)
  // A TMA load takes about 2 000 clocks from request to arrival, whatever its size.  At D = 128
  // a tile takes longer than that and three stages (all that fits) keep the loads ahead; at
  // D = 64 a tile takes about 1 600 clocks and the stages are half the size: six of them.
  static constexpr int kStages = (D == 64) ? 6 : 3;
  static_assert(kStages <= kRowMaxStages, "control block too small");
  static constexpr uint32_t kStatBytes = kAtoms * kAtomBytesStat;            // g_dQ only
  static constexpr uint32_t kStageBytes = kNStream * kAtoms * kAtomBytesStrm;
  static_assert(kStageBytes == 2 * kAtoms * kAtomBytesStat, "Q and dO are staged in one stream stage");
  static constexpr uint32_t kAuxBytes = 512;          // control block
  static constexpr uint32_t kContentBytes = kStatBytes + kStages * kStageBytes + kAuxBytes;
  static constexpr uint32_t kMaxSmem = 232448;
  static_assert(kContentBytes <= kMaxSmem, "shared memory over-subscribed");
  static_assert(kStages * kStageBytes >= BM * D * 4 && kStatBytes >= 13 * BM * 4, "room for a split tile's results");
  static constexpr uint32_t kSmemBytes = (kContentBytes + 1024 <= kMaxSmem) ? kContentBytes + 1024 : kMaxSmem;
  // At D = 64 the accumulator and the stationary operands take half the columns, which leaves
  // room for a second RB region: the RB products then run a tile ahead of the outputs instead of
  // waiting behind them, and the math warps (the bound at D = 64) never wait for RB.
  static constexpr int kRbBufs = (D == 64) ? 2 : 1;
  static constexpr int kRA = 0, kRB = 128, kOut = 128 + 128 * kRbBufs;
  static constexpr int kQT = (D == 64) ? 448 : 384, kDOT = (D == 64) ? 480 : 448;
  static_assert(kOut + D <= kQT && kQT + D / 2 <= kDOT && kDOT + D / 2 <= kTmemCols, "tensor memory over-subscribed");
  __host__ __device__ static constexpr uint32_t stream_off(int slot, int atom) {
    return (uint32_t)(slot >> 1) * (2u * kAtoms * kAtomBytesStrm) + (uint32_t)atom * 2u * kAtomBytesStrm +
           (uint32_t)(slot & 1) * kAtomBytesStrm;
  }
  __host__ __device__ static constexpr int stream_tensor(int slot) {
    return slot == 0 ? T_K : slot == 1 ? T_gK : slot == 2 ? T_V : T_gV;
  }
};

template <int MODE, int D, typename T, bool SPLIT, bool PERSIST>
__global__ void __launch_bounds__(kRowThreads, 1)
hvp_row_kernel(const __grid_constant__ TmaMaps maps, const Geometry g, const Tensors t) {
  using CF = RowCfg<D>;
  constexpr int KIND = (MODE == ROW_PREDO) ? HVP_PRE : HVP_ROW;
  constexpr int kAtoms = CF::kAtoms;
  constexpr uint32_t kIdesc64 = make_idesc(BM, 64, Pack<T>::kIsBf16, 0, 0);
  constexpr uint32_t kIdesc128 = make_idesc(BM, 128, Pack<T>::kIsBf16, 0, 0);

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  {
    uint32_t dyn_size;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_size));
    if (smem_base - smem_u32(smem_raw) + CF::kContentBytes > dyn_size) {   // uniform over the CTA
      if (threadIdx.x == 0 && t.status != nullptr) atomicCAS(t.status, 0u, wait_code(KIND, 15));
      return;
    }
  }
  const uint32_t stat_base = smem_base;
  const uint32_t strm_base = stat_base + CF::kStatBytes;
  const uint32_t aux_off = CF::kStatBytes + CF::kStages * CF::kStageBytes;
  RowControl* ctl = reinterpret_cast<RowControl*>(smem_gen + aux_off);
  // a split tile: over the g_dQ tile, which the last product has read, the row sums' exchange
  // ([2 halves][4][128] floats), this part's four sums per row and the total dot2; its result tile over
  // the stream stages
  float* part_sums = reinterpret_cast<float*>(smem_gen) + 2 * 4 * BM;       // [4][128]
  float* part_dot2 = part_sums + 4 * BM;
  float* partial = reinterpret_cast<float*>(smem_gen + CF::kStatBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = (g.N_q + BM - 1) / BM;
  const unsigned split = SPLIT ? (unsigned)g.split : 1u;      // CTAs that share this tile: a cluster (tc_common.cuh)
  const int part = SPLIT ? (int)(blockIdx.x % split) : 0;
  struct Item { int bh, r0, t_begin, n_iter; };
  auto item_of = [&](int unit) {
    Item w;
    int rank;
    tile_to_head_and_rank(g, (unsigned)unit, tiles, w.bh, rank);
    w.r0 = ((g.mask_mode != 0) ? rank : (tiles - 1 - rank)) * BM;   // heavy tiles first
    int lo, hi;
    key_range_for_queries(g, w.r0, w.r0 + BM, lo, hi);
    w.t_begin = lo / BN;
    w.n_iter = (hi > lo) ? ((hi + BN - 1) / BN - w.t_begin) : 0;
    return w;
  };
  const int first_unit = (int)(blockIdx.x / split);
  Item w = item_of(first_unit);
  // rows that see nothing
  auto write_zeros = [&](const Item& w, int threads) {
    zero_rows(MODE == ROW_PREDO ? t.out_g_dO : t.out_g_Q, w.bh, w.r0, g.N_q, g.D, threads);
    if constexpr (MODE == ROW_PREDO) {
      const int r = w.r0 + threadIdx.x;
      if (threadIdx.x < BM && r < g.N_q) {
        const size_t at = (size_t)w.bh * g.N_q + r;
        t.Dv[at] = t.dot2[at] = t.dot3[at] = 0.f;
      }
    }
  };
  if constexpr (SPLIT) {
    if (w.n_iter == 0) {
      pdl_begin(g);
      pdl_trigger();
      if (part == 0) write_zeros(w, kRowThreads);
      pdl_end(g);
      return;
    }
    take_share((int)split, part, w.t_begin, w.n_iter);      // may be none
  }

  const uint32_t bar_stat_full = smem_u32(&ctl->stat_full);
  const uint32_t bar_stat_empty = smem_u32(&ctl->stat_empty);
  const uint32_t bar_stat_tmem_ready = smem_u32(&ctl->stat_tmem_ready);
  const uint32_t bar_ra_full = smem_u32(&ctl->ra_full), bar_ra_free = smem_u32(&ctl->ra_free);
  auto bar_rb_full = [&](int b) { return smem_u32(&ctl->rb_full[b]); };
  auto bar_op_full = [&](int b) { return smem_u32(&ctl->op_full[b]); };
  const uint32_t bar_acc_done = smem_u32(&ctl->acc_done);
  constexpr int LA = CF::kRbBufs;     // tiles the RB products run ahead of the outputs
  auto bar_rb_issued = [&](int tile) { return smem_u32(&ctl->rb_issued[tile & 1]); };
  auto bar_stream_full = [&](int h, int s) { return smem_u32(&ctl->stream_full[h][s]); };
  auto bar_stream_empty = [&](int h, int s) { return smem_u32(&ctl->stream_empty[h][s]); };

  // The ring of stages.  Every item takes an entry for its Q and dO tiles (halves 0 and 1, copied to
  // tensor memory by the math warps and free again when they have said so), one for each of its tiles,
  // and one through which its result leaves (half 0; the g_dO pass first receives O there).  Entries are
  // numbered over all items of the CTA.
  constexpr int S = CF::kStages;
  auto slot_base = [&](int c) { return strm_base + (uint32_t)(c % S) * CF::kStageBytes; };
  constexpr uint32_t kHalfBytes = CF::kStageBytes / 2;
  auto entries = [](const Item& w) { return w.n_iter > 0 ? w.n_iter + (SPLIT ? 1 : 2) : 0; };
  auto load_rows128 = [&](uint32_t dst, int tensor, const Item& w, uint32_t bar) {      // a [128][D] tile of the query side
#pragma unroll
    for (int a = 0; a < kAtoms; ++a)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        tma_load_3d(dst + a * kAtomBytesStat + h * kAtomBytesStrm, &maps.m[tensor], a * 64, w.r0 + h * 64, w.bh, bar);
  };
  auto load_stationary = [&](const Item& w, int c) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mbar_arrive_expect_tx(bar_stream_full(h, c % S), kHalfBytes);
      load_rows128(slot_base(c) + h * kHalfBytes, h == 0 ? T_Q : T_dO, w, bar_stream_full(h, c % S));
    }
  };
  auto load_tile_half = [&](const Item& w, int it, int h, int c) {
    mbar_arrive_expect_tx(bar_stream_full(h, c % S), kHalfBytes);
#pragma unroll
    for (int s2 = 0; s2 < 2; ++s2)
#pragma unroll
      for (int a = 0; a < kAtoms; ++a)
        tma_load_3d(slot_base(c) + CF::stream_off(2 * h + s2, a), &maps.m[CF::stream_tensor(2 * h + s2)], a * 64, (w.t_begin + it) * BN,
                    w.bh, bar_stream_full(h, c % S));
  };
  auto load_gdq = [&](const Item& w) {
    mbar_arrive_expect_tx(bar_stat_full, CF::kStatBytes);
    load_rows128(stat_base, T_gQ, w, bar_stat_full);
  };

  // one barrier round of set-up: the producer initialises the mbarriers and, once the kernels this
  // one depends on are complete, requests the stationary tiles and the first streamed tile (their
  // latency is the longest item of the prologue); meanwhile an issuing warp allocates tensor memory
  if (warp == kProducerWarp && lane == 0) {
    for (int i = 0; i < T_COUNT; ++i) tma_prefetch_desc(&maps.m[i]);
    work_init(&ctl->work);
    mbar_init(bar_stat_full, 1);
    mbar_init(bar_stat_empty, 1);
    mbar_init(bar_stat_tmem_ready, kMathWarps);
    for (int s = 0; s < S; ++s) {
      for (int h = 0; h < 2; ++h) {
        mbar_init(bar_stream_full(h, s), 1);
        mbar_init(bar_stream_empty(h, s), 1);
      }
    }
    mbar_init(bar_ra_full, 1);
    mbar_init(bar_ra_free, kMathWarps);
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_rb_full(b), 1);
      mbar_init(bar_op_full(b), kMathWarps);
    }
    mbar_init(bar_acc_done, 1);
    mbar_init(bar_rb_issued(0), 1);
    mbar_init(bar_rb_issued(1), 1);
    ctl->abort_flag = 0u;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == kRowMmaWarp) tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols);
  pdl_begin(g);
  if (warp == kProducerWarp && lane == 0) {
    pdl_trigger();
    if (w.n_iter > 0) {
      load_stationary(w, 0);
      load_tile_half(w, 0, 0, 1);
      load_tile_half(w, 0, 1, 1);
      load_gdq(w);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile uint32_t* abort_flag = &ctl->abort_flag;

  // =========================================================================
  // TMA producer
  // =========================================================================
  if (warp == kProducerWarp) {
    if (lane == 0) {
      bool ok = true;
      int c0 = 0, items = 0;        // ring entries and items with tiles before this item
      auto wait_half = [&](int h, int c) {
        return mbar_wait(bar_stream_empty(h, c % S), ((c / S) & 1) ^ 1, abort_flag, t.status, wait_code(KIND, 1));
      };
      for (int k = 0; ok; ++k) {
        int asked = 0;
        if (w.n_iter > 0) {
          if (k > 0) {
            ok = wait_half(0, c0) && wait_half(1, c0);
            if (!ok) break;
            load_stationary(w, c0);
          }
          // The two halves of an entry are released at different times: [K, g_dK] is last read by the RA
          // products in the scalar pass (long before the outputs of the tile), [V, g_dV] by the RB
          // products in the g_Q pass.  Each half is requested as soon as its own buffer is free, so the
          // loads the first issuing warp waits for leave a tile earlier than a whole-stage release would
          // allow (a load takes about as long as a tile).
          for (int it = k > 0 ? 0 : 1; it < w.n_iter && ok; ++it) {     // the first item's first tile was requested above
            const int c = c0 + 1 + it;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (ok) ok = wait_half(h, c);
              if (ok) load_tile_half(w, it, h, c);
            }
            if (ok && it == 0) {
              ok = mbar_wait(bar_stat_empty, (items & 1) ^ 1, abort_flag, t.status, wait_code(KIND, 1));
              if (ok) load_gdq(w);
            }
            if (PERSIST && asked == 0 && it + 3 >= w.n_iter) { work_request(&ctl->work); asked = 1; }
          }
          if (!SPLIT && ok) {       // the entry of the result
            const int c = c0 + 1 + w.n_iter;
            ok = wait_half(0, c) && wait_half(1, c);
            if (!ok) break;
            if constexpr (MODE == ROW_PREDO) {
              mbar_arrive_expect_tx(bar_stream_full(0, c % S), kHalfBytes);
              load_rows128(slot_base(c), T_O, w, bar_stream_full(0, c % S));
            } else {
              mbar_arrive(bar_stream_full(0, c % S));
            }
            mbar_arrive(bar_stream_full(1, c % S));
          }
          if (!ok) break;
          ++items;
        }
        if (!PERSIST) break;
        if (asked == 0) work_request(&ctl->work);
        int unit;
        c0 += entries(w);
        ok = work_announce(&ctl->work, k, &unit, abort_flag, t.status, wait_code(KIND, 10));
        if (!ok || unit < 0) break;
        w = item_of(unit);
      }
      if (!ok) {   // give copies already in flight a bounded chance to land before the CTA exits
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) { }
      }
    }
  }
  // =========================================================================
  // MMA issuers (converged warps, one elected lane issues)
  // =========================================================================
  else if (warp == kRowMmaWarp || warp == kRowMmaWarp + 1) {
    {
      bool ok = true;
      const uint64_t d_stat = smem_desc_sw128(stat_base, 16, 1024);
      auto gq_desc = [&](int ks) {   // K-major A from shared memory: the g_dQ tile
        return d_stat + (uint64_t)(((ks >> 2) * kAtomBytesStat + (ks & 3) * 32) >> 4);
      };
      // descriptor offsets (16-byte units) within a stage: K-major B, k-step ks of slot; MN-major B,
      // 16 rows per k-step
      auto koff = [](int slot, int ks) { return (uint64_t)((CF::stream_off(slot, ks >> 2) + (ks & 3) * 32) >> 4); };
      auto moff = [](int slot, int ks) { return (uint64_t)((CF::stream_off(slot, 0) + ks * 2048) >> 4); };
      // operand written by the math warps over a 64-column score slot: the 16 elements of
      // k-step ks sit in 8 columns at 32*(ks/2) + 8*(ks%2) (owner half, then chunk)
      auto op_tmem = [&](int col0, int ks) { return tmem_base + (uint32_t)(col0 + 32 * (ks >> 1) + 8 * (ks & 1)); };
      auto commit = [&](uint32_t bar) { if (elect_one()) mma_commit(bar); };
      constexpr int KS = D / 16, KO = BN / 16;
      // a head dimension below the tile width: skip the k-steps and output columns that are padding
      const int ks_n = g.D >> 4;
      const uint32_t idesc_out = make_idesc(BM, g.D, Pack<T>::kIsBf16, 0, 1);
      const uint32_t out = tmem_base + CF::kOut;
      const uint32_t ra = tmem_base + CF::kRA, rb = tmem_base + CF::kRB;
      const uint32_t qt = tmem_base + CF::kQT, dot = tmem_base + CF::kDOT;

      // Every batch of products is issued by the elected lane inside one branch, with the
      // descriptor of the stage built once: the instruction stream between two MMAs is an add.
      // The RA batch goes out in two elected branches, the last kTail k-steps and the commit in the
      // second: the short gap lets the other issuing warp's products into the queue in between.  The
      // scalar pass takes 20 % more cycles when the whole batch is issued in one branch, 35 % more when it
      // waits in the gap for the other warp's, and 5 % more at D = 80 and 96 with kTail = 2, where the
      // second branch is left with padding steps only.
      constexpr int kTail = (D == 128) ? (MODE == ROW_PREDO ? 5 : 2) : 0;
      auto issue_ra = [&](uint32_t stage) {           // ends with the commit of the batch
        const uint64_t dk = smem_desc_sw128(stage, 16, 1024);
        if (elect_one()) {
          _Pragma("unroll") for (int ks = 0; ks < KS; ++ks)
            if (ks < ks_n) mma_ts(ra, qt + 8 * ks, dk + koff(0, ks), kIdesc128, ks > 0);
          _Pragma("unroll") for (int ks = 0; ks < KS - kTail; ++ks)
            if (ks < ks_n) mma_ss(ra + 64, gq_desc(ks), dk + koff(0, ks), kIdesc64, 1);
        }
        __syncwarp();
        if (elect_one()) {
          _Pragma("unroll") for (int ks = KS - kTail; ks < KS; ++ks)
            if (ks < ks_n) mma_ss(ra + 64, gq_desc(ks), dk + koff(0, ks), kIdesc64, 1);
          mma_commit(bar_ra_full);
        }
        __syncwarp();
      };
      auto issue_rb = [&](uint32_t stage, int b) {    // into RB buffer b; ends with its commit
        const uint64_t dk = smem_desc_sw128(stage, 16, 1024);
        const uint32_t acc = rb + 128u * (uint32_t)b;
        if (elect_one()) {
          _Pragma("unroll") for (int ks = 0; ks < KS; ++ks)
            if (ks < ks_n) mma_ts(acc, dot + 8 * ks, dk + koff(2, ks), kIdesc128, ks > 0);
          mma_commit(bar_rb_full(b));
        }
        __syncwarp();
      };
      auto issue_out = [&](uint32_t stage, bool first, int b) {   // operands in RB buffer b
        const uint64_t dm = smem_desc_sw128(stage, 2u * kAtomBytesStrm, 1024);
        constexpr int s0 = (MODE == ROW_PREDO) ? 3 : 1;     // g_dO' += P g_dV      | g_Q += dS g_dK
        constexpr int s1 = (MODE == ROW_PREDO) ? 2 : 0;     // g_dO' += (P o gdS) V | g_Q += g_S K
        if (elect_one()) {
          _Pragma("unroll") for (int ks = 0; ks < KO; ++ks)
            mma_ts(out, op_tmem(CF::kRB + 128 * b, ks), dm + moff(s0, ks), idesc_out, !(first && ks == 0));
          _Pragma("unroll") for (int ks = 0; ks < KO; ++ks)
            mma_ts(out, op_tmem(CF::kRB + 128 * b + 64, ks), dm + moff(s1, ks), idesc_out, 1);
        }
        __syncwarp();
      };

      // Two issuing warps, so that the latency of one warp's waits falls while the products of the
      // other are queued.  The tensor pipe needs no order between the two streams: RA(j+1) only
      // waits for RA(j) to have been read, and RB(j+1) follows OUT(j), which reads RB, in the
      // second warp's own order.
      auto wait_entry = [&](int h, int c) {   // half h of ring entry c has landed
        return mbar_wait(bar_stream_full(h, c % S), (c / S) & 1, abort_flag, t.status, wait_code(KIND, 3));
      };
      // which issuing warp releases which half: the one whose products read it last
      constexpr bool kRaReleasesKG = (MODE == ROW_PREDO);   // scalar pass: the outputs read V, g_dV only
      // Either warp's walk over the items: body(tiles, ring entry of the first tile, number of the first tile)
      auto walk = [&](auto role, auto&& body) {
        constexpr int kRole = decltype(role)::value;
        int c0 = 0, g0 = 0, items = 0;      // ring entries, tiles and items with tiles before this item
        for (int k = 0; ok; ++k) {
          if (w.n_iter > 0) {
            ok = mbar_wait(bar_stat_tmem_ready, items & 1, abort_flag, t.status, wait_code(KIND, 11));
            if (ok && kRole == 0) ok = mbar_wait(bar_stat_full, items & 1, abort_flag, t.status, wait_code(KIND, 2));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            if (lane == 0) mbar_arrive(bar_stream_empty(kRole, c0 % S));     // Q (first warp) and dO (second) are in tensor memory
            body(w.n_iter, c0 + 1, g0);
            g0 += w.n_iter;
            ++items;
          }
          if (!PERSIST || !ok) break;
          c0 += entries(w);
          int unit;
          ok = work_next(&ctl->work, k, &unit, abort_flag, t.status, wait_code(KIND, 14));
          if (!ok || unit < 0) break;
          w = item_of(unit);
        }
      };
      if (warp == kRowMmaWarp) {
        // ---- first warp: the RA products of every tile
        walk(Int<0>{}, [&](int n, int c1, int g0) {
          for (int j = 0; j < n && ok; ++j) {
            const int gj = g0 + j, c = c1 + j;
            ok = wait_entry(0, c);
            if (ok && gj > 0) ok = mbar_wait(bar_ra_free, (gj - 1) & 1, abort_flag, t.status, wait_code(KIND, 4));
            // ROW_Q keeps the pipe's order OUT(j-2), RB(j-1), RA(j): its second half-step is the long
            // one, and RA(j) queued any earlier delays the outputs that half-step waits behind.  The
            // scalar pass is faster with the two streams left to run freely (both measured).
            if (MODE == ROW_Q && LA == 1 && ok && gj > 0) ok = mbar_wait(bar_rb_issued(gj - 1), ((gj - 1) >> 1) & 1, abort_flag, t.status, wait_code(KIND, 13));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            issue_ra(slot_base(c));
            if (kRaReleasesKG) commit(bar_stream_empty(0, c % S));
          }
          if (ok) commit(bar_stat_empty);
        });
      } else {
        // ---- second warp: RB products (LA tiles ahead) and outputs
        walk(Int<1>{}, [&](int n, int c1, int g0) {
          for (int i = 0; i < LA && i < n && ok; ++i) {
            const int c = c1 + i;
            ok = wait_entry(1, c);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            issue_rb(slot_base(c), (g0 + i) % LA);
            if (!kRaReleasesKG) commit(bar_stream_empty(1, c % S));
            if (LA == 1 && lane == 0) mbar_arrive(bar_rb_issued(g0 + i));
          }
          for (int j = 0; j < n && ok; ++j) {
            const int gj = g0 + j, b = gj % LA, c = c1 + j, nc = c + LA;
            const bool more = j + LA < n;
            ok = mbar_wait(bar_op_full(b), (gj / LA) & 1, abort_flag, t.status, wait_code(KIND, 6));
            if (ok && more) ok = wait_entry(1, nc);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            issue_out(slot_base(c), j == 0, b);
            commit(bar_stream_empty(kRaReleasesKG ? 1 : 0, c % S));   // the half the outputs read
            if (more) {
              // buffer b again: after the outputs that read it, in this warp's own order
              issue_rb(slot_base(nc), b);
              if (!kRaReleasesKG) commit(bar_stream_empty(1, nc % S));
              if (LA == 1 && lane == 0) mbar_arrive(bar_rb_issued(gj + LA));
            }
          }
          if (ok) commit(bar_acc_done);
        });
      }
    }
  }
  // =========================================================================
  // math warps
  // =========================================================================
  else {
    const int quarter = warp & 3, half = warp >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    bool ok = true;
    int c0 = 0, g0 = 0, items = 0;      // ring entries, tiles and items with tiles before this item
    for (int k = 0; ok; ++k) {
    const int n_iter = w.n_iter, t_begin = w.t_begin, bh = w.bh, r0 = w.r0;
    if (!SPLIT && n_iter == 0) {
      write_zeros(w, kMathThreads);
    } else {
    const int gidx = r0 + row;
    const size_t row_off = (size_t)bh * g.N_q;
    // where the result leaves: its ring entry (a split tile has no such entry and does not use it)
    const int c_out = c0 + 1 + n_iter;
    const uint32_t out_tile = slot_base(c_out);
    float* row_sums = SPLIT ? reinterpret_cast<float*>(smem_gen)
                            : reinterpret_cast<float*>(smem_gen + (out_tile - smem_base) + kHalfBytes);    // the entry's other half
    (void)row_sums; (void)out_tile;

    int vlo, vhi;
    key_range_for_queries(g, gidx, gidx + 1, vlo, vhi);
    if (gidx >= g.N_q) { vlo = 0; vhi = 0; }
    const uint32_t vspan = (uint32_t)(vhi - vlo);

    // scalars of this thread's query row, negated so that every use is a packed add / fma
    float2 nL2 = make_float2(-INFINITY, -INFINITY), nDv = make_float2(0.f, 0.f);
    float2 nD2 = make_float2(0.f, 0.f), nC3 = make_float2(0.f, 0.f);
    if (gidx < g.N_q) {
      const float L2 = from_l2(t.L + row_off + gidx) * kLog2e;
      nL2 = make_float2(-L2, -L2);
      if constexpr (MODE == ROW_Q) {
        const float Dv = from_l2(t.Dv + row_off + gidx), d2 = from_l2(t.dot2 + row_off + gidx);
        const float c3 = fmaf(d2, Dv, from_l2(t.dot3 + row_off + gidx));
        nDv = make_float2(-Dv, -Dv); nD2 = make_float2(-d2, -d2); nC3 = make_float2(-c3, -c3);
      }
    }
    const float2 sl2 = make_float2(g.scale_log2e, g.scale_log2e);
    const float2 sc2 = make_float2(g.scale, g.scale);
    const float2 zero2 = make_float2(0.f, 0.f);

    // ---- copy of the stationary Q and dO rows from their ring entry to tensor memory.
    // Tile layout in shared memory: per 64-column atom, row r at r*128 bytes with its 16-byte
    // chunks XOR-swizzled by r % 8.  Tensor-memory layout of an A operand: lane = row, one
    // 32-bit column per pair of consecutive K elements.  This thread moves its row's half.
    if (n_iter > 0) {
      const uint32_t staging = slot_base(c0);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (ok) ok = mbar_wait(bar_stream_full(h, c0 % S), (c0 / S) & 1, abort_flag, t.status, wait_code(KIND, 12));
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        constexpr int kChunksPerHalf = D / 16;    // 16-byte chunks (8 halves) of this thread's half row
#pragma unroll
        for (int x = 0; x < 2; ++x) {             // 0: Q, 1: dO
          const uint32_t src = staging + x * kHalfBytes;
          const uint32_t dst = lane_addr + (x == 0 ? CF::kQT : CF::kDOT);
#pragma unroll
          for (int c = 0; c < kChunksPerHalf; c += 2) {
            uint32_t w[8];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int gc = half * kChunksPerHalf + c + u;   // chunk index within the row
              const uint32_t addr = src + (gc >> 3) * kAtomBytesStat + row * 128 + ((((uint32_t)(gc & 7)) ^ (row & 7)) << 4);
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(w[4 * u]), "=r"(w[4 * u + 1]), "=r"(w[4 * u + 2]), "=r"(w[4 * u + 3])
                           : "r"(addr));
            }
            tmem_st8(dst + 4 * (half * kChunksPerHalf + c), w);
          }
        }
        tmem_st_wait();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_stat_tmem_ready);
    }

    float2 p_[16], a_[16];   // carried from half-step 1 to half-step 2 (ROW_PREDO: a_ = p * gdS)
    float2 acc_D = zero2, acc_2 = zero2, acc_A = zero2, acc_E = zero2;   // ROW_PREDO row sums
    const uint32_t ra = lane_addr + CF::kRA;
    for (int it = 0; it < n_iter && ok; ++it) {
      const int gi = g0 + it;
      const uint32_t rb = lane_addr + CF::kRB + 128u * (uint32_t)(gi % LA);
      const int j0 = (t_begin + it) * BN;
      const int first = j0 + half * 32;
      const bool masked = !(first >= vlo && first + 31 < vhi);

      // ---------------- half-step 1: RA ------------------------------------------
      ok = mbar_wait(bar_ra_full, gi & 1, abort_flag, t.status, wait_code(KIND, 7));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      // Read this thread's 2 x 32 columns of RA in one go and release the region before the
      // arithmetic: the next tile's RA products are what the math warps wait for next.
      uint32_t s_[2][16], g_[2][16];
      tmem_ld16(ra + half * 32, s_[0]);
      tmem_ld16(ra + half * 32 + 16, s_[1]);
      tmem_ld16(ra + 64 + half * 32, g_[0]);
      tmem_ld16(ra + 64 + half * 32 + 16, g_[1]);
      tmem_ld_wait(s_[0]);
      tmem_ld_wait(s_[1]);
      tmem_ld_wait(g_[0]);
      tmem_ld_wait(g_[1]);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ra_free);
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        const int c0 = half * 32 + ch * 16;
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
          const int cc = c0 + e;
          const float2 x = __ffma2_rn(make_float2(__uint_as_float(s_[ch][e]), __uint_as_float(s_[ch][e + 1])), sl2, nL2);
          float2 pp = make_float2(ex2(x.x), ex2(x.y));
          if (masked) {
            pp.x = ((uint32_t)(j0 + cc - vlo) < vspan) ? pp.x : 0.f;
            pp.y = ((uint32_t)(j0 + cc + 1 - vlo) < vspan) ? pp.y : 0.f;
          }
          const float2 gg = make_float2(__uint_as_float(g_[ch][e]), __uint_as_float(g_[ch][e + 1]));
          p_[ch * 8 + (e >> 1)] = pp;
          if constexpr (MODE == ROW_PREDO) {
            const float2 pg = __fmul2_rn(pp, __fmul2_rn(gg, sc2));     // p * gdS
            a_[ch * 8 + (e >> 1)] = pg;
            acc_2 = __fadd2_rn(acc_2, pg);
          } else {
            a_[ch * 8 + (e >> 1)] = __ffma2_rn(gg, sc2, nD2);           // gdS - dot2
          }
        }
      }

      // ---------------- half-step 2: RB ------------------------------------------
      ok = mbar_wait(bar_rb_full(gi % LA), (gi / LA) & 1, abort_flag, t.status, wait_code(KIND, 8));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        const int c0 = half * 32 + ch * 16;
        uint32_t dp_[16], gp_[16];
        tmem_ld16(rb + c0, dp_);
        tmem_ld16(rb + 64 + c0, gp_);
        tmem_ld_wait(dp_);
        tmem_ld_wait(gp_);
        uint32_t k0[8], k1[8];
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
          const float2 pp = p_[ch * 8 + (e >> 1)], aa = a_[ch * 8 + (e >> 1)];
          const float2 dp = make_float2(__uint_as_float(dp_[e]), __uint_as_float(dp_[e + 1]));
          const float2 gp = make_float2(__uint_as_float(gp_[e]), __uint_as_float(gp_[e + 1]));
          if constexpr (MODE == ROW_PREDO) {
            acc_D = __ffma2_rn(pp, dp, acc_D);
            acc_A = __ffma2_rn(aa, dp, acc_A);
            acc_E = __ffma2_rn(pp, gp, acc_E);
            k0[e >> 1] = Pack<T>::pack(pp.x, pp.y);      // P
            k1[e >> 1] = Pack<T>::pack(aa.x, aa.y);      // P o gdS
          } else {
            const float2 dpd = __fadd2_rn(dp, nDv);
            const float2 ds = __fmul2_rn(pp, dpd);
            const float2 gs = __fmul2_rn(pp, __ffma2_rn(aa, dpd, __fadd2_rn(gp, nC3)));
            k0[e >> 1] = Pack<T>::pack(ds.x, ds.y);      // dS
            k1[e >> 1] = Pack<T>::pack(gs.x, gs.y);      // g_S
          }
        }
        // over columns this thread has just read (first half of its dP and gPdV ranges)
        tmem_st8(rb + half * 32 + ch * 8, k0);
        tmem_st8(rb + 64 + half * 32 + ch * 8, k1);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_op_full(gi % LA));
    }

    // ---------------- results ------------------------------------------------------
    float dot2_row = 0.f;
    if constexpr (!SPLIT) {       // the ring entry of the result is free, in the g_dO pass with O in it
      if (ok) ok = mbar_wait(bar_stream_full(0, c_out % S), (c_out / S) & 1, abort_flag, t.status, wait_code(KIND, 12));
      ok = __all_sync(0xffffffffu, ok);
    }
    if constexpr (MODE == ROW_PREDO) {
      // each row is summed by two threads (column halves): exchange through shared memory
      float* mine = row_sums + half * 512;
      const float sD = acc_D.x + acc_D.y, s2 = acc_2.x + acc_2.y, sA = acc_A.x + acc_A.y, sE = acc_E.x + acc_E.y;
      mine[row] = sD; mine[128 + row] = s2; mine[256 + row] = sA; mine[384 + row] = sE;
      named_barrier_sync(1, kMathThreads);
      const float* other = row_sums + (half ^ 1) * 512;
      const float Dv = sD + other[row], d2 = s2 + other[128 + row];
      const float A = sA + other[256 + row], E = sE + other[384 + row];
      dot2_row = d2;
      if constexpr (SPLIT) {
        if (half == 0) { part_sums[row] = Dv; part_sums[BM + row] = d2; part_sums[2 * BM + row] = A; part_sums[3 * BM + row] = E; }
      } else if (half == 0 && gidx < g.N_q) {
        t.Dv[row_off + gidx] = Dv;
        t.dot2[row_off + gidx] = d2;
        t.dot3[row_off + gidx] = A - 2.f * Dv * d2 + E;
      }
    }
    constexpr int kColsPerHalf = D / 2;
    constexpr int kChunks = kColsPerHalf / 16;
    const float mul = (MODE == ROW_PREDO) ? 1.f : g.scale;
    if (n_iter > 0 && ok) ok = mbar_wait(bar_acc_done, items & 1, abort_flag, t.status, wait_code(KIND, 9));
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after_sync();
    // all accumulator columns of this thread first, then the arithmetic and the stores
    uint32_t v[kChunks][16];
#pragma unroll
    for (int ch = 0; ch < kChunks; ++ch) {
      if (n_iter > 0 && ok) {
        tmem_ld16(lane_addr + CF::kOut + half * kColsPerHalf + ch * 16, v[ch]);
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[ch][e] = 0u;
      }
    }
    if (n_iter > 0 && ok) {
#pragma unroll
      for (int ch = 0; ch < kChunks; ++ch) tmem_ld_wait(v[ch]);
    }
#pragma unroll
    for (int ch = 0; ch < kChunks; ++ch) {
      if (half * kColsPerHalf + ch * 16 >= g.D) break;   // padding columns (uniform over the warp)
      if (gidx < g.N_q) {
        float f[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) f[e] = __uint_as_float(v[ch][e]) * mul;
        const int col = half * kColsPerHalf + ch * 16;
        if constexpr (SPLIT) {      // dot2 is not known yet
          store_partial16<D>(partial, row, col, f);
        } else {
          const uint32_t tile = out_tile + (uint32_t)(col >> 6) * kAtomBytesStat;
          if constexpr (MODE == ROW_PREDO) {      // g_dO = g_dO' - dot2 * O, whose element is where the result goes
            uint32_t ow[8];
            load_op16(tile, row, col & 63, ow);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float2 of = Pack<T>::unpack(ow[e]);
              f[2 * e] = fmaf(-dot2_row, of.x, f[2 * e]);
              f[2 * e + 1] = fmaf(-dot2_row, of.y, f[2 * e + 1]);
            }
          }
          uint32_t w[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) w[e] = Pack<T>::pack(f[2 * e], f[2 * e + 1]);
          store_op16(tile, row, col & 63, w);
        }
      }
    }
    if constexpr (!SPLIT) {
      store_tile_tma(&maps.out[MODE == ROW_PREDO ? TO_gdO : TO_gQ], out_tile, g.D, r0, bh, threadIdx.x == 0);
      if (threadIdx.x == 0) {
        mbar_arrive(bar_stream_empty(0, c_out % S));
        mbar_arrive(bar_stream_empty(1, c_out % S));
      }
    }
    g0 += n_iter;
    ++items;
    }
    if (!PERSIST || !ok) break;
    c0 += entries(w);
    int unit;
    ok = work_next(&ctl->work, k, &unit, abort_flag, t.status, wait_code(KIND, 14));
    if (!ok || unit < 0) break;
    w = item_of(unit);
    }
  }

  if constexpr (SPLIT) {
    cluster_barrier();
    if (warp < kMathWarps) {
      if constexpr (MODE == ROW_PREDO) {
        if (threadIdx.x < BM) {
          cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
          float sum[4] = {0.f, 0.f, 0.f, 0.f};
          for (int q = 0; q < (int)split; ++q) {
            const float* theirs = cluster.map_shared_rank(part_sums, q);
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[i] += theirs[i * BM + threadIdx.x];
          }
          part_dot2[threadIdx.x] = sum[1];
          if (part == 0 && w.r0 + threadIdx.x < g.N_q) {
            const size_t at = (size_t)w.bh * g.N_q + w.r0 + threadIdx.x;
            t.Dv[at] = sum[0];
            t.dot2[at] = sum[1];
            t.dot3[at] = sum[2] - 2.f * sum[0] * sum[1] + sum[3];
          }
        }
        named_barrier_sync(1, kMathThreads);
      }
      const size_t at = ((size_t)w.bh * g.N_q + w.r0) * g.D;
      const T* O_rows = (const T*)t.O + at;
      reduce_parts<D, T>(partial, (int)split, part, (T*)(MODE == ROW_PREDO ? t.out_g_dO : t.out_g_Q) + at, min(BM, g.N_q - w.r0), g.D,
                         [](int, int) { return 1.f; },
                         [&](int row, int col, float4& v) {
                           if constexpr (MODE == ROW_PREDO) {
                             const uint2 w = *reinterpret_cast<const uint2*>(O_rows + (size_t)row * g.D + col);
                             const float2 a = Pack<T>::unpack(w.x), b = Pack<T>::unpack(w.y);
                             const float d = -part_dot2[row];
                             v.x = fmaf(d, a.x, v.x); v.y = fmaf(d, a.y, v.y); v.z = fmaf(d, b.x, v.z); v.w = fmaf(d, b.y, v.w);
                           }
                         });
    }
    cluster_barrier();      // nobody leaves while its shared memory is being read
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kRowMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if constexpr (PERSIST) pdl_end_persistent(g);
  else pdl_end(g);
}

template <int MODE, int D, typename T>
static cudaError_t launch_row(const TmaMaps& maps, const Geometry& g_in, const Tensors& t, cudaStream_t s) {
  using CF = RowCfg<D>;
  Geometry g = g_in;
  const long long units = (long long)g.BH * ((g.N_q + BM - 1) / BM);
  g.head_group = pick_head_group(units, g.BH, 4ll * g.N_kv * g.D * 2);   // K, g_dK, V, g_dV
  // Persistent where there are more tiles of queries than SMs, long ones too: double backward, persistent
  // and not, 691 / 705 us at B8 H12 N2048 D64, 74.5 / 77 at N512, 233 / 238 at B4 H16 N1024 D128, 1034 / 1041 in
  // chunks of 1024 queries and 9216 keys (H32 D80, 121 tiles each), 728 / 725 at 5120 keys (B2 H16 D128).
  static TileKernelState states[2];
  TileKernelState& state = states[units > kSms];
  const auto whole = units > kSms ? hvp_row_kernel<MODE, D, T, false, true> : hvp_row_kernel<MODE, D, T, false, false>;
  return launch_tiles(whole, hvp_row_kernel<MODE, D, T, true, false>, maps, g, t, s, false, kRowThreads, CF::kSmemBytes,
                      2000.f, MODE == ROW_Q ? 2700.f : 0.f, state);
}

// mode 0: per-row scalars + g_dO;  mode 1: g_Q
cudaError_t launch_hvp_row(int mode, int D, int is_bf16, const TmaMaps& maps, const Geometry& g,
                           const Tensors& t, cudaStream_t s) {
  if (mode == 0) {
    if (D <= 64) return is_bf16 ? launch_row<ROW_PREDO, 64, __nv_bfloat16>(maps, g, t, s) : launch_row<ROW_PREDO, 64, __half>(maps, g, t, s);
    return is_bf16 ? launch_row<ROW_PREDO, 128, __nv_bfloat16>(maps, g, t, s) : launch_row<ROW_PREDO, 128, __half>(maps, g, t, s);
  }
  if (D <= 64) return is_bf16 ? launch_row<ROW_Q, 64, __nv_bfloat16>(maps, g, t, s) : launch_row<ROW_Q, 64, __half>(maps, g, t, s);
  return is_bf16 ? launch_row<ROW_Q, 128, __nv_bfloat16>(maps, g, t, s) : launch_row<ROW_Q, 128, __half>(maps, g, t, s);
}

}  // namespace tc
}  // namespace attn
