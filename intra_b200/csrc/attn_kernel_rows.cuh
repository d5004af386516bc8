// The attention kernel for every shape whose tiles are TMA boxes (tma_maps.h). Persistent: each CTA owns
// one SM and walks a static list of pair tiles (intra_index.h): two 128-row query sub-tiles that share
// every K / V tile brought into shared memory or (Gather-0) share those of the text only.
//
// Warp roles (512 threads):
//   warps 0-3, 4-7    softmax sets of sub-tile 0 and 1: a thread owns a query row. A set copies its scores out
//                     of the one score buffer, hands the buffer back at once and has a whole key-tile period
//                     for its phase while the other set's phase runs beside it
//   warps 8-11        epilogue: O of a finished item -> bf16 -> global while the sets are on the next item
//   warp 12           issues QK0(j) QK1(j) over the CTA's key tiles j into the shared score buffer
//   warp 13           one thread requests the Q and K tiles (bulk-tensor copies)
//   warp 14           planner: decodes the CTA's items a batch ahead into shared memory; requests the V tiles (one
//                     thread for K and V would hold up the next item's first K behind the last V's buffer)
//   warp 15           issues PV0(j) PV1(j) as the sets deliver P (a tcgen05.mma issue blocks its thread once
//                     ~5 MMAs are queued, so one warp for both kinds would let the queue drain in its waits)
// TMEM: scores cols 0-127 | P0 128-191 | P1 192-255 | O0 256-383 | O1 384-511.
//
// What the code is written for, besides the pipes, is the instruction cache: all roles run different code at
// the same time, and an earlier version of this kernel that was one body for all patterns (109 KB) spent a
// fifth to a third of its warps' time without an instruction, with the instruction cache the SMs of a GPC share
// 74-88 % busy refilling theirs. Hence one instantiation per pattern (the planner's and the epilogue's
// index arithmetic shrinks to the pattern's own), no divisions (FastDiv), per-row data evaluated by the threads
// that use it instead of by the planner, one loop over the two sub-tiles in every role that serves both, and
// rolled loops wherever registers need not be indexed.
//
// Barriers: every wait is bounded (2 s) and gives up when another thread of the CTA has. Each barrier completes
// again only after its waiter has seen the completion before, which is what lets one parity bit name a phase:
//   s_full[s][j & 1]   QK_s of key tile j has completed. Waiters: set s; warp 13 (K and Q buffers).
//                      QK_s(j + 2) needs s_taken of both sets for tile j + 1
//   s_taken[s]         set s has copied its scores of a tile (4 warps). Waiter: QK warp before the other sub-tile's QK^T
//   p_full[s]          set s has stored P of a tile (4 warps). Waiter: PV warp; the next P needs pv_done of this one
//   pv_done[s][j & 1]  PV_s of key tile j has completed. Waiters: set s before it writes the next P or rescales O;
//                      warp 14 (V buffers)
//   o_done[s], o_free[s], l_ready[s]   per item: last PV done / accumulator read / row sums published (two
//                      barriers alternate)
//   batch_ready[r], batch_free[r]   planned items
// A wait for "the phase before the first" (parity 1 of a fresh barrier) returns at once, so the first tiles and items
// need no special case.
//
// Replaces the reference's compute_attn_1rowblock_* kernels (csrc/flash_attn/src/flash_fwd_kernel.h:3970-6158).
#pragma once
#include "attn_kernel.cuh"
#include "attn_items.cuh"
#include "softmax.cuh"
#include "tma_maps.h"

namespace intra {

struct RowsCfg {
  static constexpr int SM_WARPS = 8;
  static constexpr int THREADS = 512;
  // setmaxnreg: softmax sets (a row's 128 scores live in registers), epilogue, the other warps
  static constexpr int SM_REGS = 184, EP_REGS = 64, MMA_REGS = 80;
  static_assert(256 * SM_REGS + 128 * (EP_REGS + MMA_REGS) <= 65536,
                "register budgets exceed what the CTA was launched with: setmaxnreg.inc would never return");
};
constexpr int OUT_STAGE = OUT_ROWS * 128;                  // bytes an epilogue warp stages: 64 columns of its rows
constexpr int ROWS_SMEM_BYTES = 6 * TILE_BYTES + 4 * OUT_STAGE + 1024;     // Q0 Q1 | K0 K1 | V0 V1 | output staging

// One item of the CTA's list.
struct RowSlot {
  int n_kv;              // key tiles of the item (> 0)
  int nk;                // key slots (the interval of padding rows)
  int b, hk;
  int h[2];
  int shift[2];
  Tile sub[2];
  QPlan q[2];            // TMA boxes of the two query sub-tiles
  KvPlan kv[2];          // ... and of the key tiles: [0] only, unless the sub-tiles keep their own keys
};
// The planner works out a batch of items at a time, one per lane: its code, used once per batch, is then fetched
// once per 16 items instead of once per item (2,000 cycles each time, beside which the softmax ran at half speed).
// Two batches alternate. window 16384: 158.6 -> 156.1 us, Scatter 4096 29.6 -> 29.2.
constexpr int ROW_BATCH = 16;
struct RowBatch {
  int n;                 // items in it (empty ones are left out)
  int last;              // the CTA's list ends with it
  RowSlot slot[ROW_BATCH];
};

// Token and key-slot interval of query row `row` of sub-tile `sx`: pair_q_row with the pattern known.
template <int KIND>
__device__ __forceinline__ void slot_row(const Problem& prob, const RowSlot& sl, int sx, int row, int* token, int* lo, int* hi) {
  *token = -1; *lo = 0; *hi = sl.nk - 1;
  if (sl.sub[sx].n_kv_tiles == 0) return;
  Problem p = prob;
  p.kind = KIND;
  Tile t = sl.sub[sx];
  if (KIND != KIND_IMG_GATHER0) t.kind = KIND;
  else t.kind = t.kind == KIND_IMG_GATHER0 ? KIND_IMG_GATHER0 : KIND_IMG_SCATTER;
  int tk, l, h;
  q_row(p, t, row, &tk, &l, &h);
  if (tk < 0) return;
  *token = tk;
  *lo = l + sl.shift[sx];
  *hi = h + sl.shift[sx];
}

template <int KIND>
INTRA_HD Problem kind_problem(const DualParams& p) {
  Problem pr = p.f.prob;
  pr.kind = KIND;
  return pr;
}
template <int KIND>
INTRA_HD void fill_row_slot(const Problem& pr, const DualItem& di, RowSlot& sl) {
  sl.n_kv = di.pt.kv.n_kv_tiles;
  sl.nk = di.pt.kv.nk;
  sl.b = di.b; sl.hk = di.hk;
  sl.h[0] = di.h0; sl.h[1] = di.h1;
  sl.shift[0] = di.pt.shift[0]; sl.shift[1] = di.pt.shift[1];
  sl.sub[0] = di.pt.sub[0]; sl.sub[1] = di.pt.sub[1];
  // an absent sub-tile (odd tile count) is fed the other one's rows; its results are dropped
  const bool has0 = di.pt.sub[0].n_kv_tiles > 0, has1 = di.pt.sub[1].n_kv_tiles > 0;
  const QPlan q0 = plan_q(pr, di.pt.sub[0]), q1 = plan_q(pr, di.pt.sub[1]);
  sl.q[0] = has0 ? q0 : q1;
  sl.q[1] = has1 ? q1 : q0;
  if (KIND == KIND_IMG_GATHER0) {                          // ... and reads the other one's keys, too
    const KvPlan k0 = plan_kv(pr, di.pt.sub[0]), k1 = plan_kv(pr, di.pt.sub[1]);
    sl.kv[0] = has0 ? k0 : k1;
    sl.kv[1] = has1 ? k1 : k0;
  } else {
    sl.kv[0] = plan_kv(pr, di.pt.kv);
  }
}

// Requests of one tile, completion counted in bytes on `bar`.
__device__ __forceinline__ void fetch_q_tile(const TmaMaps& maps, const QPlan& q, int head, int batch, uint32_t dst, uint32_t bar) {
  const CUtensorMap* m = &maps.view[q.which][0];
  ptx::mbar_expect_tx_at(bar, TILE_BYTES);
#pragma unroll 1
  for (int half = 0; half < 2; ++half, dst += HALF_BYTES) {
    ptx::tma_load_5d_at(dst, m, bar, half * 64, q.c1, q.c2, head, batch);
    if (q.patches) ptx::tma_load_5d_at(dst + HALF_BYTES / 2, m, bar, half * 64, q.c1b, q.c2, head, batch);
  }
}
__device__ __forceinline__ void fetch_kv_tile(const TmaMaps& maps, int operand, const KvPlan& kv, int n, int head, int batch,
                                              uint32_t dst, uint32_t bar) {
  int which, c1, c2;
  kv_box(kv, n, &which, &c1, &c2);
  const CUtensorMap* m = &maps.view[which][operand];
  ptx::mbar_expect_tx_at(bar, TILE_BYTES);
  ptx::tma_load_5d_at(dst, m, bar, 0, c1, c2, head, batch);
  ptx::tma_load_5d_at(dst + HALF_BYTES, m, bar, 64, c1, c2, head, batch);
}

// S = Q K^T and O (+)= P V of one tile as rolled loops over the eight 16-deep steps (attn_kernel.cuh has the
// operand layouts); a step's issue takes less than its MMA.
__device__ __forceinline__ void issue_qk_loop(uint64_t q_desc, uint64_t k_desc, uint32_t s_tmem) {
  constexpr uint32_t idesc = ptx::idesc_bf16_f32(TILE_M, TILE_N, 0, 0);
#pragma unroll 1
  for (int s = 0; s < HEAD_DIM / 16; ++s) {
    ptx::mma_ss(s_tmem, q_desc, k_desc, idesc, s);
    const uint64_t step = s == 3 ? (HALF_BYTES - 3 * 32) >> 4 : 32 >> 4;
    q_desc += step;
    k_desc += step;
  }
}
__device__ __forceinline__ void issue_pv_loop(uint32_t p_tmem, uint64_t v_desc, uint32_t o_tmem, uint32_t accumulate) {
  constexpr uint32_t idesc = ptx::idesc_bf16_f32(TILE_M, HEAD_DIM, 0, 1);
#pragma unroll 1
  for (int s = 0; s < TILE_N / 16; ++s) {
    ptx::mma_ts(o_tmem, p_tmem + s * 8, v_desc, idesc, accumulate | s);
    v_desc += 2048 >> 4;
  }
}

// Split key lists (Gather-0): which of the two K (or V) buffers the next tile goes to, and when that one is free.
// Image tiles: each sub-tile's own. Text tiles are the same for both sub-tiles: one load for both, 20 loads for
// the 14 products of a patch item instead of 28 (at four tiles per step the copies alone took 3,700 cycles,
// 35 B per clock and SM out of the L2). A buffer is free once the MMA that read it last has completed, sub-tile
// 1's where both read it. The next tile goes to buffer `cur`, the one that frees first: the other one after a text
// tile, sub-tile 0's after image tiles.
struct BufferUse {
  uint32_t used = 0xeu;      // two bits per buffer: the low bits of the key tile it held last (-2 and -1 to begin with)
  uint32_t reader = 3u;      // one bit per buffer: whether that was read last by sub-tile 1
  uint32_t cur = 0;
  __device__ __forceinline__ uint32_t buffer(bool shared, int sx) const { return cur ^ uint32_t(shared ? 0 : sx); }
  __device__ __forceinline__ uint32_t barrier(uint32_t x) const { return 2 * ((reader >> x) & 1u) + ((used >> (2 * x)) & 1u); }
  __device__ __forceinline__ uint32_t parity(uint32_t x) const { return (used >> (2 * x + 1)) & 1u; }
  __device__ __forceinline__ void read_by(uint32_t x, uint32_t tile, int sx) {
    used = (used & ~(3u << (2 * x))) | ((tile & 3u) << (2 * x));
    reader = (reader & ~(1u << x)) | (uint32_t(sx) << x);
  }
  __device__ __forceinline__ void next(bool shared) { cur ^= shared ? 1u : 0u; }
};

// Number of the tile buffer `x` is about to hold, counted over the CTA.
__device__ __forceinline__ uint32_t next_fill(uint32_t (&fills)[2], uint32_t x) {
  const uint32_t n = x ? fills[1] : fills[0];
  fills[0] += x ? 0 : 1;
  fills[1] += x ? 1 : 0;
  return n;
}

template <int KIND>
__global__ void __launch_bounds__(RowsCfg::THREADS, 1) intra_fwd_rows_kernel(const __grid_constant__ DualParams p) {
  using Cfg = RowsCfg;
  constexpr bool SPLIT = KIND == KIND_IMG_GATHER0;         // the sub-tiles have key lists of their own
  constexpr bool IMAGE = KIND == KIND_IMG_SCATTER || KIND == KIND_IMG_GATHER0;
  enum : int {
    Q_FULL = 0, K_FULL = 2, V_FULL = 4, S_FULL = 6, PV_DONE = 10, P_FULL = 14, S_TAKEN = 16, O_DONE = 18, O_FREE = 20,
    L_READY = 22, BATCH_READY = 26, BATCH_FREE = 28, DRAIN = 30, N_BARS = 32
  };
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[N_BARS];
  __shared__ RowBatch ring[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;
  __shared__ float row_sum[2][2][TILE_M], row_max[2][2][TILE_M];    // [item parity][sub-tile][row]

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = smem_base, k_smem = smem_base + 2 * TILE_BYTES, v_smem = smem_base + 4 * TILE_BYTES;
  const uint32_t bar0 = ptx::smem_u32(bars);
  auto bar = [&](int i) { return bar0 + 8u * uint32_t(i); };

  if (tid == 0) {
    abort_flag = 0;
    for (int i = 0; i < N_BARS; ++i) {
      int n = 1;
      if (i == P_FULL || i == P_FULL + 1 || i == S_TAKEN || i == S_TAKEN + 1 || (i >= L_READY && i < L_READY + 4)) n = 4;
      if (i == O_FREE || i == O_FREE + 1) n = 4;
      if (i == BATCH_FREE || i == BATCH_FREE + 1) n = Cfg::SM_WARPS + 4 + 2 + 1;   // sets, epilogue, issuing warps, requests
      ptx::mbar_init(&bars[i], n);
    }
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    ptx::tmem_alloc(&tmem_base_smem, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = tmem_base_smem;
  volatile int* abort_p = &abort_flag;
  bool ok = true;

#define ROWS_WAIT(index, parity, code) ptx::mbar_wait_at(bar(index), (parity) & 1, abort_p, code)
  // Loops over the items of this CTA's list (`sl`, number `seq`); the body leaves it with ok = false.
#define ROWS_ITEMS(code)                                                              \
  for (uint32_t batch = 0, seq = 0; ok; ++batch) {                                    \
    const RowBatch& rb = ring[batch & 1];                                             \
    ok = ROWS_WAIT(BATCH_READY + (batch & 1), batch >> 1, code);                      \
    if (!ok) break;                                                                   \
    _Pragma("unroll 1") for (int i = 0; i < rb.n && ok; ++i, ++seq) {                 \
      const RowSlot& sl = rb.slot[i];
  // ... and hands a batch back to the planner
#define ROWS_ITEMS_END(lanes)                                                         \
    }                                                                                 \
    if (!ok || rb.last) break;                                                        \
    __syncwarp(lanes);                                                                \
    if (lane == 0) ptx::mbar_arrive_at(bar(BATCH_FREE + (batch & 1)));                \
  }

  if (warp < Cfg::SM_WARPS) {
    // ================================ softmax sets ================================================
    ptx::setmaxnreg_inc<Cfg::SM_REGS>();
    const int sx = warp >> 2;
    const int row = tid & 127;
    const uint32_t lane_addr = tmem + (uint32_t((warp & 3) * 32) << 16);
    const uint32_t p_addr = lane_addr + 128 + sx * 64;
    const uint32_t o_addr = lane_addr + 256 + sx * 128;
    const float scale_log2 = p.f.scale_log2;
    uint32_t kt = 0;                                      // key tiles processed so far by this CTA
    ROWS_ITEMS(52)
      const int n_kv = sl.n_kv;
      int token, lo, hi;
      slot_row<KIND>(p.f.prob, sl, sx, row, &token, &lo, &hi);
      // key slots [lo_max, hi_min] are seen by every row of the warp
      const int lo_max = __reduce_max_sync(0xffffffffu, lo), hi_min = __reduce_min_sync(0xffffffffu, hi);
      float m_run = -CUDART_INF_F, l_run = 0.f;
#pragma unroll 1
      for (int n = 0; n < n_kv; ++n, ++kt) {
        ok = ROWS_WAIT(S_FULL + 2 * sx + (kt & 1), kt >> 1, 11 + sx);
        if (!ok) break;
        ptx::tc_fence_after();
        float s[TILE_N];
        uint32_t* const su = reinterpret_cast<uint32_t*>(s);
        const int u0 = n * TILE_N;
        // Chunks of 32 columns, the maximum of one worked out while the next is on its way.
        float tile_max;
        auto chunk_max = [&](int c) { return sm::row_max(*reinterpret_cast<const float(*)[32]>(&s[32 * c])); };
        if (!(u0 < lo_max || u0 + TILE_N - 1 > hi_min)) {
        ptx::tmem_ld32(lane_addr, su);
        ptx::tmem_wait_ld();
        ptx::tmem_ld32(lane_addr + 32, su + 32);
        tile_max = chunk_max(0);
        ptx::tmem_wait_ld();
        ptx::tmem_ld32(lane_addr + 64, su + 64);
        tile_max = fmaxf(tile_max, chunk_max(1));
        ptx::tmem_wait_ld();
        ptx::tmem_ld32(lane_addr + 96, su + 96);
        tile_max = fmaxf(tile_max, chunk_max(2));
        ptx::tmem_wait_ld();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_at(bar(S_TAKEN + sx));       // the other sub-tile's QK^T may overwrite the buffer
        tile_max = fmaxf(tile_max, chunk_max(3));
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) ptx::tmem_ld32(lane_addr + 32 * c, su + 32 * c);
          ptx::tmem_wait_ld();
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_at(bar(S_TAKEN + sx));
          tile_max = -CUDART_INF_F;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int a = u0 + 32 * c;
            if (a < lo_max || a + 31 > hi_min) {
              const int first = lo - a, last = hi - a;
              const uint32_t seen = (first <= 0 ? ~0u : first > 31 ? 0u : ~0u << first) & (last >= 31 ? ~0u : last < 0 ? 0u : (2u << last) - 1u);
#pragma unroll
              for (int i = 0; i < 32; ++i) s[32 * c + i] = (seen >> i) & 1u ? s[32 * c + i] : -CUDART_INF_F;
            }
            tile_max = fmaxf(tile_max, chunk_max(c));
          }
        }
        const float m_new = fmaxf(m_run, tile_max);
        // The running maximum moves only when the scores outgrow it by 2^8; until then p is merely scaled by a
        // constant that the final division by the row sum removes.
        const bool grow = (m_new - m_run) * scale_log2 > RESCALE_THRESHOLD;
        float alpha = 1.f;
        if (grow) {
          alpha = ptx::ex2((m_run - m_new) * scale_log2);  // 0 when the maximum is still -inf
          l_run *= alpha;
          m_run = m_new;
        }
        // The PV of this sub-tile's previous key tile (of this item or the one before) reads the P buffer and
        // writes O: both may be touched only once it has completed.
        ok = ROWS_WAIT(PV_DONE + 2 * sx + ((kt - 1) & 1), (kt - 1) >> 1, 13 + sx);
        if (!ok) break;
        ptx::tc_fence_after();
        if (n > 0 && __any_sync(0xffffffffu, grow)) {      // rare once the maximum has settled
#pragma unroll 1
          for (int c = 0; c < HEAD_DIM / 16; ++c) {
            uint32_t o[16];
            ptx::tmem_ld16(o_addr + c * 16, o);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            ptx::tmem_st16(o_addr + c * 16, o);
          }
        }
        const float base = (m_run == -CUDART_INF_F) ? 0.f : m_run * scale_log2;
        sm::f2 sum[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
          sm::exp_chunk<sm::EX2_FMA_PAIRS_NONE>(s, c * 32, scale_log2, base, pk, sum);
          ptx::tmem_st16(p_addr + c * 16, pk);
        }
        l_run += sm::sum4(sum);
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_at(bar(P_FULL + sx));
      }
      if (!ok) break;
      // The epilogue warps take it from here. Two barriers alternate: the report of the item after next follows the
      // next item's PV, which waited for o_free of this one, i.e. for the epilogue to have seen this report.
      row_sum[seq & 1][sx][row] = l_run;
      if (p.f.lse != nullptr) row_max[seq & 1][sx][row] = m_run;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_at(bar(L_READY + 2 * sx + (seq & 1)));
    ROWS_ITEMS_END(0xffffffffu)
  } else if (warp < Cfg::SM_WARPS + 4) {
    // ================================ epilogue =====================================================
    ptx::setmaxnreg_dec<Cfg::EP_REGS>();
    const int row = tid & 127;
    const uint32_t lane_addr = tmem + (uint32_t((warp & 3) * 32) << 16);
    ROWS_ITEMS(53)
#pragma unroll 1
      for (int sx = 0; sx < 2; ++sx) {
        const int b = sl.b, h = sl.h[sx];
        ok = ROWS_WAIT(L_READY + 2 * sx + (seq & 1), seq >> 1, 41) && ROWS_WAIT(O_DONE + sx, seq, 43 + sx);
        if (!ok) break;
        ptx::tc_fence_after();
        const float l = row_sum[seq & 1][sx][row];
        const float inv = l > 0.f ? 1.f / l : 0.f;
        const uint32_t o_addr = lane_addr + 256 + sx * 128;
        int token = -1, lo, hi;
        if (IMAGE || p.f.lse != nullptr) slot_row<KIND>(p.f.prob, sl, sx, row, &token, &lo, &hi);
        if (p.f.lse != nullptr && token >= 0)
          p.f.lse[(int64_t(b) * p.f.H + h) * p.f.prob.S + token] = row_lse(row_max[seq & 1][sx][row], l, p.f.scale_log2);
        if (IMAGE) {
          __nv_bfloat16* const dst = p.f.o + b * p.f.os.sb + int64_t(token < 0 ? 0 : token) * p.f.os.ss + h * p.f.os.sh;
          store_o_row(o_addr, HEAD_DIM, inv, dst, token >= 0, p.wide_stores != 0);
        } else {
          // A warp's 32 rows leave as two bulk stores of 64 columns each through its staging buffer (128-byte swizzle).
          // Stored by their threads, 32 bytes to 32 lines per instruction, they would hold up the sets' barrier
          // traffic behind them: GPU time of Scatter at S = 4096 30.2 -> 28.7 us, window at 16384 155.4 -> 151.2.
          // The image patterns' rows are stored by their threads: image Scatter's view has traversal strides, and for
          // Gather-0 there is no output view.
          const int w = warp & 3;
          int c1 = sl.q[sx].c1, c2 = sl.q[sx].c2;          // the query tile's place, this warp's rows on
          if (KIND == KIND_LLM_SCATTER) c2 += OUT_ROWS * w;
          if (KIND == KIND_LLM_WINDOW) c1 += OUT_ROWS * w;
          if (KIND == KIND_LLM_GATHER1) { const int seg = fdiv(OUT_ROWS * w, p.f.prob.by_G); c1 += OUT_ROWS * w - seg * p.f.prob.G; c2 += seg; }
          const bool wanted = sl.sub[sx].n_kv_tiles > 0 && sl.sub[sx].t0 + OUT_ROWS * w < sl.sub[sx].nq;
          const CUtensorMap* const m = &p.maps.view[sl.q[sx].which][3];
          const uint32_t stage = v_smem + 2 * TILE_BYTES + w * OUT_STAGE;
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            ptx::tmem_ld32(o_addr + c * 32, o);
            if ((c & 1) == 0) {                            // the staging buffer's last store has read it
              if (lane == 0) ptx::bulk_wait_read();
              __syncwarp();
            }
            ptx::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint32_t x[4];
#pragma unroll
              for (int e = 0; e < 4; ++e)
                x[e] = ptx::pack_bf16(__uint_as_float(o[8 * i + 2 * e]) * inv, __uint_as_float(o[8 * i + 2 * e + 1]) * inv);
              ptx::st_shared_v4(stage + lane * 128 + ((((c & 1) * 4 + i) ^ (lane & 7)) << 4), x[0], x[1], x[2], x[3]);
            }
            if (c & 1) {
              ptx::fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0 && wanted) {
                ptx::tma_store_5d(m, stage, (c >> 1) * 64, c1, c2, h, b);
                ptx::bulk_commit();
              }
            }
          }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_at(bar(O_FREE + sx));        // the next item's first PV may overwrite O
      }
    ROWS_ITEMS_END(0xffffffffu)
    if (!IMAGE && lane == 0) ptx::bulk_wait_read();        // the staging buffers live until their stores have read them
  } else {
    ptx::setmaxnreg_dec<Cfg::MMA_REGS>();
    if (warp == 13) {
      // ================================ requests of Q and K ==========================================
      if (lane == 0) {
        for (int i = 0; i < 2; ++i) ptx::prefetch_tensormap(&p.maps.view[VIEW_MAIN][i]);
        uint32_t j = 0;                                   // key tiles requested so far by this CTA
        BufferUse use;
        ROWS_ITEMS(55)
          const int n_kv = sl.n_kv;
#pragma unroll 1
          for (int n = 0; n < n_kv && ok; ++n, ++j) {
            // Each tile goes out as early as its buffer frees; an item's queries follow its first K tiles.
            const bool shared = !SPLIT || is_text_tile(sl.kv[0].text, n);
#pragma unroll 1
            for (int sx = 0; sx < 2 && ok; ++sx) {
              if (sx == 0 || !shared) {
                const uint32_t x = SPLIT ? use.buffer(shared, sx) : j & 1;
                ok = SPLIT ? ROWS_WAIT(S_FULL + use.barrier(x), use.parity(x), 24 + sx) : ROWS_WAIT(S_FULL + 2 + x, (j - 2) >> 1, 22);
                if (!ok) break;
                fetch_kv_tile(p.maps, 1, sl.kv[SPLIT ? sx : 0], n, sl.hk, sl.b, k_smem + x * TILE_BYTES, bar(K_FULL + x));
                if (SPLIT) use.read_by(x, j, shared ? 1 : sx);
              }
              if (n == 0) {
                ok = ROWS_WAIT(S_FULL + 2 * sx + ((j - 1) & 1), (j - 1) >> 1, 21);
                if (ok) fetch_q_tile(p.maps, sl.q[sx], sl.h[sx], sl.b, q_smem + sx * TILE_BYTES, bar(Q_FULL + sx));
              }
            }
            if (SPLIT) use.next(shared);
          }
        ROWS_ITEMS_END(1u)
      }
    } else if (warp == 14) {
      // ================================ planner, requests of V =======================================
      const Problem pr = kind_problem<KIND>(p);
      uint32_t planned = 0;                               // batches planned so far
      bool more = true;                                   // the list goes on after them
      auto plan = [&] {
        const int item = dual_item_index(planned * ROW_BATCH + lane, blockIdx.x, gridDim.x);
        const bool valid = lane < ROW_BATCH && item < p.n_items;
        const DualItem di = dual_decode(p, pr, valid ? item : 0);
        const uint32_t filled = __ballot_sync(0xffffffffu, valid && di.pt.kv.n_kv_tiles > 0);
        more = __popc(__ballot_sync(0xffffffffu, valid)) == ROW_BATCH;
        RowBatch& rb = ring[planned & 1];
        if (planned >= 2) ok = ROWS_WAIT(BATCH_FREE + (planned & 1), (planned >> 1) - 1, 51);
        if (!ok) return;
        if ((filled >> lane) & 1u) fill_row_slot<KIND>(pr, di, rb.slot[__popc(filled & ((1u << lane) - 1u))]);
        if (lane == 0) { rb.n = __popc(filled); rb.last = !more; }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_at(bar(BATCH_READY + (planned & 1)));
        ++planned;
      };
      uint32_t j = 0;
      BufferUse use;
#pragma unroll 1
      for (uint32_t step = 0, batch = 0, i = 0; ok; ++step) {
        // The next batch is planned in the middle of one, when the other roles have long left the one before, or
        // when this one is done.
        const bool done = planned > batch && int(i) == ring[batch & 1].n;
        if (planned == batch || (planned == batch + 1 && more && (i == 4 || done))) { plan(); continue; }
        if (done) {
          if (ring[batch & 1].last) break;
          ++batch;
          i = 0;
          continue;
        }
        const RowSlot& sl = ring[batch & 1].slot[i++];
        const int n_kv = sl.n_kv;
#pragma unroll 1
        for (int n = 0; n < n_kv && ok; ++n, ++j) {
          const bool shared = !SPLIT || is_text_tile(sl.kv[0].text, n);
#pragma unroll 1
          for (int sx = 0; sx < (shared ? 1 : 2); ++sx) {
            const uint32_t x = SPLIT ? use.buffer(shared, sx) : j & 1;
            ok = SPLIT ? ROWS_WAIT(PV_DONE + use.barrier(x), use.parity(x), 26 + sx) : ROWS_WAIT(PV_DONE + 2 + x, (j - 2) >> 1, 26);
            if (!ok) break;
            if (lane == 0) fetch_kv_tile(p.maps, 2, sl.kv[SPLIT ? sx : 0], n, sl.hk, sl.b, v_smem + x * TILE_BYTES, bar(V_FULL + x));
            if (SPLIT) use.read_by(x, j, shared ? 1 : sx);
          }
          if (SPLIT) use.next(shared);
        }
      }
    } else {
      // ================================ MMA issue: warp 12 QK^T, warp 15 PV ==========================
      const bool qk = warp == 12;
      const uint64_t q_desc = tile_desc_kmajor(q_smem), k_desc = tile_desc_kmajor(k_smem), v_desc = tile_desc_mnmajor(v_smem);
      constexpr uint64_t kTileStep = TILE_BYTES >> 4;      // descriptor distance between buffers
      uint32_t j = 0;                                      // key tiles so far, counted over the CTA
      uint32_t fills[2] = {0, 0}, cur = 0;                 // split key lists: tiles buffer 0 / 1 has held before; see the requests
      ROWS_ITEMS(56)
        const int n_kv = sl.n_kv;
        if (qk) {
#pragma unroll 1
          for (int n = 0; n < n_kv && ok; ++n, ++j) {
            const bool shared = !SPLIT || is_text_tile(sl.kv[0].text, n);
#pragma unroll 1
            for (int sx = 0; sx < 2; ++sx) {
              const uint32_t st = SPLIT ? cur ^ uint32_t(shared ? 0 : sx) : j & 1;
              ok = (n > 0 || ROWS_WAIT(Q_FULL + sx, seq, 31)) &&
                   ((shared && sx == 1) || ROWS_WAIT(K_FULL + st, SPLIT ? next_fill(fills, st) : j >> 1, 32)) &&
                   ROWS_WAIT(S_TAKEN + (sx ^ 1), sx ? j : j - 1, 33);   // the other set has copied its scores out
              if (!ok) break;
              ptx::tc_fence_after();
              if (ptx::elect_one()) {
                issue_qk_loop(q_desc + sx * kTileStep, k_desc + st * kTileStep, tmem);
                ptx::mma_commit_at(bar(S_FULL + 2 * sx + (j & 1)));
              }
              __syncwarp();
            }
            cur ^= SPLIT && shared ? 1 : 0;
          }
        } else {
#pragma unroll 1
          for (int n = 0; n < n_kv && ok; ++n, ++j) {
            const bool shared = !SPLIT || is_text_tile(sl.kv[0].text, n);
#pragma unroll 1
            for (int sx = 0; sx < 2; ++sx) {
              const uint32_t st = SPLIT ? cur ^ uint32_t(shared ? 0 : sx) : j & 1;
              ok = ((shared && sx == 1) || ROWS_WAIT(V_FULL + st, SPLIT ? next_fill(fills, st) : j >> 1, 40)) &&
                   (n > 0 || ROWS_WAIT(O_FREE + sx, seq - 1, 37)) &&   // O of the previous item has been read
                   ROWS_WAIT(P_FULL + sx, j, 35);
              if (!ok) break;
              ptx::tc_fence_after();
              if (ptx::elect_one()) {
                issue_pv_loop(tmem + 128 + sx * 64, v_desc + st * kTileStep, tmem + 256 + sx * 128, n);
                ptx::mma_commit_at(bar(PV_DONE + 2 * sx + (j & 1)));
                if (n == n_kv - 1) ptx::mma_commit_at(bar(O_DONE + sx));
              }
              __syncwarp();
            }
            cur ^= SPLIT && shared ? 1 : 0;
          }
        }
      ROWS_ITEMS_END(0xffffffffu)
      if (!ok) {                                           // let MMAs in flight finish before TMEM is freed
        const int drain = DRAIN + (qk ? 0 : 1);
        if (ptx::elect_one()) ptx::mma_commit_at(bar(drain));
        __syncwarp();
        int dummy = 0;
        ptx::mbar_wait(&bars[drain], 0, &dummy, 100);
      }
    }
  }
#undef ROWS_WAIT
#undef ROWS_ITEMS
#undef ROWS_ITEMS_END

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
  if (tid == 0 && abort_flag != 0) {
    ptx::drain_copies(bars, S_FULL);                       // the Q, K and V tiles that were requested before the give-up
    atomicCAS(p.f.status, 0, STATUS_WAIT_BASE + abort_flag);
  }
}

}  // namespace intra
