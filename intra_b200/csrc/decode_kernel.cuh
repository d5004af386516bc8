// One-token decode attention over a dense KV cache: every query head of a (batch, KV head) group against
// the group's S keys, K and V read once from HBM.
//
// What bounds it: reading K and V (512 bytes per key and KV head; the arithmetic is 4 FLOP per byte and
// query head), i.e. how many bytes the chip keeps in flight. So each warp streams its own blocks of 16 keys
// (8 KB of K and V) through a private ring in shared memory with cp.async, DEC_STAGES - 1 blocks ahead, and
// never waits for another warp until the end. The products run as warp-level m16n8k16 MMAs: with at most 8
// query rows there is nothing for a 128-row tcgen05 tile to do, and the unused half of the 16 rows carries
// the low-order part of the probabilities:
//
//   scores   A = Q (rows 0-7: the heads), B = K^T;
//   output   A = P, B = V. The scores' accumulator layout is P's operand layout; rows 0-7 hold P rounded to
//            bf16, rows 8-15 the rounding error in bf16, and the two row halves of the result are added at
//            the end: P keeps 16 significant bits.
//
// The blocks of 16 keys are dealt round robin to the CTAs of a thread-block cluster, which merge
// their partial results through distributed shared memory, so that a call is one launch without any
// scratch in global memory. Groups whose keys want more CTAs than a cluster has use several clusters
// and merge through a scratch buffer of the caller's and a second small launch.
//
// Measured (one B200, per call of the backend; SDPA over repeated K / V before): 1 sequence, 3001 keys, 32 heads over
// 8 KV heads 67.6 -> 13.8 us, most of it host work (8 us on the GPU); 16 sequences in a left-padded 8192-key cache
// 2287 -> 64 us, 5.2 TB/s of the keys that are visible; 4 sequences of 16384 keys 43.8 us, 6.1 TB/s.
//
// A boolean mask is looked at first: blocks without a visible key are not read, and neither are masked
// keys inside a block. Replaces the reference's dense single-token step
// (experiments/llm/intra_token_attn.py:112-134, F.scaled_dot_product_attention over repeated K / V).
#pragma once
#include <cooperative_groups.h>
#include <math_constants.h>
#include <stdint.h>

#include "attn_kernel.cuh"

namespace intra {

constexpr int DEC_WARPS = 4;
constexpr int DEC_THREADS = 32 * DEC_WARPS;
// 2 CTAs of 4 warps per SM, each warp two blocks ahead: up to 128 KB in flight per SM. Measured (us) at 16
// padded sequences in an 8192-key cache, 8 KV heads, best split of each: 71.5; 3 CTAs with one block ahead 77.5, one
// CTA with five blocks ahead 98.6 (nothing covers its start and its merge).
constexpr int DEC_CTAS_PER_SM = 2;
constexpr int DEC_STAGES = 3;                    // ring of key blocks per warp
constexpr int DEC_BLOCK = 16;                    // keys a warp takes at a time
constexpr int DEC_TILE = DEC_BLOCK * HEAD_DIM * 2;       // bytes of one block's K (or V)
constexpr int DEC_SMEM_BYTES = DEC_WARPS * DEC_STAGES * 2 * DEC_TILE;
constexpr int DEC_HEADS = 8;                     // query heads one CTA serves
constexpr int DEC_MAX_BLOCKS = DEC_THREADS;      // key blocks one CTA can be dealt (one mask-scanning thread each)
constexpr int DEC_PARTIAL = DEC_HEADS * (HEAD_DIM + 2);   // floats of one cluster's partial result in the scratch buffer

struct DecodeParams {
  const __nv_bfloat16* q;      // (B, H, 128)
  const __nv_bfloat16* k;      // (B, S, Hkv, 128) by strides
  const __nv_bfloat16* v;
  const uint8_t* mask;         // (B, S) by strides, nonzero = visible; null: every key is
  __nv_bfloat16* o;            // (B, H, 128) contiguous
  float* scratch;              // n_clusters > 1: DEC_PARTIAL floats per cluster
  int64_t q_sb, q_sh;
  TensorView ks, vs;
  int64_t mask_sb, mask_ss;
  int mask_vec;                // 16 mask bytes of a key block can be loaded at once
  int S, H, Hkv;
  int head_groups;             // groups of up to DEC_HEADS query heads per KV head
  int cluster, n_clusters;     // CTAs per cluster, clusters per (batch, KV head, head group)
  float scale_log2;
};

__device__ __forceinline__ void mma_m16n8k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// Byte offset of 16-byte piece `piece` of key row `row` in a block: the piece index is xor-ed with the row so
// that eight rows' pieces of one column lie in different banks.
__device__ __forceinline__ uint32_t dec_offset(int row, int piece) { return row * 256 + ((piece ^ (row & 7)) << 4); }
// Two probabilities as a bf16 pair and the pair of their rounding errors.
__device__ __forceinline__ void split_bf16(float p0, float p1, uint32_t& hi, uint32_t& lo) {
  hi = ptx::pack_bf16(p0, p1);
  lo = ptx::pack_bf16(p0 - __uint_as_float(hi << 16), p1 - __uint_as_float(hi & 0xffff0000u));
}
// Sum of the results of P's high and low parts. An infinite value row makes the high one infinite (or NaN, where
// infinities meet); the low one, a rounding error of either sign or zero times infinity, must not turn it into NaN.
__device__ __forceinline__ float join_parts(float hi, float lo) { return fabsf(hi) < CUDART_INF_F ? hi + lo : hi; }
// Factor that brings a partial result taken against maximum m to maximum m_all (0 for an empty one).
__device__ __forceinline__ float merge_weight(float m, float m_all) {
  return m == -CUDART_INF_F ? 0.f : ptx::ex2(m - m_all);
}

__global__ void __launch_bounds__(DEC_THREADS, DEC_CTAS_PER_SM) decode_kernel(const __grid_constant__ DecodeParams p) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(1024) uint8_t dec_smem[];            // the rings; at the end the warps' partial results
  __shared__ float part_m[DEC_WARPS][DEC_HEADS], part_l[DEC_WARPS][DEC_HEADS];
  __shared__ float cta_o[DEC_HEADS][HEAD_DIM];                     // this CTA's merged result, read by the cluster
  __shared__ float cta_m[DEC_HEADS], cta_l[DEC_HEADS];
  __shared__ int live_key[DEC_MAX_BLOCKS];                         // first key of the blocks with a visible key ...
  __shared__ uint32_t live_bits[DEC_MAX_BLOCKS];                   // ... and which of their keys are visible
  __shared__ int warp_live[DEC_WARPS];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, j = lane & 3;
  const int rank = blockIdx.x % p.cluster;
  const int group = blockIdx.x / p.cluster;                        // cluster number
  const int u = group / p.n_clusters;                              // (batch, KV head, head group)
  const int hg = u % p.head_groups;
  const int hk = (u / p.head_groups) % p.Hkv;
  const int b = u / (p.head_groups * p.Hkv);
  const int rep = p.H / p.Hkv;
  const int h0 = hk * rep + hg * DEC_HEADS;
  const int n_heads = min(rep - hg * DEC_HEADS, DEC_HEADS);

  // ---- this CTA's key blocks: every n_dealt-th one, without those a mask hides entirely ------------------
  const int n_dealt = p.cluster * p.n_clusters;
  const int first_blk = (group % p.n_clusters) * p.cluster + rank;
  const int n_blk = (p.S + DEC_BLOCK - 1) / DEC_BLOCK;
  int n_live = first_blk < n_blk ? (n_blk - 1 - first_blk) / n_dealt + 1 : 0;
  auto block_bits = [&](int key0) { return p.S - key0 >= DEC_BLOCK ? 0xffffu : (1u << (p.S - key0)) - 1u; };
  if (p.mask != nullptr) {
    uint32_t bits = 0;
    int key0 = 0;
    if (tid < n_live) {
      key0 = (first_blk + tid * n_dealt) * DEC_BLOCK;
      bits = block_bits(key0);
      const uint8_t* m = p.mask + b * p.mask_sb + key0 * p.mask_ss;
      uint32_t seen = 0;
      if (p.mask_vec && bits == 0xffffu) {
        const uint4 w = *reinterpret_cast<const uint4*>(m);
        const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < DEC_BLOCK; ++i) seen |= ((ws[i >> 2] >> (8 * (i & 3))) & 0xffu) != 0u ? 1u << i : 0u;
      } else {
        for (int i = 0; i < DEC_BLOCK; ++i)
          if ((bits >> i) & 1u) seen |= m[i * p.mask_ss] != 0 ? 1u << i : 0u;
      }
      bits &= seen;
    }
    const uint32_t vote = __ballot_sync(0xffffffffu, bits != 0u);
    if (lane == 0) warp_live[warp] = __popc(vote);
    __syncthreads();
    int at = __popc(vote & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) at += warp_live[w];
    if (bits != 0u) { live_key[at] = key0; live_bits[at] = bits; }
    __syncthreads();
    n_live = 0;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) n_live += warp_live[w];
  }
  auto block = [&](int e, uint32_t& seen) {                        // first key of the CTA's e-th block
    if (p.mask != nullptr) { seen = live_bits[e]; return live_key[e]; }
    const int key0 = (first_blk + e * n_dealt) * DEC_BLOCK;
    seen = block_bits(key0);
    return key0;
  };

  // ---- this warp streams blocks warp, warp + DEC_WARPS, ... ----------------------------------------------
  const uint32_t ring = ptx::smem_u32(dec_smem) + warp * (DEC_STAGES * 2 * DEC_TILE);
  const int half = lane >> 4, piece = lane & 15;                   // a copy instruction takes two rows
  const __nv_bfloat16* const kb = p.k + b * p.ks.sb + hk * p.ks.sh + piece * 8;
  const __nv_bfloat16* const vb = p.v + b * p.vs.sb + hk * p.vs.sh + piece * 8;
  auto fetch = [&](int e, int stage) {                             // always one commit group, possibly empty
    if (e < n_live) {
      uint32_t seen;
      const int key0 = block(e, seen);
      const uint32_t dst = ring + stage * (2 * DEC_TILE);
      const __nv_bfloat16* kr = kb + int64_t(key0 + half) * p.ks.ss;
      const __nv_bfloat16* vr = vb + int64_t(key0 + half) * p.vs.ss;
#pragma unroll
      for (int i = 0; i < DEC_BLOCK; i += 2) {                     // masked keys become zeros and are not read
        const uint32_t n = (seen >> (i + half)) & 1u ? 16u : 0u;
        const uint32_t off = dec_offset(i + half, piece);
        ptx::cp_async_16(dst + off, n ? kr + i * p.ks.ss : p.k, n);
        ptx::cp_async_16(dst + DEC_TILE + off, n ? vr + i * p.vs.ss : p.v, n);
      }
    }
    ptx::cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < DEC_STAGES - 1; ++s) fetch(warp + s * DEC_WARPS, s);

  uint32_t qf[8][2];                                               // A operand of the eight 16-dim steps, rows 0-7
  {
    const uint32_t* qp = reinterpret_cast<const uint32_t*>(p.q + b * p.q_sb + int64_t(h0 + g) * p.q_sh) + j;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      qf[t][0] = g < n_heads ? qp[8 * t] : 0u;
      qf[t][1] = g < n_heads ? qp[8 * t + 4] : 0u;
    }
  }
  float o[16][4];                                                  // dims 8 t + 2 j, + 1: rows of P's high and low parts
#pragma unroll
  for (int t = 0; t < 16; ++t) o[t][0] = o[t][1] = o[t][2] = o[t][3] = 0.f;
  float m_run = -CUDART_INF_F, l_run = 0.f;                        // of head g; l_run: this lane's keys only

  // ldmatrix row addresses: K matrices are (keys 0-7 | 8-15) x (dims 0-7 | 8-15) of a step, V the same transposed
  const int mi = lane >> 3, mr = lane & 7;
  const int k_row = (mi >> 1) * 8 + mr, v_row = (mi & 1) * 8 + mr;
  int stage = 0;
  for (int e = warp; e < n_live; e += DEC_WARPS) {
    ptx::cp_async_wait<DEC_STAGES - 2>();
    __syncwarp();                                                  // every lane's copies of this block have landed, and
    fetch(e + (DEC_STAGES - 1) * DEC_WARPS, (stage + DEC_STAGES - 1) % DEC_STAGES);   // all are done with the last one
    const uint32_t kt = ring + stage * (2 * DEC_TILE), vt = kt + DEC_TILE;
    float s[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) s[0][i] = s[1][i] = 0.f;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      uint32_t r[4];
      ldmatrix_x4(kt + dec_offset(k_row, 2 * t + (mi & 1)), r);
      mma_m16n8k16(s[0], qf[t][0], 0u, qf[t][1], 0u, r[0], r[1]);
      mma_m16n8k16(s[1], qf[t][0], 0u, qf[t][1], 0u, r[2], r[3]);
    }
    uint32_t seen;
    block(e, seen);
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int key = 2 * j + (i & 1) + 8 * (i >> 1);
      x[i] = (seen >> key) & 1u ? s[i >> 1][i & 1] * p.scale_log2 : -CUDART_INF_F;
    }
    float m_blk = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
    m_blk = fmaxf(m_blk, __shfl_xor_sync(0xffffffffu, m_blk, 1));
    m_blk = fmaxf(m_blk, __shfl_xor_sync(0xffffffffu, m_blk, 2));
    // the maximum moves only when the scores outgrow it by 2^8; until then probabilities are merely scaled
    const bool grow = m_blk > m_run + RESCALE_THRESHOLD;
    if (__any_sync(0xffffffffu, grow)) {
      const float alpha = grow ? merge_weight(m_run, m_blk) : 1.f;
      if (grow) m_run = m_blk;
      l_run *= alpha;
#pragma unroll
      for (int t = 0; t < 16; ++t) {
#pragma unroll
        for (int i = 0; i < 4; ++i) o[t][i] *= alpha;
      }
    }
    const float base = m_run == -CUDART_INF_F ? 0.f : m_run;
    float pr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) pr[i] = ptx::ex2(x[i] - base);
    l_run += (pr[0] + pr[1]) + (pr[2] + pr[3]);
    uint32_t hi0, lo0, hi1, lo1;
    split_bf16(pr[0], pr[1], hi0, lo0);
    split_bf16(pr[2], pr[3], hi1, lo1);
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      uint32_t r[4];
      ldmatrix_x4_trans(vt + dec_offset(v_row, 2 * t + (mi >> 1)), r);
      mma_m16n8k16(o[2 * t], hi0, lo0, hi1, lo1, r[0], r[1]);
      mma_m16n8k16(o[2 * t + 1], hi0, lo0, hi1, lo1, r[2], r[3]);
    }
    stage = stage + 1 == DEC_STAGES ? 0 : stage + 1;
  }
  ptx::cp_async_wait<0>();

  // ---- merge: lanes of a head, warps, CTAs of the cluster ----------------------------------------------
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
  if (j == 0) { part_m[warp][g] = m_run; part_l[warp][g] = l_run; }
  __syncthreads();                                                 // the rings are free
  constexpr int ROW = HEAD_DIM + 8;                                // rows start 8 banks apart
  float* const part_o = reinterpret_cast<float*>(dec_smem);        // [warp][head][ROW]
#pragma unroll
  for (int t = 0; t < 16; ++t)
    *reinterpret_cast<float2*>(part_o + (warp * DEC_HEADS + g) * ROW + 8 * t + 2 * j) =
        make_float2(join_parts(o[t][0], o[t][2]), join_parts(o[t][1], o[t][3]));
  __syncthreads();
  for (int h = 0; h < n_heads; ++h) {                              // thread = dim
    float m_all = -CUDART_INF_F;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) m_all = fmaxf(m_all, part_m[w][h]);
    float acc = 0.f, l_all = 0.f;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) {
      const float f = merge_weight(part_m[w][h], m_all);
      acc += f * part_o[(w * DEC_HEADS + h) * ROW + tid];
      l_all += f * part_l[w][h];
    }
    cta_o[h][tid] = acc;
    if (tid == 0) { cta_m[h] = m_all; cta_l[h] = l_all; }
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int h = rank; h < n_heads; h += p.cluster) {
    float m_all = -CUDART_INF_F;
    for (int r = 0; r < p.cluster; ++r) m_all = fmaxf(m_all, *cluster.map_shared_rank(&cta_m[h], r));
    float acc = 0.f, l_all = 0.f;
#pragma unroll 4
    for (int r = 0; r < p.cluster; ++r) {
      const float f = merge_weight(*cluster.map_shared_rank(&cta_m[h], r), m_all);
      acc += f * *cluster.map_shared_rank(&cta_o[h][tid], r);
      l_all += f * *cluster.map_shared_rank(&cta_l[h], r);
    }
    if (p.n_clusters == 1) {
      p.o[(int64_t(b) * p.H + h0 + h) * HEAD_DIM + tid] = __float2bfloat16(l_all == 0.f ? 0.f : acc / l_all);
    } else {
      float* part = p.scratch + int64_t(group) * DEC_PARTIAL + h * (HEAD_DIM + 2);
      part[tid] = acc;
      if (tid == 0) { part[HEAD_DIM] = m_all; part[HEAD_DIM + 1] = l_all; }
    }
  }
  cluster.sync();                                                  // nobody leaves while its shared memory is read
}

// The clusters' partial results of one query head -> output row. One CTA per (batch, head), thread = dim.
__global__ void __launch_bounds__(HEAD_DIM) decode_merge_kernel(const __grid_constant__ DecodeParams p) {
  const int h = blockIdx.x % p.H, b = blockIdx.x / p.H;
  const int rep = p.H / p.Hkv;
  const int hk = h / rep, hr = h % rep;
  const int u = (b * p.Hkv + hk) * p.head_groups + hr / DEC_HEADS;
  const float* part = p.scratch + int64_t(u) * p.n_clusters * DEC_PARTIAL + (hr % DEC_HEADS) * (HEAD_DIM + 2);
  float m_all = -CUDART_INF_F;
  for (int c = 0; c < p.n_clusters; ++c) m_all = fmaxf(m_all, part[int64_t(c) * DEC_PARTIAL + HEAD_DIM]);
  float acc = 0.f, l_all = 0.f;
#pragma unroll 4
  for (int c = 0; c < p.n_clusters; ++c) {
    const float* pc = part + int64_t(c) * DEC_PARTIAL;
    const float f = merge_weight(pc[HEAD_DIM], m_all);
    acc += f * pc[threadIdx.x];
    l_all += f * pc[HEAD_DIM + 1];
  }
  p.o[(int64_t(b) * p.H + h) * HEAD_DIM + threadIdx.x] = __float2bfloat16(l_all == 0.f ? 0.f : acc / l_all);
}

}  // namespace intra
