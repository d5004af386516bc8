// What the attention kernels share: the launch parameters, the items a CTA walks, and the output row stores.
#pragma once
#include "attn_kernel.cuh"
#include "tma_maps.h"

namespace intra {

struct DualParams {
  FwdParams f;
  int row_pairs;        // 0: sub-tiles are two heads of one KV group; 1: two row tiles of one head
  int n_pair_tiles;     // pair tiles per (batch, head or head pair)
  int heads_per_item;   // row_pairs ? H : H / 2  (number of items per pair tile and batch)
  int n_items;          // n_pair_tiles * B * heads_per_item
  int last_wave;        // waves alternate between heaviest and lightest first; the last one ends with the lightest
  // Items are numbered wave by wave (plan_items_order), within a wave pair tile by pair tile: divisors items per wave,
  // (batch, head) combinations per wave, heads_per_item, H / Hkv.
  FastDiv by_wave, by_tile, by_heads, by_rep;
  int split_kv;         // the two sub-tiles keep their own key lists (Gather-0): K / V buffer s belongs to sub-tile s
  int use_tma;          // tiles are fetched as TMA boxes (tma_maps.h) instead of cp.async row gathers
  int wide_stores;      // every output row is 32-byte aligned: 256-bit global stores
  TmaMaps maps;
};

struct DualItem {
  PairTile pt;
  int b, h0, h1, hk;
};

// Item number `seq` of this CTA: heaviest-first list dealt round by round, every other round reversed.
INTRA_HD int dual_item_index(int seq, int cta, int n_cta) {
  return seq * n_cta + ((seq & 1) ? (n_cta - 1 - cta) : cta);
}

INTRA_HD DualItem dual_decode(const DualParams& p, const Problem& prob, int item) {
  DualItem it;
  const int wave = fdiv(item, p.by_wave);
  const int in_wave = item - wave * int(p.by_wave.d);
  int idx = fdiv(in_wave, p.by_tile);
  const int rem = wave * int(p.by_tile.d) + in_wave - idx * int(p.by_tile.d);
  if ((p.last_wave - wave) & 1) idx = p.n_pair_tiles - 1 - idx;
  it.b = fdiv(rem, p.by_heads);
  const int hh = rem - it.b * p.heads_per_item;
  if (p.row_pairs) { it.h0 = it.h1 = hh; } else { it.h0 = 2 * hh; it.h1 = 2 * hh + 1; }
  it.hk = fdiv(it.h0, p.by_rep);
  it.pt = make_pair(prob, p.row_pairs, idx);
  return it;
}

// Normalise `ncols` (a multiple of 32) accumulator columns of this thread's TMEM lane by `inv` and store
// them as bf16 to `dst` (this row's position in the output). `wide` selects 32-byte stores, which need
// 32-byte aligned rows; tensor-memory loads are finished when the function returns.
__device__ __forceinline__ void store_o_row(uint32_t o_addr, int ncols, float inv, __nv_bfloat16* dst, bool valid,
                                            bool wide) {
#pragma unroll 1
  for (int c = 0; c < ncols / 32; ++c) {
    uint32_t o[32];
    ptx::tmem_ld32(o_addr + c * 32, o);
    ptx::tmem_wait_ld();
    if (valid) {
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 16; ++i)
        w[i] = ptx::pack_bf16(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
      __nv_bfloat16* d = dst + c * 32;
      if (wide) {
        ptx::st_global_v8(d, w);
        ptx::st_global_v8(d + 16, w + 8);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(d + i * 8) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
      }
    }
  }
}

}  // namespace intra
