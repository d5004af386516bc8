// Tensor-map (TMA) views of the Q / K / V tensors for the patterns whose row gathers are affine:
// a 128-row tile of any such pattern is one box of a <= 5-dimensional strided view of the caller's
// (batch, token, head, 128) tensor, so a single thread can fetch it with two bulk-tensor copies (one
// per 64-element half of the head dim) that land in shared memory already 128-byte swizzled.
//
//   Scatter                      dims (d, g, t, head, batch)       box (64, 1, 128)      token = t*G + g
//             S % G = r > 0: groups 0..r-1 are one token longer, so there are two such views with exact extents:
//             the "text" view holds groups 0..r-1 with S/G + 1 tokens each, the main view groups r..G-1 (base at
//             token r) with S/G. Nothing beyond token S-1 is ever read; the box rows past a group's end are
//             zero-filled. Before, these shapes took the row gathers, whose 128 threads could not keep two K / V
//             stages full: Scatter G=8, S=12345, 32/8 heads 423 us, 229 us as boxes (one launch, one B200).
//   Gather-1 (S % G^2 == 0, G|128) dims (d, w, seg, head, batch)   box (64, G, 128/G)    token = seg*G^2 + w, w = g*G + j
//   window                       dims (d, token, 1, head, batch)   box (64, 128)
//   image Scatter, image part    dims (d, c, r, head, batch), traversal strides (1, 4, 2), base at token 512
//                                box (64, W, 2*128/(W/4)): every 4th column from c = b, every 2nd row from r = a
//                text part       dims (d, token, 1, head, batch), 512 tokens, box (64, 128)
//   Gather-0 patch pairs  keys   dims (d, r, c, head, batch), box (64, 16, 8): 8 window columns, 16 rows each
//                        queries dims (d, c, r, head, batch), box (64, 8, 8): one 8x8 patch, two boxes per tile
//            text chunks         as image Scatter (the "aux" view) + the text view
//
// All views have five dimensions (one of extent 1 where four would do), so that the requesting thread has a single
// form of load to issue.
//
// Shapes outside these conditions (ragged Gather-1, odd widths) use the cp.async gathers.
// This replaces the per-thread address arithmetic of the reference's loaders
// (csrc/flash_attn/src/gmem_tile.h:481-1426, csrc/flash_attn/src/intra_copy.h:13-101).
#pragma once
#include <cuda.h>

#include "intra_index.h"

namespace intra {

enum ViewId : int {
  VIEW_MAIN = 0,    // the pattern's strided view
  VIEW_TEXT = 1,    // image kinds: the 512 text tokens; ragged Scatter: its longer groups
  VIEW_AUX = 2      // Gather-0: image-Scatter view for the keys of its text tiles
};
struct alignas(64) TmaMaps {
  CUtensorMap view[3][4];   // [ViewId][query, key, value, output (language-model patterns, boxes of 32 rows)]
};
constexpr int OUT_ROWS = 32;      // rows of an output box: what one epilogue warp stages

// Can the problem's tiles be fetched as TMA boxes?
INTRA_HD bool tma_supported(const Problem& p) {
  switch (p.kind) {
    case KIND_LLM_SCATTER: return true;
    case KIND_LLM_GATHER1: return TILE_M % p.G == 0 && p.S % (p.G * p.G) == 0;
    case KIND_LLM_WINDOW: return true;
    case KIND_IMG_SCATTER:
    case KIND_IMG_GATHER0:
      return p.W % 8 == 0 && p.W <= 256 && TILE_M % (p.W / 4) == 0 && 2 * (TILE_M / (p.W / 4)) <= 256;
    default: return false;
  }
}

// Box coordinates c1, c2 (c0 is the half of the head dim, c3 the head, c4 the batch) and view of a query tile.
struct QPlan {
  int which;         // ViewId
  int c1, c2;
  int patches;       // Gather-0: the tile is two 64-row boxes, one per 8x8 patch, the second at (c1b, c2)
  int c1b;
};
// The same of an item's key tiles: those in the set `text` are the text tokens in order, the others
// (numbered without them) lie at (c1, c2) + i * (s1, s2) of view `which`.
struct KvPlan {
  int which;
  uint32_t text;
  int c1, c2, s1, s2;
};
constexpr uint32_t TEXT_FIRST = 0xfu;      // image-Scatter keys: the text, then the group's image tokens
constexpr uint32_t TEXT_BETWEEN = 0x36u;   // Gather-0 patch pairs: image, 2 text, image, 2 text, image
INTRA_HD bool is_text_tile(uint32_t text, int n) { return n < 32 && ((text >> n) & 1u); }

// Grid rows of the image a tile of an image-Scatter group spans.
INTRA_HD int img_tile_rows(const Problem& p) { return 2 * fdiv(TILE_M, p.by_quads); }

// View and first coordinates of the rows of a Scatter / Gather-1 / window / image-Scatter tile's numbering,
// starting at its beginning.
INTRA_HD void tma_origin(const Problem& p, const Tile& t, int* which, int* c1, int* c2) {
  *which = VIEW_MAIN; *c1 = 0; *c2 = 0;
  switch (t.kind) {
    case KIND_LLM_SCATTER:
      *which = t.g < p.n_longer ? VIEW_TEXT : VIEW_MAIN;
      *c1 = t.g < p.n_longer ? t.g : t.g - p.n_longer;
      break;
    case KIND_LLM_GATHER1: *c1 = t.g * p.G; break;
    case KIND_LLM_WINDOW: *c1 = t.kbase; break;
    case KIND_IMG_SCATTER:
      *which = p.kind == KIND_IMG_GATHER0 ? VIEW_AUX : VIEW_MAIN;
      *c1 = t.g % 4; *c2 = t.g / 4;
      break;
    default: break;
  }
}

// Query sub-tile `t`.
INTRA_HD QPlan plan_q(const Problem& p, const Tile& t) {
  QPlan q;
  q.patches = 0; q.c1b = 0;
  if (t.kind == KIND_IMG_GATHER0) {
    q.which = VIEW_MAIN;
    q.c1 = PATCH * t.pcol; q.c2 = PATCH * t.prow;
    q.patches = 1;
    q.c1b = PATCH * (t.pcol + (t.nq > PATCH * PATCH ? 1 : 0));    // no right patch: the left one again
    return q;
  }
  tma_origin(p, t, &q.which, &q.c1, &q.c2);
  switch (t.kind) {
    case KIND_LLM_SCATTER: q.c2 = t.t0; break;
    case KIND_LLM_GATHER1: q.c2 = fdiv(t.t0, p.by_G); break;
    case KIND_LLM_WINDOW: q.c1 = t.t0; break;
    default:
      if (t.is_text) { q.which = VIEW_TEXT; q.c1 = t.g * TEXT_CHUNK; q.c2 = 0; }
      else q.c2 += (t.t0 / TILE_M) * img_tile_rows(p);
      break;
  }
  return q;
}

// Key tiles of key-slot map `t`.
INTRA_HD KvPlan plan_kv(const Problem& p, const Tile& t) {
  KvPlan k;
  k.text = 0; k.s1 = 0; k.s2 = 0;
  if (t.kind == KIND_IMG_GATHER0) {
    k.which = VIEW_MAIN;
    k.text = TEXT_BETWEEN;
    k.c1 = t.r0; k.c2 = t.c0; k.s2 = TILE_N / WIN;
    return k;
  }
  tma_origin(p, t, &k.which, &k.c1, &k.c2);
  switch (t.kind) {
    case KIND_LLM_SCATTER: k.s2 = TILE_N; break;
    case KIND_LLM_GATHER1: k.s2 = fdiv(TILE_N, p.by_G); break;
    case KIND_LLM_WINDOW: k.s1 = TILE_N; break;
    default: k.text = TEXT_FIRST; k.s2 = img_tile_rows(p); break;
  }
  return k;
}
INTRA_HD void kv_box(const KvPlan& k, int n, int* which, int* c1, int* c2) {
  int t = 0;                                     // text tiles before tile n
  const uint32_t before = n < 32 ? k.text & ((1u << n) - 1u) : k.text;
#ifdef __CUDA_ARCH__
  t = __popc(before);
#else
  for (uint32_t m = before; m != 0; m &= m - 1) ++t;
#endif
  const bool text = is_text_tile(k.text, n);
  *which = text ? int(VIEW_TEXT) : k.which;
  *c1 = text ? t * TILE_N : k.c1 + (n - t) * k.s1;
  *c2 = text ? 0 : k.c2 + (n - t) * k.s2;
}

}  // namespace intra
