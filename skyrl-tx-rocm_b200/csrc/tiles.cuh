// M tiles of the adapter-sorted row space and the adapters that own their rows, as the projection and GEMM
// kernels walk them.
//
// Dense lists (route_dense_kernel): tile i holds sorted rows [128 i, 128 i + 128) whatever adapters they belong
// to; its SEGMENTS are the distinct adapters of the tile, each with a 128-bit mask of the rows it owns.  A
// tcgen05.mma can leave accumulator lanes (= rows) untouched, so the rank-r contraction of every segment
// accumulates onto its own rows of one shared accumulator and no tile is ever cut at an adapter boundary: 256
// rows over 32 adapters are 2 tiles, where tiles of at most two adapters were 16.
//   entry int4 (first row, rows, segments, ~first segment)   w < 0
// Lists of the public routing entry point (at most two adapters a tile, z in two slots):
//   entry int4 (first row, rows, adapter, second)            w >= 0
// No list at all (one adapter, no ids): tile i is computed, adapter 0 owns every row.
#pragma once

#include <stdint.h>

namespace skyrl {

struct TileSource {
  const int4* tiles;            // NULL: computed tiles over rows [row0, row_end)
  const int4* seg_mask;
  const int32_t* seg_adapter;
  const int32_t* num_tiles;     // NULL: `count` is the number of tiles
  int count;
  int row0, row_end;
};

#ifdef __CUDACC__
__device__ __forceinline__ int tile_count(const TileSource& s) { return s.num_tiles != nullptr ? *s.num_tiles : s.count; }

__device__ __forceinline__ int4 tile_at(const TileSource& s, int i) {
  if (s.tiles != nullptr) return __ldg(s.tiles + i);
  const int r = s.row0 + i * 128;
  return make_int4(r, min(128, s.row_end - r), 0, 0);
}

__device__ __forceinline__ bool tile_is_dense(const int4& t) { return t.w < 0; }
__device__ __forceinline__ int tile_segments(const int4& t) { return t.w < 0 ? t.z : (t.w == 0 ? 1 : 2); }
__device__ __forceinline__ int segment_adapter(const TileSource& s, const int4& t, int j) {
  if (t.w < 0) return __ldg(s.seg_adapter + (~t.w) + j);
  return j == 0 ? t.z : (t.w & 0xffff) - 1;
}
// bit r of word r / 32: row r of the tile belongs to segment j
__device__ __forceinline__ int4 segment_mask(const TileSource& s, const int4& t, int j) {
  if (t.w < 0) return __ldg(s.seg_mask + (~t.w) + j);
  if (t.w == 0) return make_int4(-1, -1, -1, -1);
  const int split = t.w >> 16;
  int w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int n = min(max(split - 32 * q, 0), 32);
    const int low = n == 32 ? -1 : (1 << n) - 1;
    w[q] = j == 0 ? low : ~low;
  }
  return make_int4(w[0], w[1], w[2], w[3]);
}
// z slot a segment's rows keep their LoRA-A projection in
__device__ __forceinline__ int segment_slot(const int4& t, int j) { return t.w < 0 ? 0 : j; }
#endif

}  // namespace skyrl
