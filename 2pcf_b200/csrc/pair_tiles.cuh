// pair_tiles.cuh -- how a warp of the planar pair kernels walks the source rows
// of a work item as tiles of 32-source sub-chunks.
#pragma once
#include <cuda_runtime.h>

#include "tpcf_internal.cuh"

namespace tpcf {

// ------------------------------------------------------------- tile ring --
// Each warp walks the cell rows of its work item 32 at a time, lane r holding
// the source span [s0, s1) of row c0 + r.  A row's span covers the sub-chunks
// [s0 / 32, ceil(s1 / 32)); its first and last sub-chunks are partial when s0
// or s1 is not a multiple of 32.  Tile k of the pass is the (k - first)-th
// group of TCH sub-chunks of the row whose prefix of tile counts contains k.
struct TileGeom {
  int c0, n, lo0, hiL;
};
template <int TCH>
__device__ __forceinline__ int tiles_of_span(int s, int e) {
  if (e <= s) return 0;
  const int nc = ((e + kChunk - 1) >> 5) - (s >> 5);
  return (nc + TCH - 1) / TCH;
}
// Called by all 32 lanes with the same k (0 <= k < the pass's tile count);
// incl = this lane's inclusive prefix of tile counts, s0/s1 its row's span.
template <int TCH>
__device__ __forceinline__ TileGeom tile_of(int k, int incl, int ntr, int s0, int s1) {
  const int r = __popc(__ballot_sync(0xffffffffu, incl <= k));  // first row with incl > k
  const int s = __shfl_sync(0xffffffffu, s0, r);
  const int e = __shfl_sync(0xffffffffu, s1, r);
  const int first = __shfl_sync(0xffffffffu, incl - ntr, r);
  const int kk = k - first;
  const int cA = s >> 5, cB = (e + kChunk - 1) >> 5;
  TileGeom t;
  t.c0 = cA + kk * TCH;
  t.n = min(TCH, cB - t.c0);
  t.lo0 = kk == 0 ? (s & (kChunk - 1)) : 0;
  t.hiL = (t.c0 + t.n == cB && (e & (kChunk - 1))) ? (e & (kChunk - 1)) : kChunk;
  return t;
}

}  // namespace tpcf
