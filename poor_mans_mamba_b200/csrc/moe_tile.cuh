// Where a row tile of the grouped products lies, shared by their kernels.
#pragma once
#include "common.cuh"

namespace pmm {

// Finds the expert and the rows of row tile `tile` (tile_rows rows each); false when there is no such tile.  Called by whole
// warps: a lane reads one expert's bounds, so that the answer is one round trip to memory away (a search over the
// bounds is one a step, each behind the other).
__device__ __forceinline__ bool moe_tile(int tile, const int* __restrict__ offsets, const int* __restrict__ tile_start,
                                         int E, int tile_rows, int& e, int& row0, int& row1) {
  const int lane = threadIdx.x & 31;
  for (int base = 0; base < E; base += 32) {
    const int mine = base + lane;
    int first = 0, next = 0, rows0 = 0, rows1 = 0;
    if (mine < E) {
      first = tile_start[mine];
      next = tile_start[mine + 1];
      rows0 = offsets[mine];
      rows1 = offsets[mine + 1];
    }
    const unsigned hit = __ballot_sync(0xffffffffu, first <= tile && tile < next);
    if (hit == 0) continue;
    const int src = __ffs(hit) - 1;
    e = base + src;
    row0 = __shfl_sync(0xffffffffu, rows0, src) + (tile - __shfl_sync(0xffffffffu, first, src)) * tile_rows;
    row1 = min(__shfl_sync(0xffffffffu, rows1, src), row0 + tile_rows);
    return true;
  }
  return false;
}

}  // namespace pmm
