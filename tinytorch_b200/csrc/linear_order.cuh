// In which order the persistent projection kernels (linear_tc.cu, linear_tile.cu) go through the tiles of an output.
#pragma once
#include "common.cuh"

namespace ttattn {

// Tile t: groups of group_m row-tiles one after the other, within a group column by column.
__device__ __forceinline__ void tile_of(int t, int group_m, int tiles_m, int tiles_n, int* m_tile, int* n_tile) {
  const int per_group = group_m * tiles_n;
  const int g = t / per_group, in_g = t - g * per_group;
  const int first_m = g * group_m;
  const int gm = tiles_m - first_m < group_m ? tiles_m - first_m : group_m;
  *m_tile = first_m + in_g % gm;
  *n_tile = in_g / gm;
}

// Row-tiles (of `bm` rows) per group.  The pairs running at one time work on one group: its rows of x are read from HBM once as long
// as they stay in L2 while w streams by, and w once per group.  So: as many row-tiles (a power of two) as take 60 MB of
// the 126; where w itself stays in L2 (up to 40 MB), 4, so that x does not push it out.  Under sustained load, us, with 4
// before: 4096 x 4096 -> 12288 342 -> 312, 16384 x 4096 -> 12288 1341 -> 1225, 8192 cubed 893 -> 861, 2000 x 4096 -> 28672
// 387 -> 362 (and 32 or 64 instead of 16 for the second: 1377, 1625).
inline int rows_per_group(const LinearCall& c, int bm) {
  const long long x_tile = 2ll * bm * c.K, w_bytes = 2ll * c.N * c.K;
  int group_m = 4;
  if (w_bytes > 40 << 20)
    while (group_m < 64 && group_m * 2 * x_tile <= 60 << 20) group_m *= 2;
  return group_m;
}

}  // namespace ttattn
