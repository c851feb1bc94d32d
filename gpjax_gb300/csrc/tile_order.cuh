// Launch index -> output tile, shared by the tensor-core GEMMs.
#pragma once
#include <cuda_runtime.h>

namespace gpk {
namespace tc {

constexpr int BM = 128;  // output tile rows (TMEM lanes)

// Launch index -> output tile (I, J), grouped so that the CTAs resident at
// one time share operand panels in L2: groups of TILE_GROUP tile rows, walked
// column by column (consecutive CTAs take consecutive rows of one column).
// Row tiles are BM high, column tiles bn wide; for c_lower only tiles holding
// elements on or below the diagonal exist: row tile I reaches column tiles
// J < ncols(I), and column tile J starts at row tile imin(J).
constexpr int TILE_GROUP = 8;
__host__ __device__ inline int lower_ncols(int I, int tiles_n, int bn) {
  return min(tiles_n, (I * BM + BM - 1) / bn + 1);
}
__host__ __device__ inline void tile_of(int t, int c_lower, int tiles_m, int tiles_n, int bn,
                                        int& I, int& J) {
  constexpr int G = TILE_GROUP;
  if (!c_lower) {
    const int g = t / (G * tiles_n), l = t % (G * tiles_n);
    const int rows = min(G, tiles_m - g * G);
    J = l / rows;
    I = g * G + l % rows;
    return;
  }
  int g = 0, base = 0, rows = 0;
  for (;; ++g) {
    rows = min(G, tiles_m - g * G);
    int cnt = 0;
    for (int r = 0; r < rows; ++r) cnt += lower_ncols(g * G + r, tiles_n, bn);
    if (t < base + cnt) break;
    base += cnt;
  }
  int l = t - base;
  const int full_cols = lower_ncols(g * G, tiles_n, bn);  // every row of the group reaches these
  if (l < full_cols * rows) {
    J = l / rows;
    I = g * G + l % rows;
    return;
  }
  l -= full_cols * rows;
  for (J = full_cols;; ++J) {
    const int num = J * bn - BM + 1;
    const int imin = num > 0 ? (num + BM - 1) / BM : 0;
    const int r0 = max(g * G, imin);
    const int cnt = g * G + rows - r0;
    if (l < cnt) {
      I = r0 + l;
      return;
    }
    l -= cnt;
  }
}

// Number of launch indices tile_of maps (the grid of one GEMM).
__host__ __device__ inline int tile_count(int c_lower, int tiles_m, int tiles_n, int bn) {
  if (!c_lower) return tiles_m * tiles_n;
  int cnt = 0;
  for (int I = 0; I < tiles_m; ++I) cnt += lower_ncols(I, tiles_n, bn);
  return cnt;
}

}  // namespace tc
}  // namespace gpk
