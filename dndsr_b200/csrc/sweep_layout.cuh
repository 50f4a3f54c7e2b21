// Layout of the packed sweep coefficients (VRD::sweepCoef), by the rows R and the number of cells: entry (i, j) of
// A^-1 B_k for j < R, (A^-1 b_k)_i for j = R, at
//   tiled:     [tile of 32 cells][face k][j][i][32], zero beyond the last cell
//   otherwise: [cell][face k][j][i]
// The tiled kernel needs enough tiles to fill the GPU: at 36k cells it takes 33 us against 48 of the rows' layout.
#pragma once
#include <cstdint>
namespace dndsb
{
constexpr int64_t kTiledCells = 20000;
inline bool sweep_tiled(int R, int64_t nCell) { return R == 9 && nCell >= kTiledCells; }
} // namespace dndsb
