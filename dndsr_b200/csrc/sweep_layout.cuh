// Layout of the packed sweep coefficients (VRD::sweepCoef), by the rows R and the number of cells: entry (i, j) of
// A^-1 B_k for j < R, (A^-1 b_k)_i for j = R, at
//   tiled:     [tile of 32 cells][face k][j][i][32], zero beyond the last cell
//   otherwise: [cell][face k][j][i]
// The tiled kernel needs enough tiles (a block each) to fill the GPU; it is the faster one from about 10,000 cells on.
// Tiled against rows, FP64 coefficients, us: hexahedra 4,096 cells 12.8 and 11.5, 8,000 14.2 and 14.4, 10,648 17.8 and
// 18.9, 13,824 18.3 and 23.1, 17,576 19.5 and 29.3, 27,000 39.4 and 46.6, 262,144 256 and 383; quadrilaterals 10,000 13.5
// and 12.2, 14,400 13.8 and 17.0, 40,000 40.9 and 42.7; tetrahedra with the boundary term 6,912 28.8 and 26.8, 11,760 30.9
// and 33.0, 36,162 57.3 and 66.2.  FP32 coefficients: hexahedra 10,648 18.4 and 18.3, 13,824 18.4 and 20.8.
#pragma once
#include <cstdint>
namespace dndsb
{
constexpr int64_t kTiledCells = 12000;
inline bool sweep_tiled(int R, int64_t nCell) { return R == 9 && nCell >= kTiledCells; }
} // namespace dndsb
