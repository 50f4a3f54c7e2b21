// The reconstruction basis of one cell at a point, generated from the compile-time exponent table.
#pragma once
#include "fast_common.cuh"

namespace dndsb
{
// threads to a row (a boundary cell with its faces' points) of the boundary kernels of the reconstruction and its transpose:
// one per point, and with one or two points per face more, as the row's sums and its product with A^-1 are shared out over
// them.  One point per face, degree 2: the sweep of 14,112 tets takes 28 us with eight threads to a cell, 59 with one per
// point and 41 with one thread per cell and no shared memory; that of 5,760 hexahedra 27, 66 and 34; their transposes 42, 94
// and 52, and 33, 84 and 40.
inline int bnd_row_threads(int nGf) { return nGf < 3 ? 8 : nGf; }

// phi_j (moments removed) and, with GRAD, its gradient of the R reconstruction rows of cell c at point p, generated
// from the compile-time exponent table: a table filled by runtime loops lives in local memory
template <int DIM, int P, bool GRAD>
DNDSB_D void basis_rows(const GeomD &g, const VRD &vr, int64_t c, const real *p, real *phi, real (*dphi)[DIM])
{
    constexpr int NDOF = ndof_of<DIM>(P);
    real L[3];
    cell_lengths<DIM>(&g.cellScale[c * 3], vr.s.anisotropicLengths, L);
    const real *cent = &g.cellCent[c * 3], *mom = &vr.baseMoment[c * NDOF];
    const real x = (p[0] - cent[0]) / L[0], y = (p[1] - cent[1]) / L[1], z = DIM == 3 ? (p[2] - cent[2]) / L[2] : 0.0;
    const real px[4] = {1, x, x * x, x * x * x}, py[4] = {1, y, y * y, y * y * y}, pz[4] = {1, z, z * z, z * z * z};
#pragma unroll
    for (int k = 1; k < NDOF; k++)
    {
        const int e = fastc::mcode(DIM, k), ex = e & 3, ey = (e >> 2) & 3, ez = (e >> 4) & 3;
        phi[k - 1] = px[ex] * py[ey] * pz[ez] - mom[k];
        if constexpr (GRAD)
        {
            dphi[k - 1][0] = ex ? ex * px[ex ? ex - 1 : 0] * py[ey] * pz[ez] / L[0] : 0.0;
            dphi[k - 1][1] = ey ? ey * px[ex] * py[ey ? ey - 1 : 0] * pz[ez] / L[1] : 0.0;
            if constexpr (DIM == 3)
                dphi[k - 1][2] = ez ? ez * px[ex] * py[ey] * pz[ez ? ez - 1 : 0] / L[2] : 0.0;
        }
    }
}
} // namespace dndsb
