// Vector kernels of the native pseudo-time iteration (hotpath.cu), used by dndsb_eval_pseudo_iteration.
#pragma once
#include "solver.cuh"
namespace dndsb
{
// res = other - u / dt + alphaDiag rhs; dTau /= alphaDiag
int unsteady_residual(int64_t nCell, int nv, const real *other, const real *u, const real *rhs, real dt, real alphaDiag, real *res, real *dTau,
                      cudaStream_t st);
int add_increment(int64_t n, const real *inc, real *u, cudaStream_t st); // u += inc
} // namespace dndsb
