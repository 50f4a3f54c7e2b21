// The solution update of the Krylov solvers (reduce.cu): x += sum_i y_i colScale_i V_i over the valid columns gsc[2]
// (at most k), y = gsc[yOff ...]; columns krylov_ld(n) apart, 16-byte aligned; prec 0: double, 1: float.
#pragma once
#include "solver.cuh"
namespace dndsb
{
void krylov_update_x(int prec, int64_t n, int k, const void *V, const real *gsc, int yOff, const real *colScale, void *x, cudaStream_t st);
}
