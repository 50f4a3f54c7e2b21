// Cell vectors of the native linear solve: n cells of NV variables as [n][4] followed by [n][NV - 4].  The first four
// variables of a cell are one aligned vector load (the gathers of the sweeps are bound by load instructions, not by
// bytes: a row of five scalars costs five), and no pad is added to the Krylov columns.
#pragma once
#include "platform.cuh"

namespace dndsb
{
namespace vsplit
{
template <typename T>
struct Vec4;
template <>
struct Vec4<float>
{
    using type = float4;
};
template <>
struct Vec4<double>
{
    using type = double4;
};

template <int NV>
DNDSB_HD int64_t at(int64_t n, int64_t c, int v) { return v < 4 ? c * 4 + v : 4 * n + c * (NV - 4) + (v - 4); }

template <typename T, int NV>
DNDSB_D void load(const T *x, int64_t n, int64_t c, T *d)
{
    const typename Vec4<T>::type a = ((const typename Vec4<T>::type *)x)[c];
    d[0] = a.x, d[1] = a.y, d[2] = a.z, d[3] = a.w;
#pragma unroll
    for (int v = 4; v < NV; v++)
        d[v] = x[4 * n + c * (NV - 4) + (v - 4)];
}

template <typename T, int NV>
DNDSB_D void store(T *x, int64_t n, int64_t c, const T *d)
{
    typename Vec4<T>::type a;
    a.x = d[0], a.y = d[1], a.z = d[2], a.w = d[3];
    ((typename Vec4<T>::type *)x)[c] = a;
#pragma unroll
    for (int v = 4; v < NV; v++)
        x[4 * n + c * (NV - 4) + (v - 4)] = d[v];
}

// variable of flat element i
template <int NV>
DNDSB_HD int var_of(int64_t n, int64_t i) { return i < 4 * n ? (int)(i & 3) : 4 + (NV > 5 ? (int)((i - 4 * n) % (NV - 4)) : 0); }
} // namespace vsplit
} // namespace dndsb
