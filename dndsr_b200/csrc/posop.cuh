// The scalar-Jacobian LU-SGS operator of the native linear solve in colour-position order: LUSGSMatrixInit
// (src/Euler/EulerEvaluator.hxx:37-159) packed, UpdateSGS (:550-693) and LUSGSMatrixVec (:175-274) on it.
//
// Per position the neighbours are kept in compact slots ordered by when a forward sweep has passed them: first the
// `lower` ones (colour before the position's own), then the `upper` ones, then periodic images of the cell itself
// (in the product, in no sweep); slots of boundary faces are dropped.  Per slot {w n, w lambda} with
// w = alpha A_f / (2 V_c) and the neighbour's position, both in tiles of 32 positions (the 32 lanes of a warp read one
// slot of their positions as one contiguous line).  The flux Jacobian of a cell needs only its velocity and total
// enthalpy, kept as one aligned 4-vector per cell (and U5 / rho for the SA variable), and the vectors are split as in
// vec_split.cuh, so a product takes three vector loads and a scalar one per neighbour and no division:
//   A(U) dU . n:  q = dm.n - (v.n) drho, dp = (gamma - 1)(dE - v.dm + v^2 drho / 2);
//   {dm.n, dm (v.n) + v q + n dp, (dE + dp)(v.n) + H q, dU5 (v.n) + (U5 / rho) q}.
//
// With A = L + D + U (+ S, the self images) a symmetric sweep is M^-1 = (D + U)^-1 D (D + L)^-1, and
//   M^-1 A v = (D + U)^-1 D [v + (D + L)^-1 (U + S) v]
// (Eisenstat's form): the forward sweep takes the upper slots of v and the lower slots of its own result, the
// backward sweep the upper slots, so a preconditioned product reads one and a half operators instead of two and a
// half (a product, then two sweeps that each test all slots) and writes no intermediate A v.  From a zero start the
// backward sweep of a pair is x_p -= D_p^-1 sum_upper, in place, and the last colour has nothing to do.
//
// Bound by the operator stream and the neighbour gathers.  GMRES(30) preconditioned by one pair, per solve: 249,600
// tets in FP64 2.57 ms of sweeps and products before (248 + 30 launches, neighbours' conservative states gathered and
// divided, all slots tested in each sweep); 1,996,800 tets in FP32 8.28 ms.  This form: 1.69 ms and 5.15 ms, with
// the vectors as cell rows 1.89 ms and 5.36 ms.
#pragma once
#include "solver.cuh"
#include "vec_split.cuh"
#include "chain.cuh"

namespace dndsb
{
namespace posop
{
using vsplit::Vec4;

// diagonals per cell: 1, or NV with the SA source Jacobian
template <int NV>
constexpr int jd_of() { return NV == 6 ? NV : 1; }

// slot k of position p in the tiled arrays
template <int NF>
DNDSB_HD int64_t slot_at(int64_t p, int k) { return ((((p >> 5) * NF) + k) << 5) + (p & 31); }

template <typename T>
struct Op
{
    using T4 = typename Vec4<T>::type;
    int64_t n = 0;            // positions
    int32_t *nbr = nullptr;   // [tiles][NF][32] neighbour positions
    int32_t *cnt = nullptr;   // [n] lower | (lower + upper) << 8 | all << 16
    T4 *op = nullptr;         // [tiles][NF][32] {w n, w lambda}
    T *jd = nullptr;          // [n][JD] diagonal
    T *jdi = nullptr;         // [n][JD] its inverse
    T4 *vh = nullptr;         // [n] velocity and total enthalpy
    T *nu = nullptr;          // [n] U5 / rho (6 variables)
};

// Releases its successor on entry, so the next kernel of the sequence may not read the operator ahead of its wait; the
// sweeps and products do, and another kernel that waits (k_gather_T of linsolve.cu) has to stand before the first of them.
template <typename T, int NV, int NF>
DNDSB_GLOBAL void k_build(MeshD m, GeomD g, const real *lamFace, const real *dTau, real dt, real alphaDiag, real gamma, const real *u,
                          const real *jSource, const int32_t *__restrict__ cellPos, Op<T> A)
{
    chain_step();
    using T4 = typename Vec4<T>::type;
    DNDSB_KERNEL_LOOP(p, m.nCell)
    {
        const int64_t c = m.colorCells[p];
        const int col = m.cellColor[c];
        const real iv = 1.0 / g.vol[c];
        const real cf = 0.5 * alphaDiag / g.vol[c];
        real fp = 1.0 / dTau[c] + 1.0 / dt;
        T4 o4[NF];
        int o[NF], cls[NF];
#pragma unroll
        for (int k = 0; k < NF; k++)
        {
            int pk = m.cell2face[c * NF + k];
            int64_t f = pk >> 1;
            real sg = (pk & 1) ? -1.0 : 1.0;
            fp += (0.5 * alphaDiag) * g.faceArea[f] * lamFace[f] * iv;
            real w = cf * g.faceArea[f];
            o4[k].x = (T)(w * g.faceMeanNorm[f * 3] * sg);
            o4[k].y = (T)(w * g.faceMeanNorm[f * 3 + 1] * sg);
            o4[k].z = (T)(w * g.faceMeanNorm[f * 3 + 2] * sg);
            o4[k].w = (T)(w * lamFace[f]);
            o[k] = m.cellNbr[c * NF + k];
            cls[k] = o[k] < 0 ? 3 : o[k] == c ? 2 : m.cellColor[o[k]] < col ? 0 : 1;
            o[k] = o[k] < 0 ? -1 : cellPos[o[k]];
        }
        int n = 0, cnt = 0;
        for (int x = 0; x < 3; x++)
        {
#pragma unroll
            for (int k = 0; k < NF; k++)
                if (cls[k] == x)
                {
                    A.op[slot_at<NF>(p, n)] = o4[k];
                    A.nbr[slot_at<NF>(p, n)] = o[k];
                    n++;
                }
            cnt |= n << (8 * x);
        }
        A.cnt[p] = cnt;
        constexpr int JD = jd_of<NV>();
        for (int v = 0; v < JD; v++)
        {
            const T d = (T)(fp + (JD > 1 ? alphaDiag * jSource[c * NV + v] : 0.0));
            A.jd[p * JD + v] = d;
            A.jdi[p * JD + v] = T(1) / d;
        }
        const real ir = 1.0 / u[c * NV];
        const real v0 = u[c * NV + 1] * ir, v1 = u[c * NV + 2] * ir, v2 = u[c * NV + 3] * ir;
        const real pr = (gamma - 1) * (u[c * NV + 4] - 0.5 * u[c * NV] * (v0 * v0 + v1 * v1 + v2 * v2));
        T4 vh;
        vh.x = (T)v0, vh.y = (T)v1, vh.z = (T)v2, vh.w = (T)((u[c * NV + 4] + pr) * ir);
        A.vh[p] = vh;
        if (NV == 6)
            A.nu[p] = (T)(u[c * NV + 5] * ir);
    }
}

// buf += f (w A(U) - w lambda) dU for one neighbour
template <typename T, int NV>
DNDSB_D void add_jac(const typename Vec4<T>::type &o, const typename Vec4<T>::type &s, T nu, const T *d, T g1, T f, T *buf)
{
    const T vn = s.x * o.x + s.y * o.y + s.z * o.z;
    const T mn = d[1] * o.x + d[2] * o.y + d[3] * o.z;
    const T q = mn - vn * d[0];
    const T dp = g1 * (d[4] - (s.x * d[1] + s.y * d[2] + s.z * d[3]) + T(0.5) * (s.x * s.x + s.y * s.y + s.z * s.z) * d[0]);
    buf[0] += f * (mn - o.w * d[0]);
    buf[1] += f * (d[1] * (vn - o.w) + s.x * q + o.x * dp);
    buf[2] += f * (d[2] * (vn - o.w) + s.y * q + o.y * dp);
    buf[3] += f * (d[3] * (vn - o.w) + s.z * q + o.z * dp);
    buf[4] += f * ((d[4] + dp) * vn + s.w * q - o.w * d[4]);
    if (NV == 6)
        buf[NV - 1] += f * (d[NV - 1] * (vn - o.w) + nu * q);
}

// buf += sum over the slots [j0, j1) of f (w A - w lambda) x_q, with x = xa, f = fa for slots below ja and xb, fb from
// there; a group's loads are all issued before the first use.  The first group's coefficients are read ahead of the
// chain's wait; own() reads the row's own values (and may set fb) right
// after it.  What the sequence writes is passed without __restrict__, so that no load moves ahead of the wait.
template <typename T, int NV, int NF, typename F>
DNDSB_D void add_slots(const Op<T> &A, int64_t p, int j0, int j1, int ja, const T *xa, T fa, const T *xb, const T &fb, T g1, T *buf, F own)
{
    using T4 = typename Vec4<T>::type;
    constexpr int G = NF <= 4 ? NF : 3;
    int q[NF];
#pragma unroll
    for (int k = 0; k < NF; k++)
        q[k] = k >= j0 && k < j1 ? A.nbr[slot_at<NF>(p, k)] : -1;
#pragma unroll
    for (int b = 0; b < NF; b += G)
    {
        T4 o[G], s[G];
        T d[G][NV], nu[G];
#pragma unroll
        for (int k = 0; k < G; k++)
            if (q[b + k] >= 0)
            {
                o[k] = A.op[slot_at<NF>(p, b + k)];
                s[k] = A.vh[q[b + k]];
                nu[k] = NV == 6 ? A.nu[q[b + k]] : T(0);
            }
        if (b == 0)
        {
            chain_step();
            own();
        }
#pragma unroll
        for (int k = 0; k < G; k++)
            if (q[b + k] >= 0)
                vsplit::load<T, NV>(b + k < ja ? xa : xb, A.n, q[b + k], d[k]);
#pragma unroll
        for (int k = 0; k < G; k++)
            if (q[b + k] >= 0)
                add_jac<T, NV>(o[k], s[k], nu[k], d[k], g1, b + k < ja ? fa : fb, buf);
    }
}

// x_p = D_p^-1 (rhs_p - sum_lower xLow - sum_upper xUp) over positions [pBeg, pEnd); a null xLow or xUp is a zero
// vector whose slots are skipped.  xNew may be xLow or xUp (other colours' rows are read, the own row written).
template <typename T, int NV, int NF>
DNDSB_GLOBAL void k_sweep(int64_t pBeg, int64_t pEnd, Op<T> A, const T *rhs, const T *xLow, const T *xUp, T *xNew, T g1)
{
    constexpr int JD = jd_of<NV>();
    DNDSB_KERNEL_LOOP(ii, pEnd - pBeg)
    {
        const int64_t p = pBeg + ii;
        const int cnt = A.cnt[p], nl = cnt & 255, nu = (cnt >> 8) & 255;
        T buf[NV], r[NV];
#pragma unroll
        for (int v = 0; v < NV; v++)
            buf[v] = 0;
        add_slots<T, NV, NF>(A, p, xLow ? 0 : nl, xUp ? nu : nl, nl, xLow, T(1), xUp, T(1), g1, buf,
                             [&] { vsplit::load<T, NV>(rhs, A.n, p, r); });
#pragma unroll
        for (int v = 0; v < NV; v++)
            r[v] = (r[v] - buf[v]) * A.jdi[p * JD + (JD > 1 ? v : 0)];
        vsplit::store<T, NV>(xNew, A.n, p, r);
    }
}

// the backward half of a symmetric sweep whose forward half is in x: x_p -= D_p^-1 sum_upper x, one colour, in place
template <typename T, int NV, int NF>
DNDSB_GLOBAL void k_back(int64_t pBeg, int64_t pEnd, Op<T> A, T *x, T g1)
{
    constexpr int JD = jd_of<NV>();
    DNDSB_KERNEL_LOOP(ii, pEnd - pBeg)
    {
        const int64_t p = pBeg + ii;
        const int cnt = A.cnt[p], nl = cnt & 255, nu = (cnt >> 8) & 255;
        T buf[NV], r[NV];
#pragma unroll
        for (int v = 0; v < NV; v++)
            buf[v] = 0;
        add_slots<T, NV, NF>(A, p, nl, nu, nl, (const T *)x, T(1), (const T *)x, T(1), g1, buf, [&] { vsplit::load<T, NV>(x, A.n, p, r); });
#pragma unroll
        for (int v = 0; v < NV; v++)
            r[v] -= buf[v] * A.jdi[p * JD + (JD > 1 ? v : 0)];
        vsplit::store<T, NV>(x, A.n, p, r);
    }
}

// the forward half of M^-1 A (s x), s = *xs (null: 1): t_p = D_p^-1 (s sum_{upper, self} x - sum_lower t), y_p = s x_p + t_p
template <typename T, int NV, int NF>
DNDSB_GLOBAL void k_product_forward(int64_t pBeg, int64_t pEnd, Op<T> A, const T *x, T *t, T *y, T g1, const real *xs)
{
    constexpr int JD = jd_of<NV>();
    T sx = 1;
    DNDSB_KERNEL_LOOP(ii, pEnd - pBeg)
    {
        const int64_t p = pBeg + ii;
        const int cnt = A.cnt[p], nl = cnt & 255, na = cnt >> 16;
        T buf[NV], r[NV];
#pragma unroll
        for (int v = 0; v < NV; v++)
            buf[v] = 0;
        add_slots<T, NV, NF>(A, p, 0, na, nl, (const T *)t, T(-1), x, sx, g1, buf,
                             [&]
                             {
                                 sx = xs ? (T)*xs : T(1);
                                 vsplit::load<T, NV>(x, A.n, p, r);
                             });
#pragma unroll
        for (int v = 0; v < NV; v++)
        {
            buf[v] *= A.jdi[p * JD + (JD > 1 ? v : 0)];
            r[v] = sx * r[v] + buf[v];
        }
        vsplit::store<T, NV>(t, A.n, p, buf);
        vsplit::store<T, NV>(y, A.n, p, r);
    }
}

// Ax = A (s x), s = *xs (null: 1)
template <typename T, int NV, int NF>
DNDSB_GLOBAL void k_product(int64_t n, Op<T> A, const T *x, T *Ax, T g1, const real *xs)
{
    constexpr int JD = jd_of<NV>();
    T sx = 1;
    DNDSB_KERNEL_LOOP(p, n)
    {
        const int cnt = A.cnt[p];
        T buf[NV];
        add_slots<T, NV, NF>(A, p, 0, cnt >> 16, NF, x, T(1), x, T(1), g1, buf,
                             [&]
                             {
                                 sx = xs ? (T)*xs : T(1);
                                 vsplit::load<T, NV>(x, A.n, p, buf);
#pragma unroll
                                 for (int v = 0; v < NV; v++)
                                     buf[v] *= A.jd[p * JD + (JD > 1 ? v : 0)];
                             });
#pragma unroll
        for (int v = 0; v < NV; v++)
            buf[v] *= sx;
        vsplit::store<T, NV>(Ax, A.n, p, buf);
    }
}
} // namespace posop
} // namespace dndsb
