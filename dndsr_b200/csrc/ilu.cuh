// Block ILU(0) of the implicit operator: JacobianLocalLU's InPlaceDecompose and Solve (Solver/Direct.hpp:312-405,
// 487-540) for iluCode 0 (the face-neighbour pattern, no fill), run colour by colour.  A row's lower neighbours
// are those of lower rank (rank = position in colour order, or the colour); cells of one colour are never
// adjacent, so every row of a colour depends only on rows of earlier colours and a colour is factored (or
// solved) in one launch.  On a mesh numbered colour by colour this is the reference's natural-order
// factorisation.
//
// Storage: off holds per row r and slot k the block of A (then L for lower and U for upper neighbours), dinv the
// inverted pivots, D the diagonal blocks of A.  BlockLay places element e of row r (E elements per row) in tiles
// of 2^s rows: rows of a tile innermost, so that the 32 threads of a warp read one element of 32 consecutive rows
// as one contiguous 256-byte line and a warp's rows share one contiguous range; s = 0 is rows outermost
// ([row][E]).  nbr [r][NF] holds the neighbour row of each slot (-1: none).
#pragma once
#include "roejac.cuh"
#include "chain.cuh"

namespace dndsb
{
namespace ilu
{
struct BlockLay
{
    int64_t E; // elements per row
    int s;     // log2 of the rows per tile
    DNDSB_HD int64_t at(int64_t r, int64_t e) const { return ((((r >> s) * E) + e) << s) + (r & ((int64_t(1) << s) - 1)); }
};
// rows allocated for a tiled layout of n rows
inline int64_t padded_rows(int64_t n, int s) { return ((n + (int64_t(1) << s) - 1) >> s) << s; }

template <int NV>
DNDSB_HD void mul_sub(const real *A, const real *B, real *C) // C -= A B (row-major NV x NV)
{
    for (int i = 0; i < NV; i++)
        for (int j = 0; j < NV; j++)
        {
            real acc = 0;
            for (int l = 0; l < NV; l++)
                acc += A[i * NV + l] * B[l * NV + j];
            C[i * NV + j] -= acc;
        }
}

template <int NF>
DNDSB_HD int slot_of(const int32_t *nbr, int64_t r, int64_t target)
{
    for (int s = 0; s < NF; s++)
        if (nbr[r * NF + s] == target)
            return s;
    return -1;
}

// the block of elements e0 .. e0 + NV NV - 1 of row r
template <typename T, int NV>
DNDSB_HD void load(const T *src, BlockLay L, int64_t r, int e0, real *dst)
{
    for (int i = 0; i < NV * NV; i++)
        dst[i] = (real)src[L.at(r, e0 + i)];
}
template <typename T, int NV>
DNDSB_HD void store(const real *v, T *dst, BlockLay L, int64_t r, int e0)
{
    for (int i = 0; i < NV * NV; i++)
        dst[L.at(r, e0 + i)] = (T)v[i];
}

// one row of the factorisation: A (the operator's slot blocks) and D (diagonal blocks) in, off / dinv out, in the
// operator's slot order
template <typename T, int NV, int NF>
DNDSB_HD bool factor_row(int64_t r, const int32_t *nbr, const int32_t *rank, const T *A, const T *D, BlockLay offL, BlockLay dL, BlockLay DL,
                         T *off, T *dinv)
{
    constexpr int NN = NV * NV;
    auto rk = [&](int64_t x) { return rank ? (int64_t)rank[x] : x; };
    const int64_t rr = rk(r);
    int low[NF], nLow = 0, upp[NF], nUpp = 0;
    for (int k = 0; k < NF; k++)
    {
        int64_t q = nbr[r * NF + k];
        if (q < 0 || q == r)
            continue;
        if (rk(q) < rr)
        {
            // insertion in ascending rank: the order of the reference's sorted lower row
            int a = nLow++;
            while (a > 0 && rk(nbr[r * NF + low[a - 1]]) > rk(q))
                low[a] = low[a - 1], a--;
            low[a] = k;
        }
        else
            upp[nUpp++] = k;
    }
    real L[NF * NN];
    for (int a = 0; a < nLow; a++)
    {
        int64_t j = nbr[r * NF + low[a]];
        real *Lij = L + a * NN;
        load<T, NV>(A, offL, r, low[a] * NN, Lij);
        for (int b = 0; b < a; b++)
        {
            int64_t k = nbr[r * NF + low[b]];
            int s = slot_of<NF>(nbr, k, j);
            if (s >= 0)
            {
                real Ukj[NN];
                load<T, NV>(off, offL, k, s * NN, Ukj);
                mul_sub<NV>(L + b * NN, Ukj, Lij);
            }
        }
        real Dj[NN], t[NN];
        load<T, NV>(dinv, dL, j, 0, Dj);
        for (int i = 0; i < NN; i++)
            t[i] = 0;
        mul_sub<NV>(Lij, Dj, t);
        for (int i = 0; i < NN; i++)
            Lij[i] = -t[i];
    }
    real Di[NN], Dinv[NN];
    load<T, NV>(D, DL, r, 0, Di);
    for (int b = 0; b < nLow; b++)
    {
        int64_t k = nbr[r * NF + low[b]];
        int s = slot_of<NF>(nbr, k, r);
        if (s >= 0)
        {
            real Uki[NN];
            load<T, NV>(off, offL, k, s * NN, Uki);
            mul_sub<NV>(L + b * NN, Uki, Di);
        }
    }
    bool ok = roej::block_inv<NV>(Di, Dinv);
    if (!ok)
        for (int i = 0; i < NN; i++)
            Dinv[i] = 0;
    store<T, NV>(Dinv, dinv, dL, r, 0);
    for (int a = 0; a < nUpp; a++)
    {
        int64_t j = nbr[r * NF + upp[a]];
        real Uij[NN];
        load<T, NV>(A, offL, r, upp[a] * NN, Uij);
        for (int b = 0; b < nLow; b++)
        {
            int64_t k = nbr[r * NF + low[b]];
            int s = slot_of<NF>(nbr, k, j);
            if (s >= 0)
            {
                real Ukj[NN];
                load<T, NV>(off, offL, k, s * NN, Ukj);
                mul_sub<NV>(L + b * NN, Ukj, Uij);
            }
        }
        store<T, NV>(Uij, off, offL, r, upp[a] * NN);
    }
    for (int a = 0; a < nLow; a++)
        store<T, NV>(L + a * NN, off, offL, r, low[a] * NN);
    real zero[NN];
    for (int i = 0; i < NN; i++)
        zero[i] = 0;
    // slots without a neighbour (boundary faces) and a row's periodic image of itself carry nothing
    for (int k = 0; k < NF; k++)
    {
        int64_t q = nbr[r * NF + k];
        if (q < 0 || q == r)
            store<T, NV>(zero, off, offL, r, k * NN);
    }
    return ok;
}

// rows: the rows of one colour (nullptr: the contiguous range [beg, end))
template <typename T, int NV, int NF>
DNDSB_GLOBAL void k_ilu_factor(int64_t beg, int64_t end, const int32_t *__restrict__ rows, const int32_t *__restrict__ nbr,
                               const int32_t *__restrict__ rank, const T *A, const T *__restrict__ D, BlockLay offL, BlockLay dL, BlockLay DL,
                               T *off, T *dinv, int *err) // A may be off (factored in place)
{
    DNDSB_KERNEL_LOOP(ii, end - beg)
    {
        int64_t r = rows ? (int64_t)rows[beg + ii] : beg + ii;
        if (!factor_row<T, NV, NF>(r, nbr, rank, A, D, offL, dL, DL, off, dinv))
            atomicOr(err, (int)DE_SINGULAR);
    }
}

// Row-parallel kernels on tiled blocks (BlockLay s = 5): a block is NV warps on the 32 rows of one tile, warp i on
// component i of each row, lane on the row.  Warp i loads component i of the neighbours' vectors once for the whole
// block (shared memory), while every thread's NV elements per slot, one contiguous line per warp and element, are
// already in flight.  One thread per row (NV NV elements per slot each) left too few loads in flight on one colour's
// rows: 21 us per colour and solve of 249,600 tets in FP64 (1.4 TB/s), now 9 (forward) and 14 (backward), the product
// 61 -> 50 us; lanes on components with each lane gathering whole neighbour vectors multiplied the gathers by NV.
inline unsigned tile_blocks(int64_t beg, int64_t end) { return (unsigned)(((end + 31) >> 5) - (beg >> 5)); }

// Row i of the inverse of 32 blocks (lanes) whose rows i the warps i of the block hold, as roej::block_inv forms it; the
// pivot rows go through sD and sU.  False for a singular block.  Every thread of the block calls it.
template <int NV>
DNDSB_D bool tile_inv(const real *row, real (*sD)[32], real (*sU)[32], real *inv)
{
    const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
    real M[NV], X[NV], a = 0;
#pragma unroll
    for (int l = 0; l < NV; l++)
        a = l == i ? row[l] : a;
    __shared__ real sS[NV][32]; // the row scales
    sS[i][lane] = 1.0 / a;
    int ok = a != 0;
#pragma unroll
    for (int l = 0; l < NV; l++)
        M[l] = 1.0 / a * row[l], X[l] = l == i ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < NV; k++)
    {
        __syncthreads();
#pragma unroll
        for (int l = 0; l < NV; l++)
            sD[i * NV + l][lane] = M[l], sU[i * NV + l][lane] = X[l];
        __syncthreads();
        int pr = k;
        real best = fabs(sD[k * NV + k][lane]);
#pragma unroll
        for (int p = k + 1; p < NV; p++)
            if (fabs(sD[p * NV + k][lane]) > best)
                best = fabs(sD[p * NV + k][lane]), pr = p;
        ok = ok && best > 0;
        const real ip = 1.0 / sD[pr * NV + k][lane];
        if (i == pr && i != k)
#pragma unroll
            for (int l = 0; l < NV; l++)
                M[l] = sD[k * NV + l][lane], X[l] = sU[k * NV + l][lane];
        const real fct = M[k];
#pragma unroll
        for (int l = 0; l < NV; l++)
        {
            const real pm = sD[pr * NV + l][lane] * ip, px = sU[pr * NV + l][lane] * ip;
            M[l] = i == k ? pm : M[l] - fct * pm;
            X[l] = i == k ? px : X[l] - fct * px;
        }
    }
    __shared__ int sBad[32];
    if (threadIdx.x < 32)
        sBad[lane] = 0;
    __syncthreads();
    if (!ok)
        sBad[lane] = 1;
    __syncthreads();
#pragma unroll
    for (int l = 0; l < NV; l++)
        inv[l] = X[l] * sS[l][lane];
    return !sBad[lane];
}

// The factorisation in compact slot order, rows [beg, end) of one colour in position order (a row's rank is its
// position): slot j < cnlow[r] holds the j-th lower neighbour in ascending rank, the upper neighbours follow, cnbr
// [r][NF] their rows (-1 after the last), so the triangular solves read a row's lower (or upper) blocks from consecutive
// slots.  Row i of L_j, of the diagonal and of the upper blocks depends on row i of the operator's blocks alone, so warp
// i takes it; the neighbours' factors and the pivot rows go through shared memory.  The sums run in factor_row's order.
// One thread per row held its blocks in local memory: 121 us per colour of 249,600 tets in FP64, now 93.
// Bound by the gathers of the neighbours' blocks, so three blocks per SM (136 registers a thread with 5 variables, 113
// with 6) instead of the one or two that the free choice of registers leaves.  Per solve, three blocks against free
// choice: 249,600 tets 366 and 474 us in FP64, 349 and 460 in FP32; 110,592 hexahedra 223 and 516, 204 and 506; 131,072
// triangles 132 and 170, 111 and 146; 65,536 quadrilaterals 91 and 112, 81 and 100; 6 variables on 72,000 hexahedra 231
// and 404, 215 and 383.
template <typename T, int NV, int NF>
DNDSB_GLOBAL void __launch_bounds__(32 * NV, 3) k_ilu_factor_c(int64_t beg, int64_t end, const int32_t *__restrict__ nbr, const T *__restrict__ A,
                                                           const T *__restrict__ D, BlockLay offL, BlockLay dL, BlockLay DL, T *off, T *dinv,
                                                           int *err, int32_t *cnbr, int32_t *cnlow)
{
    constexpr int NN = NV * NV;
    __shared__ real sD[NN][32], sU[NN][32]; // of the current lower neighbour: its inverse diagonal, its block towards this row
    const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
    const int64_t r = (((beg >> 5) + blockIdx.x) << 5) + lane;
    const bool on = r >= beg && r < end;
    // the slots in compact order: lower neighbours by rank (equal ranks in slot order), then the upper ones in slot order
    int qs[NF], slot[NF], q[NF], nLow = 0, nAll = 0;
#pragma unroll
    for (int k = 0; k < NF; k++)
    {
        qs[k] = on ? nbr[r * NF + k] : -1;
        if (qs[k] == r)
            qs[k] = -1;
        slot[k] = 0, q[k] = -1;
        nLow += qs[k] >= 0 && qs[k] < r;
        nAll += qs[k] >= 0;
    }
    int nUpp = 0;
#pragma unroll
    for (int k = 0; k < NF; k++)
    {
        if (qs[k] < 0)
            continue;
        int at = 0;
        if (qs[k] < r)
        {
#pragma unroll
            for (int l = 0; l < NF; l++)
                at += qs[l] >= 0 && qs[l] < r && (qs[l] < qs[k] || (qs[l] == qs[k] && l < k));
        }
        else
            at = nLow + nUpp++;
#pragma unroll
        for (int a = 0; a < NF; a++)
            if (a == at)
                slot[a] = k, q[a] = qs[k];
    }
    auto opRow = [&](int k, real *o)
    {
#pragma unroll
        for (int l = 0; l < NV; l++)
            o[l] = (real)A[offL.at(r, k * NN + i * NV + l)];
    };
    real L[NF][NV], Di[NV] = {};
    // o -= sum over the first nb lower neighbours of L_b U_(b, j), where b and j are neighbours
    auto eliminate = [&](int nb, int j, real *o)
    {
#pragma unroll
        for (int b = 0; b < NF; b++)
            if (b < nb)
            {
                const int s = slot_of<NF>(cnbr, q[b], j);
                if (s >= 0)
#pragma unroll
                    for (int c = 0; c < NV; c++)
                    {
                        real acc = 0;
#pragma unroll
                        for (int l = 0; l < NV; l++)
                            acc += L[b][l] * (real)off[offL.at(q[b], s * NN + l * NV + c)];
                        o[c] -= acc;
                    }
            }
    };
    if (on)
#pragma unroll
        for (int l = 0; l < NV; l++)
            Di[l] = (real)D[DL.at(r, i * NV + l)];
#pragma unroll
    for (int a = 0; a < NF; a++)
    {
        const bool has = a < nLow;
        if (!__syncthreads_or(has))
            break;
        const int s = has ? slot_of<NF>(cnbr, q[a], r) : -1;
        if (has)
#pragma unroll
            for (int l = 0; l < NV; l++)
            {
                sD[i * NV + l][lane] = (real)dinv[dL.at(q[a], i * NV + l)];
                if (s >= 0)
                    sU[i * NV + l][lane] = (real)off[offL.at(q[a], s * NN + i * NV + l)];
            }
        __syncthreads();
        if (has)
        {
            real o[NV];
            opRow(slot[a], o);
            eliminate(a, q[a], o);
#pragma unroll
            for (int c = 0; c < NV; c++)
            {
                real acc = 0;
#pragma unroll
                for (int l = 0; l < NV; l++)
                    acc += o[l] * sD[l * NV + c][lane];
                L[a][c] = acc;
            }
            if (s >= 0)
#pragma unroll
                for (int c = 0; c < NV; c++)
                {
                    real acc = 0;
#pragma unroll
                    for (int l = 0; l < NV; l++)
                        acc += L[a][l] * sU[l * NV + c][lane];
                    Di[c] -= acc;
                }
        }
    }
    real inv[NV];
    const bool ok = tile_inv<NV>(Di, sD, sU, inv);
    if (!on)
        return;
    if (!ok && i == 0)
        atomicOr(err, (int)DE_SINGULAR);
#pragma unroll
    for (int l = 0; l < NV; l++)
        dinv[dL.at(r, i * NV + l)] = ok ? (T)inv[l] : T(0);
#pragma unroll
    for (int a = 0; a < NF; a++)
    {
        real o[NV];
#pragma unroll
        for (int c = 0; c < NV; c++)
            o[c] = a < nLow ? L[a][c] : 0.0;
        if (a >= nLow && a < nAll)
        {
            opRow(slot[a], o);
            eliminate(nLow, q[a], o);
        }
#pragma unroll
        for (int c = 0; c < NV; c++)
            off[offL.at(r, a * NN + i * NV + c)] = (T)o[c];
        if (i == 0)
            cnbr[r * NF + a] = q[a];
    }
    if (i == 0)
        cnlow[r] = nLow;
}

// the triangular solves on compact factors (cnbr / cnlow of k_ilu_factor_c), rows [beg, end) of one colour:
// forward y_r = b_r - sum_{j < nLow} L_j y_q; backward x_r = dinv_r (y_r - sum_{j >= nLow} U_j x_q), in place
// (add: also added to xAdd)
template <typename T, int NV, int NF>
DNDSB_GLOBAL void __launch_bounds__(32 * NV) k_ilu_lower_c(int64_t beg, int64_t end, const int32_t *__restrict__ cnbr,
                                                          const int32_t *__restrict__ cnlow, const T *__restrict__ off, BlockLay offL, const T *b,
                                                          T *x) // b may be x
{
    constexpr int NN = NV * NV;
    __shared__ T sx[NF][NV][32];
    const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
    const int64_t r = (((beg >> 5) + blockIdx.x) << 5) + lane;
    const bool on = r >= beg && r < end;
    const int nl = on ? cnlow[r] : 0;
    T f[NF][NV];
    int q[NF];
#pragma unroll
    for (int j = 0; j < NF; j++)
        if (j < nl)
        {
            q[j] = cnbr[r * NF + j];
#pragma unroll
            for (int l = 0; l < NV; l++)
                f[j][l] = off[offL.at(r, j * NN + i * NV + l)];
        }
    chain_step();
    T acc = on ? b[r * NV + i] : T(0);
#pragma unroll
    for (int j = 0; j < NF; j++)
        if (j < nl)
            sx[j][i][lane] = x[(int64_t)q[j] * NV + i];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NF; j++)
        if (j < nl)
        {
            T s = 0;
#pragma unroll
            for (int l = 0; l < NV; l++)
                s += f[j][l] * sx[j][l][lane];
            acc -= s;
        }
    if (on)
        x[r * NV + i] = acc;
}

template <typename T, int NV, int NF>
DNDSB_GLOBAL void __launch_bounds__(32 * NV) k_ilu_upper_c(int64_t beg, int64_t end, const int32_t *__restrict__ cnbr,
                                                          const int32_t *__restrict__ cnlow, const T *__restrict__ off, BlockLay offL,
                                                          const T *__restrict__ dinv, BlockLay dL, T *x, T *xAdd)
{
    constexpr int NN = NV * NV;
    __shared__ T sx[NF + 1][NV][32];
    const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
    const int64_t r = (((beg >> 5) + blockIdx.x) << 5) + lane;
    const bool on = r >= beg && r < end;
    const int nl = on ? cnlow[r] : NF;
    T f[NF][NV], d[NV];
    int q[NF];
#pragma unroll
    for (int j = 0; j < NF; j++)
    {
        q[j] = j >= nl ? cnbr[r * NF + j] : -1;
        if (q[j] >= 0)
        {
#pragma unroll
            for (int l = 0; l < NV; l++)
                f[j][l] = off[offL.at(r, j * NN + i * NV + l)];
        }
    }
    if (on)
#pragma unroll
        for (int l = 0; l < NV; l++)
            d[l] = dinv[dL.at(r, i * NV + l)];
    chain_step();
    T acc = on ? x[r * NV + i] : T(0);
#pragma unroll
    for (int j = 0; j < NF; j++)
        if (q[j] >= 0)
            sx[j][i][lane] = x[(int64_t)q[j] * NV + i];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NF; j++)
        if (q[j] >= 0)
        {
            T s = 0;
#pragma unroll
            for (int l = 0; l < NV; l++)
                s += f[j][l] * sx[j][l][lane];
            acc -= s;
        }
    sx[NF][i][lane] = acc;
    __syncthreads();
    if (!on)
        return;
    T s = 0;
#pragma unroll
    for (int l = 0; l < NV; l++)
        s += d[l] * sx[NF][l][lane];
    x[r * NV + i] = s;
    if (xAdd)
        xAdd[r * NV + i] += s;
}

// y = A (s x) of the block operator (diagonal blocks jdB, slot blocks opB, neighbours nbr [r][NF]), s = *xs (null: 1);
// with rhs: y = rhs - A x
template <typename T, int NV, int NF>
DNDSB_GLOBAL void __launch_bounds__(32 * NV) k_block_product(int64_t n, const int32_t *__restrict__ nbr, const T *__restrict__ opB,
                                                            const T *__restrict__ jdB, const T *x, T *y, const real *xs, const T *rhs)
{
    constexpr int NN = NV * NV;
    const BlockLay oL{NF * NN, 5}, dL{2 * NN, 5};
    __shared__ T sx[NF + 1][NV][32];
    const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
    const int64_t r = ((int64_t)blockIdx.x << 5) + lane;
    const bool on = r < n;
    T f[NF][NV], d[NV];
    int q[NF];
#pragma unroll
    for (int j = 0; j < NF; j++)
    {
        q[j] = on ? nbr[r * NF + j] : -1;
        if (q[j] >= 0)
        {
#pragma unroll
            for (int l = 0; l < NV; l++)
                f[j][l] = opB[oL.at(r, j * NN + i * NV + l)];
        }
    }
    if (on)
    {
#pragma unroll
        for (int l = 0; l < NV; l++)
            d[l] = jdB[dL.at(r, i * NV + l)];
    }
    chain_step();
    const T sc = xs ? (T)*xs : T(1);
#pragma unroll
    for (int j = 0; j < NF; j++)
        if (q[j] >= 0)
            sx[j][i][lane] = x[(int64_t)q[j] * NV + i];
    if (on)
        sx[NF][i][lane] = x[r * NV + i];
    __syncthreads();
    if (!on)
        return;
    T acc = 0;
#pragma unroll
    for (int l = 0; l < NV; l++)
        acc += d[l] * sx[NF][l][lane];
#pragma unroll
    for (int j = 0; j < NF; j++)
        if (q[j] >= 0)
        {
            T s = 0;
#pragma unroll
            for (int l = 0; l < NV; l++)
                s += f[j][l] * sx[j][l][lane];
            acc += s;
        }
    y[r * NV + i] = rhs ? rhs[r * NV + i] - acc : sc * acc;
}

// forward: y_r = b_r - sum over lower slots of L y_q;  backward: x_r = dinv_r (y_r - sum over upper slots of U x_q),
// in place on x (= y)
template <typename T, int NV, int NF>
DNDSB_GLOBAL void k_ilu_lower(int64_t beg, int64_t end, const int32_t *__restrict__ rows, const int32_t *__restrict__ nbr,
                              const int32_t *__restrict__ rank, const T *__restrict__ off, BlockLay offL, const T *b, T *x) // b may be x
{
    constexpr int NN = NV * NV;
    DNDSB_KERNEL_LOOP(ii, end - beg)
    {
        int64_t r = rows ? (int64_t)rows[beg + ii] : beg + ii;
        int64_t rr = rank ? (int64_t)rank[r] : r;
        T acc[NV];
        for (int v = 0; v < NV; v++)
            acc[v] = b[r * NV + v];
#pragma unroll
        for (int k = 0; k < NF; k++)
        {
            int64_t q = nbr[r * NF + k];
            if (q < 0 || q == r || (rank ? (int64_t)rank[q] : q) >= rr)
                continue;
            T xq[NV];
            for (int l = 0; l < NV; l++)
                xq[l] = x[q * NV + l];
            for (int i = 0; i < NV; i++)
            {
                T s = 0;
                for (int l = 0; l < NV; l++)
                    s += off[offL.at(r, k * NN + i * NV + l)] * xq[l];
                acc[i] -= s;
            }
        }
        for (int v = 0; v < NV; v++)
            x[r * NV + v] = acc[v];
    }
}

template <typename T, int NV, int NF>
DNDSB_GLOBAL void k_ilu_upper(int64_t beg, int64_t end, const int32_t *__restrict__ rows, const int32_t *__restrict__ nbr,
                              const int32_t *__restrict__ rank, const T *__restrict__ off, BlockLay offL, const T *__restrict__ dinv, BlockLay dL,
                              T *x)
{
    constexpr int NN = NV * NV;
    DNDSB_KERNEL_LOOP(ii, end - beg)
    {
        int64_t r = rows ? (int64_t)rows[beg + ii] : beg + ii;
        int64_t rr = rank ? (int64_t)rank[r] : r;
        T acc[NV];
        for (int v = 0; v < NV; v++)
            acc[v] = x[r * NV + v];
#pragma unroll
        for (int k = 0; k < NF; k++)
        {
            int64_t q = nbr[r * NF + k];
            if (q < 0 || q == r || (rank ? (int64_t)rank[q] : q) <= rr)
                continue;
            T xq[NV];
            for (int l = 0; l < NV; l++)
                xq[l] = x[q * NV + l];
            for (int i = 0; i < NV; i++)
            {
                T s = 0;
                for (int l = 0; l < NV; l++)
                    s += off[offL.at(r, k * NN + i * NV + l)] * xq[l];
                acc[i] -= s;
            }
        }
        for (int i = 0; i < NV; i++)
        {
            T s = 0;
            for (int l = 0; l < NV; l++)
                s += dinv[dL.at(r, i * NV + l)] * acc[l];
            x[r * NV + i] = s;
        }
    }
}
} // namespace ilu
} // namespace dndsb
