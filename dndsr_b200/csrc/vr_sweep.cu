// VR Jacobi sweep (VariationalReconstruction_Reconstruction.hxx:485-615), interior faces:
//   uRecNew_c = (1 - w) uRec_c + w sum_k (A^-1 B_k uRec_o + A^-1 b_k (u_o - u_c)),
// with recordInc the preconditioned residual uRec_c - sum_k (...).
//
// Two kernels, each with its layout of the packed coefficients (sweep_layout.cuh: by the rows R and the cells).
//
// k_vr_sweep_staged (R = 9, from kTiledCells cells on): coefficients in tiles of 32 cells [tile][face k][j][i][32], the 32
// lanes of a warp the cells of a tile, so every coefficient load is one contiguous line; a thread takes three rows of
// its cell, three warps share a tile.  The rows of the neighbours (uRec_o and u_o, 50 doubles) are copied into shared
// memory by asynchronous copies that run along each row, three stages deep (the own row, then the faces), and the
// result leaves through shared memory the same way.  HBM bound on the coefficients: 450 -> 260 us on the 64^3
// Taylor-Green mesh (1.33 GB, 5.1 TB/s), 48 -> 33 us on 36k tets.  What bounded the sweep before was L1: with R threads
// per cell reading the neighbour's row as broadcasts, every double of every neighbour row cost a tag lookup.  With the
// 3 rows of degree 1 the same staging is slower than reading (78 us against 67 on 250k tets: short rows, one warp per
// tile), so those keep
//
// k_vr_sweep_rows: R neighbouring lanes per cell, lane i on row i, coefficients [cell][face k][j][i]; lane i loads row i
// of the neighbour and the lanes exchange rows by shuffles, so a row costs NV loads instead of R NV broadcasts.
#include "solver.cuh"
#include "sweep_layout.cuh"
#include "fast_common.cuh"
#include "chain.cuh"

namespace dndsb
{
namespace
{
using fastc::copies_commit;
using fastc::copies_wait;
using fastc::copy8_async;

template <int R, int NV>
struct Stage
{
    static constexpr int W = R * NV, N = W + NV, SW = N | 1; // an odd stride: the lanes' rows start in different banks
    static constexpr int LEN = 32 * SW;
};

constexpr int kStagedRows = 3; // rows a thread of the staged kernel takes

template <int R, int NV, int NF, typename TC>
__global__ void __launch_bounds__(32 * (R / kStagedRows))
    k_vr_sweep_staged(int64_t nCell, const int32_t *__restrict__ nbr, const TC *__restrict__ coef, const real *uRec,
                      real *uRecNew, const real *u, real relax, int recordInc, int uRecIsZero)
{
    chain_step();
    using St = Stage<R, NV>;
    constexpr int RT = kStagedRows, G = R / RT;
    extern __shared__ real sb[]; // three stages
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, i0 = g * RT;
    const int64_t tile = blockIdx.x;
    const int64_t c = tile * 32 + lane;
    int src[NF + 1]; // rows of the stages: the cell's own, then its neighbours' (-1: none)
    src[0] = c < nCell ? (int)c : -1;
#pragma unroll
    for (int k = 0; k < NF; k++)
        src[k + 1] = c < nCell ? nbr[c * NF + k] : -1;
    const bool useRec = !(recordInc && uRecIsZero);
    auto stage = [&](int s, int mine)
    {
        real *dst = sb + (s % 3) * St::LEN;
        if (!useRec)
        {
            // from a zero reconstruction the sweep reads the means alone: each lane's row by the threads of its cell
            if (mine >= 0)
                for (int v = g; v < NV; v += G)
                    copy8_async(dst + lane * St::SW + St::W + v, u + (int64_t)mine * NV + v);
            copies_commit();
            return;
        }
#pragma unroll 4
        for (int m = g; m < 32; m += G)
        {
            const int o = __shfl_sync(0xffffffffu, mine, m);
            if (o < 0)
                continue;
#pragma unroll
            for (int e0 = 0; e0 < St::N; e0 += 32)
            {
                const int e = e0 + lane;
                if (e < St::N)
                    copy8_async(dst + m * St::SW + e, e < St::W ? uRec + (int64_t)o * St::W + e : u + (int64_t)o * NV + (e - St::W));
            }
        }
        copies_commit();
    };
    stage(0, src[0]);
    stage(1, src[1]);
    real acc[RT][NV], ui[NV];
    const real sgn = recordInc ? -1.0 : relax;
    const TC *cb = coef + tile * NF * (R + 1) * R * 32 + i0 * 32 + lane; // entry (face k, j, row i0 + r) at cb[((k (R + 1) + j) R + r) 32]
#pragma unroll
    for (int s = 0; s <= NF; s++)
    {
        TC M[R + 1][RT];
        if (s > 0)
        {
#pragma unroll
            for (int j = 0; j <= R; j++)
#pragma unroll
                for (int r = 0; r < RT; r++)
                    M[j][r] = (useRec || j == R) ? cb[(((s - 1) * (R + 1) + j) * R + r) * 32] : TC(0);
        }
        copies_wait<1>();
        __syncthreads();
        // the buffer of stage s - 1: every thread of the tile is past it
        if (s + 2 <= NF)
            stage(s + 2, src[s + 2 <= NF ? s + 2 : 0]);
        else
            copies_commit();
        const real *row = sb + (s % 3) * St::LEN + lane * St::SW;
        if (src[s] < 0)
            continue;
        if (s == 0)
        {
#pragma unroll
            for (int v = 0; v < NV; v++)
            {
                ui[v] = row[St::W + v];
#pragma unroll
                for (int r = 0; r < RT; r++)
                {
                    const real x = row[(i0 + r) * NV + v];
                    acc[r][v] = recordInc ? (uRecIsZero ? 0.0 : x) : x * (1 - relax);
                }
            }
            continue;
        }
        real t[RT][NV];
#pragma unroll
        for (int v = 0; v < NV; v++)
        {
            const real du = row[St::W + v] - ui[v];
#pragma unroll
            for (int r = 0; r < RT; r++)
                t[r][v] = (real)M[R][r] * du;
        }
        if (useRec)
        {
#pragma unroll
            for (int j = 0; j < R; j++)
#pragma unroll
                for (int v = 0; v < NV; v++)
                {
                    const real x = row[j * NV + v];
#pragma unroll
                    for (int r = 0; r < RT; r++)
                        t[r][v] += (real)M[j][r] * x;
                }
        }
#pragma unroll
        for (int r = 0; r < RT; r++)
#pragma unroll
            for (int v = 0; v < NV; v++)
                acc[r][v] += sgn * t[r][v];
    }
    // out through the buffer that the last stage did not use
    real *ob = sb + ((NF + 1) % 3) * St::LEN;
    if (c < nCell)
    {
#pragma unroll
        for (int r = 0; r < RT; r++)
#pragma unroll
            for (int v = 0; v < NV; v++)
                ob[lane * St::SW + (i0 + r) * NV + v] = acc[r][v];
    }
    __syncthreads();
    for (int m = g; m < 32; m += G)
    {
        if (tile * 32 + m >= nCell)
            break;
#pragma unroll
        for (int e0 = 0; e0 < St::W; e0 += 32)
            if (e0 + lane < St::W)
                uRecNew[(tile * 32 + m) * St::W + e0 + lane] = ob[m * St::SW + e0 + lane];
    }
}

// cells of a warp of the row kernel
template <int R>
constexpr int warp_cells() { return 32 / R; }
constexpr int kRowWarps = 4;

template <int R, int NV, int NF, typename TC>
__global__ void __launch_bounds__(32 * kRowWarps)
    k_vr_sweep_rows(int64_t nCell, const int32_t *__restrict__ nbr, const TC *__restrict__ coef, const real *uRec,
                    real *uRecNew, const real *u, real relax, int recordInc, int uRecIsZero)
{
    chain_step();
    constexpr int CW = warp_cells<R>();
    const int lane = threadIdx.x & 31, cl = lane / R, i = lane - cl * R, lane0 = lane - i;
    const int64_t c = ((int64_t)blockIdx.x * kRowWarps + (threadIdx.x >> 5)) * CW + cl;
    const bool on = cl < CW && c < nCell;
    const int64_t cc = on ? c : 0; // idle lanes shuffle along on cell 0
    const bool useRec = !(recordInc && uRecIsZero);
    real acc[NV], ui[NV];
#pragma unroll
    for (int v = 0; v < NV; v++)
    {
        const real x = uRec[(cc * R + i) * NV + v];
        acc[v] = recordInc ? (uRecIsZero ? 0.0 : x) : x * (1 - relax);
        ui[v] = u[cc * NV + v];
    }
    const real sgn = recordInc ? -1.0 : relax;
    int src[NF];
#pragma unroll
    for (int k = 0; k < NF; k++)
        src[k] = nbr[cc * NF + k];
    const TC *cb = coef + cc * NF * (R + 1) * R + i; // entry (face k, j) at cb[(k (R+1) + j) R]
#pragma unroll
    for (int k = 0; k < NF; k++)
    {
        const int o = src[k] < 0 ? (int)cc : src[k]; // a boundary face's coefficients are not applied
        TC M[R + 1];
#pragma unroll
        for (int j = 0; j <= R; j++)
            M[j] = (useRec || j == R) ? cb[(k * (R + 1) + j) * R] : TC(0);
        real row[NV], uo[NV];
#pragma unroll
        for (int v = 0; v < NV; v++)
        {
            row[v] = useRec ? uRec[((int64_t)o * R + i) * NV + v] : 0.0;
            uo[v] = u[(int64_t)o * NV + v];
        }
        real t[NV];
#pragma unroll
        for (int v = 0; v < NV; v++)
            t[v] = (real)M[R] * (uo[v] - ui[v]);
        if (useRec)
        {
#pragma unroll
            for (int j = 0; j < R; j++)
#pragma unroll
                for (int v = 0; v < NV; v++)
                    t[v] += (real)M[j] * __shfl_sync(0xffffffffu, row[v], lane0 + j);
        }
        if (src[k] >= 0)
        {
#pragma unroll
            for (int v = 0; v < NV; v++)
                acc[v] += sgn * t[v];
        }
    }
    if (!on)
        return;
#pragma unroll
    for (int v = 0; v < NV; v++)
        uRecNew[(c * R + i) * NV + v] = acc[v];
}

template <int R, int NV, int NF, typename TC>
int launch(int64_t nCell, const int32_t *nbr, const TC *coef, const real *uRec, real *uRecNew, const real *u, real relax, int recordInc,
           int uRecIsZero, cudaStream_t st)
{
    if constexpr (R == 9)
        if (sweep_tiled(R, nCell))
        {
            constexpr size_t sh = sizeof(real) * 3 * Stage<R, NV>::LEN;
            static unsigned long long attrSet = 0; // one bit per device: dynamic shared memory limit raised
            int dev = 0;
            cudaGetDevice(&dev);
            if (dev >= 64 || !((attrSet >> dev) & 1ULL))
            {
                if (cudaFuncSetAttribute(k_vr_sweep_staged<R, NV, NF, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh) != cudaSuccess)
                    return ST_CUDA;
                if (dev < 64)
                    attrSet |= 1ULL << dev;
            }
            launch_chained_shared(k_vr_sweep_staged<R, NV, NF, TC>, (unsigned)((nCell + 31) / 32), 32 * (R / kStagedRows), sh, st, nCell, nbr, coef, uRec, uRecNew, u, relax,
                                                                                                             recordInc, uRecIsZero);
            return last_error() == cudaSuccess ? ST_OK : ST_CUDA;
        }
    const int64_t warps = (nCell + warp_cells<R>() - 1) / warp_cells<R>();
    launch_chained(k_vr_sweep_rows<R, NV, NF, TC>, (unsigned)((warps + kRowWarps - 1) / kRowWarps), 32 * kRowWarps, st, nCell, nbr, coef, uRec, uRecNew, u, relax,
                                                                                                            recordInc, uRecIsZero);
    return last_error() == cudaSuccess ? ST_OK : ST_CUDA;
}

template <typename TC>
int dispatch(const MeshD &m, const VRD &vr, int nv, const TC *coef, const real *uRec, real *uRecNew, const real *u, int recordInc, int uRecIsZero,
             cudaStream_t st)
{
#define DNDSB_VRS(R_, NV_, NF_)                       \
    if (vr.R == R_ && nv == NV_ && m.nf == NF_)       \
        return launch<R_, NV_, NF_, TC>(m.nCell, m.cellNbr, coef, uRec, uRecNew, u, vr.s.jacobiRelax, recordInc, uRecIsZero, st);
    DNDSB_VRS(2, 5, 3)
    DNDSB_VRS(2, 5, 4)
    DNDSB_VRS(5, 5, 3)
    DNDSB_VRS(5, 5, 4)
    DNDSB_VRS(9, 5, 3)
    DNDSB_VRS(9, 5, 4)
    DNDSB_VRS(9, 5, 6)
    DNDSB_VRS(3, 5, 4)
    DNDSB_VRS(3, 5, 6)
    DNDSB_VRS(3, 6, 4) // the SA model at degree 1 in 3-D
    DNDSB_VRS(3, 6, 6)
#undef DNDSB_VRS
    return ST_UNSUPPORTED;
}
} // namespace

int vr_iter_fast(const MeshD &m, const VRD &vr, int nv, const real *uRec, real *uRecNew, const real *u, int recordInc, int uRecIsZero,
                 int useFP32, cudaStream_t st)
{
    if (!vr.sweepCoef)
        return ST_UNSUPPORTED;
    return useFP32 ? dispatch<float>(m, vr, nv, vr.sweepCoef32, uRec, uRecNew, u, recordInc, uRecIsZero, st)
                   : dispatch<real>(m, vr, nv, vr.sweepCoef, uRec, uRecNew, u, recordInc, uRecIsZero, st);
}
} // namespace dndsb
