// Cell-side kernels of the derivatives shared by the 5- and 6-variable families (adjoint.cu, adjoint_generic.cuh): the
// gather of the face cotangents and the transposed reconstruction sweep.
#pragma once
#include "solver.cuh"
#include "basis_rows.cuh"
#include "bc.cuh"
#include "dual.cuh"
#include "chain.cuh"

namespace dndsb
{
namespace
{
// (du, duRec)_c = sum over the cell's faces of the face cotangents of its side (fixed face order); W = (R + 1) NV.
// One thread per entry, so the lanes read along the face records: HBM bound.  A thread per cell read 4 or 6 records in
// strides (81 us for 249,600 tets at W = 20, now 46).
template <int W, int NV>
DNDSB_GLOBAL void k_adj_gather(int64_t nCell, int nf, const int32_t *__restrict__ c2f, const real *__restrict__ faceAdj, real *du, real *duRec)
{
    DNDSB_KERNEL_LOOP(e, nCell * W)
    {
        const int64_t c = e / W;
        const int i = (int)(e - c * W);
        real acc = 0;
        for (int k = 0; k < nf; k++)
            acc += faceAdj[(int64_t)c2f[c * nf + k] * W + i]; // (face << 1 | side) numbers the records
        if (i < NV)
            du[c * NV + i] = acc;
        else
            duRec[c * (W - NV) + i - NV] = acc;
    }
}

// VJP of the sweep uRecNew_i = (1-w) uRec_i + w sum_k [M_ik uRec_k + b_ik (u_k - u_i)] (interior faces):
// v = cotangent of uRecNew -> vRec (of uRec), vU (of u), gathered per cell.
// R neighbouring lanes per cell, lane r on row r of vRec: it reads column r of the neighbour's block (the lanes of a cell
// read along its rows), row r of the neighbour's cotangent, and takes the other rows from its neighbours by shuffles.
// A thread per cell read whole blocks and rows in strides and carried the boundary cells' ghost derivatives: 156 us for
// 249,600 tets at R = 3 and 697 us at R = 9, now 75 and 367, and 31 and 70 in the boundary kernel.
template <int R, int NV>
DNDSB_GLOBAL void __launch_bounds__(128) k_vr_vjp_rows(MeshD m, VRD vr, const real *__restrict__ v, real *__restrict__ vRec, real *__restrict__ vU)
{
    chain_release(); // the boundary kernel waits before it adds to what this one writes
    constexpr int CW = 32 / R;
    const int lane = threadIdx.x & 31, cl = lane / R, r = lane - cl * R, lane0 = lane - r, nf = m.nf;
    const int64_t o = ((int64_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * CW + cl;
    const bool on = cl < CW && o < m.nCell;
    const int64_t oc = on ? o : 0; // idle lanes shuffle along on cell 0
    const real om = vr.s.jacobiRelax;
    real vo[NV], aRec[NV], pU[NV];
#pragma unroll
    for (int x = 0; x < NV; x++)
        vo[x] = v[(oc * R + r) * NV + x], aRec[x] = 0, pU[x] = 0;
    for (int j = 0; j < nf; j++)
    {
        const int nb = m.cellNbr[oc * nf + j];
        const int64_t i = nb < 0 ? oc : nb;
        const int k = nb < 0 ? 0 : m.nbrSlot[oc * nf + j];
        const real *M = vr.AAInvB + (i * (nf + 1) + 1 + k) * R * R + r;
        const real b = vr.AInvb[(i * nf + k) * R + r], bo = vr.AInvb[(oc * nf + j) * R + r];
        real vi[NV], t[NV];
#pragma unroll
        for (int x = 0; x < NV; x++)
            vi[x] = v[(i * R + r) * NV + x], t[x] = 0;
#pragma unroll
        for (int l = 0; l < R; l++)
        {
            const real ml = M[l * R];
#pragma unroll
            for (int x = 0; x < NV; x++)
                t[x] += ml * __shfl_sync(0xffffffffu, vi[x], lane0 + l);
        }
        if (nb >= 0)
        {
#pragma unroll
            for (int x = 0; x < NV; x++)
                aRec[x] += t[x], pU[x] += b * vi[x] - bo * vo[x];
        }
    }
#pragma unroll
    for (int x = 0; x < NV; x++)
    {
        real s = 0;
#pragma unroll
        for (int l = 0; l < R; l++)
            s += __shfl_sync(0xffffffffu, pU[x], lane0 + l);
        if (on)
        {
            vRec[(o * R + r) * NV + x] = (1 - om) * vo[x] + om * aRec[x];
            if (r == 0)
                vU[o * NV + x] = om * s;
        }
    }
}

// adds the boundary term's share: t = w A_c^-T v_c is the cotangent of BCC = sum_q w0^2 |J| w phi_q (UB_q - u_c) with
// UB_q = ghost(compress(u_c, u_c + phi_q . uRec_c)); the ghost is differentiated in dual numbers with respect to the
// point state and the mean.  One thread per (boundary cell, point), more where the points are few (bnd_row_threads), the
// block's sums in point order (as k_vr_bc).  Chained to k_vr_vjp_rows, which is launched after all that this kernel reads is
// complete: only the sums at the end wait for its results (on small meshes a launch of its own cost a tenth of the whole
// transpose: 14,112 tets of degree 1 24.9 us in one kernel, 26.6 in two).
template <int DIM, int P, int NV>
DNDSB_GLOBAL void k_vr_vjp_bnd(MeshD m, GeomD g, VRD vr, const real *__restrict__ v, const real *__restrict__ uRec, const real *__restrict__ u,
                               real *vRec, real *vU, int tpr)
{
    constexpr int NDOF = ndof_of<DIM>(P), R = NDOF - 1, RV = R * NV, ROW = R + 2 * NV;
    using DV = Dual<NV>;
    extern __shared__ real smVb[];
    const int nG = g.nGf, cl = threadIdx.x / tpr, q = threadIdx.x - cl * tpr, rows = blockDim.x / tpr;
    const int64_t ii = (int64_t)blockIdx.x * rows + cl;
    const int64_t c = ii < m.nBndCell ? m.bndCell[ii] : -1;
    real *sT = smVb + cl * (RV + RV + NV + nG * ROW); // [R][NV] the cotangent of BCC
    real *sA = sT + RV;                                // [R][NV] and [NV]: the sums for vRec and vU
    real *row = sA + RV + NV + q * ROW;                // per point: phi, the cotangents of the point state and of the mean
    const real *row0 = sA + RV + NV;
    if (c >= 0)
    {
        const real *Ai = vr.AAInvB + c * (m.nf + 1) * R * R, *vc = v + c * RV;
        for (int e = q; e < RV + NV; e += tpr)
        {
            sA[e] = 0;
            if (e < RV)
            {
                const int r = e / NV, x = e - r * NV;
                real a = 0;
                for (int l = 0; l < R; l++)
                    a += Ai[l * R + r] * vc[l * NV + x];
                sT[e] = vr.s.jacobiRelax * a;
            }
        }
    }
    for (int k = 0; k < m.nf; k++)
    {
        int64_t f = 0;
        real w0 = 0;
        if (c >= 0 && m.cellNbr[c * m.nf + k] < 0)
        {
            f = m.cell2face[c * m.nf + k] >> 1;
            w0 = vr.faceWeight[f * (P + 1)];
        }
        if (!__syncthreads_or(w0 != 0)) // also orders the sums of the last slot and the points of this one
            continue;
        if (w0 != 0 && q < nG)
        {
            const real *uc = u + c * NV, *rc = uRec + c * RV, *n = &g.faceNorm[(f * nG + q) * 3];
            const int zone = m.faceZone[f];
            real phi[R], UL[NV], UBbar[NV];
            basis_rows<DIM, P, false>(g, vr, c, &g.facePP[(f * nG + q) * 3], phi, nullptr);
            const real JW = g.faceJDet[f * nG + q] * g.faceQw[q] * w0 * w0;
#pragma unroll
            for (int x = 0; x < NV; x++)
            {
                real a = uc[x], t = 0;
#pragma unroll
                for (int j = 0; j < R; j++)
                    a += phi[j] * rc[j * NV + x], t += phi[j] * sT[j * NV + x];
                UL[x] = a, UBbar[x] = t * JW;
            }
#pragma unroll
            for (int j = 0; j < R; j++)
                row[j] = phi[j];
#pragma unroll 1
            for (int pass = 0; pass < 2; pass++) // seeds: the point state, then the mean
            {
                DV ULd[NV], umd[NV], ULf[NV], UB[NV];
                for (int x = 0; x < NV; x++)
                    ULd[x] = DV::var(UL[x], pass == 0 ? x : -1), umd[x] = DV::var(uc[x], pass == 1 ? x : -1);
                compress_rec<NV>(umd, ULd, ULf);
                if (!bc_value_fix<NV>(vr.bnd, zone, ULf, n, UB))
                    for (int x = 0; x < NV; x++)
                        UB[x] = ULf[x];
                for (int i = 0; i < NV; i++)
                {
                    real a = 0;
                    for (int x = 0; x < NV; x++)
                        a += UB[x].d[i] * UBbar[x];
                    row[R + pass * NV + i] = pass == 0 ? a : a - UBbar[i];
                }
            }
        }
        __syncthreads();
        if (w0 != 0)
            for (int e = q; e < RV + NV; e += tpr)
            {
                const int j = e / NV, x = e - j * NV; // j = R: vU
                real a = sA[e];
                for (int p = 0; p < nG; p++)
                {
                    const real *pr = row0 + p * ROW;
                    a += j < R ? pr[j] * pr[R + x] : pr[R + x] + pr[R + NV + x];
                }
                sA[e] = a;
            }
    }
    chain_wait();
    __syncthreads();
    if (c < 0)
        return;
    for (int e = q; e < RV + NV; e += tpr)
        if (e < RV)
            vRec[c * RV + e] += sA[e];
        else
            vU[c * NV + e - RV] += sA[e];
}

template <int DIM, int P, int NV>
void launch_vr_vjp(const MeshD &m, const GeomD &g, const VRD &vr, const real *v, const real *uRec, const real *u, real *vRec, real *vU, cudaStream_t st)
{
    constexpr int R = ndof_of<DIM>(P) - 1, CW = 32 / R;
    const int64_t warps = (m.nCell + CW - 1) / CW;
    k_vr_vjp_rows<R, NV><<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(m, vr, v, vRec, vU);
    if (m.nBndCell > 0 && vr.bnd.nZone > 0)
    {
        // about 32 threads, and no more rows than the 48 KB of shared memory that a launch has without asking hold
        const size_t rowBytes = sizeof(real) * (2 * R * NV + NV + g.nGf * (R + 2 * NV));
        const int tpr = bnd_row_threads(g.nGf), want = tpr < 32 ? 32 / tpr : 1, fit = (int)(48 * 1024 / rowBytes), rows = want < fit ? want : fit;
        const size_t sh = rows * rowBytes;
        launch_chained_shared(k_vr_vjp_bnd<DIM, P, NV>, (unsigned)((m.nBndCell + rows - 1) / rows), rows * tpr, sh, st, m, g, vr, v, uRec, u, vRec, vU, tpr);
    }
}
} // namespace
} // namespace dndsb
