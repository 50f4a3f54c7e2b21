// Deterministic column reductions (sum / min / max) over cell rows: a fixed
// partition into kRedBlocks chunks, a fixed shared-memory tree per chunk and
// a single-block final pass, so results do not depend on scheduling.
#include "solver.cuh"
#include "krylov_update.cuh"
#include "vec_split.cuh"
#include "chain.cuh"
#include <type_traits>

namespace dndsb
{
namespace
{
constexpr int kRedBlock = 256;

// deterministic reductions: fixed block partition, fixed shared-memory tree

template <int OP /*0 sum, 1 min, 2 max*/>
DNDSB_D real red_op(real a, real b) { return OP == 0 ? a + b : OP == 1 ? dmin(a, b) : dmax(a, b); }

template <int OP>
DNDSB_D real warp_red(real x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        x = red_op<OP>(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

// partial[block][col] over the block's rows; x is [n][ncol], ncol at most 8, optional row weight w.  One pass for all
// columns, a thread per row: a tree per column over 592 blocks took 6.3 us for 8,192 rows of 5 and the final one 5.6.
template <int OP>
DNDSB_GLOBAL void k_reduce_cols(int64_t n, int ncol, const real *x, const real *__restrict__ w, int powP, real *partial)
{
    chain_step();
    __shared__ real sh[kRedBlock / 32][8];
    real a[8];
#pragma unroll
    for (int v = 0; v < 8; v++)
        a[v] = OP == 0 ? 0.0 : OP == 1 ? kVeryLarge : -kVeryLarge;
    DNDSB_KERNEL_LOOP(i, n)
    {
        const real wi = w ? w[i] : 1.0;
#pragma unroll
        for (int v = 0; v < 8; v++)
            if (v < ncol)
            {
                real xv = x[i * ncol + v];
                xv = powP == 1 ? fabs(xv) : powP == 2 ? xv * xv : xv;
                a[v] = red_op<OP>(a[v], xv * wi);
            }
    }
#pragma unroll
    for (int v = 0; v < 8; v++)
    {
        const real r = warp_red<OP>(a[v]);
        if ((threadIdx.x & 31) == 0)
            sh[threadIdx.x >> 5][v] = r;
    }
    __syncthreads();
    if ((int)threadIdx.x < ncol)
    {
        real r = sh[0][threadIdx.x];
        for (int k = 1; k < kRedBlock / 32; k++)
            r = red_op<OP>(r, sh[k][threadIdx.x]);
        partial[blockIdx.x * ncol + threadIdx.x] = r;
    }
}

// one warp per column
template <int OP>
DNDSB_GLOBAL void k_reduce_final(int nb, int ncol, const real *partial, real *out)
{
    chain_step();
    const int col = threadIdx.x >> 5, lane = threadIdx.x & 31;
    real a = OP == 0 ? 0.0 : OP == 1 ? kVeryLarge : -kVeryLarge;
    for (int i = lane; i < nb; i += 32)
        a = red_op<OP>(a, partial[i * ncol + col]);
    a = warp_red<OP>(a);
    if (lane == 0)
        out[col] = a;
}

} // namespace

real *reduce_cols(int op, int64_t n, int ncol, const real *x, const real *w, int powP, real *redBuf, cudaStream_t st)
{
    real *out = redBuf + kRedBlocks * 8;
    const int64_t want = (n + kRedBlock - 1) / kRedBlock;
    const int nb = want < 1 ? 1 : want < kRedBlocks ? (int)want : kRedBlocks;
    if (op == 0)
    {
        launch_chained(k_reduce_cols<0>, nb, kRedBlock, st, n, ncol, x, w, powP, redBuf);
        launch_chained(k_reduce_final<0>, 1, 32 * ncol, st, nb, ncol, redBuf, out);
    }
    else if (op == 1)
    {
        launch_chained(k_reduce_cols<1>, nb, kRedBlock, st, n, ncol, x, w, powP, redBuf);
        launch_chained(k_reduce_final<1>, 1, 32 * ncol, st, nb, ncol, redBuf, out);
    }
    else
    {
        launch_chained(k_reduce_cols<2>, nb, kRedBlock, st, n, ncol, x, w, powP, redBuf);
        launch_chained(k_reduce_final<2>, 1, 32 * ncol, st, nb, ncol, redBuf, out);
    }
    return out;
}
// ---------------------------------------------------------------------------
// Krylov reductions for the native GMRES (weighted dots, Gram-Schmidt).
// Vectors are flat [n] arrays of T, cell rows of NV variables or (SPLIT) laid out as in vec_split.cuh;
// element i carries the weight s2 of its variable; sums accumulate in FP64 over the same fixed partition.
// ---------------------------------------------------------------------------
namespace
{
DNDSB_D void block_sum4(real (*sh)[kRedBlock], real a0, real a1, real a2, real a3)
{
    sh[0][threadIdx.x] = a0, sh[1][threadIdx.x] = a1, sh[2][threadIdx.x] = a2, sh[3][threadIdx.x] = a3;
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1)
    {
        if (threadIdx.x < st)
            for (int q = 0; q < 4; q++)
                sh[q][threadIdx.x] += sh[q][threadIdx.x + st];
        __syncthreads();
    }
}

// Quads of 4 consecutive elements, loaded as one 16-byte (float) or two 16-byte (double) loads.
template <typename T>
struct Quad;
template <>
struct Quad<float>
{
    using raw = float4;
    static DNDSB_D raw load_raw(const float *p) { return *(const float4 *)p; }
    static DNDSB_D real dot(const raw &v, const real (&w)[4]) { return (real)v.x * w[0] + (real)v.y * w[1] + (real)v.z * w[2] + (real)v.w * w[3]; }
    static DNDSB_D void load(const float *p, real (&o)[4])
    {
        float4 v = *(const float4 *)p;
        o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
    }
    // stores x rounded to float and returns the stored values
    static DNDSB_D void store(float *p, const real (&x)[4], real (&r)[4])
    {
        float4 v = make_float4((float)x[0], (float)x[1], (float)x[2], (float)x[3]);
        *(float4 *)p = v;
        r[0] = v.x, r[1] = v.y, r[2] = v.z, r[3] = v.w;
    }
};
template <>
struct Quad<double>
{
    struct raw
    {
        double2 a, b;
    };
    static DNDSB_D raw load_raw(const double *p) { return raw{((const double2 *)p)[0], ((const double2 *)p)[1]}; }
    static DNDSB_D real dot(const raw &v, const real (&w)[4]) { return v.a.x * w[0] + v.a.y * w[1] + v.b.x * w[2] + v.b.y * w[3]; }
    static DNDSB_D void load(const double *p, real (&o)[4])
    {
        double2 a = ((const double2 *)p)[0], b = ((const double2 *)p)[1];
        o[0] = a.x, o[1] = a.y, o[2] = b.x, o[3] = b.y;
    }
    static DNDSB_D void store(double *p, const real (&x)[4], real (&r)[4])
    {
        ((double2 *)p)[0] = make_double2(x[0], x[1]);
        ((double2 *)p)[1] = make_double2(x[2], x[3]);
        r[0] = x[0], r[1] = x[1], r[2] = x[2], r[3] = x[3];
    }
};

// sum over the block in a fixed order: xor-shuffle tree inside each warp (lane 0's value is
// used), then the warps in index order by one thread; valid in thread 0 (and for column k in
// thread k of the multi-column form below)
DNDSB_D real warp_sum(real x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

constexpr int kKG = 8; // most columns a block of the multi-dot takes

// Called by every block after it has written its partials [nb][ncol]: the block that arrives last
// (a ticket on *cnt, which it resets for the next launch) sums them per column in a fixed order (lanes
// over a fixed stride of the blocks, then a fixed xor tree, lane 0's value), the order the separate
// final pass used, so the result does not depend on which block finishes last.  out[col] = the sum
// (its square root with takeSqrt) times colScale[col] (when given).  Returns true in that block
// (uniformly over its threads).
DNDSB_D bool last_block_final(int nb, int ncol, const real *partial, real *out, const real *colScale, int takeSqrt, unsigned *cnt)
{
    __shared__ unsigned ticket;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        ticket = atomicAdd(cnt, 1u);
    __syncthreads();
    if (ticket != gridDim.x - 1)
        return false;
    __threadfence();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int col = wid; col < ncol; col += nw)
    {
        real a = 0;
        for (int i = lane; i < nb; i += 32)
            a += __ldcg(partial + (int64_t)i * ncol + col);
        a = warp_sum(a);
        if (lane == 0)
        {
            real r = takeSqrt ? sqrt(a) : a;
            out[col] = colScale ? r * colScale[col] : r;
        }
    }
    if (threadIdx.x == 0)
        *cnt = 0;
    __syncthreads();
    return true;
}

// weights of the four elements of quad q, for quads q0, q0 + dq, ... (dq of either sign): split vectors hold a quad within the first four
// variables of a cell or within the rest, plain ones start it at variable (4 q) % NV
template <int NV, bool SPLIT>
struct QuadWeights
{
    const real *ss;
    int64_t nCell;
    int r, dr;
    DNDSB_D QuadWeights(const real *ss_, int64_t n, int64_t q0, int dq)
        : ss(ss_), nCell(n / NV), r(SPLIT ? 0 : (int)((4 * q0) % NV)), dr(SPLIT ? 0 : ((4 * dq) % NV + NV) % NV)
    {
    }
    DNDSB_D real at(int64_t q, int e) const
    {
        if constexpr (SPLIT)
            return ss[q < nCell ? e : NV == 5 ? 4 : 4 + (e & 1)];
        else
            return ss[r + e < NV ? r + e : r + e - NV];
    }
    DNDSB_D void next()
    {
        if constexpr (!SPLIT)
            r = r + dr >= NV ? r + dr - NV : r + dr;
    }
};

// sums of NK columns from V against w over the quads q0, q0 + dq, ...: warp sums into sh[column][warp]
template <typename T, int NV, bool SPLIT, int NK>
DNDSB_D void mdot_group(int64_t n, int64_t q0, int dq, int64_t ld, const T *V, const T *w, const real *ss,
                        real (*sh)[kRedBlock / 32])
{
    real a[NK];
#pragma unroll
    for (int k = 0; k < NK; k++)
        a[k] = 0;
    const int64_t nq = (n + 3) >> 2;
    QuadWeights<NV, SPLIT> qw(ss, n, q0, dq);
    for (int64_t q = q0; q < nq; q += dq, qw.next())
    {
        // every load issued (in its storage type) before the first use
        typename Quad<T>::raw v[NK];
#pragma unroll
        for (int k = 0; k < NK; k++)
            v[k] = Quad<T>::load_raw(V + k * ld + 4 * q);
        real wv[4];
        Quad<T>::load(w + 4 * q, wv);
#pragma unroll
        for (int e = 0; e < 4; e++)
            wv[e] *= qw.at(q, e);
#pragma unroll
        for (int k = 0; k < NK; k++)
            a[k] += Quad<T>::dot(v[k], wv);
    }
#pragma unroll
    for (int k = 0; k < NK; k++)
    {
        const real x = warp_sum(a[k]);
        if ((threadIdx.x & 31) == 0)
            sh[k][threadIdx.x >> 5] = x;
    }
}

// out[col] = colScale[col] sum_i V[col][i] w[i] s2[var(i)] (the basis columns are stored unnormalised; colScale holds
// their normalising factors).  Columns are ld apart (ld a multiple of 4, the pad beyond n zero).
// HBM bound on the basis.  The kRedBlocks blocks split into nG groups of at most kKG columns (their widths differ by
// at most one) times chunks of quads, block = chunk nG + group, so the blocks of a chunk share its w in L2 and every
// block makes one pass: 592 blocks that each walked all column groups over a chunk of 592 paid a block reduction per
// group for one or two quads per thread (30 steps of 249,600 tets in FP64: 1.30 -> 1.08 ms).  partial [chunks][ncol]; the
// last block to finish sums the chunks.
// All chunks advance together through the vector (a chunk's threads take every nChunk-th group of 256 quads), so what the
// caches hold at the end is the end of every column: k_kmaxpy_norm walks back from there.  With each block on a range of
// its own and both kernels forwards, GMRES(30) took 3.49 ms for 249,600 tets in FP64 and 12.45 ms for 1,996,800 in FP32,
// now 3.30 and 12.10.
template <typename T, int NV, bool SPLIT>
DNDSB_GLOBAL void __launch_bounds__(kRedBlock, 4) k_kmdot(int64_t n, int64_t ld, int ncol, int nG, const T *V, const T *w,
                                                       const real *__restrict__ s2, real *partial, real *out, const real *colScale,
                                                       unsigned *cnt)
{
    chain_step();
    __shared__ real sh[kKG][kRedBlock / 32];
    __shared__ real ss[8];
    if (threadIdx.x < NV)
        ss[threadIdx.x] = s2[threadIdx.x];
    __syncthreads();
    const int grp = blockIdx.x % nG, chunk = blockIdx.x / nG, nChunk = gridDim.x / nG;
    const int base = ncol / nG, extra = ncol - base * nG; // the first `extra` groups have one column more
    const int c0 = grp * base + (grp < extra ? grp : extra), nk = base + (grp < extra ? 1 : 0);
    const int64_t q0 = (int64_t)chunk * blockDim.x + threadIdx.x;
    const int dq = nChunk * (int)blockDim.x;
    const T *Vc = V + (int64_t)c0 * ld;
    switch (nk)
    {
    case 1: mdot_group<T, NV, SPLIT, 1>(n, q0, dq, ld, Vc, w, ss, sh); break;
    case 2: mdot_group<T, NV, SPLIT, 2>(n, q0, dq, ld, Vc, w, ss, sh); break;
    case 3: mdot_group<T, NV, SPLIT, 3>(n, q0, dq, ld, Vc, w, ss, sh); break;
    case 4: mdot_group<T, NV, SPLIT, 4>(n, q0, dq, ld, Vc, w, ss, sh); break;
    case 5: mdot_group<T, NV, SPLIT, 5>(n, q0, dq, ld, Vc, w, ss, sh); break;
    case 6: mdot_group<T, NV, SPLIT, 6>(n, q0, dq, ld, Vc, w, ss, sh); break;
    case 7: mdot_group<T, NV, SPLIT, 7>(n, q0, dq, ld, Vc, w, ss, sh); break;
    default: mdot_group<T, NV, SPLIT, 8>(n, q0, dq, ld, Vc, w, ss, sh); break;
    }
    __syncthreads();
    if ((int)threadIdx.x < nk)
    {
        real t = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++)
            t += sh[threadIdx.x][q];
        partial[(int64_t)chunk * ncol + c0 + threadIdx.x] = t;
    }
    last_block_final(nChunk, ncol, partial, out, colScale, 0, cnt);
}

// w -= sum_c h[c] colScale[c] V[c] (columns subtracted in index order), the quads from the last to the first (see k_kmdot);
// the last block writes
// *outNorm = sqrt(sum_i w_i^2 s2[var(i)]) of the stored w.  w is column ncol of the same basis (not read
// through V).  With gsc (the GMRES scalars: [0] scale, [2] valid columns) it also sets the normalising
// factor of the new column, *scaleNext = 1 / norm, or 0 at a breakdown (norm <= 1e-32 scale), which it
// records in gsc[2] = j (GMRES_LeftPreconditioned::solve, Linear.hpp:100-108).
template <typename T, int NV, bool SPLIT>
DNDSB_GLOBAL void __launch_bounds__(kRedBlock, 4) k_kmaxpy_norm(int64_t n, int64_t ld, int ncol, const T *V, const real *h,
                                                             const real *colScale, T *w, const real *__restrict__ s2, real *partial,
                                                             real *outNorm, unsigned *cnt, real *gsc, int j, real *scaleNext)
{
    chain_step();
    __shared__ real hs[32];
    __shared__ real ss[8];
    __shared__ real sh[kRedBlock / 32];
    if (threadIdx.x < ncol)
        hs[threadIdx.x] = h[threadIdx.x] * (colScale ? colScale[threadIdx.x] : 1.0);
    if (threadIdx.x < NV)
        ss[threadIdx.x] = s2[threadIdx.x];
    __syncthreads();
    const int64_t nq = (n + 3) >> 2, dq = (int64_t)gridDim.x * blockDim.x, at = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t q1 = at + (nq - 1) / dq * dq; // the thread's last quad, or one dq beyond
    real a = 0;
    QuadWeights<NV, SPLIT> qw(ss, n, q1, -(int)dq);
    for (int64_t q = q1; q >= 0; q -= dq, qw.next())
    {
        if (q >= nq)
            continue;
        real x[4];
        Quad<T>::load(w + 4 * q, x);
        int c = 0;
        for (; c + 4 <= ncol; c += 4)
        {
            real v[4][4];
#pragma unroll
            for (int k = 0; k < 4; k++)
                Quad<T>::load(V + (int64_t)(c + k) * ld + 4 * q, v[k]);
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                const real hc = hs[c + k];
#pragma unroll
                for (int e = 0; e < 4; e++)
                    x[e] -= hc * v[k][e];
            }
        }
        for (; c < ncol; c++)
        {
            real v[4];
            Quad<T>::load(V + (int64_t)c * ld + 4 * q, v);
            const real hc = hs[c];
#pragma unroll
            for (int e = 0; e < 4; e++)
                x[e] -= hc * v[e];
        }
        if (4 * q + 4 > n) // the pad stays zero also where a factor is not finite: later solves read it
        {
#pragma unroll
            for (int e = 1; e < 4; e++)
                x[e] = 4 * q + e < n ? x[e] : 0.0;
        }
        real xr[4];
        Quad<T>::store(w + 4 * q, x, xr);
#pragma unroll
        for (int e = 0; e < 4; e++)
            a += xr[e] * xr[e] * qw.at(q, e);
    }
    const real x = warp_sum(a);
    if ((threadIdx.x & 31) == 0)
        sh[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        real t = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++)
            t += sh[q];
        partial[blockIdx.x] = t;
    }
    if (last_block_final(gridDim.x, 1, partial, outNorm, nullptr, 1, cnt) && gsc && threadIdx.x == 0)
    {
        real hn = *outNorm;
        bool broken = !(hn > gsc[0] * 1e-32) || gsc[2] <= j;
        *scaleNext = broken ? 0.0 : 1.0 / hn;
        if (broken && gsc[2] > j)
            gsc[2] = j;
    }
}

// x += sum_c y_c colScale_c V_c over the valid columns (gsc[2], at most k), y = gsc[yOff ...].  HBM bound on the
// basis: quads of a column as in the multi-dot, four columns in flight (one element per thread and column at a time
// took 371 us at 2 million cells, FP32; now 185).  x needs no alignment or pad: its ragged end goes by elements.
template <typename T>
DNDSB_GLOBAL void __launch_bounds__(kRedBlock) k_kupdate(int64_t n, int64_t ld, int k, const T *__restrict__ V, const real *__restrict__ gsc, int yOff,
                                                        const real *__restrict__ colScale, T *x)
{
    __shared__ real hs[32];
    const int nv = dmin(gsc[2], k);
    if ((int)threadIdx.x < nv)
        hs[threadIdx.x] = gsc[yOff + threadIdx.x] * colScale[threadIdx.x];
    __syncthreads();
    DNDSB_KERNEL_LOOP(q, (n + 3) >> 2)
    {
        const int m = n - 4 * q < 4 ? (int)(n - 4 * q) : 4;
        real a[4];
#pragma unroll
        for (int e = 0; e < 4; e++)
            a[e] = e < m ? (real)x[4 * q + e] : 0.0;
        int c = 0;
        for (; c + 4 <= nv; c += 4)
        {
            real v[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                Quad<T>::load(V + (int64_t)(c + i) * ld + 4 * q, v[i]);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    a[e] += hs[c + i] * v[i][e];
        }
        for (; c < nv; c++)
        {
            real v[4];
            Quad<T>::load(V + (int64_t)c * ld + 4 * q, v);
#pragma unroll
            for (int e = 0; e < 4; e++)
                a[e] += hs[c] * v[e];
        }
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (e < m)
                x[4 * q + e] = (T)a[e];
    }
}

// partial[block] = sum_i x_i^2 s2[var(i)] (any length, any alignment)
template <typename T, int NV, bool SPLIT>
DNDSB_GLOBAL void k_knorm2(int64_t n, const T *__restrict__ x, const real *__restrict__ s2, real *partial, real *outNorm, unsigned *cnt)
{
    __shared__ real sh[4][kRedBlock];
    int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    int64_t b0 = blockIdx.x * chunk, b1 = b0 + chunk < n ? b0 + chunk : n;
    real a = 0;
    for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x)
    {
        real d = (real)x[i];
        a += d * d * s2[SPLIT ? vsplit::var_of<NV>(n / NV, i) : (int)(i % NV)];
    }
    block_sum4(sh, a, 0, 0, 0);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = sh[0][0];
    last_block_final(gridDim.x, 1, partial, outNorm, nullptr, 1, cnt);
}

// partial[block] = sum_i (a_i - b_i)^2 s2[var(i)]
template <typename T, int NV, bool SPLIT>
DNDSB_GLOBAL void k_kdiff_norm(int64_t n, const T *__restrict__ x, const T *__restrict__ y, const real *__restrict__ s2, real *partial,
                               real *outNorm, unsigned *cnt)
{
    __shared__ real sh[4][kRedBlock];
    int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    int64_t b0 = blockIdx.x * chunk, b1 = b0 + chunk < n ? b0 + chunk : n;
    real a = 0;
    for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x)
    {
        real d = (real)x[i] - (real)y[i];
        a += d * d * s2[SPLIT ? vsplit::var_of<NV>(n / NV, i) : (int)(i % NV)];
    }
    block_sum4(sh, a, 0, 0, 0);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = sh[0][0];
    last_block_final(gridDim.x, 1, partial, outNorm, nullptr, 1, cnt);
}

// blocks of kRedBlock threads for n elements, at most `most`, each thread with the same number of quads where it can be
unsigned even_blocks(int64_t n, int most)
{
    const int64_t nq = (n + 3) >> 2, rounds = (nq + (int64_t)most * kRedBlock - 1) / ((int64_t)most * kRedBlock);
    return (unsigned)((nq + rounds * kRedBlock - 1) / (rounds * kRedBlock));
}

template <typename T, int NV, bool SPLIT>
void kmdot(int64_t n, int64_t ld, int ncol, const void *V, const void *w, const real *s2, real *red, real *out, const real *colScale,
           unsigned *cnt, cudaStream_t st)
{
    const int nG = (ncol + kKG - 1) / kKG;
    launch_chained(k_kmdot<T, NV, SPLIT>, even_blocks(n, kRedBlocks / nG) * nG, kRedBlock, st, n, ld, ncol, nG, (const T *)V, (const T *)w, s2, red, out, colScale, cnt);
}

template <typename T, int NV, bool SPLIT>
void kmaxpy(int64_t n, int64_t ld, int ncol, const void *V, const real *h, const real *colScale, void *w, const real *s2, real *red,
            real *outNorm, unsigned *cnt, real *gsc, int j, real *scaleNext, cudaStream_t st)
{
    launch_chained(k_kmaxpy_norm<T, NV, SPLIT>, even_blocks(n, kRedBlocks), kRedBlock, st, n, ld, ncol, (const T *)V, h, colScale, (T *)w, s2, red, outNorm, cnt, gsc, j,
                                                           scaleNext);
}

template <typename T, int NV, bool SPLIT>
void knorm(int64_t n, const void *x, const real *s2, real *red, real *outNorm, unsigned *cnt, cudaStream_t st)
{
    k_knorm2<T, NV, SPLIT><<<kRedBlocks, kRedBlock, 0, st>>>(n, (const T *)x, s2, red, outNorm, cnt);
}

template <typename T, int NV, bool SPLIT>
void kdiff(int64_t n, const void *x, const void *y, const real *s2, real *red, real *outNorm, unsigned *cnt, cudaStream_t st)
{
    k_kdiff_norm<T, NV, SPLIT><<<kRedBlocks, kRedBlock, 0, st>>>(n, (const T *)x, (const T *)y, s2, red, outNorm, cnt);
}

template <typename F>
void for_kind(int prec, int nv, bool split, F f)
{
    using std::integral_constant;
    auto nvs = [&](auto t, auto sp) { nv == 5 ? f(t, integral_constant<int, 5>(), sp) : f(t, integral_constant<int, 6>(), sp); };
    auto sps = [&](auto t) { split ? nvs(t, std::true_type()) : nvs(t, std::false_type()); };
    prec ? sps(float()) : sps(double());
}
#define DNDSB_KDISPATCH(FN, ...) \
    for_kind(prec, nv, split, [&](auto t, auto v, auto sp) { FN<decltype(t), decltype(v)::value, decltype(sp)::value>(__VA_ARGS__); })
} // namespace

// V: ncol columns ld apart (ld a multiple of 4, 16-byte aligned, zero beyond n); w: a column of the same storage
void krylov_mdot(int prec, int64_t n, int64_t ld, int nv, bool split, int ncol, const void *V, const void *w, const real *s2, real *red, real *out,
                 const real *colScale, unsigned *cnt, cudaStream_t st)
{
    DNDSB_KDISPATCH(kmdot, n, ld, ncol, V, w, s2, red, out, colScale, cnt, st);
}

void krylov_maxpy_norm(int prec, int64_t n, int64_t ld, int nv, bool split, int ncol, const void *V, const real *h, const real *colScale, void *w,
                       const real *s2, real *red, real *outNorm, unsigned *cnt, real *gsc, int j, real *scaleNext, cudaStream_t st)
{
    DNDSB_KDISPATCH(kmaxpy, n, ld, ncol, V, h, colScale, w, s2, red, outNorm, cnt, gsc, j, scaleNext, st);
}

void krylov_update_x(int prec, int64_t n, int k, const void *V, const real *gsc, int yOff, const real *colScale, void *x, cudaStream_t st)
{
    const int64_t nq = (n + 3) >> 2;
    if (prec)
        DNDSB_LAUNCH(k_kupdate<float>, nq, kRedBlock, st, n, krylov_ld(n), k, (const float *)V, gsc, yOff, colScale, (float *)x);
    else
        DNDSB_LAUNCH(k_kupdate<double>, nq, kRedBlock, st, n, krylov_ld(n), k, (const double *)V, gsc, yOff, colScale, (double *)x);
}

void krylov_norm(int prec, int64_t n, int nv, bool split, const void *x, const real *s2, real *red, real *outNorm, unsigned *cnt, cudaStream_t st)
{
    DNDSB_KDISPATCH(knorm, n, x, s2, red, outNorm, cnt, st);
}

void krylov_diff_norm(int prec, int64_t n, int nv, bool split, const void *x, const void *y, const real *s2, real *red, real *outNorm, unsigned *cnt,
                      cudaStream_t st)
{
    DNDSB_KDISPATCH(kdiff, n, x, y, s2, red, outNorm, cnt, st);
}
} // namespace dndsb
