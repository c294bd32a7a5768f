/*
 * igab_spmv.cuh -- the product of the structured CSR matrix with a vector, one warp per control point
 * (see igab_krylov.cu for the layout), shared by the Krylov solvers and the multigrid smoothers.
 */
#ifndef IGAB_SPMV_CUH
#define IGAB_SPMV_CUH

#include "igab_device.cuh"

namespace {

/* the window of control points a row couples to (csr_pos) */
__device__ __forceinline__ void row_window(const igab_geom &g, long r, int &x0, int &y0, int &z0, int &nxb, int &nyb,
                                           int &nzb, int &x1, int &y1, int &z1, int &k1)
{
    /* 32-bit divisions: the nonzeros, 27 per row and more, are counted in 31 bits */
    const unsigned row = (unsigned)r, cp = row / 3u, n2 = (unsigned)g.nb[2], n1 = (unsigned)g.nb[1], xy = cp / n2;
    k1 = (int)(row - 3u * cp);
    z1 = (int)(cp - xy * n2);
    x1 = (int)(xy / n1);
    y1 = (int)(xy - (unsigned)x1 * n1);
    x0 = x1 > 2 ? x1 - 2 : 0;
    y0 = y1 > 2 ? y1 - 2 : 0;
    z0 = z1 > 2 ? z1 - 2 : 0;
    const int xe = x1 + 2 < g.nb[0] - 1 ? x1 + 2 : g.nb[0] - 1;
    const int ye = y1 + 2 < g.nb[1] - 1 ? y1 + 2 : g.nb[1] - 1;
    const int ze = z1 + 2 < g.nb[2] - 1 ? z1 + 2 : g.nb[2] - 1;
    nxb = xe - x0 + 1;
    nyb = ye - y0 + 1;
    nzb = ze - z0 + 1;
}

/* rows 3 cp, 3 cp + 1, 3 cp + 2 of K x, in every lane of the warp; x may be another kernel's output that this one has
 * waited for, so it comes without __restrict__ (ordinary loads) */
template <typename T>
__device__ __forceinline__ void spmv_rows(const igab_geom &g, const T *__restrict__ vals, const double *x, long cp,
                                          int lane, double &a0, double &a1, double &a2)
{
    int x0, y0, z0, nxb, nyb, nzb, x1, y1, z1, k1;
    row_window(g, 3 * cp, x0, y0, z0, nxb, nyb, nzb, x1, y1, z1, k1);
    const int L = 3 * nzb, total = nxb * nyb * L;   /* L in {9, 12, 15}, total <= 375 */
    /* lane j < nxb * nyb (<= 25) holds the first column of run j */
    const long base_own = lane < nxb * nyb ? 3 * cp_index(g, x0 + lane / nyb, y0 + lane % nyb, z0) : 0;
    /* run = p / L as (p * ceil(2^16 / L)) >> 16, exact for L in {9, 12, 15} and p < 375 */
    const unsigned invL = (65536u + (unsigned)L - 1u) / (unsigned)L;
    /* the three rows of the control point share the columns; row k starts k * total later */
    const T *v0 = vals + g.rowptr[3 * cp], *v1 = v0 + total, *v2 = v1 + total;
    a0 = a1 = a2 = 0.0;
    /* four 32-entry chunks per pass: every load of the pass is issued before the first
     * multiply, so a warp keeps 16 loads in flight; the additions keep the chunk order */
    for (int p0 = 0; p0 < total; p0 += 128) {
        double xv[4];
        T w0[4], w1[4], w2[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int p = p0 + 32 * c + lane;
            const bool in = p < total;
            const int run = (int)(((unsigned)(in ? p : 0) * invL) >> 16);
            const long base = __shfl_sync(0xffffffffu, base_own, run);
            xv[c] = in ? x[base + (p - run * L)] : 0.0;
            w0[c] = in ? v0[p] : T(0);
            w1[c] = in ? v1[p] : T(0);
            w2[c] = in ? v2[p] : T(0);
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (p0 + 32 * c + lane < total) {
                a0 += double(w0[c]) * xv[c];
                a1 += double(w1[c]) * xv[c];
                a2 += double(w2[c]) * xv[c];
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
}

/* the same with the matrix loaded whole (375 entries at most, 12 chunks: a lane's 36 loads are in flight at once), which
 * needs no x, so that a kernel can do it before it waits for the one that writes x.  For a matrix of few waves of
 * blocks: spmv_rows takes half the registers and streams a large one.  The additions are in spmv_rows' order. */
#define SPMV_CHUNKS 12
template <typename T>
struct spmv_part {
    T w[3][SPMV_CHUNKS];
    unsigned col[SPMV_CHUNKS];
    int total;
};
template <typename T>
__device__ __forceinline__ void spmv_load(const igab_geom &g, const T *__restrict__ vals, long cp, int lane,
                                          spmv_part<T> &P)
{
    int x0, y0, z0, nxb, nyb, nzb, x1, y1, z1, k1;
    row_window(g, 3 * cp, x0, y0, z0, nxb, nyb, nzb, x1, y1, z1, k1);
    const int L = 3 * nzb, total = nxb * nyb * L;
    const unsigned base_own = lane < nxb * nyb ? (unsigned)(3 * cp_index(g, x0 + lane / nyb, y0 + lane % nyb, z0)) : 0u;
    const unsigned invL = (65536u + (unsigned)L - 1u) / (unsigned)L;
    const T *v = vals + g.rowptr[3 * cp];
    P.total = total;
#pragma unroll
    for (int c = 0; c < SPMV_CHUNKS; c++) {
        const int p = 32 * c + lane;
        const bool in = p < total;
        const int run = (int)(((unsigned)(in ? p : 0) * invL) >> 16);
        P.col[c] = __shfl_sync(0xffffffffu, base_own, run) + (unsigned)(p - run * L);
#pragma unroll
        for (int k = 0; k < 3; k++) P.w[k][c] = in ? v[k * total + p] : T(0);
    }
}
template <typename T>
__device__ __forceinline__ void spmv_mult(const spmv_part<T> &P, const double *x, int lane, double a[3])
{
    double xv[SPMV_CHUNKS];
#pragma unroll
    for (int c = 0; c < SPMV_CHUNKS; c++) xv[c] = 32 * c + lane < P.total ? x[P.col[c]] : 0.0;
    a[0] = a[1] = a[2] = 0.0;
#pragma unroll
    for (int c = 0; c < SPMV_CHUNKS; c++)
        if (32 * c + lane < P.total)
#pragma unroll
            for (int k = 0; k < 3; k++) a[k] += double(P.w[k][c]) * xv[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; k++) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
}

} /* namespace */

#endif
