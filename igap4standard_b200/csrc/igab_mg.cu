/*
 * Geometric multigrid on nested spline spaces, as the preconditioner of a GMRES or
 * conjugate gradient solve with the assembled tangent (no reference counterpart: it
 * stands in for the PETSc KSP of the reference application, src/snes_init.c:24-39,
 * which is outside the assembly path).
 *
 * Why: the phys/ge tangent is a fourth-order operator (the strain-gradient term
 * le^2 |grad grad u|^2), so its condition number grows like h^-4; Jacobi-preconditioned
 * Krylov iterations stall at 32^3 and 64^3.  Multigrid keeps the iteration count flat.
 *
 * Hierarchy.  Level 0 is the caller's mesh.  Level l+1 removes every other interior
 * knot of level l in each direction (n elements -> n / 2), so its spline space is a
 * subspace of level l's: the prolongation is knot insertion of the removed knots
 * (Boehm's algorithm for p = 2, built on the host as three 1-D matrices, applied on
 * the device as their tensor product), the restriction its transpose.  Coarsening stops
 * at about a thousand dofs, or where a direction has an odd element count.  Coarse
 * operators are rediscretised: each coarse level is an igab context with the same
 * material, boundary tables and (averaged) element scales, whose tangent is assembled
 * at the zero state by the library's own kernels (a preconditioner, so the state it is
 * linearised at only affects the convergence rate).  The coarsest level is solved
 * directly (its inverse, below).  Dirichlet rows, identity rows
 * of every level's tangent, are masked out of the restricted residuals and of the
 * prolonged corrections, which keeps the V-cycle symmetric.
 *
 * Smoother: Chebyshev polynomial of degree 6 in D^-1 K on [1.1 lmax / 100, 1.1 lmax], lmax
 * by 40 power iterations; the same polynomial before and after the coarse
 * correction, so the V-cycle is a symmetric preconditioner and CG applies.
 *
 * Coarsest level: its tangent (symmetric positive definite: the zero-state tangent with
 * unit Dirichlet rows and columns) is inverted on the device by Gauss-Jordan elimination
 * without pivoting, one launch per pivot, and each V-cycle applies the inverse as a dense
 * product with a fixed summation order (no host round trip).  A pivot that is not
 * positive and finite (an unstable material) falls back to a dense LU with partial
 * pivoting on the host.
 *
 * Operators: every level's is the tangent at the zero state (the fine one in FP32, the
 * coarse ones in FP64), symmetric positive definite for a stable material, so the V-cycle
 * does not depend on the Newton iterate.  The hierarchy is rebuilt when the material, the
 * boundary tables' values or the element scales change (the context's parameter
 * version).  Every dot product is a fixed-order reduction: solves are bitwise repeatable.
 *
 * On meshes of some ten thousand dofs a solve is bound by the number of its short kernels, not by their bytes.  The
 * smoother's vector updates ride on its products: a level but the coarsest takes 12 products and two transfers per
 * V-cycle.  The V-cycle is one graph launch, a Gram-Schmidt step keeps its coefficients on the device and is read once,
 * each kernel is launched, and its matrix rows and tables loaded, under the one before (mg_launch), the Gram-Schmidt
 * products of all vectors run side by side, and a kernel has blocks for the dofs there are.  GMRES of three Newton steps
 * at 8^3 / 16^3 / 24^3 / 32^3: 3.1 / 9.4 / 28.1 / 70.6 ms, 30 / 47 / 63 / 80 iterations of 104 / 199 / 446 / 883 us.
 * What is left at 16^3 are 12 fine products of 9 us (6 us of them latency: three passes of loads on 1.2 waves of blocks)
 * and some 26 other kernels of 3-5 us.
 * The parts of it, measured at degree 3 (6 products per level) at 16^3: fused updates, graph and device coefficients
 * 465 -> 175 us per iteration, launches under one another 175 -> 127 us (8^3: 6.5 -> 4.6 ms, 32^3, 185 iterations:
 * 110.5 -> 95.2 ms); left out: more blocks per SM by fewer registers (spills, 14.0-19.6 ms against 13.7), rows cut at
 * whole runs of columns (half the instructions, no faster, 32^3 101.6).
 * Measured and rejected: the smoothing operators stored in half precision (64^3: 4.58 ->
 * 4.36 ms per GMRES iteration, but one more iteration per solve; no gain per Newton step).
 */
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include <cuda_runtime.h>
#include <type_traits>
#include "igab_internal.h"
#include "igab_reduce.cuh"
#include "igab_spmv.cuh"

namespace {

#define MG_THREADS 256
#define MG_BLOCKS 296
#define MG_ALL 4096            /* control points up to which a product loads its rows whole, before the wait (mg_spmv) */
#define MG_SPMV 128            /* block of the smoother's products: small, so that a coarse level spreads over the SMs */
#define MG_MAX_LEVELS 8
#define MG_DEGREE 6            /* Chebyshev degree per smoothing */
#define MG_RATIO 100.0         /* largest to smallest eigenvalue of its interval (mg_cheb) */
#define MG_POWER_ITERS 40      /* power iterations for lmax of D^-1 K (estimate_lmax) */
#define MG_POWER_NORM 10       /* normalised after so many */
#define GM_RESTART 50          /* GMRES restart length */
#define MG_COARSE_DOF 1200     /* the coarsest level is solved directly below this size */

/* 1-D prolongation along one direction: fine coefficient i = sum_a w[i][a] coarse idx[i][a]
 * (kp entries per fine point), restriction coarse j = sum_b rw[j][b] fine ridx[j][b] */
struct mg_dir {
    int nf = 0, nc = 0, kp = 0, kr = 0;
    int *p_idx = nullptr;
    double *p_w = nullptr;
    int *r_idx = nullptr;
    double *r_w = nullptr;
};

struct mg_level {
    igab_ctx *ctx = nullptr;       /* level 0: the caller's; coarser: owned */
    long n = 0;
    const void *vals = nullptr;    /* the level's tangent values */
    int prec = IGAB_PREC_FP64;
    double *own_vals = nullptr;    /* coarse levels: FP64 tangent at the zero state */
    double *dinv = nullptr;
    double lmax = 0.0;
    double *x = nullptr, *b = nullptr, *r = nullptr, *d = nullptr, *t = nullptr;
    unsigned char *mask = nullptr; /* 1 on the Dirichlet rows */
    mg_dir dir[3];                 /* transfer between this level (coarse) and the one above */
};

__global__ void k_mg_diag_inv(igab_geom g, const void *__restrict__ vals, int prec, double *__restrict__ dinv)
{
    const long r = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (r >= g.ndof) return;
    const long cp = r / 3;
    const int k1 = (int)(r % 3);
    const int z1 = (int)(cp % g.nb[2]), y1 = (int)((cp / g.nb[2]) % g.nb[1]), x1 = (int)(cp / ((long)g.nb[2] * g.nb[1]));
    const int x0 = x1 > 2 ? x1 - 2 : 0, y0 = y1 > 2 ? y1 - 2 : 0, z0 = z1 > 2 ? z1 - 2 : 0;
    const int ye = y1 + 2 < g.nb[1] - 1 ? y1 + 2 : g.nb[1] - 1;
    const int ze = z1 + 2 < g.nb[2] - 1 ? z1 + 2 : g.nb[2] - 1;
    const int nyb = ye - y0 + 1, nzb = ze - z0 + 1;
    const long pos = g.rowptr[r] + (((long)(x1 - x0) * nyb + (y1 - y0)) * nzb + (z1 - z0)) * 3 + k1;
    const double dv = prec == IGAB_PREC_FP64 ? ((const double *)vals)[pos] : (double)((const float *)vals)[pos];
    dinv[r] = dv != 0.0 ? 1.0 / dv : 1.0;
}

#define MG_LOOP(i, n) for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < (n); i += (long)gridDim.x * blockDim.x)

/* Programmatic dependent launch.  The kernels of a V-cycle and of a Gram-Schmidt step follow one another in a stream
 * and take 2-7 us each, so a kernel is launched (mg_launch) while the one before it still runs: it loads what no kernel
 * of the solve writes (the matrix, the tables), then mg_wait() returns when the kernel before has completed and its
 * writes are visible, and lets the next one be launched.  A kernel of the chain therefore starts only after the one
 * two before it has completed.  Vectors are read after mg_wait() and through pointers without __restrict__, which
 * keeps them off the read-only path. */
__device__ __forceinline__ void mg_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... K, class... A>
void mg_launch(void (*k)(K...), dim3 grid, int block, cudaStream_t st, A... a)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, k, K(a)...);   /* an error stays for the callers' cudaGetLastError() */
}

/* d = s * dinv * r */
__global__ void k_mg_jac(long n, const double *__restrict__ dinv, const double *__restrict__ r, double s,
                         double *__restrict__ d)
{
    MG_LOOP(i, n) d[i] = s * dinv[i] * r[i];
}

/* b = r = in, d = s dinv in: a V-cycle's right-hand side and its first Chebyshev direction */
__global__ void k_mg_start(long n, const double *__restrict__ in, const double *__restrict__ dinv, double s,
                           double *__restrict__ b, double *__restrict__ r, double *__restrict__ d)
{
    MG_LOOP(i, n)
    {
        const double v = in[i];
        b[i] = v;
        r[i] = v;
        d[i] = s * dinv[i] * v;
    }
}

/* A product with the level's operator and what the smoother does with it, row by row (the level is a few kernels
 * of a few microseconds: the vector passes between its products cost as much as the products):
 *   MG_STEP        t = K d: x += d (x = d when first), r -= t, d' = a d + c dinv r
 *   MG_LAST_PRE    t = K d: x += d, r -= t with the Dirichlet rows masked (what the restriction takes)
 *   MG_RESID       t = K x: r = b - t, d' = a dinv r
 *   MG_LAST_POST   t = K d: x += d + d', the residual after the last step is not needed
 * d' goes to another vector than d, whose neighbours the other rows still read. */
enum { MG_STEP = 0, MG_LAST_PRE = 1, MG_RESID = 2, MG_LAST_POST = 3 };
template <typename T, int OP, bool ALL>
__global__ void __launch_bounds__(MG_SPMV, ALL ? 4 : 8) k_mg_spmv(igab_geom g, const T *__restrict__ vals, const double *in,
                                                     const double *b, const double *__restrict__ dinv,
                                                     const unsigned char *__restrict__ mask, double a, double c,
                                                     int first, double *x, double *r, double *dn)
{
    const long cp = (long)blockIdx.x * (MG_SPMV / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (3 * cp >= g.ndof) return;   /* warp-uniform */
    const long i = 3 * cp + lane;
    spmv_part<T> P;
    if (ALL) spmv_load<T>(g, vals, cp, lane, P);
    double di = 0.0, u = 0.0, ro = 0.0, xo = 0.0, s[3];
    int dirichlet = 0;
    if (lane < 3) {
        di = dinv[i];
        if (OP == MG_LAST_PRE) dirichlet = mask[i];
    }
    mg_wait();
    if (lane < 3) {
        ro = OP == MG_RESID ? b[i] : r[i];
        if (OP != MG_RESID) u = in[i];
        if (OP != MG_RESID && !first) xo = x[i];
    }
    if (ALL) spmv_mult<T>(P, in, lane, s);
    else spmv_rows<T>(g, vals, in, cp, lane, s[0], s[1], s[2]);
    if (lane >= 3) return;
    const double ri = ro - (lane == 0 ? s[0] : (lane == 1 ? s[1] : s[2]));
    if (OP == MG_RESID) {
        r[i] = ri;
        dn[i] = a * di * ri;
        return;
    }
    const double xn = first ? u : xo + u;
    if (OP == MG_LAST_POST) {
        x[i] = xn + (a * u + c * di * ri);
        return;
    }
    x[i] = xn;
    r[i] = OP == MG_LAST_PRE && dirichlet ? 0.0 : ri;
    if (OP == MG_STEP) dn[i] = a * u + c * di * ri;
}

/* r = b - t */
__global__ void k_mg_sub(long n, const double *__restrict__ b, const double *__restrict__ t, double *__restrict__ r)
{
    MG_LOOP(i, n) r[i] = b[i] - t[i];
}

/* y = a x + b y */
__global__ void k_mg_axpby(long n, double a, const double *__restrict__ x, double b, double *__restrict__ y)
{
    MG_LOOP(i, n) y[i] = a * x[i] + b * y[i];
}

__global__ void k_mg_copy(long n, const double *__restrict__ x, double *__restrict__ y)
{
    MG_LOOP(i, n) y[i] = x[i];
}

__global__ void k_mg_mask(long nd, const int *__restrict__ rows, unsigned char *__restrict__ mask)
{
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t < nd) mask[rows[t]] = 1;
}

struct mg_dirs_dev {
    const int *p_idx[3];
    const double *p_w[3];
    const int *r_idx[3];
    const double *r_w[3];
    int kp[3], kr[3];
    int nbf[3], nbc[3];
};

/* xf += P xc off the Dirichlet rows (tensor product of the three 1-D prolongations, per displacement component) */
__global__ void __launch_bounds__(MG_THREADS) k_mg_prolong(mg_dirs_dev D, const double *xc,
                                                           const unsigned char *__restrict__ mask, double *xf)
{
    const long n = 3L * D.nbf[0] * D.nbf[1] * D.nbf[2], i = blockIdx.x * (long)MG_THREADS + threadIdx.x;
    if (i >= n) return;
    const int dirichlet = mask[i];
    const long f = i / 3;
    const int k = (int)(i - 3 * f);
    const int iz = (int)(f % D.nbf[2]), iy = (int)((f / D.nbf[2]) % D.nbf[1]), ix = (int)(f / ((long)D.nbf[2] * D.nbf[1]));
    /* the first two of each direction's points (there are no more with every other knot removed) before the wait */
    int j[3][2];
    double w[3][2];
#pragma unroll
    for (int d = 0; d < 3; d++)
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const int o = (d == 0 ? ix : (d == 1 ? iy : iz)) * D.kp[d] + a;
            const bool in = a < D.kp[d];
            j[d][a] = in ? D.p_idx[d][o] : 0;
            w[d][a] = in ? D.p_w[d][o] : 0.0;
        }
    mg_wait();   /* also where nothing is added: each grid of the chain has to wait somewhere */
    if (dirichlet) return;
    const double old = xf[i];
    double s = 0.0;
    if (D.kp[0] <= 2 && D.kp[1] <= 2 && D.kp[2] <= 2) {
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int c = 0; c < 2; c++)
                    s += w[0][a] * w[1][b] * w[2][c] *
                         xc[3 * (((long)j[0][a] * D.nbc[1] + j[1][b]) * D.nbc[2] + j[2][c]) + k];
    } else {
        for (int a = 0; a < D.kp[0]; a++) {
            const double wa = D.p_w[0][ix * D.kp[0] + a];
            const int ja = D.p_idx[0][ix * D.kp[0] + a];
            for (int b = 0; b < D.kp[1]; b++) {
                const double wab = wa * D.p_w[1][iy * D.kp[1] + b];
                const long jab = ((long)ja * D.nbc[1] + D.p_idx[1][iy * D.kp[1] + b]) * D.nbc[2];
                for (int c = 0; c < D.kp[2]; c++)
                    s += wab * D.p_w[2][iz * D.kp[2] + c] * xc[3 * (jab + D.p_idx[2][iz * D.kp[2] + c]) + k];
            }
        }
    }
    xf[i] = old + s;
}

/* b = r = P^T rf, zero on the Dirichlet rows, d = s dinv b (the coarse level's right-hand side and first direction) */
__global__ void __launch_bounds__(MG_THREADS) k_mg_restrict(mg_dirs_dev D, const double *rf,
                                                            const unsigned char *__restrict__ mask,
                                                            const double *__restrict__ dinv, double s, double *b,
                                                            double *r, double *d)
{
    const long nc = (long)D.nbc[0] * D.nbc[1] * D.nbc[2];
    const long j = (long)blockIdx.x * (MG_THREADS / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (j >= nc) return;   /* warp-uniform */
    const int jz = (int)(j % D.nbc[2]), jy = (int)((j / D.nbc[2]) % D.nbc[1]), jx = (int)(j / ((long)D.nbc[2] * D.nbc[1]));
    const long i = 3 * j + lane;
    const double di = lane < 3 ? dinv[i] : 0.0;
    const int dirichlet = lane < 3 ? mask[i] : 0;
    double v[3] = {0.0, 0.0, 0.0};
    bool waited = false;
    /* a lane takes every 32nd of the (a, e) pairs of fine lines, then a fixed shuffle tree */
    for (int p0 = 0; p0 < D.kr[0] * D.kr[1]; p0 += 32) {
        const int p = p0 + lane, a = p / D.kr[1], e = p - a * D.kr[1];
        const bool in = p < D.kr[0] * D.kr[1];
        const double wab = in ? D.r_w[0][jx * D.kr[0] + a] * D.r_w[1][jy * D.kr[1] + e] : 0.0;
        const long iab = in ? ((long)D.r_idx[0][jx * D.kr[0] + a] * D.nbf[1] + D.r_idx[1][jy * D.kr[1] + e]) * D.nbf[2] : 0;
        for (int c0 = 0; c0 < D.kr[2]; c0 += 4) {
            double w[4];
            int o[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const bool inc = c0 + c < D.kr[2];
                w[c] = inc ? wab * D.r_w[2][jz * D.kr[2] + c0 + c] : 0.0;
                o[c] = inc ? D.r_idx[2][jz * D.kr[2] + c0 + c] : -1;
            }
            if (!waited) mg_wait();   /* warp-uniform */
            waited = true;
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (in && o[c] >= 0) {
                    const double *u = rf + 3 * (iab + o[c]);
                    v[0] += w[c] * u[0];
                    v[1] += w[c] * u[1];
                    v[2] += w[c] * u[2];
                }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane >= 3) return;
    const double u = dirichlet ? 0.0 : (lane == 0 ? v[0] : (lane == 1 ? v[1] : v[2]));
    b[i] = u;
    r[i] = u;
    d[i] = s * di * u;
}

} /* namespace */

/* 1-D prolongation by knot insertion (Boehm, p = 2): the coarse knot vector kc (open)
 * refined by the knots `ins` (ascending, inside the open interval) into the fine one.
 * P[i][j] (nb_f x nb_c, row-major) maps coarse spline coefficients to fine ones. */
static void igab_mg_knot_prolongation(const std::vector<double> &kc, const std::vector<double> &ins,
                                      std::vector<double> &P, int &nbf, int &nbc)
{
    std::vector<double> kv = kc;
    nbc = (int)kc.size() - 3;
    std::vector<std::vector<double>> M(nbc, std::vector<double>(nbc, 0.0));
    for (int j = 0; j < nbc; j++) M[j][j] = 1.0;
    for (double t : ins) {
        const int nk = (int)kv.size(), nb = nk - 3;
        int k = 2;
        while (k + 1 < nk - 3 && !(kv[k] <= t && t < kv[k + 1])) k++;
        std::vector<std::vector<double>> Q(nb + 1, std::vector<double>(nbc, 0.0));
        for (int i = 0; i <= nb; i++) {
            if (i <= k - 2) Q[i] = M[i];
            else if (i >= k + 1) Q[i] = M[i - 1];
            else {
                const double a = (t - kv[i]) / (kv[i + 2] - kv[i]);
                for (int j = 0; j < nbc; j++) Q[i][j] = a * M[i][j] + (1.0 - a) * M[i - 1][j];
            }
        }
        M.swap(Q);
        kv.insert(kv.begin() + k + 1, t);
    }
    nbf = (int)M.size();
    P.assign((size_t)nbf * nbc, 0.0);
    for (int i = 0; i < nbf; i++)
        for (int j = 0; j < nbc; j++) P[(size_t)i * nbc + j] = M[i][j];
}

struct igab_mg {
    int nlev = 0;
    mg_level L[MG_MAX_LEVELS];
    long version = -1;
    bool direct = false;            /* coarsest level solved directly */
    bool dev_inv = false;           /* by the device inverse (else by the host LU) */
    int nd = 0;                     /* its size */
    std::vector<double> lu;
    std::vector<int> piv;
    double *h_vec = nullptr;        /* pinned nd doubles */
    double *inv = nullptr;          /* nd x nd inverse of the coarsest tangent (row-major) */
    double *gj = nullptr;           /* Gauss-Jordan pivot row and column buffers, 2 x 2 x nd */
    int *gj_flag = nullptr;         /* set by a pivot that is not positive and finite */
    double *part = nullptr, *dots = nullptr, *h_dots = nullptr;
    double *zero = nullptr;         /* zero state (fine size) */
    long zero_n = 0;
    void *fine_vals = nullptr;      /* the caller's tangent at the zero state, FP32 */
    double *kv = nullptr;           /* Krylov vectors of the caller's mesh */
    long kv_n = 0;
    double *mpart = nullptr;        /* multi-dot partial sums [GM_RESTART + 1][RD_BLOCKS] and results */
    double *h_md = nullptr;         /* pinned: the coefficients of a Gram-Schmidt step */
    cudaGraphExec_t vexec = nullptr;   /* the V-cycle from L[0].b, r, d to L[0].x */
    int vlaunches = 0;
    int launches = 0;
};

namespace {

int mg_free_level(mg_level &L, bool own)
{
    if (own && L.ctx) igab_destroy(L.ctx);
    cudaFree(L.own_vals);
    cudaFree(L.dinv);
    cudaFree(L.mask);
    cudaFree(L.x);
    for (int d = 0; d < 3; d++) {
        cudaFree(L.dir[d].p_idx);
        cudaFree(L.dir[d].p_w);
        cudaFree(L.dir[d].r_idx);
        cudaFree(L.dir[d].r_w);
    }
    L = mg_level();
    return 0;
}

void mg_free(igab_mg *m)
{
    if (!m) return;
    if (m->vexec) cudaGraphExecDestroy(m->vexec);
    for (int l = 0; l < m->nlev; l++) mg_free_level(m->L[l], l > 0);
    cudaFree(m->part);
    cudaFree(m->zero);
    cudaFree(m->fine_vals);
    cudaFree(m->kv);
    cudaFree(m->mpart);
    cudaFreeHost(m->h_md);
    cudaFreeHost(m->h_vec);
    cudaFree(m->inv);
    cudaFree(m->gj);
    cudaFree(m->gj_flag);
    cudaFreeHost(m->h_dots);
    delete m;
}

int mg_vectors(mg_level &L)
{
    const size_t bytes = (size_t)L.n * sizeof(double);
    IGAB_CUDA_TRY(cudaMalloc((void **)&L.x, 5 * bytes));
    L.b = L.x + L.n;
    L.r = L.b + L.n;
    L.d = L.r + L.n;
    L.t = L.d + L.n;
    IGAB_CUDA_TRY(cudaMalloc((void **)&L.dinv, bytes));
    IGAB_CUDA_TRY(cudaMalloc((void **)&L.mask, (size_t)L.n));
    return 0;
}

/* mask = 1 on the level's Dirichlet rows */
int mg_mask(mg_level &L, cudaStream_t st)
{
    IGAB_CUDA_TRY(cudaMemsetAsync(L.mask, 0, (size_t)L.n, st));
    if (L.ctx->nd > 0)
        k_mg_mask<<<(unsigned)((L.ctx->nd + 255) / 256), 256, 0, st>>>(L.ctx->nd, L.ctx->d_drow, L.mask);
    IGAB_CUDA_TRY(cudaGetLastError());
    return 0;
}

int mg_upload_dir(mg_dir &D, const std::vector<double> &P, int nbf, int nbc)
{
    std::vector<std::vector<std::pair<int, double>>> rows(nbf), cols(nbc);
    for (int i = 0; i < nbf; i++)
        for (int j = 0; j < nbc; j++) {
            const double w = P[(size_t)i * nbc + j];
            if (w != 0.0) {
                rows[i].push_back({j, w});
                cols[j].push_back({i, w});
            }
        }
    int kp = 1, kr = 1;
    for (auto &r : rows) kp = std::max(kp, (int)r.size());
    for (auto &c : cols) kr = std::max(kr, (int)c.size());
    std::vector<int> pi((size_t)nbf * kp, 0), ri((size_t)nbc * kr, 0);
    std::vector<double> pw((size_t)nbf * kp, 0.0), rw((size_t)nbc * kr, 0.0);
    for (int i = 0; i < nbf; i++)
        for (size_t a = 0; a < rows[i].size(); a++) {
            pi[(size_t)i * kp + a] = rows[i][a].first;
            pw[(size_t)i * kp + a] = rows[i][a].second;
        }
    for (int j = 0; j < nbc; j++)
        for (size_t b = 0; b < cols[j].size(); b++) {
            ri[(size_t)j * kr + b] = cols[j][b].first;
            rw[(size_t)j * kr + b] = cols[j][b].second;
        }
    D.nf = nbf;
    D.nc = nbc;
    D.kp = kp;
    D.kr = kr;
    IGAB_CUDA_TRY(cudaMalloc((void **)&D.p_idx, pi.size() * sizeof(int)));
    IGAB_CUDA_TRY(cudaMalloc((void **)&D.p_w, pw.size() * sizeof(double)));
    IGAB_CUDA_TRY(cudaMalloc((void **)&D.r_idx, ri.size() * sizeof(int)));
    IGAB_CUDA_TRY(cudaMalloc((void **)&D.r_w, rw.size() * sizeof(double)));
    IGAB_CUDA_TRY(cudaMemcpy(D.p_idx, pi.data(), pi.size() * sizeof(int), cudaMemcpyHostToDevice));
    IGAB_CUDA_TRY(cudaMemcpy(D.p_w, pw.data(), pw.size() * sizeof(double), cudaMemcpyHostToDevice));
    IGAB_CUDA_TRY(cudaMemcpy(D.r_idx, ri.data(), ri.size() * sizeof(int), cudaMemcpyHostToDevice));
    IGAB_CUDA_TRY(cudaMemcpy(D.r_w, rw.data(), rw.size() * sizeof(double), cudaMemcpyHostToDevice));
    return 0;
}

mg_dirs_dev dirs_view(const mg_level &C)
{
    mg_dirs_dev D;
    for (int d = 0; d < 3; d++) {
        D.p_idx[d] = C.dir[d].p_idx;
        D.p_w[d] = C.dir[d].p_w;
        D.r_idx[d] = C.dir[d].r_idx;
        D.r_w[d] = C.dir[d].r_w;
        D.kp[d] = C.dir[d].kp;
        D.kr[d] = C.dir[d].kr;
        D.nbf[d] = C.dir[d].nf;
        D.nbc[d] = C.dir[d].nc;
    }
    return D;
}

/* dense LU with partial pivoting (column-major n x n in a), in place */
bool lu_factor(int n, std::vector<double> &a, std::vector<int> &piv)
{
    piv.resize(n);
    for (int k = 0; k < n; k++) {
        int p = k;
        double mx = std::fabs(a[(size_t)k * n + k]);
        for (int i = k + 1; i < n; i++)
            if (std::fabs(a[(size_t)k * n + i]) > mx) { mx = std::fabs(a[(size_t)k * n + i]); p = i; }
        if (mx == 0.0) return false;
        piv[k] = p;
        if (p != k)
            for (int j = 0; j < n; j++) std::swap(a[(size_t)j * n + k], a[(size_t)j * n + p]);
        const double inv = 1.0 / a[(size_t)k * n + k];
        for (int i = k + 1; i < n; i++) a[(size_t)k * n + i] *= inv;
        for (int j = k + 1; j < n; j++) {
            const double akj = a[(size_t)j * n + k];
            if (akj != 0.0)
                for (int i = k + 1; i < n; i++) a[(size_t)j * n + i] -= a[(size_t)k * n + i] * akj;
        }
    }
    return true;
}

void lu_solve(int n, const std::vector<double> &a, const std::vector<int> &piv, double *x)
{
    for (int k = 0; k < n; k++) std::swap(x[k], x[piv[k]]);
    for (int j = 0; j < n; j++)
        for (int i = j + 1; i < n; i++) x[i] -= a[(size_t)j * n + i] * x[j];
    for (int j = n - 1; j >= 0; j--) {
        x[j] /= a[(size_t)j * n + j];
        for (int i = 0; i < j; i++) x[i] -= a[(size_t)j * n + i] * x[j];
    }
}

int spmv(igab_mg *m, mg_level &L, const double *x, double *y)
{
    const int rc = igab_launch_spmv(L.ctx, L.vals, L.prec, x, y);
    m->launches++;
    return rc;
}

/* lmax of D^-1 K by power iteration from a fixed start vector.  The smoother amplifies what lies above 1.01 times its
 * interval, steeply so at its degree, and a V-cycle that does is not positive definite: CG then breaks down.  So the
 * estimate has to be within the 10% that the interval adds.  Over 48 meshes (4 to 64 elements a side, even, graded,
 * stretched, uneven materials) 12 iterations fell short by up to 12.8%, 24 by 6.0%, 40 by 3.5%, 80 by 2.0%.  Both norms
 * are read after every tenth iteration only (lmax^10 is far from the range's end): four reads, where 12 iterations with
 * a read each took longer at 16^3; a large mesh pays for the products, once per material. */
int estimate_lmax(igab_mg *m, mg_level &L)
{
    cudaStream_t st = L.ctx->stream;
    const long n = L.n;
    std::vector<double> v0((size_t)n);
    unsigned s = 12345u;
    for (long i = 0; i < n; i++) {
        s = s * 1664525u + 1013904223u;
        v0[(size_t)i] = 0.5 + (double)(s >> 8) / (double)(1u << 24);
    }
    IGAB_CUDA_TRY(cudaMemcpyAsync(L.d, v0.data(), (size_t)n * sizeof(double), cudaMemcpyHostToDevice, st));
    double lam = 0.0, dd[2];
    for (int it = 0; it < MG_POWER_ITERS; it++) {
        int rc = spmv(m, L, L.d, L.t);
        if (rc) return rc;
        if ((it + 1) % MG_POWER_NORM) {
            k_mg_jac<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, L.dinv, L.t, 1.0, L.d);
            m->launches++;
            continue;
        }
        k_mg_jac<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, L.dinv, L.t, 1.0, L.r);   /* r = D^-1 K d */
        IGAB_CUDA_TRY(rd_dot2(st, n, L.r, L.r, L.d, L.d, m->part, m->dots, m->h_dots, dd));
        const double nr = std::sqrt(dd[0]);
        lam = dd[1] > 0.0 ? nr / std::sqrt(dd[1]) : 0.0;
        if (nr == 0.0) break;
        k_mg_axpby<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, 1.0 / nr, L.r, 0.0, L.d);   /* d = r / ||r|| */
        m->launches += 4;
    }
    static_assert(MG_POWER_ITERS % MG_POWER_NORM == 0, "the last iteration reads the norms");
    L.lmax = lam > 0.0 ? lam : 1.0;
    return 0;
}

/* The interval is wide and the degree high, as the operator is of fourth order: an error of half the coarse mesh's
 * resolution has 2^-4 or less of lmax, and the rediscretised coarse operator corrects the modes near that poorly.
 * GMRES of three Newton steps at 8^3 / 16^3 / 32^3 (ms; iterations at 16^3; lmax of 12 power iterations, 4% lower than
 * now at 16^3): degree 3, ratio 10: 4.6 / 13.8 / 95.2
 * (108); degree 3, ratio 30: 16^3 11.7, 32^3 79.7 (91); degree 4, 30: 11.0, 78.6 (73); degree 6: ratio 40 10.4, 80.2,
 * 80 2.8 / 9.3 / 70.7 (47), 120 3.3 / 8.7 / 68.2 (44), 200 4.1 / 8.9 / 64.6; degree 8: ratio 100 2.8 / 8.7 / 71.7 (35),
 * 200 3.7 / 8.6 / 65.1; degree 10, 200: 3.5 / 8.8 / 67.4; degree 2, 10: 15.0, 92.2 (140).
 * The Chebyshev recurrence on [1.1 lmax / ratio, 1.1 lmax]: the first direction is dinv r / theta, step i makes the next one
 * a d + c dinv r */
struct mg_cheb {
    double theta, a[MG_DEGREE], c[MG_DEGREE];
    explicit mg_cheb(double lmax)
    {
        const double hi = 1.1 * lmax, lo = hi / MG_RATIO, delta = 0.5 * (hi - lo);
        theta = 0.5 * (hi + lo);
        const double sigma = theta / delta;
        double rho = 1.0 / sigma;
        for (int i = 0; i < MG_DEGREE; i++) {
            const double rn = 1.0 / (2.0 * sigma - rho);
            a[i] = rn * rho;
            c[i] = 2.0 * rn / delta;
            rho = rn;
        }
    }
};

template <int OP>
void mg_spmv(igab_mg *m, mg_level &L, cudaStream_t st, const double *in, double a, double c, int first, double *dn)
{
    const unsigned nblk = (unsigned)((L.n / 3 + MG_SPMV / 32 - 1) / (MG_SPMV / 32));
    const igab_geom g = L.ctx->geom();
    const auto go = [&](auto *vals, auto all) {
        using T = std::remove_const_t<std::remove_pointer_t<decltype(vals)>>;
        mg_launch(k_mg_spmv<T, OP, decltype(all)::value>, nblk, MG_SPMV, st, g, vals, in, L.b, L.dinv, L.mask, a, c, first,
                  L.x, L.r, dn);
    };
    /* up to about two waves of blocks (148 SMs x 16 warps) the rows are loaded whole under the kernel before; beyond,
     * the registers that takes cost more than the wait: 1,000 points (8^3) 4.7 against 5.2 us, the 2,744 of 12^3 within
     * a 24^3 solve 39.3 against 40.8 ms, but 5,832 (16^3) 15.5 against 13.7 ms and 32^3 120 against 95 ms a solve */
    const bool all = L.n / 3 <= MG_ALL;
    if (L.prec == IGAB_PREC_FP64) {
        if (all) go((const double *)L.vals, std::true_type());
        else go((const double *)L.vals, std::false_type());
    } else {
        if (all) go((const float *)L.vals, std::true_type());
        else go((const float *)L.vals, std::false_type());
    }
    m->launches++;
}

/* A (row-major n x n) from the structured CSR of the coarsest level: one thread per row */
__global__ void k_mg_dense(int n, const int *__restrict__ rowptr, const int *__restrict__ cols,
                           const double *__restrict__ vals, double *__restrict__ A)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    for (int k = rowptr[r]; k < rowptr[r + 1]; k++) A[(size_t)r * n + cols[k]] = vals[k];
}

/* pivot row and column 0 into the step buffers */
__global__ void k_mg_gj_init(int n, const double *__restrict__ A, double *__restrict__ row, double *__restrict__ col)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    row[i] = A[i];
    col[i] = A[(size_t)i * n];
}

/* Gauss-Jordan step k in place (row-major A), from the old pivot row / column (row, col);
 * writes row / column k + 1 of the result into (nrow, ncol) for the next step.  Each
 * entry is computed by one thread from the old values only. */
__global__ void k_mg_gj_step(int n, int k, double *A, const double *row,
                             const double *col, double *nrow, double *ncol, int *flag)
{
    mg_wait();
    const int t = blockIdx.x * MG_THREADS + threadIdx.x, i = t / n, j = t - i * n;   /* n <= MG_COARSE_DOF */
    if (i >= n) return;
    const double p = col[k];
    if (i == k && j == k && !(p > 0.0 && isfinite(p))) *flag = 1;
    const double ip = 1.0 / p;
    double v;
    if (i == k) v = j == k ? ip : row[j] * ip;
    else if (j == k) v = -col[i] * ip;
    else v = A[(size_t)i * n + j] - col[i] * (row[j] * ip);
    A[(size_t)i * n + j] = v;
    if (i == k + 1) nrow[j] = v;
    if (j == k + 1) ncol[i] = v;
}

/* x = Ainv b: one warp per row (the first 24 x 32 of its entries before the wait), lane-strided partial sums then a
 * fixed shuffle tree */
__global__ void __launch_bounds__(128) k_mg_gemv(long n, const double *__restrict__ Ai, const double *b, double *x)
{
    const long r = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    const double *row = Ai + r * n;
    double w[24], s = 0.0;
#pragma unroll
    for (int c = 0; c < 24; c++) w[c] = 32 * c + lane < n ? row[32 * c + lane] : 0.0;
    mg_wait();
    double v[24];
#pragma unroll
    for (int c = 0; c < 24; c++) v[c] = 32 * c + lane < n ? b[32 * c + lane] : 0.0;
#pragma unroll
    for (int c = 0; c < 24; c++) s += w[c] * v[c];
    for (long j = 768 + lane; j < n; j += 32) s += row[j] * b[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) x[r] = s;
}

/* x_l = V-cycle approximation of K_l^-1 b_l; b, r = b and the first direction d in the level's vectors */
int vcycle(igab_mg *m, int l, cudaStream_t st)
{
    static_assert(MG_DEGREE >= 2, "the last step after the correction is folded into the one before");
    mg_level &L = m->L[l];
    if (l == m->nlev - 1) {
        if (m->direct && m->dev_inv) {
            mg_launch(k_mg_gemv, (unsigned)((L.n + 3) / 4), 128, st, L.n, m->inv, L.b, L.x);
            m->launches++;
        } else if (m->direct) {
            IGAB_CUDA_TRY(cudaMemcpyAsync(m->h_vec, L.b, (size_t)L.n * sizeof(double), cudaMemcpyDeviceToHost, st));
            IGAB_CUDA_TRY(cudaStreamSynchronize(st));
            lu_solve(m->nd, m->lu, m->piv, m->h_vec);
            IGAB_CUDA_TRY(cudaMemcpyAsync(L.x, m->h_vec, (size_t)L.n * sizeof(double), cudaMemcpyHostToDevice, st));
        } else {
            k_mg_jac<<<MG_BLOCKS, MG_THREADS, 0, st>>>(L.n, L.dinv, L.b, 1.0, L.x);
            m->launches++;
        }
        IGAB_CUDA_TRY(cudaGetLastError());
        return 0;
    }
    mg_level &C = m->L[l + 1];
    const mg_cheb p(L.lmax);
    double *d = L.d, *dn = L.t;
    for (int i = 0; i + 1 < MG_DEGREE; i++) {
        mg_spmv<MG_STEP>(m, L, st, d, p.a[i], p.c[i], i == 0, dn);
        std::swap(d, dn);
    }
    mg_spmv<MG_LAST_PRE>(m, L, st, d, 0.0, 0.0, 0, dn);
    /* coarse correction with the Dirichlet rows of both levels masked (symmetric; a coarse x is zero on them, as its
     * right-hand side is and the operators have unit rows and columns there) */
    const mg_dirs_dev D = dirs_view(C);
    mg_launch(k_mg_restrict, (unsigned)((C.n / 3 + MG_THREADS / 32 - 1) / (MG_THREADS / 32)), MG_THREADS, st, D, L.r, C.mask,
              C.dinv, 1.0 / mg_cheb(C.lmax).theta, C.b, C.r, C.d);
    m->launches++;
    int rc = vcycle(m, l + 1, st);
    if (rc) return rc;
    mg_launch(k_mg_prolong, (unsigned)((L.n + MG_THREADS - 1) / MG_THREADS), MG_THREADS, st, D, C.x, L.mask, L.x);
    m->launches++;
    /* r = b - K x, then the same smoother again */
    d = L.d;
    dn = L.t;
    mg_spmv<MG_RESID>(m, L, st, L.x, 1.0 / p.theta, 0.0, 0, d);
    for (int i = 0; i + 2 < MG_DEGREE; i++) {
        mg_spmv<MG_STEP>(m, L, st, d, p.a[i], p.c[i], 0, dn);
        std::swap(d, dn);
    }
    mg_spmv<MG_LAST_POST>(m, L, st, d, p.a[MG_DEGREE - 2], p.c[MG_DEGREE - 2], 0, dn);
    IGAB_CUDA_TRY(cudaGetLastError());
    return 0;
}

/* the coarse levels for the context's current parameters */
int mg_build(igab_ctx *c, igab_mg *m)
{
    if (m->vexec) {
        cudaGraphExecDestroy(m->vexec);
        m->vexec = nullptr;
    }
    for (int l = 1; l < m->nlev; l++) mg_free_level(m->L[l], true);
    m->nlev = 1;
    m->direct = false;
    mg_level &F = m->L[0];
    F.ctx = c;
    F.n = c->ndof;
    if (!F.x) {
        int rc = mg_vectors(F);
        if (rc) return rc;
    }
    /* the preconditioner's fine operator: the caller's tangent at the zero state (FP32),
     * symmetric positive definite for a stable material whatever the current state is */
    if (!m->zero || m->zero_n < F.n) {
        cudaFree(m->zero);
        m->zero = nullptr;
        IGAB_CUDA_TRY(cudaMalloc((void **)&m->zero, (size_t)F.n * sizeof(double)));
        IGAB_CUDA_TRY(cudaMemset(m->zero, 0, (size_t)F.n * sizeof(double)));
        m->zero_n = F.n;
    }
    if (!m->fine_vals) IGAB_CUDA_TRY(cudaMalloc(&m->fine_vals, (size_t)c->nnz * sizeof(float)));
    {
        int rc = igab_launch_tangent(c, m->zero, m->fine_vals, IGAB_PREC_FP32);
        if (rc) return rc;
    }
    F.vals = m->fine_vals;
    F.prec = IGAB_PREC_FP32;
    {
        int rc = mg_mask(F, c->stream);
        if (rc) return rc;
    }
    k_mg_diag_inv<<<(unsigned)((F.n + 255) / 256), 256, 0, c->stream>>>(c->geom(), F.vals, F.prec, F.dinv);
    IGAB_CUDA_TRY(cudaGetLastError());
    {
        int rc = estimate_lmax(m, F);
        if (rc) return rc;
    }
    /* element log-scales of the caller's context (averaged per coarse element below) */
    std::vector<double> s_f;
    if (c->escale_on) {
        s_f.resize((size_t)c->nel);
        IGAB_CUDA_TRY(cudaMemcpy(s_f.data(), c->d_escale, (size_t)c->nel * sizeof(double), cudaMemcpyDeviceToHost));
    }
    while (m->nlev < MG_MAX_LEVELS) {
        igab_ctx *f = m->L[m->nlev - 1].ctx;
        if (f->ndof <= MG_COARSE_DOF) break;
        bool ok = true;
        for (int d = 0; d < 3; d++) ok = ok && f->ne[d] % 2 == 0 && f->ne[d] >= 4;
        if (!ok) break;
        igab_mesh_desc desc;
        memset(&desc, 0, sizeof(desc));
        desc.phys = f->phys;
        std::vector<double> kn;
        std::vector<double> knc[3], ins[3];
        for (int d = 0; d < 3; d++) {
            const std::vector<double> &kf = f->knots[d];
            const int n = f->ne[d];
            desc.nelem[d] = n / 2;
            knc[d].assign(kf.begin(), kf.begin() + 3);
            for (int i = 1; i < n; i++) {   /* interior knot i sits at kf[2 + i] */
                if (i % 2 == 0) knc[d].push_back(kf[2 + i]);
                else ins[d].push_back(kf[2 + i]);
            }
            knc[d].insert(knc[d].end(), kf.end() - 3, kf.end());
            kn.insert(kn.end(), knc[d].begin(), knc[d].end());
        }
        desc.knots = kn.data();
        memcpy(desc.par_mat, f->par_mat, sizeof(desc.par_mat));
        memcpy(desc.bc_type, f->bc_type, sizeof(desc.bc_type));
        memcpy(desc.par_periodic, f->par_periodic, sizeof(desc.par_periodic));
        memcpy(desc.par_dirichlet, f->par_dirichlet, sizeof(desc.par_dirichlet));
        igab_ctx *cc = nullptr;
        int rc = igab_create(&desc, f->device, &cc);
        if (rc) return rc;
        mg_level &C = m->L[m->nlev];
        C.ctx = cc;
        m->nlev++;
        if ((rc = igab_set_stream(cc, c->stream))) return rc;
        C.n = cc->ndof;
        C.prec = IGAB_PREC_FP64;
        for (int d = 0; d < 3; d++) {
            std::vector<double> P;
            int nbf = 0, nbc = 0;
            igab_mg_knot_prolongation(knc[d], ins[d], P, nbf, nbc);
            if (nbf != f->nb[d] || nbc != cc->nb[d]) {
                igab_set_error("multigrid: prolongation size %d x %d, expected %d x %d", nbf, nbc, f->nb[d], cc->nb[d]);
                return IGAB_ERR_ARG;
            }
            if ((rc = mg_upload_dir(C.dir[d], P, nbf, nbc))) return rc;
        }
        if ((rc = mg_vectors(C))) return rc;
        if ((rc = mg_mask(C, c->stream))) return rc;
        /* element scales: the mean of the eight fine elements of each coarse element */
        if (!s_f.empty()) {
            const int *nf = f->ne, *nc = cc->ne;
            std::vector<double> gc((size_t)cc->nel);
            for (int ex = 0; ex < nc[0]; ex++)
                for (int ey = 0; ey < nc[1]; ey++)
                    for (int ez = 0; ez < nc[2]; ez++) {
                        double sum = 0.0;
                        for (int k = 0; k < 8; k++) {
                            const long fe = ((long)(2 * ex + (k >> 2)) * nf[1] + 2 * ey + ((k >> 1) & 1)) * nf[2] +
                                            2 * ez + (k & 1);
                            sum += s_f[(size_t)fe];
                        }
                        gc[((size_t)ex * nc[1] + ey) * nc[2] + ez] = std::log(sum / 8.0);
                    }
            std::vector<double> sc((size_t)cc->nel);
            for (size_t e = 0; e < sc.size(); e++) sc[e] = std::exp(gc[e]);
            s_f.swap(sc);
            if ((rc = igab_set_element_log_scale(cc, gc.data(), 0))) return rc;
        }
        /* the coarse tangent at the zero state (m->zero holds the fine level's zeros) */
        IGAB_CUDA_TRY(cudaMalloc((void **)&C.own_vals, (size_t)cc->nnz * sizeof(double)));
        if ((rc = igab_launch_tangent(cc, m->zero, C.own_vals, IGAB_PREC_FP64))) return rc;
        C.vals = C.own_vals;
        k_mg_diag_inv<<<(unsigned)((C.n + 255) / 256), 256, 0, c->stream>>>(cc->geom(), C.vals, C.prec, C.dinv);
        IGAB_CUDA_TRY(cudaGetLastError());
        if ((rc = estimate_lmax(m, C))) return rc;
        igab_scratch_free(cc);   /* one assembly per build (the estimate has waited for it) */
    }
    /* the coarsest level directly, when small: the device inverse */
    mg_level &B = m->L[m->nlev - 1];
    m->dev_inv = false;
    if (m->nlev > 1 && B.n <= MG_COARSE_DOF) {
        igab_ctx *cc = B.ctx;
        const int n = (int)B.n;
        cudaFree(m->inv);
        cudaFree(m->gj);
        m->inv = nullptr;
        m->gj = nullptr;
        IGAB_CUDA_TRY(cudaMalloc((void **)&m->inv, (size_t)n * n * sizeof(double)));
        IGAB_CUDA_TRY(cudaMalloc((void **)&m->gj, (size_t)4 * n * sizeof(double)));
        if (!m->gj_flag) IGAB_CUDA_TRY(cudaMalloc((void **)&m->gj_flag, sizeof(int)));
        int *dcols = nullptr;
        IGAB_CUDA_TRY(cudaMalloc((void **)&dcols, (size_t)cc->nnz * sizeof(int)));
        int rc = igab_launch_csr_cols(cc, dcols);
        if (!rc) {
            cudaStream_t st = c->stream;
            cudaError_t e = cudaMemsetAsync(m->inv, 0, (size_t)n * n * sizeof(double), st);
            if (e == cudaSuccess) e = cudaMemsetAsync(m->gj_flag, 0, sizeof(int), st);
            if (e == cudaSuccess) {
                k_mg_dense<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, cc->d_rowptr, dcols, B.own_vals, m->inv);
                k_mg_gj_init<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, m->inv, m->gj, m->gj + n);
                const unsigned blocks = (unsigned)(((long)n * n + MG_THREADS - 1) / MG_THREADS);
                for (int k = 0; k < n; k++) {
                    double *rk = m->gj + (size_t)(k & 1) * 2 * n, *nx = m->gj + (size_t)((k + 1) & 1) * 2 * n;
                    mg_launch(k_mg_gj_step, blocks, MG_THREADS, st, n, k, m->inv, rk, rk + n, nx, nx + n, m->gj_flag);
                }
                e = cudaGetLastError();
            }
            int flag = 1;
            if (e == cudaSuccess) e = cudaMemcpyAsync(&flag, m->gj_flag, sizeof(int), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) {
                igab_set_error("multigrid coarse inverse: %s", cudaGetErrorString(e));
                rc = IGAB_ERR_CUDA;
            } else if (!flag) {
                m->dev_inv = true;
            }
        }
        cudaFree(dcols);
        if (rc) return rc;
    }
    if (m->nlev > 1 && B.n <= MG_COARSE_DOF && m->dev_inv) {
        m->direct = true;
        m->nd = (int)B.n;
    } else if (m->nlev > 1 && B.n <= MG_COARSE_DOF) {   /* not positive definite: host LU */
        igab_ctx *cc = B.ctx;
        const int n = (int)B.n;
        std::vector<int> cols((size_t)cc->nnz);
        int rc = igab_csr_pattern(cc, nullptr, cols.data());
        if (rc) return rc;
        std::vector<double> v((size_t)cc->nnz);
        IGAB_CUDA_TRY(cudaStreamSynchronize(c->stream));
        IGAB_CUDA_TRY(cudaMemcpy(v.data(), B.vals, (size_t)cc->nnz * sizeof(double), cudaMemcpyDeviceToHost));
        m->lu.assign((size_t)n * n, 0.0);
        for (int r = 0; r < n; r++)
            for (int k = cc->rowptr_h[r]; k < cc->rowptr_h[r + 1]; k++) m->lu[(size_t)cols[k] * n + r] = v[k];
        if (!lu_factor(n, m->lu, m->piv)) {
            igab_set_error("multigrid: the coarsest tangent is singular");
            return IGAB_ERR_NONFINITE;
        }
        m->direct = true;
        m->nd = n;
        cudaFreeHost(m->h_vec);
        m->h_vec = nullptr;
        IGAB_CUDA_TRY(cudaMallocHost((void **)&m->h_vec, (size_t)n * sizeof(double)));
    }
    m->version = c->param_version;
    return 0;
}

} /* namespace */

void igab_mg_release(igab_ctx *c)
{
    mg_free(c->mg);
    c->mg = nullptr;
}

int igab_mg_levels(igab_ctx *c, int *levels)
{
    *levels = c->mg ? c->mg->nlev : 0;
    return 0;
}


namespace {

/* partial sums of V_i . w for the four i from 4 blockIdx.y (V_i = V + i n, i < k), per block into part[i][RD_BLOCKS] */
__global__ void __launch_bounds__(RD_THREADS) k_md_partial(long n, const double *V, int k, const double *w, double *part)
{
    __shared__ double red[4][RD_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i0 = 4 * blockIdx.y;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    mg_wait();
    MG_LOOP(t, n)
    {
        const double x = w[t];
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (i0 + i < k) s[i] += V[(size_t)(i0 + i) * n + t] * x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
    if (lane < 4) red[lane][warp] = lane == 0 ? s[0] : (lane == 1 ? s[1] : (lane == 2 ? s[2] : s[3]));
    __syncthreads();
    if (threadIdx.x < 4 && i0 + threadIdx.x < k) {
        double q = 0.0;
#pragma unroll
        for (int e = 0; e < RD_THREADS / 32; e++) q += red[threadIdx.x][e];
        part[(size_t)(i0 + threadIdx.x) * RD_BLOCKS + blockIdx.x] = q;
    }
}

/* the sum of part[0..nb) in a fixed order, in every thread of the block (nb <= RD_BLOCKS <= 2 RD_THREADS) */
__device__ __forceinline__ double md_sum(const double *part, int nb)
{
    __shared__ double red[RD_THREADS / 32];
    const int t = threadIdx.x;
    double s = t < nb ? part[t] : 0.0;
    if (t + RD_THREADS < nb) s += part[t + RD_THREADS];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((t & 31) == 0) red[t >> 5] = s;
    __syncthreads();
    double q = 0.0;
#pragma unroll
    for (int e = 0; e < RD_THREADS / 32; e++) q += red[e];
    return q;
}
static_assert(RD_BLOCKS <= 2 * RD_THREADS, "two partial sums per thread");

/* out[i] = sum of part[i][0..nb), one block per i */
__global__ void __launch_bounds__(RD_THREADS) k_md_finish(const double *part, int nb, double *out)
{
    mg_wait();
    const double q = md_sum(part + (size_t)blockIdx.x * RD_BLOCKS, nb);
    if (threadIdx.x == 0) out[blockIdx.x] = q;
}

/* w -= sum_{i<k} h_i V_i (h on the device); with part: the blocks' partial sums of w . w */
__global__ void __launch_bounds__(RD_THREADS) k_md_update(long n, const double *V, int k, const double *h, double *w,
                                                          double *part)
{
    __shared__ double red[RD_THREADS / 32];
    double q = 0.0;
    mg_wait();
    MG_LOOP(t, n)
    {
        double s = w[t];
#pragma unroll 8
        for (int i = 0; i < k; i++) s -= h[i] * V[(size_t)i * n + t];
        w[t] = s;
        q += s * s;
    }
    if (!part) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = q;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < RD_THREADS / 32; i++) s += red[i];
        part[blockIdx.x] = s;
    }
}

/* *nn = w . w from the nb partial sums (every block adds them up in the same order), v = w / ||w|| */
__global__ void __launch_bounds__(RD_THREADS) k_md_scale(long n, const double *w, const double *part, int nb, double *nn,
                                                         double *v)
{
    mg_wait();
    const double q = md_sum(part, nb);
    if (blockIdx.x == 0 && threadIdx.x == 0) *nn = q;
    const double inv = q > 0.0 ? 1.0 / sqrt(q) : 0.0;
    MG_LOOP(t, n) v[t] = inv * w[t];
}

/* u = sum_{i<k} y_i V_i  (y on the device) */
__global__ void k_md_combine(long n, const double *__restrict__ V, int k, const double *__restrict__ y, double *u)
{
    MG_LOOP(t, n)
    {
        double s = 0.0;
        for (int i = 0; i < k; i++) s += y[i] * V[(size_t)i * n + t];
        u[t] = s;
    }
}

/* the blocks of a vector kernel: no more than the vector fills */
int md_blocks(long n) { return (int)std::min<long>(RD_BLOCKS, (n + RD_THREADS - 1) / RD_THREADS); }

/* out = V[0..k)^T w, on the device */
void mdot(igab_mg *m, cudaStream_t st, long n, const double *V, int k, const double *w, double *out)
{
    const int nb = md_blocks(n);
    mg_launch(k_md_partial, dim3((unsigned)nb, (unsigned)((k + 3) / 4)), RD_THREADS, st, n, V, k, w, m->mpart);
    mg_launch(k_md_finish, (unsigned)k, RD_THREADS, st, m->mpart, nb, out);
    m->launches += 2;
}

/* the V-cycle as the preconditioner: L[0].x = M r.  Its kernels are replayed from a graph, captured after each build of
 * the hierarchy (not with the host LU, which reads and writes in between, nor on the legacy stream, which cannot be
 * captured). */
int precond(igab_mg *m, const double *r)
{
    mg_level &F = m->L[0];
    cudaStream_t st = F.ctx->stream;
    k_mg_start<<<MG_BLOCKS, MG_THREADS, 0, st>>>(F.n, r, F.dinv, 1.0 / mg_cheb(F.lmax).theta, F.b, F.r, F.d);
    m->launches++;
    if ((m->direct && !m->dev_inv) || st == cudaStreamLegacy) return vcycle(m, 0, st);
    if (!m->vexec) {
        const int l0 = m->launches;
        cudaGraph_t gr = nullptr;
        IGAB_CUDA_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        const int rc = vcycle(m, 0, st);
        cudaError_t e = cudaStreamEndCapture(st, &gr);
        if (!rc && e == cudaSuccess) e = cudaGraphInstantiate(&m->vexec, gr, 0);
        if (gr) cudaGraphDestroy(gr);
        if (rc) return rc;
        IGAB_CUDA_TRY(e);
        m->vlaunches = m->launches - l0;
        m->launches = l0;
    }
    IGAB_CUDA_TRY(cudaGraphLaunch(m->vexec, st));
    m->launches += m->vlaunches;
    return 0;
}

int dot1(igab_mg *m, cudaStream_t st, long n, const double *a, const double *b, double *out)
{
    double d2[2];
    IGAB_CUDA_TRY(rd_dot2(st, n, a, b, nullptr, nullptr, m->part, m->dots, m->h_dots, d2));
    *out = d2[0];
    return 0;
}

/* preconditioned CG on K (vals, prec); breakdown when p.Kp <= 0 */
int solve_cg(igab_mg *m, igab_ctx *c, const void *vals, int prec, const double *b, double *x, double tol, int maxit,
             int *iterations, int *converged, double *rnorm, int *breakdown)
{
    cudaStream_t st = c->stream;
    const long n = c->ndof;
    double *r = m->kv, *z = m->L[0].x, *p = r + n, *q = p + n;
    int rc = 0;
    k_mg_copy<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, b, r);
    if ((rc = precond(m, r))) return rc;
    k_mg_copy<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, z, p);
    double rz = 0.0;
    if ((rc = dot1(m, st, n, r, z, &rz))) return rc;
    for (int it = 1; it <= maxit; it++) {
        if ((rc = igab_launch_spmv(c, vals, prec, p, q))) return rc;
        double pq = 0.0, rr = 0.0;
        if ((rc = dot1(m, st, n, p, q, &pq))) return rc;
        if (!(pq > 0.0) || !(rz > 0.0)) {
            *breakdown = 1;
            return 0;
        }
        const double alpha = rz / pq;
        k_mg_axpby<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, alpha, p, 1.0, x);
        k_mg_axpby<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, -alpha, q, 1.0, r);
        if ((rc = dot1(m, st, n, r, r, &rr))) return rc;
        *iterations = it;
        *rnorm = std::sqrt(rr);
        if (*rnorm <= tol) {
            *converged = 1;
            return 0;
        }
        if ((rc = precond(m, r))) return rc;
        double rz1 = 0.0;
        if ((rc = dot1(m, st, n, r, z, &rz1))) return rc;
        k_mg_axpby<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, 1.0, z, rz1 / rz, p);
        rz = rz1;
        m->launches += 4;
    }
    return 0;
}

/* right-preconditioned GMRES(GM_RESTART) on K with the V-cycle M: x = M u, u in the
 * Krylov space of K M; classical Gram-Schmidt with one reorthogonalisation (CGS2), Givens
 * rotations; the true residual is recomputed at every restart */
int solve_gmres(igab_mg *m, igab_ctx *c, const void *vals, int prec, const double *b, double *x, double tol,
                int maxit, int *iterations, int *converged, double *rnorm)
{
    cudaStream_t st = c->stream;
    const long n = c->ndof;
    const int mr = GM_RESTART, nb = md_blocks(n);
    double *V = m->kv, *w = V + (size_t)(mr + 1) * n, *r = w + n;
    const double *t = m->L[0].x;   /* the preconditioner's result */
    /* device: h of the first and of the second projection, ||w||^2; h_md receives the three */
    double *dev_h = m->mpart + (size_t)(GM_RESTART + 1) * RD_BLOCKS, *dev_h2 = dev_h + mr + 1, *dev_nn = dev_h2 + mr + 1;
    const double *ph = m->h_md, *ph2 = ph + mr + 1, *pnn = ph2 + mr + 1;
    std::vector<double> H((size_t)(mr + 1) * mr), cs(mr), sn(mr), g(mr + 1), h(mr + 1), y(mr);
    int rc = 0, its = 0;
    k_mg_copy<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, b, r);
    double beta = 0.0;
    if ((rc = dot1(m, st, n, r, r, &beta))) return rc;
    beta = std::sqrt(beta);
    *rnorm = beta;
    while (its < maxit) {
        if (beta <= tol) {
            *converged = 1;
            break;
        }
        k_mg_axpby<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, 1.0 / beta, r, 0.0, V);
        std::fill(g.begin(), g.end(), 0.0);
        g[0] = beta;
        int j = 0;
        for (; j < mr && its < maxit; j++) {
            if ((rc = precond(m, V + (size_t)j * n))) return rc;
            if ((rc = igab_launch_spmv(c, vals, prec, t, w))) return rc;
            /* CGS2: h = V^T w, w -= V h, twice; the next basis vector w / ||w||; one read of the coefficients */
            double *part = m->mpart;
            mdot(m, st, n, V, j + 1, w, dev_h);
            mg_launch(k_md_update, nb, RD_THREADS, st, n, V, j + 1, dev_h, w, nullptr);
            mdot(m, st, n, V, j + 1, w, dev_h2);
            mg_launch(k_md_update, nb, RD_THREADS, st, n, V, j + 1, dev_h2, w, part);
            mg_launch(k_md_scale, nb, RD_THREADS, st, n, w, part, nb, dev_nn, V + (size_t)(j + 1) * n);
            IGAB_CUDA_TRY(cudaGetLastError());
            IGAB_CUDA_TRY(cudaMemcpyAsync(m->h_md, dev_h, (size_t)(2 * mr + 3) * sizeof(double), cudaMemcpyDeviceToHost, st));
            IGAB_CUDA_TRY(cudaStreamSynchronize(st));
            for (int i = 0; i <= j; i++) h[i] = ph[i] + ph2[i];
            const double hn = std::sqrt(*pnn);
            m->launches += 4;
            its++;
            /* apply the previous rotations, then a new one that zeroes hn */
            for (int i = 0; i < j; i++) {
                const double a = h[i], bb = h[i + 1];
                h[i] = cs[i] * a + sn[i] * bb;
                h[i + 1] = -sn[i] * a + cs[i] * bb;
            }
            const double den = std::sqrt(h[j] * h[j] + hn * hn);
            if (den == 0.0) {
                cs[j] = 1.0;
                sn[j] = 0.0;
            } else {
                cs[j] = h[j] / den;
                sn[j] = hn / den;
            }
            h[j] = den;
            for (int i = 0; i <= j; i++) H[(size_t)i * mr + j] = h[i];
            g[j + 1] = -sn[j] * g[j];
            g[j] = cs[j] * g[j];
            *rnorm = std::fabs(g[j + 1]);
            if (*rnorm <= tol || hn == 0.0) {
                j++;
                break;
            }
        }
        /* y = H^-1 g, x += M (V y) */
        for (int i = j - 1; i >= 0; i--) {
            double sacc = g[i];
            for (int k = i + 1; k < j; k++) sacc -= H[(size_t)i * mr + k] * y[k];
            y[i] = H[(size_t)i * mr + i] != 0.0 ? sacc / H[(size_t)i * mr + i] : 0.0;
        }
        IGAB_CUDA_TRY(cudaMemcpyAsync(dev_h, y.data(), (size_t)j * sizeof(double), cudaMemcpyHostToDevice, st));
        k_md_combine<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, V, j, dev_h, w);
        if ((rc = precond(m, w))) return rc;
        k_mg_axpby<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, 1.0, t, 1.0, x);
        /* true residual */
        if ((rc = igab_launch_spmv(c, vals, prec, x, w))) return rc;
        k_mg_sub<<<MG_BLOCKS, MG_THREADS, 0, st>>>(n, b, w, r);
        m->launches += 4;
        if ((rc = dot1(m, st, n, r, r, &beta))) return rc;
        beta = std::sqrt(beta);
        *rnorm = beta;
    }
    if (beta <= tol) *converged = 1;
    *iterations = its;
    IGAB_CUDA_TRY(cudaGetLastError());
    return 0;
}

} /* namespace */

int igab_mg_solve(igab_ctx *c, int method, const void *vals, int prec, const double *b, double *x, double rtol,
                  double atol, int maxit, int *iterations, int *converged, double *rnorm, double *bnorm, int *breakdown)
{
    if (!c->mg) {
        c->mg = new igab_mg();
        IGAB_CUDA_TRY(cudaMalloc((void **)&c->mg->part, (2 * RD_BLOCKS + 2) * sizeof(double)));
        c->mg->dots = c->mg->part + 2 * RD_BLOCKS;
        IGAB_CUDA_TRY(cudaMallocHost((void **)&c->mg->h_dots, 2 * sizeof(double)));
        IGAB_CUDA_TRY(cudaMalloc((void **)&c->mg->mpart,
                                 ((size_t)(GM_RESTART + 1) * RD_BLOCKS + 2 * (GM_RESTART + 1) + 1) * sizeof(double)));
        IGAB_CUDA_TRY(cudaMemset(c->mg->mpart, 0,
                                 ((size_t)(GM_RESTART + 1) * RD_BLOCKS + 2 * (GM_RESTART + 1) + 1) * sizeof(double)));
        IGAB_CUDA_TRY(cudaMallocHost((void **)&c->mg->h_md, (2 * (GM_RESTART + 1) + 1) * sizeof(double)));
    }
    igab_mg *m = c->mg;
    m->launches = 0;
    int rc = 0;
    if (m->version != c->param_version || m->nlev == 0)
        if ((rc = mg_build(c, m))) return rc;
    const long n = c->ndof;
    const long need = (long)(GM_RESTART + 4) * n;
    if (m->kv_n != need) {
        cudaFree(m->kv);
        m->kv = nullptr;
        m->kv_n = 0;
        IGAB_CUDA_TRY(cudaMalloc((void **)&m->kv, (size_t)need * sizeof(double)));
        m->kv_n = need;
    }
    cudaStream_t st = c->stream;
    IGAB_CUDA_TRY(cudaMemsetAsync(x, 0, (size_t)n * sizeof(double), st));
    double bb = 0.0;
    if ((rc = dot1(m, st, n, b, b, &bb))) return rc;
    const double bn = std::sqrt(bb);
    const double tol = std::max(rtol * bn, atol);
    *bnorm = bn;
    *rnorm = bn;
    *iterations = 0;
    *converged = bn <= tol ? 1 : 0;
    *breakdown = 0;
    if (!*converged) {
        if (method == IGAB_KSP_MG_CG)
            rc = solve_cg(m, c, vals, prec, b, x, tol, maxit, iterations, converged, rnorm, breakdown);
        else
            rc = solve_gmres(m, c, vals, prec, b, x, tol, maxit, iterations, converged, rnorm);
        if (rc) return rc;
    }
    IGAB_CUDA_TRY(cudaGetLastError());
    IGAB_CUDA_TRY(cudaStreamSynchronize(st));
    c->last_launches = m->launches;
    return 0;
}

extern "C" int igab_mg_prolongation_1d(const double *coarse_knots, int n_coarse_elements, const double *inserted,
                                       int n_inserted, double *P)
{
    if (!coarse_knots || !P || n_coarse_elements < 1 || n_inserted < 0 || (n_inserted > 0 && !inserted)) {
        igab_set_error("igab_mg_prolongation_1d: bad argument");
        return IGAB_ERR_ARG;
    }
    std::vector<double> kc(coarse_knots, coarse_knots + n_coarse_elements + 5);
    std::vector<double> ins(inserted, inserted + n_inserted);
    for (int i = 0; i < n_inserted; i++)
        if (!(ins[i] > kc[2] && ins[i] < kc[kc.size() - 3]) || (i > 0 && ins[i] < ins[i - 1])) {
            igab_set_error("igab_mg_prolongation_1d: inserted knots must be ascending and interior");
            return IGAB_ERR_ARG;
        }
    std::vector<double> M;
    int nbf = 0, nbc = 0;
    igab_mg_knot_prolongation(kc, ins, M, nbf, nbc);
    memcpy(P, M.data(), M.size() * sizeof(double));
    return 0;
}
