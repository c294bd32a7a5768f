/*
 * Tangent volume kernel by sum factorisation on the FP64 tensor path (mma.sync m8n8k4 f64).
 *
 * Per element (src/snesiga_Tangent.c:104-190), with the 27 x 27 point matrix D (component k,
 * derivative m = 0..8; igab_math.cuh),
 *   K(a,k; b,l) = sum_q sum_{m,n} N_a^m(q) w_q D_{km,ln}(q) N_b^n(q),   N_a^m = X_ax Y_ay Z_az.
 * For each of the six component pairs k <= l the three directions are contracted one after the
 * other.  A derivative m has orders (kx, ky, kz); z first, over the 4 Gauss points qz:
 *   T1[(kx,ky),(lx,ly)](qx,qy; az,bz) = sum_{kz,lz} sum_qz Z_az^kz Z_bz^lz D_mn(q)
 *   T2[kx,lx](qx; ay,by; az,bz)       = sum_{ky,ly} sum_qy Y_ay^ky Y_by^ly T1
 *   K(ax,bx; ay,by; az,bz)            = sum_{kx,lx} sum_qx X_ax^kx X_bx^lx T2.
 * 69 of the 81 (m, n) are nonzero, in 34 of 36 class pairs of T1 and 9 of T2; for k = l the matrix is
 * P + P^T with P over m <= n only (39, 20, 6).  About 1,900 m8n8k4 products (0.97 MFLOP) per element
 * against 6.98 MFLOP of the rank-12 form X^T Phi'' X it replaces.
 *
 * Each step is a product W (pairs x 4 points) B (4 points x columns): the 9 pairs (a, b) of a direction
 * are one m8 tile without the pair (1, 1), plus the total sum_q B.  As the three functions sum to 1 (in
 * the tables that the kernel uses, sf_sum) and their derivatives to 0, the entry (1, 1) is the total minus the other eight, so the eight rows
 * come out as they are, one product serves all nine pairs, and the totals only need the terms without a
 * derivative in that direction (a sum over four lanes).  The totals are carried as row / column 4 through
 * all steps and turned into the entries (1, 1) on the finished element matrix, direction by direction.
 *
 * In the first step a lane is one Gauss point (qz = lane % 4, column = lane / 4): it computes its
 * point's D_mn in registers, which is the B fragment.  8 warps: two halves of the 16 columns (qx, qy) x
 * four groups of classes; then (qx) x two halves of the (kx, lx); then one tile of eight (az, bz) per
 * (ay, by).  One 256-thread block per tile of 2 x 2 x 2 elements, two blocks per SM (114 KB, 128
 * registers).  The phases of a pair are separated by block barriers; the last step of a pair runs
 * beside the first step of the next, and the read-out of one component row and the next element's
 * field beside later pairs.
 *
 * phys/getime uses the same kernel (NR = 2): its Hessian is a weighted sum over the Taylor orders of the segment
 * from t_n-1/2 to t_n+1/2, which is the static form summed over two fields (sf_coef), plus the inertia term on
 * the value components; the additional work is in the point matrices only.  FP64 throughout; FP32 values round
 * at the store.
 *
 * Measured (tangent alone).  64^3: 20.5 ms FP64, 19.9 ms FP32 values, against 96.1 ms for the rank-12 form on the
 * same pipe and 41.1 ms for its TF32 tcgen05 form.  Error of the FP32 values against FP64, in the norm of all and the
 * worst entry over its row's largest: 7.6e-8 and 5.4e-7, TF32 form 1.3e-6 and 2.8e-6.  32^3 transient: 4.7 ms against
 * 35.3 ms for the rank-24 form.  Bound by instruction latency in the short
 * barrier phases (IPC 0.36 per scheduler; tensor and FP64 pipe 47%).  Measured and left out: the second step fed
 * from the first one's accumulators in registers, without T1 (23.0 ms: it moves the third step into the same
 * warps' serial chain); totals by shuffles instead of a product with ones (+0.7 ms); one copy of each part
 * of the code under run-time slots and phases (54 instead of 85 KB of code, +2.5 ms); padding of the element
 * matrices against bank conflicts (no change).
 */
#include <algorithm>
#include <cuda_runtime.h>
#include <type_traits>
#include "igab_device.cuh"

namespace {

#define SF_THR 256
#define SF_TE 2
/* Meshes up to this many elements go through a scratch array of element matrices (143 MB at most) and a gather,
 * which lets every element run at once; larger ones add tile after tile, colour after colour.  One mesh on one
 * stream: 8^3 1,079 -> 80 us, 12^3 1,081 -> 213, 16^3 1,096 -> 493, 20^3 1,109 -> 933, 24^3 1,570 -> 1,605
 * (transient 8^3 1,207 -> 109, 16^3 1,216 -> 695); three meshes on three streams, which fill one another's gaps:
 * 12^3 369 -> 215 us each, 16^3 476 -> 503, 20^3 648 -> 972. */
#define SF_ELEM_MAX 4096
#define SF_STEP 1184                     /* elements of a step of the host entry point: four of two blocks per SM */
#define SF_LAYER_MAX (SF_ELEM_MAX / 3)   /* its largest layer: a step and the two layers before it fit */

/* ---- derivative components m = 0..8: x y z xx xy xz yy yz zz; class = (kx, ky) in the order
 * 0:(0,0) 1:(0,1) 2:(0,2) 3:(1,0) 4:(1,1) 5:(2,0) */
__host__ __device__ constexpr int sf_kz(int m) { return a_kz(m + 1); }
__host__ __device__ constexpr int sf_cls(int m)
{
    const int kx = a_kx(m + 1), ky = a_ky(m + 1);
    return kx == 0 ? ky : (kx == 1 ? 3 + ky : 5);
}
__host__ __device__ constexpr int cls_kx(int c) { return c < 3 ? 0 : (c < 5 ? 1 : 2); }
__host__ __device__ constexpr int cls_ky(int c) { return c < 3 ? c : (c < 5 ? c - 3 : 0); }
/* the two indices of a second derivative c = m - 3 */
__host__ __device__ constexpr int s_i(int c) { return c < 3 ? 0 : (c < 5 ? 1 : 2); }
__host__ __device__ constexpr int s_k(int c) { return c == 0 ? 0 : (c == 1 || c == 3 ? 1 : 2); }
__host__ __device__ constexpr int sym6(int I, int K)
{
    return I == 0 ? K : (K == 0 ? I : (I == 1 ? 2 + K : (K == 1 ? 2 + I : 5)));
}
/* the component of class c with z order kz, or -1 */
__host__ __device__ constexpr int sf_comp(int c, int kz)
{
    for (int m = 0; m < 9; m++)
        if (sf_cls(m) == c && sf_kz(m) == kz) return m;
    return -1;
}
/* two second derivatives couple only through a shared index */
__host__ __device__ constexpr bool mn_nonzero(int m, int n)
{
    return m < 3 || n < 3 || s_i(m - 3) == s_i(n - 3) || s_i(m - 3) == s_k(n - 3) || s_k(m - 3) == s_i(n - 3) ||
           s_k(m - 3) == s_k(n - 3);
}
__host__ __device__ constexpr bool cls_nonzero(int c, int d) { return !((c == 5 && d == 2) || (c == 2 && d == 5)); }
/* m <= n in the order of (class, kz) */
__host__ __device__ constexpr bool mn_upper(int m, int n)
{
    return sf_cls(m) < sf_cls(n) || (sf_cls(m) == sf_cls(n) && sf_kz(m) <= sf_kz(n));
}
/* the group of warps that owns class pair (c, d) in the first step: 15 / 17 / 17 / 20 products of a pair
 * k < l, 11 / 12 / 10 / 6 of a pair k = l */
__host__ __device__ constexpr int cls_group(bool diag, int c, int d)
{
    if (!diag) return c == 0 ? 0 : (c == 3 ? 1 : (c == 1 ? 2 : 3));
    if (c == 0) return d == 0 || d == 1 || d == 3 ? 0 : 2;
    return c == 1 ? 1 : (c == 3 ? 2 : 3);
}
/* the half of the warps that owns (kx, lx) in the second step: 17 / 17, or 10 / 10 */
__host__ __device__ constexpr int x_half(bool diag, int X)
{
    if (!diag) return X < 3 ? 0 : 1;
    return X == 0 || X == 2 || X == 5 ? 0 : 1;
}
/* the qx (warp of the half) that forms the z-total column of (kx, lx) */
__host__ __device__ constexpr int x_zwarp(bool diag, int X)
{
    if (!diag) return X < 3 ? X : (X == 3 ? 0 : (X == 4 ? 1 : (X == 5 || X == 8 ? 2 : 3)));
    return X == 0 || X == 1 ? 0 : (X == 2 || X == 4 ? 1 : (X == 5 ? 2 : 3));
}

/* point data, [item][64 points], point = 4 (4 qx + qy) + qz; CN, S and TAU times the weight */
template <int NR>
struct pt_at {   /* NR = 1: phys/ge; 2: phys/getime, the two fields of the hat form */
    static constexpr int NC = NR == 1 ? 1 : 3;   /* CN of the field pairs (0,0), (0,1), (1,1) */
    static constexpr int F = 0, G = 9 * NR, W = 27 * NR, CN = W + 1, S = CN + 6 * NC, TAU = S + 6, N = TAU + 9;
};

/* material constants of D, and the hat form of the transient tangent: with the weights tw of the Hessian's
 * Taylor coefficients, tw0 a a + 2 tw1 a b + tw2 b b = (r00 a + r01 b)^2 + (r11 b)^2, so that every term with a
 * constant Phi'' is the static one summed over the two fields r00 m + r01 h and r11 h (igab_math.cuh: m, h);
 * (al, be, ga) is the inverse map, mass the coefficient of the value components */
struct sf_coef {
    double aon, aoff, ash;
    double r00, r01, r11, al, be, ga, mass;
};
__host__ __device__ inline sf_coef sf_coef_ge(const igab_geom &g)
{
    sf_coef C = {};
    C.aon = g.coef.p4sq * (4.0 / 3.0);
    C.aoff = g.coef.p4sq * (-2.0 / 3.0);
    C.ash = g.coef.p3 * 0.5;
    return C;
}

struct __align__(16) sf_row { long rb; int rsx, rsy; };

template <int NR>
struct sf_smem {
    double pt[pt_at<NR>::N * 64];
    double T1[36 * 128];     /* [class pair][8 pairs (az,bz)][16 columns], 16-byte chunks swizzled */
    double T1x[(24 + NR) * 16];   /* z totals of the class pairs without z derivative (and of the values) */
    double T2[9 * 288];      /* [kx,lx][9 (ay,by)][4 qx][8 (az,bz)], swizzled */
    double T2x[9 * 36];      /* z totals [kx,lx][9 (ay,by)][4 qx] */
    double K[4 * 729];       /* element matrices of component pairs, [9 (ax,bx)][9 (ay,by)][9 (az,bz)] */
    double tab[2][3][IGAB_TAB1D];
    double wh[2][3][IGAB_NQ];
    double esc[2];
    sf_row row[3][27];
};
static_assert(sizeof(sf_smem<1>) + 1024 + 384 <= 233472 / 2, "two blocks per SM");
/* the control values and the interpolation of the next element's field and the fifth element-matrix slot use
 * T1x and T1, which are free then */
#define SF_U(S, f) ((S).T1x + 82 * (f))
#define SF_A(S) ((S).T1)
#define SF_C(S) ((S).T1 + 648)
#define SF_KSLOT(S, s) ((s) < 4 ? (S).K + 729 * (s) : (S).T1 + 2400)

/* f(integral_constant 0), ..., f(integral_constant N - 1) */
template <int I, int N, class F>
__device__ __forceinline__ void static_for(F &&f)
{
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(f);
    }
}

__device__ __forceinline__ void sf_dmma(double &c0, double &c1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}
/* the pair index 3 a + b of row r of an m8 tile (all but 4 = (1, 1)) */
__device__ __forceinline__ int pair_id(int r) { return r + (r >> 2); }

/* A fragments of the 9 derivative combinations of one direction: W[3 k + l] = B_a^k(q) B_b^l(q),
 * (a, b) = pair of row lane / 4, q = lane % 4 */
__device__ __forceinline__ void sf_weights(const double *tab, int lane, double w[9])
{
    const int id = pair_id(lane >> 2), q = lane & 3;
    const double *ta = tab + q * 9 + (id / 3) * 3, *tb = tab + q * 9 + (id % 3) * 3;
    const double a0 = ta[0], a1 = ta[1], a2 = ta[2], b0 = tb[0], b1 = tb[1], b2 = tb[2];
    w[0] = a0 * b0; w[1] = a0 * b1; w[2] = a0 * b2;
    w[3] = a1 * b0; w[4] = a1 * b1; w[5] = a1 * b2;
    w[6] = a2 * b0; w[7] = a2 * b1; w[8] = a2 * b2;
}

/* one point's data of a component pair */
template <int NR>
struct sf_point {
    double f[NR][3], h[NR][3], g[NR][6], y[NR][6];   /* F and second derivatives of k and l */
    double won, woff, wsh;                           /* w * 2 le^2 (2/3, -1/3), w * e345 / 2 */
    double cn[pt_at<NR>::NC][6], s[6], tau[9];
};

/* w D_mn of the point */
template <int NR, bool DG, int m, int n>
__device__ __forceinline__ double sf_d(const sf_point<NR> &P)
{
    double v = 0.0;
    if constexpr (m < 3 && n < 3) {
        constexpr int I = m, J = n, M1 = (I + 1) % 3, M2 = (I + 2) % 3, IJ = sym6(I, J);
        double t = 0.0, u = 0.0;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            t += P.g[r][sym6(I, 0)] * P.y[r][sym6(J, 0)] + P.g[r][sym6(I, 1)] * P.y[r][sym6(J, 1)] +
                 P.g[r][sym6(I, 2)] * P.y[r][sym6(J, 2)];
            if constexpr (I != J) u += P.f[r][J] * P.h[r][I];
            else u += P.f[r][M1] * P.h[r][M1] + P.f[r][M2] * P.h[r][M2];
        }
        v = (I == J ? P.won : P.woff) * t + P.cn[0][IJ] * (P.f[0][I] * P.h[0][J]);
        v += P.wsh * u;
        if constexpr (NR == 2)
            v += P.cn[1][IJ] * (P.f[0][I] * P.h[1][J] + P.f[1][I] * P.h[0][J]) + P.cn[2][IJ] * (P.f[1][I] * P.h[1][J]);
        if constexpr (DG) v += P.s[IJ];
    } else if constexpr (m < 3) {
        constexpr int I = m, J = s_i(n - 3), K = s_k(n - 3);
#pragma unroll
        for (int r = 0; r < NR; r++) {
            v += P.g[r][sym6(I, K)] * ((I == J ? P.won : P.woff) * P.h[r][J]);
            if constexpr (J != K) v += P.g[r][sym6(I, J)] * ((I == K ? P.won : P.woff) * P.h[r][K]);
        }
        if constexpr (DG && I == J) v += P.tau[3 * I + K];
        else if constexpr (DG && I == K) v += P.tau[3 * I + J];
    } else if constexpr (n < 3) {
        constexpr int J = n, I = s_i(m - 3), K = s_k(m - 3);
#pragma unroll
        for (int r = 0; r < NR; r++) {
            v += ((I == J ? P.won : P.woff) * P.f[r][I]) * P.y[r][sym6(J, K)];
            if constexpr (I != K) v += ((K == J ? P.won : P.woff) * P.f[r][K]) * P.y[r][sym6(J, I)];
        }
        if constexpr (DG && J == I) v += P.tau[3 * J + K];
        else if constexpr (DG && J == K) v += P.tau[3 * J + I];
    } else {
        /* over the orderings (I, K) of m and (J, L) of n with K = L: A_IJ f_I h_J */
        constexpr int i0 = s_i(m - 3), k0 = s_k(m - 3), j0 = s_i(n - 3), l0 = s_k(n - 3);
#pragma unroll
        for (int r = 0; r < NR; r++) {
            if constexpr (k0 == l0) v += P.f[r][i0] * ((i0 == j0 ? P.won : P.woff) * P.h[r][j0]);
            if constexpr (i0 != k0 && i0 == l0) v += P.f[r][k0] * ((k0 == j0 ? P.won : P.woff) * P.h[r][j0]);
            if constexpr (j0 != l0 && k0 == j0) v += P.f[r][i0] * ((i0 == l0 ? P.won : P.woff) * P.h[r][l0]);
            if constexpr (i0 != k0 && j0 != l0 && i0 == j0)
                v += P.f[r][k0] * ((k0 == l0 ? P.won : P.woff) * P.h[r][l0]);
        }
    }
    return v;
}

/* first step: the class pairs of group G, for the 8 columns of half h */
template <int NR, int G, bool DG>
__device__ __forceinline__ void sf_s1(sf_smem<NR> &S, const double *tz, int lane, int h, int k, int l, const sf_coef &C)
{
    double w[9];
    sf_weights(tz, lane, w);
    const double *p = S.pt + h * 32 + lane;
    using A = pt_at<NR>;
    sf_point<NR> P;
#pragma unroll
    for (int r = 0; r < NR; r++) {
#pragma unroll
        for (int J = 0; J < 3; J++) {
            P.f[r][J] = p[(A::F + 9 * r + 3 * k + J) * 64];
            P.h[r][J] = DG ? P.f[r][J] : p[(A::F + 9 * r + 3 * l + J) * 64];
        }
#pragma unroll
        for (int c = 0; c < 6; c++) {
            P.g[r][c] = p[(A::G + 18 * r + 6 * k + c) * 64];
            P.y[r][c] = DG ? P.g[r][c] : p[(A::G + 18 * r + 6 * l + c) * 64];
        }
    }
#pragma unroll
    for (int c = 0; c < 6; c++) {
#pragma unroll
        for (int r = 0; r < A::NC; r++) P.cn[r][c] = p[(A::CN + 6 * r + c) * 64];
        P.s[c] = DG ? p[(A::S + c) * 64] : 0.0;
    }
#pragma unroll
    for (int c = 0; c < 9; c++) P.tau[c] = DG ? p[(A::TAU + c) * 64] : 0.0;
    const double wq = p[A::W * 64];
    P.won = wq * C.aon;
    P.woff = wq * C.aoff;
    P.wsh = wq * C.ash;
    const int r = lane >> 2, q = lane & 3;
    /* row r, chunk 4 h + lane % 4 of two columns; chunks are XORed so that these stores and the second
     * step's loads (4 rows x 4 qy) hit distinct banks */
    double *t1 = S.T1 + r * 16 + 2 * ((4 * h + q) ^ (4 * (r & 1) + (r & 2)));
    double *t1x = S.T1x + 8 * h + 2 * q;
    static_for<0, 36>([&](auto cd_) {
        constexpr int cd = decltype(cd_)::value, c = cd / 6, d = cd % 6;
        if constexpr (cls_nonzero(c, d) && !(DG && c > d) && cls_group(DG, c, d) == G) {
            double c0 = 0.0, c1 = 0.0;
            if constexpr (NR == 2 && DG && cd == 0) {
                /* inertia / damping: the value components, T1x row 25 */
                const double v = 0.5 * C.mass * wq;
                double t0 = 0.0, t1v = 0.0;
                sf_dmma(c0, c1, w[0], v);
                sf_dmma(t0, t1v, 1.0, v);
                if (r == 0) *reinterpret_cast<double2 *>(t1x + 25 * 16) = make_double2(t0, t1v);
            }
            static_for<0, 9>([&](auto kk_) {
                constexpr int kk = decltype(kk_)::value, m = sf_comp(c, kk / 3), n = sf_comp(d, kk % 3);
                if constexpr (m >= 0 && n >= 0) {
                    if constexpr (mn_nonzero(m, n) && !(DG && !mn_upper(m, n))) {
                        double v = sf_d<NR, DG, m, n>(P);
                        if constexpr (DG && m == n) v *= 0.5;
                        sf_dmma(c0, c1, w[kk], v);
                        if constexpr (kk == 0) {
                            double t0 = 0.0, t1v = 0.0;
                            sf_dmma(t0, t1v, 1.0, v);
                            if (r == 0)
                                *reinterpret_cast<double2 *>(t1x + ((c - 1) * 5 + d - 1) * 16) = make_double2(t0, t1v);
                        }
                    }
                }
            });
            *reinterpret_cast<double2 *>(t1 + cd * 128) = make_double2(c0, c1);
        }
    });
}

/* second step: the (kx, lx) of the half, for one qx; the z totals of a (kx, lx) by one warp of the half, with
 * the four qx as columns */
template <int NR, int HALF, bool DG>
__device__ __forceinline__ void sf_s2(sf_smem<NR> &S, const double *ty, int lane, int qx)
{
    double w[9];
    sf_weights(ty, lane, w);
    const int n = lane >> 2, q = lane & 3;
    const double *t1 = S.T1 + n * 16 + 2 * ((2 * qx + (q >> 1)) ^ (4 * (n & 1) + (n & 2))) + (q & 1);
    const int id = pair_id(n);
    /* T2 row (ay,by), 8 doubles per qx: qx flips with the row's parity and the (az,bz) halves with qx / 2,
     * so that 2-row stores and 4-qx loads hit distinct banks */
    const int sw = (2 * q) ^ (4 * (qx >> 1));
    double *t2 = S.T2 + id * 32 + ((qx ^ (id & 1)) << 3) + sw;
    double *t2y = S.T2 + 4 * 32 + (qx << 3) + sw;
    static_for<0, 9>([&](auto X_) {
        constexpr int X = decltype(X_)::value, kx = X / 3, lx = X % 3;
        if constexpr (!(DG && kx > lx) && x_half(DG, X) == HALF) {
            double c0 = 0.0, c1 = 0.0;
            static_for<0, 36>([&](auto cd_) {
                constexpr int cd = decltype(cd_)::value, c = cd / 6, d = cd % 6, kl = 3 * cls_ky(c) + cls_ky(d);
                if constexpr (cls_kx(c) == kx && cls_kx(d) == lx && cls_nonzero(c, d) && !(DG && c > d)) {
                    const double b = t1[cd * 128];
                    sf_dmma(c0, c1, w[kl], b);
                    if constexpr (kl == 0) {
                        double t0 = 0.0, t1v = 0.0;
                        sf_dmma(t0, t1v, 1.0, b);
                        if (n == 0) *reinterpret_cast<double2 *>(t2y + X * 288) = make_double2(t0, t1v);
                    }
                }
            });
            *reinterpret_cast<double2 *>(t2 + X * 288) = make_double2(c0, c1);
            if (qx == x_zwarp(DG, X)) {
                const double *t1x = S.T1x + (n & 3) * 4 + q;
                c0 = c1 = 0.0;
                static_for<0, 36>([&](auto cd_) {
                    constexpr int cd = decltype(cd_)::value, c = cd / 6, d = cd % 6, kl = 3 * cls_ky(c) + cls_ky(d);
                    constexpr bool mass = NR == 2 && DG && cd == 0;
                    if constexpr (((c > 0 && d > 0) || mass) && cls_kx(c) == kx && cls_kx(d) == lx &&
                                  cls_nonzero(c, d) && !(DG && c > d)) {
                        const double b = n < 4 ? t1x[(mass ? 25 : (c - 1) * 5 + d - 1) * 16] : 0.0;
                        sf_dmma(c0, c1, w[kl], b);
                        if constexpr (kl == 0) {
                            double t0 = 0.0, t1v = 0.0;
                            sf_dmma(t0, t1v, 1.0, b);
                            if (lane < 2)
                                *reinterpret_cast<double2 *>(S.T2x + X * 36 + 16 + 2 * q) = make_double2(t0, t1v);
                        }
                    }
                });
                if (q < 2) *reinterpret_cast<double2 *>(S.T2x + X * 36 + id * 4 + 2 * q) = make_double2(c0, c1);
            }
        }
    });
}

/* third step: the tile of eight (az,bz) columns of (ay,by) t; all loads first, then two product chains */
template <bool DG>
__device__ __forceinline__ void sf_s3(const double *T2, const double w[9], double *K, int t, int lane)
{
    const int n = lane >> 2, q = lane & 3;
    const double *t2 = T2 + t * 32 + ((q ^ (t & 1)) << 3) + (n ^ (4 * (q >> 1)));
    double b[9], c0 = 0.0, c1 = 0.0, d0 = 0.0, d1 = 0.0, x0 = 0.0, x1 = 0.0;
#pragma unroll
    for (int X = 0; X < 9; X++)
        if (!(DG && X / 3 > X % 3)) b[X] = t2[X * 288];
#pragma unroll
    for (int X = 0; X < 9; X++) {
        if (DG && X / 3 > X % 3) continue;
        if (X & 1) sf_dmma(d0, d1, w[X], b[X]);
        else sf_dmma(c0, c1, w[X], b[X]);
        if (X == 0) sf_dmma(x0, x1, 1.0, b[X]);
    }
    const int z0 = pair_id(2 * q), z1 = pair_id(2 * q + 1);
    double *o = K + pair_id(n) * 81 + t * 9;
    o[z0] = c0 + d0;
    o[z1] = c1 + d1;
    if (n == 0) {
        K[4 * 81 + t * 9 + z0] = x0;
        K[4 * 81 + t * 9 + z1] = x1;
    }
}

/* third step of the z totals: job 9 the eight (ay,by), job 10 the total in y and z (only where both
 * derivatives are in x, or of the values) */
template <int NR, bool DG>
__device__ __forceinline__ void sf_s3z(const double *T2x, const double w[9], double *K, int job, int lane)
{
    const int n = lane >> 2, q = lane & 3, xr = pair_id(n) * 81;
    double c0 = 0.0, c1 = 0.0;
    if (job == 9) {
        const double *t2 = T2x + pair_id(n) * 4 + q;
        double t0 = 0.0, t1 = 0.0;
#pragma unroll
        for (int X = 0; X < 9; X++) {
            if (DG && X / 3 > X % 3) continue;
            const double b = t2[X * 36];
            sf_dmma(c0, c1, w[X], b);
            if (X == 0) sf_dmma(t0, t1, 1.0, b);
        }
        K[xr + pair_id(2 * q) * 9 + 4] = c0;
        K[xr + pair_id(2 * q + 1) * 9 + 4] = c1;
        if (n == 0) {
            K[4 * 81 + pair_id(2 * q) * 9 + 4] = t0;
            K[4 * 81 + pair_id(2 * q + 1) * 9 + 4] = t1;
        }
    } else {
        double t0 = 0.0, t1 = 0.0;
#pragma unroll
        for (int X = 0; X < 9; X++) {
            const bool mass = NR == 2 && DG && X == 0;
            if (!mass && (X / 3 == 0 || X % 3 == 0 || (DG && X / 3 > X % 3))) continue;
            const double b = n == 0 ? T2x[X * 36 + 16 + q] : 0.0;
            sf_dmma(c0, c1, w[X], b);
            if (mass) sf_dmma(t0, t1, 1.0, b);
        }
        if (q == 0) K[xr + 4 * 9 + 4] = c0;
        if (lane == 0) K[4 * 81 + 4 * 9 + 4] = t0;
    }
}

/* third step of a pair into an element-matrix slot: tiles 0-8, then the z totals, over the warps */
template <int NR, bool DG>
__device__ __forceinline__ void sf_s3_all(sf_smem<NR> &S, const double *tx, double *K, int warp, int lane)
{
    double w[9];
    sf_weights(tx, lane, w);
#pragma unroll 1
    for (int t = warp; t < 11; t += 8) {
        if (t < 9) sf_s3<DG>(S.T2, w, K, t, lane);
        else sf_s3z<NR, DG>(S.T2x, w, K, t, lane);
    }
}

/* totals -> entries (1, 1) in z, then y, of slots s0, s1, s2 (the first ns): a warp per three (ax,bx) */
template <int NR>
__device__ __forceinline__ void sf_fix_zy(sf_smem<NR> &S, int s0, int s1, int s2, int ns, int warp, int lane)
{
    for (int u = warp; u < 3 * ns; u += 8) {
        const int sl = u / 3;
        double *K = SF_KSLOT(S, sl == 0 ? s0 : (sl == 1 ? s1 : s2)) + (3 * (u - 3 * sl) + lane / 9) * 81;
        const int e = lane % 9;
        if (lane < 27) {
            double *z = K + e * 9;
            z[4] -= ((z[0] + z[1]) + (z[2] + z[3])) + ((z[5] + z[6]) + (z[7] + z[8]));
        }
        __syncwarp();
        if (lane < 27) {
            double *z = K + e;
            z[36] -= ((z[0] + z[9]) + (z[18] + z[27])) + ((z[45] + z[54]) + (z[63] + z[72]));
        }
    }
}
/* and in x */
template <int NR>
__device__ __forceinline__ void sf_fix_x(sf_smem<NR> &S, int s0, int s1, int s2, int ns, int tid)
{
    if (tid < 81 * ns) {
        const int sl = tid / 81;
        double *z = SF_KSLOT(S, sl == 0 ? s0 : (sl == 1 ? s1 : s2)) + (tid - 81 * sl);
        z[324] -= ((z[0] + z[81]) + (z[162] + z[243])) + ((z[405] + z[486]) + (z[567] + z[648]));
    }
}

/* Add rows (a, k), a = 0..26, into the CSR values; slot s_l holds pair (min(k,l), max(k,l)).  A thread owns one column c2 = 3 b + l and walks the 9
 * rows of one ax, so consecutive lanes add to runs of 9 consecutive values and the index arithmetic of a row
 * is two multiply-adds. */
template <typename T, int NR>
__device__ __forceinline__ void sf_scatter(sf_smem<NR> &S, T *__restrict__ vals, int k, int s0, int s1, int s2, int tid)
{
    if (tid >= 243) return;
    const int j = tid / 81, c = tid - 81 * j, l = c % 3, b = c / 3;
    const int bx = b / 9, by = (b / 3) % 3, bz = b % 3;
    const double *Kl = SF_KSLOT(S, l == 0 ? s0 : (l == 1 ? s1 : s2));
    const double *Kn = Kl + (3 * j + bx) * 81 + by * 9 + bz;       /* (a, b), + 27 ay + 3 az */
    const double *Kt = Kl + (3 * bx + j) * 81 + by * 27 + bz * 3;  /* (b, a), + 9 ay + az */
    const bool up = l >= k, dg = l == k;
    const double *Ka = up ? Kn : Kt;
    const int sy = up ? 27 : 9, sz = up ? 3 : 1;
    double x[9];
#pragma unroll
    for (int a = 0; a < 9; a++) x[a] = Ka[(a / 3) * sy + (a % 3) * sz];
    if (dg)
#pragma unroll
        for (int a = 0; a < 9; a++) x[a] += Kt[9 * (a / 3) + a % 3];
    T *v = vals + c % 9;
#pragma unroll
    for (int a = 0; a < 9; a++) {
        const sf_row R = S.row[k][9 * j + a];
        atomicAdd(v + R.rb + (bx * R.rsx + by * R.rsy), T(x[a]));
    }
}

/* ---- the field of an element: loads, three interpolation steps, point data */
struct sf_elem { int ex, ey, ez; };

__device__ __forceinline__ void sf_copy8(double *dst, const double *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void sf_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
/* asynchronous loads of an element: U (and the two history levels), the 1-D tables, weights, the scale */
template <int NR>
__device__ __forceinline__ void sf_load(sf_smem<NR> &S, const igab_geom &g, const double *__restrict__ U, const sf_elem &E,
                                        int buf, int tid)
{
    if (tid < 81) {
        const int i = tid % 3, a = tid / 3;
        const long o = 3 * cp_index(g, E.ex + a / 9, E.ey + (a / 3) % 3, E.ez + a % 3) + i;
        sf_copy8(SF_U(S, 0) + tid, U + o);
        if constexpr (NR == 2) {
            sf_copy8(SF_U(S, 1) + tid, g.hist1 + o);
            sf_copy8(SF_U(S, 2) + tid, g.hist0 + o);
        }
    } else if (tid < 189) {
        const int d = (tid - 81) / 36, o = (tid - 81) % 36, e = d == 0 ? E.ex : (d == 1 ? E.ey : E.ez);
        sf_copy8(&S.tab[buf][d][o], g.tab[d] + (long)e * IGAB_TAB1D + o);
    } else if (tid < 201) {
        const int d = (tid - 189) >> 2, o = (tid - 189) & 3, e = d == 0 ? E.ex : (d == 1 ? E.ey : E.ez);
        sf_copy8(&S.wh[buf][d][o], g.wh[d] + (long)e * IGAB_NQ + o);
    } else if (tid == 201) {
        if (g.escale) sf_copy8(&S.esc[buf], g.escale + ((long)E.ex * g.ne[1] + E.ey) * g.ne[2] + E.ez);
        else S.esc[buf] = 1.0;
    }
}
/* field r of control value o: U, or the middle (u0 + u1) / 2 and the half step (u - u0) / 2 */
template <int NR>
__device__ __forceinline__ double sf_value(const sf_smem<NR> &S, int r, int o)
{
    if (NR == 1) return SF_U(S, 0)[o];
    return 0.5 * (r == 0 ? SF_U(S, 2)[o] + SF_U(S, 1)[o] : SF_U(S, 0)[o] - SF_U(S, 2)[o]);
}
template <int NR>
__device__ __forceinline__ void sf_interp_z(sf_smem<NR> &S, int buf, int tid)
{
    const double *Bz = S.tab[buf][2];
    for (int o = tid; o < 324 * NR; o += SF_THR) {
        const int f = o / 324, e = o - 324 * f, i = e % 3, kz = (e / 3) % 3, a = ((e / 9) % 9) * 9 + i, q = e / 81;
        SF_A(S)[o] = Bz[q * 9 + kz] * sf_value<NR>(S, f, a) + Bz[q * 9 + 3 + kz] * sf_value<NR>(S, f, a + 3) +
                     Bz[q * 9 + 6 + kz] * sf_value<NR>(S, f, a + 6);
    }
}
template <int NR>
__device__ __forceinline__ void sf_interp_y(sf_smem<NR> &S, int buf, int tid)
{
    const double *By = S.tab[buf][1];
    for (int o = tid; o < 864 * NR; o += SF_THR) {
        const int f = o / 864, e = o - 864 * f;
        const int i = e % 3, kk = (e / 3) % 6, ax = (e / 18) % 3, qq = e / 54;
        const int qy = qq & 3, qz = qq >> 2, ky = kk_ky(kk), kz = kk_kz(kk);
        const double *a0 = SF_A(S) + 324 * f + ((qz * 3 + ax) * 3) * 9 + kz * 3 + i;
        SF_C(S)[o] = By[qy * 9 + ky] * a0[0] + By[qy * 9 + 3 + ky] * a0[9] + By[qy * 9 + 6 + ky] * a0[18];
    }
}
/* The basis's denominators carry a guard of 1e-15 (igab_bspline_p2), so the three functions sum to 1 only within 1e-15
 * over the element's width (their derivatives do sum to 0).  The totals need 1, so the tables are divided by the sum
 * and the weights multiplied by its square, which leaves the products as they are.  Without it the values were 1e-12
 * of the row's largest off at 64^3 on the unit cube, and 2e-7 on a cube of 1e-6; now 3e-15.  It costs nothing that
 * shows (64^3 20.5 ms): both steps run on threads that wait; the totals weighted with the sum's square instead, a
 * register more in each step, took 2.6%.
 * The sum of thread i < 12: direction i / 4, point i % 4; an empty element has any sum and no weight. */
template <int NR>
__device__ __forceinline__ double sf_sum(const sf_smem<NR> &S, int buf, int i)
{
    const double *t = S.tab[buf][i >> 2] + (i & 3) * 9;
    const double s = t[0] + t[3] + t[6];
    return s > 1e-3 ? s : 1.0;
}
/* beside the last interpolation, which still needs the tables as they are */
template <int NR>
__device__ __forceinline__ void sf_norm_weights(sf_smem<NR> &S, int buf, int i)
{
    if (i < 0 || i >= 12) return;
    const double s = sf_sum<NR>(S, buf, i);
    S.wh[buf][i >> 2][i & 3] *= s * s;
}
/* and beside the point data, which does not */
template <int NR>
__device__ __forceinline__ void sf_norm_tab(sf_smem<NR> &S, int buf, int i)
{
    if (i < 0 || i >= 12) return;
    const double r = 1.0 / sf_sum<NR>(S, buf, i);
    double *t = S.tab[buf][i >> 2] + (i & 3) * 9;
#pragma unroll
    for (int k = 0; k < 9; k++) t[k] *= r;
}
/* F and G of component tid / 64 at point tid % 64; for NR = 2 of the hat fields r00 m + r01 h, r11 h */
template <int NR>
__device__ __forceinline__ void sf_interp_x(sf_smem<NR> &S, const igab_geom &g, const sf_coef &R, int buf, int tid)
{
    if (tid >= 192) {
        sf_norm_weights<NR>(S, buf, tid - 192);
        return;
    }
    using A = pt_at<NR>;
    const int i = tid >> 6, p = tid & 63, qz = p & 3, qy = (p >> 2) & 3, qx = p >> 4;
    const double *Bx = S.tab[buf][0] + qx * 9;
    double b[3][3], u[NR][9];
#pragma unroll
    for (int ax = 0; ax < 3; ax++)
#pragma unroll
        for (int k = 0; k < 3; k++) b[ax][k] = Bx[ax * 3 + k];
#pragma unroll
    for (int f = 0; f < NR; f++) {
        const double *C = SF_C(S) + 864 * f + (qy + 4 * qz) * 54 + i;
        double c[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ax++)
#pragma unroll
            for (int k = 0; k < 6; k++) c[ax][k] = C[(ax * 6 + k) * 3];
#pragma unroll
        for (int a = 1; a < 10; a++) {
            double s = 0.0;
#pragma unroll
            for (int ax = 0; ax < 3; ax++) s += b[ax][a_kx(a)] * c[ax][a_kk(a)];
            if (a < 4 && f == 0) {
                if (g.periodic) s += g.pp[3 * i + a - 1];
                if (i == a - 1) s += 1.0;
            }
            u[f][a - 1] = s;
        }
    }
#pragma unroll
    for (int a = 0; a < 9; a++) {
        double v0 = u[0][a];
        if constexpr (NR == 2) {
            v0 = R.r00 * v0 + R.r01 * u[NR - 1][a];
            S.pt[(a < 3 ? A::F + 9 + 3 * i + a : A::G + 18 + 6 * i + a - 3) * 64 + p] = R.r11 * u[NR - 1][a];
        }
        S.pt[(a < 3 ? A::F + 3 * i + a : A::G + 6 * i + a - 3) * 64 + p] = v0;
    }
}
/* CN_IJ (the normal strains' Hessian from those of (vvol, va, vb)) times w */
__device__ __forceinline__ void sf_store_cn(double *cn, double w, double h0, double haa, double hbb, double hab)
{
    const double a0 = h0 * (1.0 / 3.0), a1 = haa * 0.5, a2 = hbb * (1.0 / 6.0),
                 a3 = hab * (IGAB_INV_SQRT2 * IGAB_INV_SQRT6);
    cn[0 * 64] = w * (a0 + a1 + a2 + 2.0 * a3);
    cn[1 * 64] = w * (a0 - a1 + a2);
    cn[2 * 64] = w * (a0 - 2.0 * a2 - 2.0 * a3);
    cn[3 * 64] = w * (a0 + a1 + a2 - 2.0 * a3);
    cn[4 * 64] = w * (a0 - 2.0 * a2 + 2.0 * a3);
    cn[5 * 64] = w * (a0 + 4.0 * a2);
}
/* strains and stresses: warps 0-1 the strain part (CN, S), warps 2-7 TAU for one K each */
template <int NR>
__device__ __forceinline__ void sf_point_data(sf_smem<NR> &S, const igab_geom &g, const sf_coef &R, int buf, int tid)
{
    using A = pt_at<NR>;
    sf_norm_tab<NR>(S, buf, tid - 224);
    const int p = tid & 63, qz = p & 3, qy = (p >> 2) & 3, qx = p >> 4;
    double *pt = S.pt + p;
    const double w = S.wh[buf][0][qx] * S.wh[buf][1][qy] * S.wh[buf][2][qz] * S.esc[buf];
    double F[NR][3][3];
#pragma unroll
    for (int r = 0; r < NR; r++)
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
            for (int J = 0; J < 3; J++) F[r][k][J] = pt[(A::F + 9 * r + 3 * k + J) * 64];
    if (tid < 64) {
        const double is2 = IGAB_INV_SQRT2, is3 = IGAB_INV_SQRT3, is6 = IGAB_INV_SQRT6;
        const double c36 = g.coef.c36, c37 = g.coef.c37, c38 = g.coef.c38, p3 = g.coef.p3;
        pt[A::W * 64] = w;
        double sv, sa, sb, sh[3];   /* Phi' of (vvol, va, vb) and the shear stresses E_01, E_02, E_12 */
        if constexpr (NR == 1) {
            double e[6];
#pragma unroll
            for (int c = 0; c < 6; c++) {
                const int I = s_i(c), J = s_k(c);
                e[c] = 0.5 * (F[0][0][I] * F[0][0][J] + F[0][1][I] * F[0][1][J] + F[0][2][I] * F[0][2][J] -
                              (I == J ? 1.0 : 0.0));
            }
            const double vv = (e[0] + e[3] + e[5]) * is3, va = (e[0] - e[3]) * is2,
                         vb = (e[0] + e[3] - 2.0 * e[5]) * is6;
            const double s2 = va * va + vb * vb;
            sv = 2.0 * g.coef.p2 * vv;
            sa = -6.0 * c36 * va * vb + 2.0 * c37 * va + 4.0 * c38 * s2 * va;
            sb = 3.0 * c36 * (vb * vb - va * va) + 2.0 * c37 * vb + 4.0 * c38 * s2 * vb;
            const double haa = -6.0 * c36 * vb + 2.0 * c37 + 4.0 * c38 * (3.0 * va * va + vb * vb);
            const double hbb = 6.0 * c36 * vb + 2.0 * c37 + 4.0 * c38 * (va * va + 3.0 * vb * vb);
            const double hab = -6.0 * c36 * va + 8.0 * c38 * va * vb;
            sf_store_cn(pt + A::CN * 64, w, 2.0 * g.coef.p2, haa, hbb, hab);
            sh[0] = e[1]; sh[1] = e[2]; sh[2] = e[4];
        } else {
            /* E(s) = E0 + s E1 + s^2 E2 along u(s) = m + s h, from F0 = al F^0 + be F^1, F1 = ga F^1 */
            igab_tay<4> v[3];
            double e[3][3];
#pragma unroll
            for (int I = 0; I < 3; I++) {
                double x0 = 0.0, x1 = 0.0, x2 = 0.0;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const double a = R.al * F[0][k][I] + R.be * F[NR - 1][k][I], b = R.ga * F[NR - 1][k][I];
                    x0 += a * a;
                    x1 += a * b;
                    x2 += b * b;
                }
                e[0][I] = 0.5 * (x0 - 1.0);
                e[1][I] = x1;
                e[2][I] = 0.5 * x2;
            }
#pragma unroll
            for (int j = 0; j < 3; j++) {
                v[0].c[j] = (e[j][0] + e[j][1] + e[j][2]) * is3;
                v[1].c[j] = (e[j][0] - e[j][1]) * is2;
                v[2].c[j] = (e[j][0] + e[j][1] - 2.0 * e[j][2]) * is6;
            }
            v[0].c[3] = v[1].c[3] = v[2].c[3] = 0.0;
            const igab_tay<4> aa = v[1] * v[1], bb = v[2] * v[2], ab = v[1] * v[2], s2 = aa + bb;
            const igab_tay<4> sa3 = s2 * v[1], sb3 = s2 * v[2];
            sv = sa = sb = 0.0;
            /* N_j = sum_b tw[j + b] f_b of the parts of Phi'' that vary along s; the constant part is the same
             * in both hat fields and does not couple them */
            double na[3] = {0.0, 0.0, 0.0}, nb[3] = {0.0, 0.0, 0.0}, nab[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const double fa = -6.0 * c36 * v[2].c[b] + 4.0 * c38 * (3.0 * aa.c[b] + bb.c[b]);
                const double fb = 6.0 * c36 * v[2].c[b] + 4.0 * c38 * (aa.c[b] + 3.0 * bb.c[b]);
                const double fab = -6.0 * c36 * v[1].c[b] + 8.0 * c38 * ab.c[b];
                sv += g.tw[b] * (2.0 * g.coef.p2 * v[0].c[b]);
                sa += g.tw[b] * (-6.0 * c36 * ab.c[b] + 2.0 * c37 * v[1].c[b] + 4.0 * c38 * sa3.c[b]);
                sb += g.tw[b] * (3.0 * c36 * (bb.c[b] - aa.c[b]) + 2.0 * c37 * v[2].c[b] + 4.0 * c38 * sb3.c[b]);
#pragma unroll
                for (int j = 0; j < 3; j++)
                    if (j + b < 4) {
                        na[j] += g.tw[j + b] * fa;
                        nb[j] += g.tw[j + b] * fb;
                        nab[j] += g.tw[j + b] * fab;
                    }
            }
            const double q00 = R.al * R.al, q01a = R.al * R.be, q01b = R.al * R.ga, q11a = R.be * R.be,
                         q11b = 2.0 * R.be * R.ga, q11c = R.ga * R.ga, h0 = 2.0 * g.coef.p2, hc = 2.0 * c37;
            double *cn = pt + A::CN * 64;
            sf_store_cn(cn, w, h0, hc + q00 * na[0], hc + q00 * nb[0], q00 * nab[0]);
            sf_store_cn(cn + 6 * 64, w, 0.0, q01a * na[0] + q01b * na[1], q01a * nb[0] + q01b * nb[1],
                        q01a * nab[0] + q01b * nab[1]);
            sf_store_cn(cn + 12 * 64, w, h0, hc + q11a * na[0] + q11b * na[1] + q11c * na[2],
                        hc + q11a * nb[0] + q11b * nb[1] + q11c * nb[2],
                        q11a * nab[0] + q11b * nab[1] + q11c * nab[2]);
            sh[0] = sh[1] = sh[2] = 0.0;
#pragma unroll
            for (int r = 0; r < NR; r++)
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    sh[0] += 0.5 * F[r][k][0] * F[r][k][1];
                    sh[1] += 0.5 * F[r][k][0] * F[r][k][2];
                    sh[2] += 0.5 * F[r][k][1] * F[r][k][2];
                }
        }
        pt[(A::S + 0) * 64] = w * (sv * is3 + sa * is2 + sb * is6);
        pt[(A::S + 3) * 64] = w * (sv * is3 - sa * is2 + sb * is6);
        pt[(A::S + 5) * 64] = w * (sv * is3 - 2.0 * sb * is6);
        pt[(A::S + 1) * 64] = w * p3 * sh[0];
        pt[(A::S + 2) * 64] = w * p3 * sh[1];
        pt[(A::S + 4) * 64] = w * p3 * sh[2];
    } else {
        const int K = (tid >> 6) - 1;
        double ek[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int r = 0; r < NR; r++)
#pragma unroll
            for (int I = 0; I < 3; I++) {
                const double *G = pt + (A::G + 18 * r + igab_idx6(I, K)) * 64;
                ek[I] += F[r][0][I] * G[0] + F[r][1][I] * G[6 * 64] + F[r][2][I] * G[12 * 64];
            }
        const double m = (ek[0] + ek[1] + ek[2]) * (1.0 / 3.0), wa = w * 2.0 * g.coef.p4sq;
#pragma unroll
        for (int I = 0; I < 3; I++) pt[(A::TAU + 3 * I + K) * 64] = wa * (ek[I] - m);
    }
}
/* where the rows (a, k) of the element lie in the CSR values */
template <int NR>
__device__ __forceinline__ void sf_rows(sf_smem<NR> &S, const igab_geom &g, const sf_elem &E, int tid)
{
    if (tid >= 81) return;
    sf_row R;
    elem_row_base(g, E.ex, E.ey, E.ez, 3 * (tid % 27) + tid / 27, R.rb, R.rsx, R.rsy);
    (&S.row[0][0])[tid] = R;
}

/* which elements a block does, and where their matrices go: the elements of a 2 x 2 x 2 tile (position
 * 4 dx + 2 dy + dz ascending) into the CSR values ... */
template <typename T>
struct sf_tile_io {
    tile_t Tl;
    T *vals;
    int le;
    __device__ __forceinline__ bool next(const igab_geom &, sf_elem &E)
    {
        do le++;
        while (le < 8 && ((le >> 2) >= Tl.nv[0] || ((le >> 1) & 1) >= Tl.nv[1] || (le & 1) >= Tl.nv[2]));
        E = {Tl.e0[0] + (le >> 2), Tl.e0[1] + ((le >> 1) & 1), Tl.e0[2] + (le & 1)};
        return le < 8;
    }
    template <int NR>
    __device__ __forceinline__ void out(sf_smem<NR> &S, const igab_geom &, const sf_elem &, int k, int s0, int s1, int s2,
                                        int tid)
    {
        sf_scatter<T, NR>(S, vals, k, s0, s1, s2, tid);
    }
};
/* ... or every gridDim-th element of the mesh into a scratch array [element][6 pairs][729] */
/* Where the scratch holds a layer of elements: layer ex at ex % ring, for the layers of one launch, from `first` on,
 * which wrap once at most (a division per element cost 3% at 8^3) */
struct sf_ring {
    int wrap, below, above;
    sf_ring(int first, int ring) : wrap(first / ring * ring + ring), below(ring - wrap), above(-wrap) {}
    __device__ __forceinline__ int slot(int ex) const { return ex + (ex < wrap ? below : above); }
};

struct sf_elem_io {
    double *ke;
    long e, ne;
    const sf_ring &ring;
    __device__ __forceinline__ bool next(const igab_geom &g, sf_elem &E)
    {
        e += gridDim.x;
        const int i = (int)(e < ne ? e : 0), yz = g.ne[1] * g.ne[2];
        E = {i / yz, (i % yz) / g.ne[2], i % g.ne[2]};
        return e < ne;
    }
    template <int NR>
    __device__ __forceinline__ void out(sf_smem<NR> &S, const igab_geom &g, const sf_elem &E, int k, int s0, int s1,
                                        int s2, int tid)
    {
        /* rows 0 bring the pairs (0,0) (0,1) (0,2), rows 1 (1,1) (1,2), rows 2 (2,2): slot s_l, l >= k */
        double *o = ke + (((long)ring.slot(E.ex) * g.ne[1] + E.ey) * g.ne[2] + E.ez) * 4374 + (k == 0 ? 0 : (k == 1 ? 3 : 5)) * 729;
        for (int l = k; l < 3; l++, o += 729) {
            const double *K = SF_KSLOT(S, l == 0 ? s0 : (l == 1 ? s1 : s2));
            for (int i = tid; i < 729; i += SF_THR) o[i] = K[i];
        }
    }
};

template <int NR, class IO>
__device__ __forceinline__ void sf_run(const igab_geom &g, const sf_coef &C, IO &io, const double *__restrict__ U,
                                       sf_smem<NR> &S)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int buf = 0;
    sf_elem E;
    if (!io.next(g, E)) return;
    sf_load<NR>(S, g, U, E, buf, tid);
    sf_copy_wait();
    __syncthreads();
    sf_interp_z<NR>(S, buf, tid);
    __syncthreads();
    sf_interp_y<NR>(S, buf, tid);
    __syncthreads();
    sf_interp_x<NR>(S, g, C, buf, tid);
    __syncthreads();
    sf_point_data<NR>(S, g, C, buf, tid);
    __syncthreads();

#define SF_S1_(DG, k, l)                                                             \
    switch (warp >> 1) {                                                             \
    case 0: sf_s1<NR, 0, DG>(S, tab[2], lane, warp & 1, k, l, C); break;             \
    case 1: sf_s1<NR, 1, DG>(S, tab[2], lane, warp & 1, k, l, C); break;             \
    case 2: sf_s1<NR, 2, DG>(S, tab[2], lane, warp & 1, k, l, C); break;             \
    default: sf_s1<NR, 3, DG>(S, tab[2], lane, warp & 1, k, l, C); break;            \
    }
#define SF_S2_(DG)                                                                   \
    if (warp < 4) sf_s2<NR, 0, DG>(S, tab[1], lane, warp & 3);                       \
    else sf_s2<NR, 1, DG>(S, tab[1], lane, warp & 3);

    while (true) {
        sf_elem En;
        const bool more = io.next(g, En);
        const double(*tab)[IGAB_TAB1D] = S.tab[buf];
        /* pairs in the order (0,0) (0,1) (0,2) (1,1) (1,2) (2,2), slots 0 1 2 3 0 4 */
        for (int p = 0; p < 6; p++) {
            const int k = p < 3 ? 0 : (p < 5 ? 1 : 2), l = p < 3 ? p : (p < 5 ? p - 2 : 2);
            const bool dg = k == l;
            if (p > 0) {
                double *Ks = SF_KSLOT(S, p == 5 ? 0 : p - 1);
                if (p == 1 || p == 4) sf_s3_all<NR, true>(S, tab[0], Ks, warp, lane);
                else sf_s3_all<NR, false>(S, tab[0], Ks, warp, lane);
            }
            if (dg) { SF_S1_(true, k, l) } else { SF_S1_(false, k, l) }
            if (p == 4) sf_fix_x<NR>(S, 0, 1, 2, 3, tid);
            __syncthreads();
            if (dg) { SF_S2_(true) } else { SF_S2_(false) }
            if (p == 0) sf_rows<NR>(S, g, E, tid);
            if (p == 3) sf_fix_zy<NR>(S, 0, 1, 2, 3, warp, lane);
            if (p == 4) io.out(S, g, E, 0, 0, 1, 2, tid);
            if (p == 5) sf_fix_zy<NR>(S, 3, 0, 0, 2, warp, lane);
            __syncthreads();
        }
        if (more) sf_load<NR>(S, g, U, En, buf ^ 1, tid);
        sf_s3_all<NR, true>(S, tab[0], SF_KSLOT(S, 4), warp, lane);
        sf_fix_x<NR>(S, 3, 0, 0, 2, tid);
        sf_copy_wait();
        __syncthreads();
        sf_fix_zy<NR>(S, 4, 4, 4, 1, warp, lane);
        io.out(S, g, E, 1, 1, 3, 0, tid);
        if (more) sf_interp_z<NR>(S, buf ^ 1, tid);
        __syncthreads();
        sf_fix_x<NR>(S, 4, 4, 4, 1, tid);
        if (more) sf_interp_y<NR>(S, buf ^ 1, tid);
        __syncthreads();
        io.out(S, g, E, 2, 2, 0, 4, tid);
        if (more) sf_interp_x<NR>(S, g, C, buf ^ 1, tid);
        __syncthreads();
        if (!more) break;
        buf ^= 1;
        E = En;
        sf_point_data<NR>(S, g, C, buf, tid);
        __syncthreads();
    }
#undef SF_S1_
#undef SF_S2_
}

/* two blocks per SM for phys/ge; the transient point data (45 KB) and its registers leave room for one */
template <typename T, int NR>
__global__ void __launch_bounds__(SF_THR, NR == 1 ? 2 : 1) k_tan_sf(igab_geom g, sf_coef C,
                                                                    const double *__restrict__ U,
                                                                    T *__restrict__ vals, int colour, int tile0)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    sf_smem<NR> &S = *reinterpret_cast<sf_smem<NR> *>(smem_raw);
    sf_tile_io<T> io;
    if (!decode_tile(g, SF_TE, colour, tile0 + blockIdx.x, io.Tl)) return;
    io.vals = vals;
    io.le = -1;
    sf_run<NR>(g, C, io, U, S);
}

/* the matrices of elements e0 .. ne - 1 into a scratch array */
template <int NR>
__global__ void __launch_bounds__(SF_THR, NR == 1 ? 2 : 1) k_tan_sf_elem(igab_geom g, sf_coef C,
                                                                         const double *__restrict__ U,
                                                                         double *__restrict__ ke, long e0, long ne,
                                                                         sf_ring ring)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    sf_smem<NR> &S = *reinterpret_cast<sf_smem<NR> *>(smem_raw);
    sf_elem_io io = {ke, e0 + (long)blockIdx.x - (long)gridDim.x, ne, ring};
    sf_run<NR>(g, C, io, U, S);
}

/* CSR values from the scratch array.  One block per control point, one thread per column (cx, cy, cz, l) of its
 * rows, the three rows together (one index computation, four loads per element).  An entry receives its at most
 * 27 element values one by one in the order of the coloured launches (colour position, then position in the
 * tile) and in the same precision, so the values equal theirs bit for bit. */
template <typename T>
__global__ void __launch_bounds__(384) k_tan_gather(igab_geom g, const double *__restrict__ ke, T *__restrict__ vals,
                                                    int order, int cp0, sf_ring ring)
{
    const int cp = cp0 + blockIdx.x, s = threadIdx.x;
    const int z = cp % g.nb[2], y = (cp / g.nb[2]) % g.nb[1], x = cp / (g.nb[2] * g.nb[1]);
    const int x0 = max(x - 2, 0), y0 = max(y - 2, 0), y1 = min(y + 2, g.nb[1] - 1);
    const int z0 = max(z - 2, 0), z1 = min(z + 2, g.nb[2] - 1);
    const int nyb = y1 - y0 + 1, nzb = z1 - z0 + 1;
    const int r0 = g.rowptr[3 * cp], len = g.rowptr[3 * cp + 1] - r0;
    if (s >= len) return;
    const int l = s % 3, c = s / 3, cz = z0 + c % nzb, cy = y0 + (c / nzb) % nyb, cx = x0 + c / (nzb * nyb);
    /* per direction the elements that hold both points, by the parity of their tile */
    const int P[3] = {x, y, z}, Q[3] = {cx, cy, cz};
    int lo[3][2], hi[3][2];
#pragma unroll
    for (int d = 0; d < 3; d++)
        elem_parity_ranges(max(max(P[d], Q[d]) - 2, 0), min(min(P[d], Q[d]), g.ne[d] - 1) + 1, lo[d], hi[d]);
    int off[3];   /* pair (min(k,l), max(k,l)) */
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int u = min(k, l), v = max(k, l);
        off[k] = 729 * (2 * u - (u >> 1) + v);
    }
    T acc[3] = {T(0), T(0), T(0)};
#pragma unroll 1
    for (int kp = 0; kp < 8; kp++) {
        const int col = igab_colour_at(order, kp), px = col >> 2, py = (col >> 1) & 1, pz = col & 1;
        for (int ex = px ? lo[0][1] : lo[0][0]; ex < (px ? hi[0][1] : hi[0][0]); ex++) {
            const int slot = ring.slot(ex);
            for (int ey = py ? lo[1][1] : lo[1][0]; ey < (py ? hi[1][1] : hi[1][0]); ey++)
                for (int ez = pz ? lo[2][1] : lo[2][0]; ez < (pz ? hi[2][1] : hi[2][0]); ez++) {
                    const double *K = ke + (((long)slot * g.ne[1] + ey) * g.ne[2] + ez) * 4374;
                    const int ax = x - ex, ay = y - ey, az = z - ez, bx = cx - ex, by = cy - ey, bz = cz - ez;
                    const int i = (3 * ax + bx) * 81 + (3 * ay + by) * 9 + 3 * az + bz;
                    const int it = (3 * bx + ax) * 81 + (3 * by + ay) * 9 + 3 * bz + az;
                    double v[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) v[k] = __ldg(K + off[k] + (k <= l ? i : it));
                    const double w = __ldg(K + off[l == 0 ? 0 : (l == 1 ? 1 : 2)] + it);
#pragma unroll
                    for (int k = 0; k < 3; k++) acc[k] += T(k == l ? v[k] + w : v[k]);
                }
        }
    }
    T *o = vals + r0 + s;
#pragma unroll
    for (int k = 0; k < 3; k++) o[(long)k * len] = acc[k];
}

/* One tile of one colour of a batch's instances per block, items from `item0` on.  A launch holds one colour position of
 * a group of instances, so the launches order the colours and neither fences nor real waits are left: one fence per
 * tile between a tile's reductions and its flag (waits inside one launch) cost 13% (48^3 as a batch of one: 10.3 ms
 * against 9.1 for the single mesh, 8.9 without fences), as it stands until the SM's reductions have drained. */
template <typename T>
__global__ void __launch_bounds__(SF_THR, 2) k_tan_sf_batch(igab_batch_dev B, int item0, const double *__restrict__ U,
                                                            T *__restrict__ vals)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    sf_smem<1> &S = *reinterpret_cast<sf_smem<1> *>(smem_raw);
    __shared__ batch_slot sl;
    if (threadIdx.x == 0) batch_item(B, sl, item0 + (int)blockIdx.x);
    __syncthreads();
    batch_stage(B, sl, false);
    sf_tile_io<T> io;
    decode_tile(sl.g, SF_TE, sl.colour, sl.tile, io.Tl);
    io.vals = vals + B.nnz_off[sl.inst];
    io.le = -1;
    const sf_coef C = sf_coef_ge(sl.g);
    sf_run<1>(sl.g, C, io, U + B.dof_off[sl.inst], S);
    batch_done(B, sl, false);
}

int sm_count(int device)
{
    int n = 0;
    return cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && n > 0 ? n : 148;
}

/* element layers ex0 .. ex1 - 1 into the scratch (of `ring` layers), then the rows they complete: those of the control
 * points x = ex0 .. ex1 - 1, of all the rest with the last layer */
template <typename T, int NR>
int launch_sf_layers(igab_ctx *c, const igab_geom &g, const sf_coef &C, const double *dU, T *dv, double *ke, int ex0,
                     int ex1, int ring)
{
    const size_t sm = sizeof(sf_smem<NR>);
    const long layer = (long)g.ne[1] * g.ne[2], ne = (ex1 - ex0) * layer, cap = (NR == 1 ? 2L : 1L) * sm_count(c->device);
    const int plane = g.nb[1] * g.nb[2], x1 = ex1 == g.ne[0] ? g.nb[0] : ex1;
    IGAB_CUDA_TRY(cudaFuncSetAttribute(k_tan_sf_elem<NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_tan_sf_elem<NR><<<(unsigned)(ne < cap ? ne : cap), SF_THR, sm, c->stream>>>(g, C, dU, ke, ex0 * layer, ex1 * layer,
                                                                                  sf_ring(ex0, ring));
    k_tan_gather<T><<<(unsigned)((x1 - ex0) * plane), 384, 0, c->stream>>>(g, ke, dv, c->colour_order, ex0 * plane,
                                                                         sf_ring(std::max(ex0 - 2, 0), ring));
    c->last_launches += 2;
    IGAB_CUDA_TRY(cudaGetLastError());
    return 0;
}

/* tx0 .. tx1: tiles along x; with ke: element layers tx0 .. tx1 through that scratch (igab_launch_tan_sf_layers) */
template <typename T, int NR>
int launch_sf(igab_ctx *c, const igab_geom &g, const sf_coef &C, const double *dU, T *dv, int tx0, int tx1, bool zero,
              double *ke = nullptr, int ring = 0)
{
    if (ke) return launch_sf_layers<T, NR>(c, g, C, dU, dv, ke, tx0, tx1, ring);
    const size_t sm = sizeof(sf_smem<NR>);
    if (tx0 == 0 && tx1 == (g.ne[0] + 1) / 2 && c->nel <= SF_ELEM_MAX) {
        int rc = igab_scratch(c, IGAB_SCRATCH_TAN, (size_t)c->nel * 4374 * sizeof(double), &ke);
        if (rc) return rc;
    }
    if (ke) {
        const int rc = launch_sf_layers<T, NR>(c, g, C, dU, dv, ke, 0, g.ne[0], g.ne[0]);
        return rc ? rc : igab_scratch_used(c);
    }
    if (zero) {
        IGAB_CUDA_TRY(cudaMemsetAsync(dv, 0, (size_t)c->nnz * sizeof(T), c->stream));
        igab_mark(c, 3);
    }
    IGAB_CUDA_TRY(cudaFuncSetAttribute(k_tan_sf<T, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    for (int k = 0; k < 8; k++) {
        const int colour = igab_colour_at(c->colour_order, k);
        long first = 0;
        const long nt = tiles_of_colour_in(g, SF_TE, colour, tx0, tx1, &first);
        if (nt == 0) continue;
        k_tan_sf<T, NR><<<(unsigned)nt, SF_THR, sm, c->stream>>>(g, C, dU, dv, colour, (int)first);
        c->last_launches++;
    }
    IGAB_CUDA_TRY(cudaGetLastError());
    return 0;
}

} /* namespace */

/* the coefficients of the transient integrand's derivative by the newest (0) or an older level; g gets its weights */
static sf_coef sf_coef_getime(igab_geom &g, int level)
{
    if (level == 1) {          /* d r / d u1 */
        const double w[4] = {0.5, 0.25, 1.0 / 6.0, 0.125};
        for (int j = 0; j < 4; j++) g.tw[j] = w[j];
        g.tmass = -2.0 * g.rho / (g.dt * g.dt);
    } else if (level == 2) {   /* d r / d u0 */
        const double w[4] = {0.25, 1.0 / 12.0, 1.0 / 24.0, 0.125};
        for (int j = 0; j < 4; j++) g.tw[j] = w[j];
        g.tmass = g.rho / (g.dt * g.dt) - g.cii / (2.0 * g.dt);
    }
    sf_coef C = sf_coef_ge(g);
    C.mass = g.tmass;
    C.r00 = sqrt(g.tw[0]);
    C.r01 = g.tw[1] / C.r00;
    C.r11 = sqrt(g.tw[2] - C.r01 * C.r01);
    C.al = 1.0 / C.r00;
    C.ga = 1.0 / C.r11;
    C.be = -C.r01 * C.al * C.ga;
    return C;
}

static int launch_sf_any(igab_ctx *c, const double *dU, void *dv, int prec, int level, int tx0, int tx1, bool zero,
                         double *ke = nullptr, int ring = 0)
{
    igab_geom g = c->geom();
    if (c->phys == IGAB_PHYS_GETIME) {
        const sf_coef C = sf_coef_getime(g, level);
        return prec == IGAB_PREC_FP64 ? launch_sf<double, 2>(c, g, C, dU, (double *)dv, tx0, tx1, zero, ke, ring)
                                      : launch_sf<float, 2>(c, g, C, dU, (float *)dv, tx0, tx1, zero, ke, ring);
    }
    const sf_coef C = sf_coef_ge(g);
    return prec == IGAB_PREC_FP64 ? launch_sf<double, 1>(c, g, C, dU, (double *)dv, tx0, tx1, zero, ke, ring)
                                  : launch_sf<float, 1>(c, g, C, dU, (float *)dv, tx0, tx1, zero, ke, ring);
}

int igab_launch_tan_sf(igab_ctx *c, const double *dU, void *dv, int prec, int tx0, int tx1, bool zero)
{
    return launch_sf_any(c, dU, dv, prec, 0, tx0, tx1, zero);
}

int igab_launch_tan_getime_level(igab_ctx *c, const double *dU, void *dv, int prec, int level, int tx0, int tx1,
                                 bool zero)
{
    return launch_sf_any(c, dU, dv, prec, level, tx0, tx1, zero);
}

/* The host entry point's tangent goes through the scratch in steps of some layers of elements along x, so that the
 * download starts after the first: a step has some four waves of elements, and the scratch holds a step and the two
 * layers before it, which its first rows need too.  An element costs 119 ns this way and 78 in large slabs of tiles, but
 * a launch of few tiles takes 133 us however few they are, and the bus 174 ns (FP64) or 87 (FP32) per element: layers
 * too large for the scratch, or half that for FP32, go by tiles.  Whole call: 24 x 21 x 26 FP64 4.0 -> 2.8 ms, FP32 3.5
 * -> 2.3, transient 4.5 -> 3.3; 16^3 1.54 -> 1.21; 40 x 36 x 36 FP64 12.1 -> 9.6, but FP32 7.9 by tiles, 8.7 this way. */
int igab_tan_sf_steps(igab_ctx *c, int prec, int *step, int *ring, double **ke)
{
    *ke = nullptr;
    const long layer = (long)c->ne[1] * c->ne[2];
    if (layer > (prec == IGAB_PREC_FP64 ? SF_LAYER_MAX : SF_LAYER_MAX / 2)) return 0;
    const long s = std::max(1L, SF_STEP / layer), r = c->nel <= SF_ELEM_MAX ? c->ne[0] : SF_ELEM_MAX / layer;
    *ring = (int)r;
    *step = (int)(r < c->ne[0] ? std::min(s, r - 2) : s);
    return igab_scratch(c, IGAB_SCRATCH_TAN, (size_t)(r * layer) * 4374 * sizeof(double), ke);
}

int igab_launch_tan_sf_layers(igab_ctx *c, const double *dU, void *dv, int prec, double *ke, int ex0, int ex1, int ring)
{
    return launch_sf_any(c, dU, dv, prec, 0, ex0, ex1, false, ke, ring);
}

template <typename T>
static int launch_sf_batch(const igab_batch_dev &B, int item0, int n, cudaStream_t st, const double *dU, T *dv)
{
    const size_t sm = sizeof(sf_smem<1>);
    if (n <= 0) return 0;
    IGAB_CUDA_TRY(cudaFuncSetAttribute(k_tan_sf_batch<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_tan_sf_batch<T><<<n, SF_THR, sm, st>>>(B, item0, dU, dv);
    IGAB_CUDA_TRY(cudaGetLastError());
    return 0;
}

int igab_launch_tan_sf_batch(const igab_batch_dev &B, int item0, int n, cudaStream_t st, const double *dU, void *dv,
                             int prec)
{
    return prec == IGAB_PREC_FP64 ? launch_sf_batch<double>(B, item0, n, st, dU, (double *)dv)
                                  : launch_sf_batch<float>(B, item0, n, st, dU, (float *)dv);
}
