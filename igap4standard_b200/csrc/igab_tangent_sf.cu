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
 * are one m8 tile without the pair (1, 1), plus the total sum_q B.  As the three functions sum to 1
 * (and their derivatives to 0), the entry (1, 1) is the total minus the other eight, so the eight rows
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
 * Measured at 64^3 (tangent alone): 22.3 ms, FP64 and FP32 values, against 96.6 ms for the rank-12 form
 * on the same pipe and 40.4 ms for its TF32 tcgen05 form; the FP32 values' error against 64 bits falls
 * from 1.3e-6 to 8e-8.  Bound by shared memory (17,300 wavefronts per element, 60-70% of the rate);
 * the products take 7,500 cycles of the pipe.
 */
#include <cuda_runtime.h>
#include <type_traits>
#include "igab_device.cuh"

namespace {

#define SF_THR 256
#define SF_TE 2

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
enum { P_F = 0, P_G = 9, P_W = 27, P_CN = 28, P_S = 34, P_TAU = 40, P_N = 49 };

struct sf_row { long rb; int rsx, rsy, len, pad; };

struct sf_smem {
    double pt[P_N * 64];
    double T1[36 * 128];     /* [class pair][8 pairs (az,bz)][16 columns], 16-byte chunks swizzled */
    double T1x[25 * 16];     /* z totals of the class pairs without z derivative */
    double T2[9 * 288];      /* [kx,lx][9 (ay,by)][4 qx][8 (az,bz)], swizzled */
    double T2x[9 * 36];      /* z totals [kx,lx][9 (ay,by)][4 qx] */
    double K[4 * 729];       /* element matrices of component pairs, [9 (ax,bx)][9 (ay,by)][9 (az,bz)] */
    double tab[2][3][IGAB_TAB1D];
    double wh[2][3][IGAB_NQ];
    double esc[2];
    sf_row row[27];
};
/* the staging of the next element's field and the fifth element-matrix slot use T1 / T1x, which are free then */
#define SF_A(S) ((S).T1)
#define SF_C(S) ((S).T1 + 972)
#define SF_U(S) ((S).T1x)
#define SF_KSLOT(S, s) ((s) < 4 ? (S).K + 729 * (s) : (S).T1 + 2048)

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
__device__ __forceinline__ double sum4(double v)
{
    v += shfl_xor(v, 1);
    return v + shfl_xor(v, 2);
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
struct sf_point {
    double f[3], h[3], g[6], y[6];   /* F and second derivatives of k and l */
    double won, woff, wsh;           /* w * 2 le^2 (2/3, -1/3), w * e345 / 2 */
    double cn[6], s[6], tau[9];
};

/* w D_mn of the point */
template <bool DG, int m, int n>
__device__ __forceinline__ double sf_d(const sf_point &P)
{
    if constexpr (m < 3 && n < 3) {
        constexpr int I = m, J = n, M1 = (I + 1) % 3, M2 = (I + 2) % 3;
        const double t = P.g[sym6(I, 0)] * P.y[sym6(J, 0)] + P.g[sym6(I, 1)] * P.y[sym6(J, 1)] +
                         P.g[sym6(I, 2)] * P.y[sym6(J, 2)];
        double v = (I == J ? P.won : P.woff) * t + P.cn[sym6(I, J)] * (P.f[I] * P.h[J]);
        if constexpr (I != J) v += P.wsh * (P.f[J] * P.h[I]);
        else v += P.wsh * (P.f[M1] * P.h[M1] + P.f[M2] * P.h[M2]);
        if constexpr (DG) v += P.s[sym6(I, J)];
        return v;
    } else if constexpr (m < 3) {
        constexpr int I = m, J = s_i(n - 3), K = s_k(n - 3);
        double v = P.g[sym6(I, K)] * ((I == J ? P.won : P.woff) * P.h[J]);
        if constexpr (J != K) v += P.g[sym6(I, J)] * ((I == K ? P.won : P.woff) * P.h[K]);
        if constexpr (DG && I == J) v += P.tau[3 * I + K];
        else if constexpr (DG && I == K) v += P.tau[3 * I + J];
        return v;
    } else if constexpr (n < 3) {
        constexpr int J = n, I = s_i(m - 3), K = s_k(m - 3);
        double v = ((I == J ? P.won : P.woff) * P.f[I]) * P.y[sym6(J, K)];
        if constexpr (I != K) v += ((K == J ? P.won : P.woff) * P.f[K]) * P.y[sym6(J, I)];
        if constexpr (DG && J == I) v += P.tau[3 * J + K];
        else if constexpr (DG && J == K) v += P.tau[3 * J + I];
        return v;
    } else {
        /* over the orderings (I, K) of m and (J, L) of n with K = L: A_IJ f_I h_J */
        constexpr int i0 = s_i(m - 3), k0 = s_k(m - 3), j0 = s_i(n - 3), l0 = s_k(n - 3);
        double v = 0.0;
        if constexpr (k0 == l0) v += P.f[i0] * ((i0 == j0 ? P.won : P.woff) * P.h[j0]);
        if constexpr (i0 != k0 && i0 == l0) v += P.f[k0] * ((k0 == j0 ? P.won : P.woff) * P.h[j0]);
        if constexpr (j0 != l0 && k0 == j0) v += P.f[i0] * ((i0 == l0 ? P.won : P.woff) * P.h[l0]);
        if constexpr (i0 != k0 && j0 != l0 && i0 == j0) v += P.f[k0] * ((k0 == l0 ? P.won : P.woff) * P.h[l0]);
        return v;
    }
}

/* first step: the class pairs of group G, for the 8 columns of half h */
template <int G, bool DG>
__device__ __forceinline__ void sf_s1(sf_smem &S, const double *tz, int lane, int h, int k, int l, double aon,
                                      double aoff, double ash)
{
    double w[9];
    sf_weights(tz, lane, w);
    const double *p = S.pt + h * 32 + lane;
    sf_point P;
#pragma unroll
    for (int J = 0; J < 3; J++) {
        P.f[J] = p[(P_F + 3 * k + J) * 64];
        P.h[J] = DG ? P.f[J] : p[(P_F + 3 * l + J) * 64];
    }
#pragma unroll
    for (int c = 0; c < 6; c++) {
        P.g[c] = p[(P_G + 6 * k + c) * 64];
        P.y[c] = DG ? P.g[c] : p[(P_G + 6 * l + c) * 64];
        P.cn[c] = p[(P_CN + c) * 64];
        P.s[c] = DG ? p[(P_S + c) * 64] : 0.0;
    }
#pragma unroll
    for (int c = 0; c < 9; c++) P.tau[c] = DG ? p[(P_TAU + c) * 64] : 0.0;
    const double wq = p[P_W * 64];
    P.won = wq * aon;
    P.woff = wq * aoff;
    P.wsh = wq * ash;
    const int r = lane >> 2;
    /* row r, chunk 4 h + lane % 4 of two columns; chunks are XORed so that these stores and the second
     * step's loads (4 rows x 4 qy) hit distinct banks */
    double *t1 = S.T1 + r * 16 + 2 * ((4 * h + (lane & 3)) ^ (4 * (r & 1) + (r & 2)));
    double *t1x = S.T1x + 8 * h + r;
    static_for<0, 36>([&](auto cd_) {
        constexpr int cd = decltype(cd_)::value, c = cd / 6, d = cd % 6;
        if constexpr (cls_nonzero(c, d) && !(DG && c > d) && cls_group(DG, c, d) == G) {
            double c0 = 0.0, c1 = 0.0;
            static_for<0, 9>([&](auto kk_) {
                constexpr int kk = decltype(kk_)::value, kz = kk / 3, lz = kk % 3, m = sf_comp(c, kz), n = sf_comp(d, lz);
                if constexpr (m >= 0 && n >= 0) {
                    if constexpr (mn_nonzero(m, n) && !(DG && !mn_upper(m, n))) {
                        double v = sf_d<DG, m, n>(P);
                        if constexpr (DG && m == n) v *= 0.5;
                        sf_dmma(c0, c1, w[kk], v);
                        if constexpr (kk == 0) {
                            const double t = sum4(v);
                            if ((lane & 3) == 0) t1x[((c - 1) * 5 + d - 1) * 16] = t;
                        }
                    }
                }
            });
            *reinterpret_cast<double2 *>(t1 + cd * 128) = make_double2(c0, c1);
        }
    });
}

/* second step: the (kx, lx) of the half, for one qx */
template <int HALF, bool DG>
__device__ __forceinline__ void sf_s2(sf_smem &S, const double *ty, int lane, int qx)
{
    double w[9];
    sf_weights(ty, lane, w);
    const int n = lane >> 2, q = lane & 3;
    const double *t1 = S.T1 + n * 16 + 2 * ((2 * qx + (q >> 1)) ^ (4 * (n & 1) + (n & 2))) + (q & 1);
    const int id = pair_id(n);
    /* T2 row (ay,by), 8 doubles per qx: qx flips with the row's parity and the (az,bz) halves with qx / 2,
     * so that 2-row stores and 4-qx loads hit distinct banks */
    double *t2 = S.T2 + id * 32 + ((qx ^ (id & 1)) << 3) + ((2 * q) ^ (4 * (qx >> 1)));
    double *t2y = S.T2 + 4 * 32 + (qx << 3) + (n ^ (4 * (qx >> 1)));
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
                        const double t = sum4(b);
                        if (q == 0) t2y[X * 288] = t;
                    }
                }
            });
            *reinterpret_cast<double2 *>(t2 + X * 288) = make_double2(c0, c1);
            if (qx == x_zwarp(DG, X)) {
                /* z totals, all four qx as columns */
                const double *t1x = S.T1x + (n & 3) * 4 + q;
                c0 = c1 = 0.0;
                static_for<0, 36>([&](auto cd_) {
                    constexpr int cd = decltype(cd_)::value, c = cd / 6, d = cd % 6, kl = 3 * cls_ky(c) + cls_ky(d);
                    if constexpr (c > 0 && d > 0 && cls_kx(c) == kx && cls_kx(d) == lx && cls_nonzero(c, d) &&
                                  !(DG && c > d)) {
                        const double b = n < 4 ? t1x[((c - 1) * 5 + d - 1) * 16] : 0.0;
                        sf_dmma(c0, c1, w[kl], b);
                        if constexpr (kl == 0) {
                            const double t = sum4(b);
                            if (q == 0 && n < 4) S.T2x[X * 36 + 16 + n] = t;
                        }
                    }
                });
                if (q < 2) *reinterpret_cast<double2 *>(S.T2x + X * 36 + id * 4 + 2 * q) = make_double2(c0, c1);
            }
        }
    });
}

/* third step into an element-matrix slot: one tile of eight (az,bz) columns per (ay,by), then the z totals */
template <bool DG>
__device__ __forceinline__ void sf_s3(sf_smem &S, const double *tx, double *K, int warp, int lane)
{
    double w[9];
    sf_weights(tx, lane, w);
    const int n = lane >> 2, q = lane & 3;
    const int xr = pair_id(n) * 81;
    for (int t = warp; t < 11; t += 8) {
        double c0 = 0.0, c1 = 0.0;
        if (t < 9) {
            const double *t2 = S.T2 + t * 32 + ((q ^ (t & 1)) << 3) + (n ^ (4 * (q >> 1)));
#pragma unroll
            for (int X = 0; X < 9; X++) {
                if (DG && X / 3 > X % 3) continue;
                const double b = t2[X * 288];
                sf_dmma(c0, c1, w[X], b);
                if (X == 0) {
                    const double s = sum4(b);
                    if (q == 0) K[4 * 81 + t * 9 + pair_id(n)] = s;
                }
            }
            K[xr + t * 9 + pair_id(2 * q)] = c0;
            K[xr + t * 9 + pair_id(2 * q + 1)] = c1;
        } else if (t == 9) {
            const double *t2 = S.T2x + pair_id(n) * 4 + q;
#pragma unroll
            for (int X = 0; X < 9; X++) {
                if (DG && X / 3 > X % 3) continue;
                const double b = t2[X * 36];
                sf_dmma(c0, c1, w[X], b);
                if (X == 0) {
                    const double s = sum4(b);
                    if (q == 0) K[4 * 81 + pair_id(n) * 9 + 4] = s;
                }
            }
            K[xr + pair_id(2 * q) * 9 + 4] = c0;
            K[xr + pair_id(2 * q + 1) * 9 + 4] = c1;
        } else {
            /* totals in y and z: only where both derivatives are in x */
#pragma unroll
            for (int X = 0; X < 9; X++) {
                if (X / 3 == 0 || X % 3 == 0 || (DG && X / 3 > X % 3)) continue;
                const double b = n == 0 ? S.T2x[X * 36 + 16 + q] : 0.0;
                sf_dmma(c0, c1, w[X], b);
            }
            if (q == 0) K[xr + 4 * 9 + 4] = c0;
            if (lane == 0) K[4 * 81 + 4 * 9 + 4] = 0.0;
        }
    }
}

/* totals -> entries (1, 1) in z, then y, of slots s0, s1, s2 (the first ns): a warp per three (ax,bx) */
__device__ __forceinline__ void sf_fix_zy(sf_smem &S, int s0, int s1, int s2, int ns, int warp, int lane)
{
    for (int u = warp; u < 3 * ns; u += 8) {
        const int sl = u / 3, j = u % 3;
        double *K = SF_KSLOT(S, sl == 0 ? s0 : (sl == 1 ? s1 : s2)) + (3 * j + lane / 9) * 81;
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
__device__ __forceinline__ void sf_fix_x(sf_smem &S, int s0, int s1, int s2, int ns, int tid)
{
    if (tid < 81 * ns) {
        const int sl = tid / 81;
        double *z = SF_KSLOT(S, sl == 0 ? s0 : (sl == 1 ? s1 : s2)) + tid % 81;
        z[324] -= ((z[0] + z[81]) + (z[162] + z[243])) + ((z[405] + z[486]) + (z[567] + z[648]));
    }
}

/* Add rows (a, k), a = 0..26, into the CSR values: sl[l] is the slot of pair (min(k,l), max(k,l)).
 * A thread owns one column c2 = 3 b + l and walks the 9 rows of one ax, so consecutive lanes add to runs
 * of 9 consecutive values and the index arithmetic of a row is three multiply-adds. */
template <typename T>
__device__ __forceinline__ void sf_scatter(sf_smem &S, T *__restrict__ vals, int k, int s0, int s1, int s2, int tid)
{
    if (tid >= 243) return;
    const int j = tid / 81, c = tid - 81 * j, l = c % 3, b = c / 3;
    const int bx = b / 9, by = (b / 3) % 3, bz = b % 3;
    const double *Kl = SF_KSLOT(S, l == 0 ? s0 : (l == 1 ? s1 : s2));
    const double *Kn = Kl + (3 * j + bx) * 81 + by * 9 + bz;       /* (a, b), + 27 ay + 3 az */
    const double *Kt = Kl + (3 * bx + j) * 81 + by * 27 + bz * 3;  /* (b, a), + 9 ay + az */
    T *v = vals + c % 9;
#pragma unroll
    for (int ay = 0; ay < 3; ay++)
#pragma unroll
        for (int az = 0; az < 3; az++) {
            const sf_row &R = S.row[9 * j + 3 * ay + az];
            double x = l >= k ? Kn[27 * ay + 3 * az] : Kt[9 * ay + az];
            if (l == k) x += Kt[9 * ay + az];
            atomicAdd(v + R.rb + k * R.len + bx * R.rsx + by * R.rsy, T(x));
        }
}

/* ---- the field of an element: loads, three interpolation steps, point data */
struct sf_elem { int ex, ey, ez; };

/* one value per thread: 81 of U, 108 of the 1-D tables, 12 weights, the element scale */
__device__ __forceinline__ double sf_prefetch(const igab_geom &g, const double *__restrict__ U, const sf_elem &E,
                                              int tid)
{
    if (tid < 81) {
        const int i = tid % 3, a = tid / 3;
        return U[3 * cp_index(g, E.ex + a / 9, E.ey + (a / 3) % 3, E.ez + a % 3) + i];
    }
    if (tid < 189) {
        const int d = (tid - 81) / 36, o = (tid - 81) % 36, e = d == 0 ? E.ex : (d == 1 ? E.ey : E.ez);
        return g.tab[d][(long)e * IGAB_TAB1D + o];
    }
    if (tid < 201) {
        const int d = (tid - 189) >> 2, o = (tid - 189) & 3, e = d == 0 ? E.ex : (d == 1 ? E.ey : E.ez);
        return g.wh[d][(long)e * IGAB_NQ + o];
    }
    return tid == 201 ? elem_scale(g, E.ex, E.ey, E.ez) : 0.0;
}
__device__ __forceinline__ void sf_stage(sf_smem &S, double v, int buf, int tid)
{
    if (tid < 81) SF_U(S)[tid] = v;
    else if (tid < 189) (&S.tab[buf][0][0])[tid - 81] = v;
    else if (tid < 201) (&S.wh[buf][0][0])[tid - 189] = v;
    else if (tid == 201) S.esc[buf] = v;
}
__device__ __forceinline__ void sf_interp_z(sf_smem &S, int buf, int tid)
{
    const double *Bz = S.tab[buf][2];
    for (int o = tid; o < 972; o += SF_THR) {
        const int i = o % 3, kz = (o / 3) % 3, a = (o / 9) % 9, q = o / 81;
        const double *u0 = SF_U(S) + a * 9 + i;
        SF_A(S)[o] = Bz[q * 9 + kz] * u0[0] + Bz[q * 9 + 3 + kz] * u0[3] + Bz[q * 9 + 6 + kz] * u0[6];
    }
}
__device__ __forceinline__ void sf_interp_y(sf_smem &S, int buf, int tid)
{
    const double *By = S.tab[buf][1];
    for (int o = tid; o < 864; o += SF_THR) {
        const int i = o % 3, kk = (o / 3) % 6, ax = (o / 18) % 3, qq = o / 54;
        const int qy = qq & 3, qz = qq >> 2, ky = kk_ky(kk), kz = kk_kz(kk);
        const double *a0 = SF_A(S) + ((qz * 3 + ax) * 3) * 9 + kz * 3 + i;
        SF_C(S)[o] = By[qy * 9 + ky] * a0[0] + By[qy * 9 + 3 + ky] * a0[9] + By[qy * 9 + 6 + ky] * a0[18];
    }
}
/* F and G of component tid / 64 at point tid % 64 */
__device__ __forceinline__ void sf_interp_x(sf_smem &S, const igab_geom &g, int buf, int tid)
{
    if (tid >= 192) return;
    const int i = tid >> 6, p = tid & 63, qz = p & 3, qy = (p >> 2) & 3, qx = p >> 4;
    const double *C = SF_C(S) + (qy + 4 * qz) * 54 + i;
    const double *Bx = S.tab[buf][0] + qx * 9;
    double b[3][3];
#pragma unroll
    for (int ax = 0; ax < 3; ax++)
#pragma unroll
        for (int k = 0; k < 3; k++) b[ax][k] = Bx[ax * 3 + k];
#pragma unroll
    for (int a = 1; a < 10; a++) {
        double s = 0.0;
#pragma unroll
        for (int ax = 0; ax < 3; ax++) s += b[ax][a_kx(a)] * C[(ax * 6 + a_kk(a)) * 3];
        if (a < 4) {
            if (g.periodic) s += g.pp[3 * i + a - 1];
            if (i == a - 1) s += 1.0;
            S.pt[(P_F + 3 * i + a - 1) * 64 + p] = s;
        } else
            S.pt[(P_G + 6 * i + a - 4) * 64 + p] = s;
    }
}
/* strains and stresses: warps 0-1 the strain part (CN, S), warps 2-7 TAU for one K each */
__device__ __forceinline__ void sf_point_data(sf_smem &S, const igab_geom &g, const sf_elem &E, int buf, int tid)
{
    const int p = tid & 63, qz = p & 3, qy = (p >> 2) & 3, qx = p >> 4;
    double *pt = S.pt + p;
    const double w = S.wh[buf][0][qx] * S.wh[buf][1][qy] * S.wh[buf][2][qz] * S.esc[buf];
    double F[3][3];
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int J = 0; J < 3; J++) F[k][J] = pt[(P_F + 3 * k + J) * 64];
    if (tid < 64) {
        const double is2 = IGAB_INV_SQRT2, is3 = IGAB_INV_SQRT3, is6 = IGAB_INV_SQRT6;
        double e[6];
#pragma unroll
        for (int c = 0; c < 6; c++) {
            const int I = s_i(c), J = s_k(c);
            e[c] = 0.5 * (F[0][I] * F[0][J] + F[1][I] * F[1][J] + F[2][I] * F[2][J] - (I == J ? 1.0 : 0.0));
        }
        const double vv = (e[0] + e[3] + e[5]) * is3, va = (e[0] - e[3]) * is2, vb = (e[0] + e[3] - 2.0 * e[5]) * is6;
        const double c36 = g.coef.c36, c37 = g.coef.c37, c38 = g.coef.c38;
        const double s2 = va * va + vb * vb;
        const double d0 = 2.0 * g.coef.p2 * vv;
        const double da = -6.0 * c36 * va * vb + 2.0 * c37 * va + 4.0 * c38 * s2 * va;
        const double db = 3.0 * c36 * (vb * vb - va * va) + 2.0 * c37 * vb + 4.0 * c38 * s2 * vb;
        const double h0 = 2.0 * g.coef.p2;
        const double haa = -6.0 * c36 * vb + 2.0 * c37 + 4.0 * c38 * (3.0 * va * va + vb * vb);
        const double hbb = 6.0 * c36 * vb + 2.0 * c37 + 4.0 * c38 * (va * va + 3.0 * vb * vb);
        const double hab = -6.0 * c36 * va + 8.0 * c38 * va * vb;
        /* CN_IJ = d2 Phi / dE_II dE_JJ through (vvol, va, vb) */
        const double a0 = h0 * (1.0 / 3.0), a1 = haa * 0.5, a2 = hbb * (1.0 / 6.0), a3 = hab * (is2 * is6);
        pt[P_W * 64] = w;
        pt[(P_CN + 0) * 64] = w * (a0 + a1 + a2 + 2.0 * a3);
        pt[(P_CN + 1) * 64] = w * (a0 - a1 + a2);
        pt[(P_CN + 2) * 64] = w * (a0 - 2.0 * a2 - 2.0 * a3);
        pt[(P_CN + 3) * 64] = w * (a0 + a1 + a2 - 2.0 * a3);
        pt[(P_CN + 4) * 64] = w * (a0 - 2.0 * a2 + 2.0 * a3);
        pt[(P_CN + 5) * 64] = w * (a0 + 4.0 * a2);
        pt[(P_S + 0) * 64] = w * (d0 * is3 + da * is2 + db * is6);
        pt[(P_S + 3) * 64] = w * (d0 * is3 - da * is2 + db * is6);
        pt[(P_S + 5) * 64] = w * (d0 * is3 - 2.0 * db * is6);
        pt[(P_S + 1) * 64] = w * g.coef.p3 * e[1];
        pt[(P_S + 2) * 64] = w * g.coef.p3 * e[2];
        pt[(P_S + 4) * 64] = w * g.coef.p3 * e[4];
    } else {
        const int K = (tid >> 6) - 1;
        double ek[3];
#pragma unroll
        for (int I = 0; I < 3; I++) {
            const int c = igab_idx6(I, K);
            ek[I] = F[0][I] * pt[(P_G + c) * 64] + F[1][I] * pt[(P_G + 6 + c) * 64] + F[2][I] * pt[(P_G + 12 + c) * 64];
        }
        const double m = (ek[0] + ek[1] + ek[2]) * (1.0 / 3.0), wa = w * 2.0 * g.coef.p4sq;
#pragma unroll
        for (int I = 0; I < 3; I++) pt[(P_TAU + 3 * I + K) * 64] = wa * (ek[I] - m);
    }
    if (tid < 27) {
        sf_row &R = S.row[tid];
        elem_row_base(g, E.ex, E.ey, E.ez, 3 * tid, R.rb, R.rsx, R.rsy);
        const int x = E.ex + tid / 9;
        const int x0 = x > 2 ? x - 2 : 0, x1 = x + 2 < g.nb[0] - 1 ? x + 2 : g.nb[0] - 1;
        R.len = (x1 - x0 + 1) * R.rsx;
    }
}

/* the element of a tile at or after position le (8: none), le = 4 dx + 2 dy + dz */
__device__ __forceinline__ int sf_next(const tile_t &T, int le)
{
    while (le < 8 && ((le >> 2) >= T.nv[0] || ((le >> 1) & 1) >= T.nv[1] || (le & 1) >= T.nv[2])) le++;
    return le;
}

template <typename T>
__device__ __forceinline__ void sf_tile(const igab_geom &g, const tile_t &Tl, const double *__restrict__ U,
                                        T *__restrict__ vals, sf_smem &S)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const double aon = g.coef.p4sq * (4.0 / 3.0), aoff = g.coef.p4sq * (-2.0 / 3.0), ash = g.coef.p3 * 0.5;
    int le = sf_next(Tl, 0), buf = 0;
    sf_elem E = {Tl.e0[0] + (le >> 2), Tl.e0[1] + ((le >> 1) & 1), Tl.e0[2] + (le & 1)};
    sf_stage(S, sf_prefetch(g, U, E, tid), buf, tid);
    __syncthreads();
    sf_interp_z(S, buf, tid);
    __syncthreads();
    sf_interp_y(S, buf, tid);
    __syncthreads();
    sf_interp_x(S, g, buf, tid);
    __syncthreads();
    sf_point_data(S, g, E, buf, tid);
    __syncthreads();

#define SF_S1_(DG, k, l)                                                                              \
    switch (warp >> 1) {                                                                              \
    case 0: sf_s1<0, DG>(S, S.tab[buf][2], lane, warp & 1, k, l, aon, aoff, ash); break;              \
    case 1: sf_s1<1, DG>(S, S.tab[buf][2], lane, warp & 1, k, l, aon, aoff, ash); break;              \
    case 2: sf_s1<2, DG>(S, S.tab[buf][2], lane, warp & 1, k, l, aon, aoff, ash); break;              \
    default: sf_s1<3, DG>(S, S.tab[buf][2], lane, warp & 1, k, l, aon, aoff, ash); break;             \
    }
#define SF_S2_(DG)                                                                                    \
    if (warp < 4) sf_s2<0, DG>(S, S.tab[buf][1], lane, warp & 3);                                     \
    else sf_s2<1, DG>(S, S.tab[buf][1], lane, warp & 3);

    while (true) {
        const int ln = sf_next(Tl, le + 1);
        double pre = 0.0;
        sf_elem En = E;
        /* pairs in the order (0,0) (0,1) (0,2) (1,1) (1,2) (2,2), slots 0 1 2 3 0 4 */
        for (int p = 0; p < 6; p++) {
            const int k = p < 3 ? 0 : (p < 5 ? 1 : 2), l = p < 3 ? p : (p < 5 ? p - 2 : 2);
            const bool dg = k == l;
            if (p > 0) {
                double *Ks = SF_KSLOT(S, p == 5 ? 0 : p - 1);
                if (p == 1 || p == 4) sf_s3<true>(S, S.tab[buf][0], Ks, warp, lane);
                else sf_s3<false>(S, S.tab[buf][0], Ks, warp, lane);
            }
            if (dg) { SF_S1_(true, k, l) } else { SF_S1_(false, k, l) }
            if (p == 4) sf_fix_x(S, 0, 1, 2, 3, tid);
            __syncthreads();
            if (dg) { SF_S2_(true) } else { SF_S2_(false) }
            if (p == 3) sf_fix_zy(S, 0, 1, 2, 3, warp, lane);
            if (p == 4) sf_scatter<T>(S, vals, 0, 0, 1, 2, tid);
            if (p == 5) {
                sf_fix_zy(S, 3, 0, 0, 2, warp, lane);
                if (ln < 8) {
                    En = {Tl.e0[0] + (ln >> 2), Tl.e0[1] + ((ln >> 1) & 1), Tl.e0[2] + (ln & 1)};
                    pre = sf_prefetch(g, U, En, tid);
                }
            }
            __syncthreads();
        }
        sf_s3<true>(S, S.tab[buf][0], SF_KSLOT(S, 4), warp, lane);
        sf_fix_x(S, 3, 0, 0, 2, tid);
        if (ln < 8) sf_stage(S, pre, buf ^ 1, tid);
        __syncthreads();
        sf_fix_zy(S, 4, 4, 4, 1, warp, lane);
        sf_scatter<T>(S, vals, 1, 1, 3, 0, tid);
        if (ln < 8) sf_interp_z(S, buf ^ 1, tid);
        __syncthreads();
        sf_fix_x(S, 4, 4, 4, 1, tid);
        if (ln < 8) sf_interp_y(S, buf ^ 1, tid);
        __syncthreads();
        sf_scatter<T>(S, vals, 2, 2, 0, 4, tid);
        if (ln < 8) sf_interp_x(S, g, buf ^ 1, tid);
        __syncthreads();
        if (ln >= 8) break;
        buf ^= 1;
        le = ln;
        E = En;
        sf_point_data(S, g, E, buf, tid);
        __syncthreads();
    }
#undef SF_S1_
#undef SF_S2_
}

template <typename T>
__global__ void __launch_bounds__(SF_THR, 2) k_tan_sf(igab_geom g, const double *__restrict__ U, T *__restrict__ vals,
                                                      int colour, int tile0)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    sf_smem &S = *reinterpret_cast<sf_smem *>(smem_raw);
    tile_t Tl;
    if (!decode_tile(g, SF_TE, colour, tile0 + blockIdx.x, Tl)) return;
    sf_tile<T>(g, Tl, U, vals, S);
}

/* persistent over the tiles of every instance of a batch */
template <typename T>
__global__ void __launch_bounds__(SF_THR, 2) k_tan_sf_batch(igab_batch_dev B, const double *__restrict__ U,
                                                            T *__restrict__ vals)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    sf_smem &S = *reinterpret_cast<sf_smem *>(smem_raw);
    __shared__ batch_slot sl;
    while (batch_next(B, sl)) {
        tile_t Tl;
        decode_tile(sl.g, SF_TE, sl.colour, sl.tile, Tl);
        sf_tile<T>(sl.g, Tl, U + B.dof_off[sl.inst], vals + B.nnz_off[sl.inst], S);
        batch_done(B, sl);
    }
}

template <typename T>
int launch_sf(igab_ctx *c, const double *dU, T *dv, int tx0, int tx1)
{
    const igab_geom g = c->geom();
    const size_t sm = sizeof(sf_smem);
    IGAB_CUDA_TRY(cudaFuncSetAttribute(k_tan_sf<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    for (int k = 0; k < 8; k++) {
        const int colour = igab_colour_at(c->colour_order, k);
        long first = 0;
        const long nt = tiles_of_colour_in(g, SF_TE, colour, tx0, tx1, &first);
        if (nt == 0) continue;
        k_tan_sf<T><<<(unsigned)nt, SF_THR, sm, c->stream>>>(g, dU, dv, colour, (int)first);
        c->last_launches++;
    }
    IGAB_CUDA_TRY(cudaGetLastError());
    return 0;
}

} /* namespace */

int igab_launch_tan_sf(igab_ctx *c, const double *dU, void *dv, int prec, int tx0, int tx1)
{
    return prec == IGAB_PREC_FP64 ? launch_sf<double>(c, dU, (double *)dv, tx0, tx1)
                                  : launch_sf<float>(c, dU, (float *)dv, tx0, tx1);
}

template <typename T>
static int launch_sf_batch(const igab_batch_dev &B, int grid, cudaStream_t st, const double *dU, T *dv)
{
    const size_t sm = sizeof(sf_smem);
    IGAB_CUDA_TRY(cudaFuncSetAttribute(k_tan_sf_batch<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_tan_sf_batch<T><<<grid, SF_THR, sm, st>>>(B, dU, dv);
    IGAB_CUDA_TRY(cudaGetLastError());
    return 0;
}

int igab_launch_tan_sf_batch(const igab_batch_dev &B, int grid, cudaStream_t st, const double *dU, void *dv, int prec)
{
    return prec == IGAB_PREC_FP64 ? launch_sf_batch<double>(B, grid, st, dU, (double *)dv)
                                  : launch_sf_batch<float>(B, grid, st, dU, (float *)dv);
}

template <typename T>
static int occupancy_sf(int *per_sm)
{
    const size_t sm = sizeof(sf_smem);
    IGAB_CUDA_TRY(cudaFuncSetAttribute(k_tan_sf_batch<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    IGAB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_tan_sf_batch<T>, SF_THR, sm));
    return 0;
}

int igab_batch_occupancy_tan(int prec, int *per_sm)
{
    return prec == IGAB_PREC_FP64 ? occupancy_sf<double>(per_sm) : occupancy_sf<float>(per_sm);
}
