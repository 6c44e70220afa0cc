// eri_low.cuh -- contracted integrals of the classes of total angular
// momentum up to 4 (low_class), from Boys functions instead of Rys quadrature; included by
// gtf_dev.cuh.
//
// (ss|ss) (ps|ss) (ps|ps) (pp|ss) (ds|ss) (ds|ps) (pp|ps) (dp|ss), most of a
// build's quartets, and (dp|ps) (ds|pp) (ds|ds) (dd|ss).  Per primitive quartet, with S_m = pref F_m(T), the
// Obara-Saika recurrences (S. Obara, A. Saika, J. Chem. Phys. 84, 3963 (1986))
// build only (a s|c s); (pp|, (dp| and (dd| follow from these by
// the horizontal transfer (a b+1| = (a+1 b| + (A - B)(a b|, which does not
// depend on the primitives and is applied once, to the contracted sums.
//
// Why: the Rys kernels of these classes kept the L1 pipe 65-81% busy and the
// FP64 pipe below 50%: each primitive quartet read 10 pairs of 16 bytes per
// root from the table in shared memory.  One Boys polynomial and one
// exponential read 88 bytes whatever the class, from a table of 8 KB, and
// the recurrences take fewer operations than the products of the 2-D integrals.
#pragma once

// H_m = F_m / (2m - 1)!! on the table's intervals: row of polynomial
// coefficients in s = T - T_mid, then exp(-T_mid)
template <typename R>
struct BoysTab;
template <>
struct BoysTab<double> {
    static constexpr int DEG = BOYS_DEG, EDEG = BOYS_EXP_DEG, ROW = BOYS_DEG + 2, LEN = ROW * BOYS_NINT;
    static __device__ __forceinline__ const double *ptr(int m) { return BOYS_TABLE + m * LEN; }
    static __host__ __device__ constexpr double ecoef(int j)
    {
        constexpr double c[] = {BOYS_EXP_LIST};
        return c[j];
    }
};
template <>
struct BoysTab<float> {
    static constexpr int DEG = BOYS32_DEG, EDEG = BOYS32_EXP_DEG, ROW = BOYS32_DEG + 2, LEN = ROW * BOYS_NINT;
    static __device__ __forceinline__ const float *ptr(int m) { return BOYS32_TABLE + m * LEN; }
    static __host__ __device__ constexpr float ecoef(int j)
    {
        constexpr float c[] = {BOYS32_EXP_LIST};
        return c[j];
    }
};

// (2m - 1)!!, m <= 4 (no recursion: it must fold in the unrolled loops)
__host__ __device__ constexpr double boys_dfac(int m) { return m <= 1 ? 1.0 : m == 2 ? 3.0 : m == 3 ? 15.0 : 105.0; }

// F[0..M] at T; row0: the rows of H_M (global or shared).  Above BOYS_TMAX
// exp(-T) is below the rounding of every F_m, m <= 4.  Within 3 units in the
// last place below it; above, the rounding of 1 / T enters F_m m times.
template <int M, typename R>
__device__ __forceinline__ void boys(R T, R (&F)[M + 1], const R *row0)
{
    typedef BoysTab<R> Tab;
    static_assert(M <= BOYS_MMAX, "table");
    if (T >= (R)BOYS_TMAX) {
        const R rs = grsqrt(T);
        R it = rs * rs;
        it = gfma(it, gfma(-T, it, (R)1), it);   // 1 / T: one Newton step takes rsqrt's rounding out
        F[0] = (R)0.886226925452758014 * rs;   // sqrt(pi) / 2
#pragma unroll
        for (int m = 0; m < M; m++) F[m + 1] = F[m] * ((R)(m + 0.5) * it);
        return;
    }
    const int k = (int)(T * (R)(1.0 / BOYS_H));
    const R s = T - ((R)k * (R)BOYS_H + (R)(0.5 * BOYS_H));
    const R *c = row0 + k * Tab::ROW;
    R h = c[Tab::DEG];
#pragma unroll
    for (int j = Tab::DEG - 1; j >= 0; j--) h = gfma(h, s, c[j]);
    F[M] = M > 1 ? h * (R)boys_dfac(M) : h;
    if constexpr (M > 0) {
        R q = Tab::ecoef(Tab::EDEG);
#pragma unroll
        for (int j = Tab::EDEG - 1; j >= 0; j--) q = gfma(q, s, Tab::ecoef(j));
        const R E = c[Tab::DEG + 1], e = gfma(E * s, q, E);
        const R t2 = (R)2 * T;
#pragma unroll
        for (int m = M; m > 0; m--) {
            h = gfma(t2, h, m > 1 ? e * (R)(1.0 / boys_dfac(m)) : e);
            F[m - 1] = m > 2 ? h * (R)boys_dfac(m - 1) : h;
        }
    }
}

// total angular momentum up to 3, and at 4 all but (pp|pp), whose 81 sums
// outgrow the registers
__host__ __device__ constexpr bool low_class(int LA, int LB, int LC, int LD)
{
    return LA + LB + LC + LD <= 3 || (LA + LB + LC + LD == 4 && !(LA == 1 && LB == 1));
}

// index of the d component ij and of the f component ijk (x = 0, y = 1, z = 2):
// with ny and nz of its factors y and z, (ny + nz)(ny + nz + 1) / 2 + nz
__host__ __device__ constexpr int cart_of(int ny, int nz) { return (ny + nz) * (ny + nz + 1) / 2 + nz; }
__host__ __device__ constexpr int d_of(int i, int j) { return cart_of((i == 1) + (j == 1), (i == 2) + (j == 2)); }
__host__ __device__ constexpr int f_of(int i, int j, int k)
{
    return cart_of((i == 1) + (j == 1) + (k == 1), (i == 2) + (j == 2) + (k == 2));
}

// index of the g component ijkl
__host__ __device__ constexpr int g_of(int i, int j, int k, int l)
{
    return cart_of((i == 1) + (j == 1) + (k == 1) + (l == 1), (i == 2) + (j == 2) + (k == 2) + (l == 2));
}

// contracted sums the primitive loops keep: the (a s|c s) with a from LA to
// LA + LB (all three of (dd|) on LC + LD, for (ds|pp) also on LC
__host__ __device__ constexpr int low_nsum(int LA, int LB, int LC, int LD)
{
    const int l = LA + LB;
    if (LC + LD == 2) return ncart(l) * (ncart(2) + (LD == 1 ? ncart(1) : 0));
    int n = 0;
    for (int a = LA; a <= l; a++) n += ncart(a) * ncart(LC);
    return n;
}

// one primitive quartet: S[m] = pref F_m, m <= LA + LB + LC + LD
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void low_prim(R (&v)[low_nsum(LA, LB, LC, LD)], const R (&S)[LA + LB + LC + LD + 1],
                                         const R (&PA)[3], const R (&QC)[3], const R (&PQ)[3], R qf, R pf, R h2p,
                                         R h2q, R hpq)
{
    constexpr int L = LA + LB, LT = L + LC + LD;
    if constexpr (LT == 0) {
        v[0] += S[0];
    } else {
        R WP[3], P[LT][3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            WP[i] = -qf * PQ[i];
#pragma unroll
            for (int m = 0; m < LT; m++) P[m][i] = gfma(PA[i], S[m], WP[i] * S[m + 1]);
        }
        R WQ[3];
#pragma unroll
        for (int k = 0; k < 3; k++) WQ[k] = pf * PQ[k];
        if constexpr (L == 1) {
            if constexpr (LC == 0) {
#pragma unroll
                for (int i = 0; i < 3; i++) v[i] += P[0][i];
            } else {
#pragma unroll
                for (int k = 0; k < 3; k++)
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        R t = gfma(QC[k], P[0][i], v[i + 3 * k]);
                        if (i == k) t = gfma(hpq, S[1], t);
                        v[i + 3 * k] = gfma(WQ[k], P[1][i], t);
                    }
            }
        } else {
            R D[LT - 1][6];
#pragma unroll
            for (int m = 0; m < LT - 1; m++) {
                const R e = h2p * gfma(-qf, S[m + 1], S[m]);
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = i; j < 3; j++) {
                        R t = WP[j] * P[m + 1][i];
                        if (i == j) t += e;
                        D[m][d_of(i, j)] = gfma(PA[j], P[m][i], t);
                    }
            }
            if constexpr (L >= 3) {
                // (fs|ss)^m, each component from the (ds|ss) one that needs
                // no delta term where there is such a one
                R F[LT - 2][10];
#pragma unroll
                for (int m = 0; m < LT - 2; m++) {
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            R t = WP[k] * D[m + 1][d_of(i, i)];
                            if (i == k) t = gfma((R)2 * h2p, gfma(-qf, P[m + 1][k], P[m][k]), t);
                            F[m][f_of(i, i, k)] = gfma(PA[k], D[m][d_of(i, i)], t);
                        }
                    F[m][4] = gfma(PA[2], D[m][1], WP[2] * D[m + 1][1]);   // xyz
                }
                if constexpr (L == 4) {
                    // (gs|ss): xxxx.. from xxx, the others with as few delta terms as possible
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            const int f = f_of(i, i, i);
                            R t = gfma(PA[k], F[0][f], v[g_of(i, i, i, k)]);
                            if (i == k) t = gfma((R)3 * h2p, gfma(-qf, D[1][d_of(i, i)], D[0][d_of(i, i)]), t);
                            v[g_of(i, i, i, k)] = gfma(WP[k], F[1][f], t);
                        }
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const int j = (i + 1) % 3, k = (i + 2) % 3;
                        // iijj from iij, iijk from iij
                        const int f = f_of(i, i, j);
                        R t = gfma(PA[j], F[0][f], v[g_of(i, i, j, j)]);
                        t = gfma(h2p, gfma(-qf, D[1][d_of(i, i)], D[0][d_of(i, i)]), t);
                        v[g_of(i, i, j, j)] = gfma(WP[j], F[1][f], t);
                        v[g_of(i, i, j, k)] = gfma(WP[k], F[1][f], gfma(PA[k], F[0][f], v[g_of(i, i, j, k)]));
                    }
#pragma unroll
                    for (int f = 0; f < 10; f++) v[15 + f] += F[0][f];
#pragma unroll
                    for (int d = 0; d < 6; d++) v[25 + d] += D[0][d];
                } else if constexpr (LC == 0) {
#pragma unroll
                    for (int f = 0; f < 10; f++) v[f] += F[0][f];
#pragma unroll
                    for (int d = 0; d < 6; d++) v[10 + d] += D[0][d];
                } else {
#pragma unroll
                    for (int c = 0; c < 3; c++) {
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = i; j < 3; j++) {
                                R t = gfma(QC[c], D[0][d_of(i, j)], v[30 + d_of(i, j) + 6 * c]);
                                if (i == c) t = gfma(hpq, P[1][j], t);
                                if (j == c) t = gfma(hpq, P[1][i], t);
                                v[30 + d_of(i, j) + 6 * c] = gfma(WQ[c], D[1][d_of(i, j)], t);
#pragma unroll
                                for (int k = j; k < 3; k++) {
                                    const int f = f_of(i, j, k);
                                    R u = gfma(QC[c], F[0][f], v[f + 10 * c]);
                                    if (i == c) u = gfma(hpq, D[1][d_of(j, k)], u);
                                    if (j == c) u = gfma(hpq, D[1][d_of(i, k)], u);
                                    if (k == c) u = gfma(hpq, D[1][d_of(i, j)], u);
                                    v[f + 10 * c] = gfma(WQ[c], F[1][f], u);
                                }
                            }
                    }
                }
            } else if constexpr (LC + LD == 2) {
                // (ds|p_k s)^m, then (ds|d_kl s) with l >= k
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    R DP[2][6], PP[3];
#pragma unroll
                    for (int m = 0; m < 2; m++)
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = i; j < 3; j++) {
                                R t = WQ[k] * D[m + 1][d_of(i, j)];
                                if (i == k) t = gfma(hpq, P[m + 1][j], t);
                                if (j == k) t = gfma(hpq, P[m + 1][i], t);
                                DP[m][d_of(i, j)] = gfma(QC[k], D[m][d_of(i, j)], t);
                            }
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        R t = WQ[k] * P[2][i];
                        if (i == k) t = gfma(hpq, S[2], t);
                        PP[i] = gfma(QC[k], P[1][i], t);
                    }
#pragma unroll
                    for (int l = k; l < 3; l++)
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = i; j < 3; j++) {
                                const int d = d_of(i, j), o = d + 6 * d_of(k, l);
                                R t = gfma(QC[l], DP[0][d], v[o]);
                                if (k == l) t = gfma(h2q, gfma(-pf, D[1][d], D[0][d]), t);
                                if (i == l) t = gfma(hpq, PP[j], t);
                                if (j == l) t = gfma(hpq, PP[i], t);
                                v[o] = gfma(WQ[l], DP[1][d], t);
                            }
                    if constexpr (LD == 1) {
#pragma unroll
                        for (int d = 0; d < 6; d++) v[36 + d + 6 * k] += DP[0][d];
                    }
                }
            } else if constexpr (LC == 0) {
#pragma unroll
                for (int d = 0; d < 6; d++) v[d] += D[0][d];
                if constexpr (LB == 1) {
#pragma unroll
                    for (int i = 0; i < 3; i++) v[6 + i] += P[0][i];
                }
            } else {
#pragma unroll
                for (int k = 0; k < 3; k++) {
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = i; j < 3; j++) {
                            const int d = d_of(i, j);
                            R t = gfma(QC[k], D[0][d], v[d + 6 * k]);
                            if (i == k) t = gfma(hpq, P[1][j], t);
                            if (j == k) t = gfma(hpq, P[1][i], t);
                            v[d + 6 * k] = gfma(WQ[k], D[1][d], t);
                        }
                    if constexpr (LB == 1) {
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            R t = gfma(QC[k], P[0][i], v[18 + i + 3 * k]);
                            if (i == k) t = gfma(hpq, S[1], t);
                            v[18 + i + 3 * k] = gfma(WQ[k], P[1][i], t);
                        }
                    }
                }
            }
        }
    }
}

// the quartet's integrals from the contracted sums:
// acc[ia + NA*(ib + NB*(ic + NC*id))]
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void low_finish(const R (&v)[low_nsum(LA, LB, LC, LD)], const R (&AB)[3], const R (&CD)[3],
                                           R (&acc)[ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD)])
{
    constexpr int NA = ncart(LA);
    if constexpr (LD == 1) {
#pragma unroll
        for (int id = 0; id < 3; id++)
#pragma unroll
            for (int ic = 0; ic < 3; ic++)
#pragma unroll
                for (int ia = 0; ia < NA; ia++)
                    acc[ia + NA * (ic + 3 * id)] = gfma(CD[id], v[NA * 6 + ia + NA * ic], v[ia + NA * d_of(ic, id)]);
    } else if constexpr (LB == 0) {
#pragma unroll
        for (int k = 0; k < NA * ncart(LC); k++) acc[k] = v[k];
    } else if constexpr (LB == 1) {
        constexpr int NU = ncart(LA + 1) * ncart(LC);
#pragma unroll
        for (int k = 0; k < ncart(LC); k++)
#pragma unroll
            for (int ib = 0; ib < 3; ib++)
#pragma unroll
                for (int ia = 0; ia < NA; ia++) {
                    // component a + 1_b (ncart(LA + 1) of them)
                    const int up = cart_of(cart_y(LA, ia) + (ib == 1), cart_z(LA, ia) + (ib == 2));
                    acc[ia + NA * (ib + 3 * k)] = gfma(AB[ib], v[NU + ia + NA * k], v[up + ncart(LA + 1) * k]);
                }
    } else {
        // (d d_jk| = (d+1_k p_j| + AB_k (d p_j|, (x p_j| = (x+1_j| + AB_j (x|
#pragma unroll
        for (int j = 0; j < 3; j++)
#pragma unroll
            for (int k = j; k < 3; k++)
#pragma unroll
                for (int ia = 0; ia < 6; ia++) {
                    const int y = cart_y(2, ia), z = cart_z(2, ia);
                    const R fj = v[15 + cart_of(y + (j == 1), z + (j == 2))], fk = v[15 + cart_of(y + (k == 1), z + (k == 2))];
                    const R gjk = v[cart_of(y + (j == 1) + (k == 1), z + (j == 2) + (k == 2))];
                    const R up = gfma(AB[j], fk, gjk), low = gfma(AB[j], v[25 + ia], fj);
                    acc[ia + 6 * d_of(j, k)] = gfma(AB[k], low, up);
                }
    }
}
