// eri_low.cuh -- contracted integrals of the classes of total angular
// momentum up to 3, from Boys functions instead of Rys quadrature; included by
// gtf_dev.cuh.
//
// (ss|ss) (ps|ss) (ps|ps) (pp|ss) (ds|ss) (ds|ps) (pp|ps) (dp|ss), most of a
// build's quartets.  Per primitive quartet, with S_m = pref F_m(T), the
// Obara-Saika recurrences (S. Obara, A. Saika, J. Chem. Phys. 84, 3963 (1986))
// build only (a s|c s); (pp| and (dp| follow from (ds|, (ps| and (fs|, (ds| by
// the horizontal transfer (a b+1| = (a+1 b| + (A - B)(a b|, which does not
// depend on the primitives and is applied once, to the contracted sums.
//
// Why: the Rys kernels of these classes kept the L1 pipe 65-81% busy and the
// FP64 pipe below 50%: each primitive quartet read 10 pairs of 16 bytes per
// root from the table in shared memory.  One Boys polynomial and one
// exponential read 88 bytes whatever the class, from a table of 8 KB, and
// the recurrences take fewer operations than the products of the 2-D integrals.
#pragma once

// F_0 .. F_m of the table's intervals: row of polynomial coefficients of F_m
// in s = T - T_mid, then exp(-T_mid)
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

// F[0..M] at T; row0: the F_M rows (global or shared).  Above BOYS_TMAX exp(-T) is below the rounding of every F_m, m <= 3.
template <int M, typename R>
__device__ __forceinline__ void boys(R T, R (&F)[M + 1], const R *row0)
{
    typedef BoysTab<R> Tab;
    static_assert(M <= BOYS_MMAX, "table");
    if (T >= (R)BOYS_TMAX) {
        const R rs = grsqrt(T), it = rs * rs;
        F[0] = (R)0.886226925452758014 * rs;   // sqrt(pi) / 2
#pragma unroll
        for (int m = 0; m < M; m++) F[m + 1] = F[m] * ((R)(m + 0.5) * it);
        return;
    }
    const int k = (int)(T * (R)(1.0 / BOYS_H));
    const R s = T - ((R)k * (R)BOYS_H + (R)(0.5 * BOYS_H));
    const R *c = row0 + k * Tab::ROW;
    R f = c[Tab::DEG];
#pragma unroll
    for (int j = Tab::DEG - 1; j >= 0; j--) f = gfma(f, s, c[j]);
    F[M] = f;
    if constexpr (M > 0) {
        R e = Tab::ecoef(Tab::EDEG);
#pragma unroll
        for (int j = Tab::EDEG - 1; j >= 0; j--) e = gfma(e, s, Tab::ecoef(j));
        e *= c[Tab::DEG + 1];
        const R t2 = (R)2 * T;
#pragma unroll
        for (int m = M; m > 0; m--) {
            const R v = gfma(t2, F[m], e);
            F[m - 1] = m == 1 ? v : v * (R)(1.0 / (2 * m - 1));
        }
    }
}

__host__ __device__ constexpr bool low_class(int LA, int LB, int LC, int LD) { return LA + LB + LC + LD <= 3; }

// index of the d component ij and of the f component ijk (x = 0, y = 1, z = 2):
// with ny and nz of its factors y and z, (ny + nz)(ny + nz + 1) / 2 + nz
__host__ __device__ constexpr int cart_of(int ny, int nz) { return (ny + nz) * (ny + nz + 1) / 2 + nz; }
__host__ __device__ constexpr int d_of(int i, int j) { return cart_of((i == 1) + (j == 1), (i == 2) + (j == 2)); }
__host__ __device__ constexpr int f_of(int i, int j, int k)
{
    return cart_of((i == 1) + (j == 1) + (k == 1), (i == 2) + (j == 2) + (k == 2));
}

// contracted sums the primitive loops keep
__host__ __device__ constexpr int low_nsum(int LA, int LB, int LC)
{
    const int l = LA + LB;
    return LB == 0 ? ncart(l) * ncart(LC) : (ncart(l) + ncart(l - 1)) * ncart(LC);
}

// one primitive quartet: S[m] = pref F_m, m <= LA + LB + LC
template <int LA, int LB, int LC, typename R>
__device__ __forceinline__ void low_prim(R (&v)[low_nsum(LA, LB, LC)], const R (&S)[LA + LB + LC + 1], const R (&PA)[3],
                                         const R (&QC)[3], const R (&PQ)[3], R qf, R pf, R h2p, R hpq)
{
    constexpr int L = LA + LB, LT = L + LC;
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
            if constexpr (L == 3) {
                // (fs|ss), each component from the (ds|ss) one that needs no
                // delta term where there is such a one, and (ds|ss)
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const int d = d_of(i, i), f = f_of(i, i, k);
                        R t = gfma(PA[k], D[0][d], v[f]);
                        if (i == k) t = gfma((R)2 * h2p, gfma(-qf, P[1][k], P[0][k]), t);
                        v[f] = gfma(WP[k], D[1][d], t);
                    }
                v[4] = gfma(WP[2], D[1][1], gfma(PA[2], D[0][1], v[4]));   // xyz
#pragma unroll
                for (int d = 0; d < 6; d++) v[10 + d] += D[0][d];
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

// the quartet's integrals from the contracted sums: acc[ia + NA*(ib + NB*ic)]
template <int LA, int LB, int LC, typename R>
__device__ __forceinline__ void low_finish(const R (&v)[low_nsum(LA, LB, LC)], const R (&AB)[3],
                                           R (&acc)[ncart(LA) * ncart(LB) * ncart(LC)])
{
    if constexpr (LB == 0) {
#pragma unroll
        for (int k = 0; k < ncart(LA) * ncart(LC); k++) acc[k] = v[k];
    } else {
        constexpr int NA = ncart(LA), NU = ncart(LA + 1) * ncart(LC);
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
    }
}
