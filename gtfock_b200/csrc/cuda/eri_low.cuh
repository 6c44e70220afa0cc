// eri_low.cuh -- contracted integrals of the classes of total angular
// momentum up to 4 (low_class), from Boys functions instead of Rys quadrature; included by
// gtf_dev.cuh.
//
// (ss|ss) (ps|ss) (ps|ps) (pp|ss) (ds|ss) (ds|ps) (pp|ps) (dp|ss), most of a
// build's quartets, and (dp|ps) (ds|pp) (ds|ds) (dd|ss).  Per primitive
// quartet, with S_m = pref F_m(T), the Obara-Saika recurrences (S. Obara,
// A. Saika, J. Chem. Phys. 84, 3963 (1986)) raise every index about its own
// centre.
//
// Why: the Rys kernels of these classes kept the L1 pipe 65-81% busy and the
// FP64 pipe below 50%: each primitive quartet read 10 pairs of 16 bytes per
// root from the table in shared memory.  One Boys polynomial and one
// exponential read 88 bytes whatever the class, from a table of 8 KB, and
// the recurrences take fewer operations than the products of the 2-D integrals.
//
// Accuracy: over random contracted quartets (tests/host/eri_accuracy.cpp) the
// error relative to a quartet's largest integral is 0.7 to 1.0 times that of
// the Rys form in FP64 and in FP32, for two reasons.  (pp|, (dp|, (dd| and |pp)
// are raised with P - B (Q - D); moving the second index by the horizontal
// transfer (a b+1| = (a+1 b| + (A - B)(a b|, on the contracted sums, cancels
// where P is close to B: 1.3 to 2.8 times the error of the Rys form.  And the
// last step to an integral is summed before it is added to acc, one rounding
// of the contracted sum instead of one per term (1.0 to 1.2 times otherwise),
// but for (ds|pp) and (dd|ss), which stay below 1.0 without and whose sums
// fill the registers.  C54H18 / cc-pVDZ: 181.2 ms against 176.4 with the
// transfer, (H2O)64 / 6-31G 30.0 against 29.7.
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

// index of the d component ij (x = 0, y = 1, z = 2): with ny and nz of its
// factors y and z, (ny + nz)(ny + nz + 1) / 2 + nz
__host__ __device__ constexpr int cart_of(int ny, int nz) { return (ny + nz) * (ny + nz + 1) / 2 + nz; }
__host__ __device__ constexpr int d_of(int i, int j) { return cart_of((i == 1) + (j == 1), (i == 2) + (j == 2)); }

// adds one primitive quartet to acc[ia + NA*(ib + NB*(ic + NC*id))]:
// S[m] = pref F_m, m <= LA + LB + LC + LD
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void low_prim(R (&v)[ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD)],
                                         const R (&S)[LA + LB + LC + LD + 1], const R (&PA)[3], const R (&AB)[3],
                                         const R (&QC)[3], const R (&CD)[3], const R (&PQ)[3], R qf, R pf, R h2p,
                                         R h2q, R hpq)
{
    constexpr int L = LA + LB, LT = L + LC + LD;
    if constexpr (LT == 0) {
        v[0] += S[0];
    } else {
        // (ps|ss)^m
        R WP[3], P[LT][3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            WP[i] = -qf * PQ[i];
#pragma unroll
            for (int m = 0; m < LT; m++) P[m][i] = gfma(PA[i], S[m], WP[i] * S[m + 1]);
        }
        R WQ[3], PB[3], QD[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            WQ[k] = pf * PQ[k];
            PB[k] = PA[k] + AB[k];
            QD[k] = QC[k] + CD[k];
        }
        // h2p (S_m - qf S_m+1)
        R e[LT];
#pragma unroll
        for (int m = 0; m < LT; m++) e[m] = h2p * gfma(-qf, S[m + 1], S[m]);
        if constexpr (L == 1) {
            if constexpr (LC == 0) {
#pragma unroll
                for (int i = 0; i < 3; i++) v[i] += P[0][i];
            } else {
#pragma unroll
                for (int k = 0; k < 3; k++)
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        R t = WQ[k] * P[1][i];
                        if (i == k) t = gfma(hpq, S[1], t);
                        v[i + 3 * k] += gfma(QC[k], P[0][i], t);
                    }
            }
        } else if constexpr (LA == 1) {
            // (pp_j|ss)^m of one j at a time
            constexpr int M = LC + 1;
#pragma unroll
            for (int j = 0; j < 3; j++) {
                R PP[M][3];
#pragma unroll
                for (int m = 0; m < M; m++)
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        R t = WP[j] * P[m + 1][i];
                        if (i == j) t += e[m];
                        PP[m][i] = gfma(PB[j], P[m][i], t);
                    }
                if constexpr (LC == 0) {
#pragma unroll
                    for (int i = 0; i < 3; i++) v[i + 3 * j] += PP[0][i];
                } else {
                    const R sp = gfma(PB[j], S[1], WP[j] * S[2]);   // (s p_j|ss)^1
#pragma unroll
                    for (int c = 0; c < 3; c++)
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            const int o = i + 3 * j + 9 * c;
                            R t = WQ[c] * PP[1][i];
                            if (i == c) t = gfma(hpq, sp, t);
                            if (j == c) t = gfma(hpq, P[1][i], t);
                            v[o] += gfma(QC[c], PP[0][i], t);
                        }
                }
            }
        } else {
            // (ds|ss)^m
            R D[LT - 1][6];
#pragma unroll
            for (int m = 0; m < LT - 1; m++)
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = i; j < 3; j++) {
                        R t = WP[j] * P[m + 1][i];
                        if (i == j) t += e[m];
                        D[m][d_of(i, j)] = gfma(PA[j], P[m][i], t);
                    }
            if constexpr (LB > 0) {
                // (dp_k|ss)^m of one k at a time
                constexpr int M = LT - 2;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    R DP[M][6];
#pragma unroll
                    for (int m = 0; m < M; m++) {
                        R pe[3];
#pragma unroll
                        for (int i = 0; i < 3; i++) pe[i] = h2p * gfma(-qf, P[m + 1][i], P[m][i]);
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = i; j < 3; j++) {
                                R t = WP[k] * D[m + 1][d_of(i, j)];
                                if (i == k) t += pe[j];
                                if (j == k) t += pe[i];
                                DP[m][d_of(i, j)] = gfma(PB[k], D[m][d_of(i, j)], t);
                            }
                    }
                    if constexpr (LT == 3) {
#pragma unroll
                        for (int d = 0; d < 6; d++) v[d + 6 * k] += DP[0][d];
                    } else {
                        // (p_i p_k|ss)^m, from which the terms of a lowered d component follow
                        R PP[2][3];
#pragma unroll
                        for (int m = 0; m < 2; m++)
#pragma unroll
                            for (int i = 0; i < 3; i++) {
                                R t = WP[k] * P[m + 1][i];
                                if (i == k) t += e[m];
                                PP[m][i] = gfma(PB[k], P[m][i], t);
                            }
                        if constexpr (LC == 1) {
#pragma unroll
                            for (int c = 0; c < 3; c++)
#pragma unroll
                                for (int i = 0; i < 3; i++)
#pragma unroll
                                    for (int j = i; j < 3; j++) {
                                        const int d = d_of(i, j), o = d + 6 * k + 18 * c;
                                        R t = WQ[c] * DP[1][d];
                                        if (k == c) t = gfma(hpq, D[1][d], t);
                                        if (i == c) t = gfma(hpq, PP[1][j], t);
                                        if (j == c) t = gfma(hpq, PP[1][i], t);
                                        v[o] += gfma(QC[c], DP[0][d], t);
                                    }
                        } else {
                            R pe[3];
#pragma unroll
                            for (int i = 0; i < 3; i++) pe[i] = h2p * gfma(-qf, PP[1][i], PP[0][i]);
#pragma unroll
                            for (int l = k; l < 3; l++)
#pragma unroll
                                for (int i = 0; i < 3; i++)
#pragma unroll
                                    for (int j = i; j < 3; j++) {
                                        const int d = d_of(i, j), o = d + 6 * d_of(k, l);
                                        R t = gfma(PB[l], DP[0][d], v[o]);
                                        if (k == l) t = gfma(h2p, gfma(-qf, D[1][d], D[0][d]), t);
                                        if (i == l) t += pe[j];
                                        if (j == l) t += pe[i];
                                        v[o] = gfma(WP[l], DP[1][d], t);
                                    }
                        }
                    }
                }
            } else if constexpr (LC + LD == 2) {
                // (ds|p_k s)^m, then (ds|d_kl s) with l >= k or (ds|p_k p_l)
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
                    for (int l = LD == 1 ? 0 : k; l < 3; l++)
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = i; j < 3; j++) {
                                const int d = d_of(i, j), o = d + 6 * (LD == 1 ? k + 3 * l : d_of(k, l));
                                R t = LD == 1 ? gfma(QD[l], DP[0][d], v[o]) : WQ[l] * DP[1][d];
                                if (k == l) t = gfma(h2q, gfma(-pf, D[1][d], D[0][d]), t);
                                if (i == l) t = gfma(hpq, PP[j], t);
                                if (j == l) t = gfma(hpq, PP[i], t);
                                if constexpr (LD == 1) v[o] = gfma(WQ[l], DP[1][d], t);
                                else v[o] += gfma(QC[l], DP[0][d], t);
                            }
                }
            } else if constexpr (LC == 0) {
#pragma unroll
                for (int d = 0; d < 6; d++) v[d] += D[0][d];
            } else {
#pragma unroll
                for (int k = 0; k < 3; k++)
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = i; j < 3; j++) {
                            const int d = d_of(i, j);
                            R t = WQ[k] * D[1][d];
                            if (i == k) t = gfma(hpq, P[1][j], t);
                            if (j == k) t = gfma(hpq, P[1][i], t);
                            v[d + 6 * k] += gfma(QC[k], D[0][d], t);
                        }
            }
        }
    }
}
