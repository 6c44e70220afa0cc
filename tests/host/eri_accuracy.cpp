// Rounding errors of the integral building blocks, compiled for the host,
// against 113-bit references.
//   eri <class 0..11> <quartets>: one line "LA LB LC LD e64_rys e64_low
//     e32_low", geometric means over random contracted quartets of the
//     error relative to the quartet's largest integral, of the Rys form and of
//     the form of eri_low.cuh (the reference: McMurchie-Davidson)
//   boys: lines "m bits below above", largest error of F_m, m <= 4, in units of
//     half a last place, below and above BOYS_TMAX, for every M >= m
#include <cuda_runtime.h>
#define asm(...)
#define volatile
#include "gtf_dev.cuh"
#undef volatile
#undef asm
#include <quadmath.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

typedef __float128 Q;
static std::mt19937_64 rng;
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }

// F_M by its series of positive terms, the others by downward recursion
static void boys_ref(int M, Q T, Q *F)
{
    const Q e = expq(-T);
    Q t = (Q)1 / (2 * M + 1), s = t;
    if (T > 120) {   // exp(-T) is below 1e-52
        F[0] = sqrtq(M_PIq / T) / 2;
        for (int m = 0; m < M; m++) F[m + 1] = (2 * m + 1) * F[m] / (2 * T);
        return;
    }
    for (int i = 1; i < 2000 && t > s * 1e-36Q; i++) {
        t *= 2 * T / (2 * M + 2 * i + 1);
        s += t;
    }
    F[M] = e * s;
    for (int m = M; m > 0; m--) F[m - 1] = (2 * T * F[m] + e) / (2 * m - 1);
}

struct Prim {
    Q p, h, K, P[3];
};

// Hermite coefficients E_t^{ij} of one direction
static void hermite(int la, int lb, Q PA, Q PB, Q h, Q (&E)[3][3][6])
{
    memset(E, 0, sizeof(E));
    E[0][0][0] = 1;
    for (int i = 0; i <= la; i++)
        for (int j = 0; j <= lb; j++)
            for (int t = 0; t <= i + j && i + j > 0; t++) {
                const Q *s = i > 0 ? E[i - 1][j] : E[i][j - 1];
                E[i][j][t] = (t > 0 ? h * s[t - 1] : 0) + (i > 0 ? PA : PB) * s[t] + (t + 1) * s[t + 1];
            }
}

static Q hermite_r(int t, int u, int v, int n, const Q *PQ, const Q *f)
{
    if (t < 0 || u < 0 || v < 0) return 0;
    if (t > 0) return (t - 1) * hermite_r(t - 2, u, v, n + 1, PQ, f) + PQ[0] * hermite_r(t - 1, u, v, n + 1, PQ, f);
    if (u > 0) return (u - 1) * hermite_r(t, u - 2, v, n + 1, PQ, f) + PQ[1] * hermite_r(t, u - 1, v, n + 1, PQ, f);
    if (v > 0) return (v - 1) * hermite_r(t, u, v - 2, n + 1, PQ, f) + PQ[2] * hermite_r(t, u, v - 1, n + 1, PQ, f);
    return f[n];
}

static int power(int L, int c, int d) { return d == 0 ? cart_x(L, c) : d == 1 ? cart_y(L, c) : cart_z(L, c); }

static void reference(const int (&l)[4], const PairRec &pb, const PairRec &pk, const std::vector<Prim> &b,
                      const std::vector<Prim> &k, std::vector<Q> &out)
{
    const int na = ncart(l[0]), nb = ncart(l[1]), nc = ncart(l[2]), nd = ncart(l[3]), L = l[0] + l[1] + l[2] + l[3];
    const Q A[3] = {pb.Ax, pb.Ay, pb.Az}, AB[3] = {pb.ABx, pb.ABy, pb.ABz};
    const Q C[3] = {pk.Ax, pk.Ay, pk.Az}, CD[3] = {pk.ABx, pk.ABy, pk.ABz};
    out.assign(na * nb * nc * nd, 0);
    for (const Prim &x : b)
        for (const Prim &y : k) {
            Q Eb[3][3][3][6], Ek[3][3][3][6], PQ[3], f[9], R[5][5][5];
            for (int d = 0; d < 3; d++) {
                hermite(l[0], l[1], x.P[d] - A[d], x.P[d] - A[d] + AB[d], x.h, Eb[d]);
                hermite(l[2], l[3], y.P[d] - C[d], y.P[d] - C[d] + CD[d], y.h, Ek[d]);
                PQ[d] = x.P[d] - y.P[d];
            }
            const Q rho = x.p * y.p / (x.p + y.p);
            boys_ref(L, rho * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]), f);
            Q w = x.K * y.K / sqrtq(x.p + y.p);
            for (int m = 0; m <= L; m++, w *= -2 * rho) f[m] *= w;
            for (int t = 0; t <= L; t++)
                for (int u = 0; t + u <= L; u++)
                    for (int v = 0; t + u + v <= L; v++) R[t][u][v] = hermite_r(t, u, v, 0, PQ, f);
            for (int q = 0; q < na * nb * nc * nd; q++) {
                const int c[4] = {q % na, q / na % nb, q / (na * nb) % nc, q / (na * nb * nc)};
                const Q *eb[3], *ek[3];
                int mb[3], mk[3];
                for (int d = 0; d < 3; d++) {
                    const int i = power(l[0], c[0], d), j = power(l[1], c[1], d);
                    const int m = power(l[2], c[2], d), n = power(l[3], c[3], d);
                    eb[d] = Eb[d][i][j];
                    ek[d] = Ek[d][m][n];
                    mb[d] = i + j;
                    mk[d] = m + n;
                }
                Q s = 0;
                for (int t = 0; t <= mb[0]; t++)
                    for (int u = 0; u <= mb[1]; u++)
                        for (int v = 0; v <= mb[2]; v++)
                            for (int t2 = 0; t2 <= mk[0]; t2++)
                                for (int u2 = 0; u2 <= mk[1]; u2++)
                                    for (int v2 = 0; v2 <= mk[2]; v2++) {
                                        const Q e = eb[0][t] * eb[1][u] * eb[2][v] * ek[0][t2] * ek[1][u2] * ek[2][v2];
                                        s += ((t2 + u2 + v2) & 1 ? -e : e) * R[t + t2][u + u2][v + v2];
                                    }
                out[q] += s;
            }
        }
}

struct Shell {
    double c[3];
    std::vector<double> e, w;
};

// 1 to 6 primitives (d shells 1 to 3) of exponents 0.1 to 30, normalised, one weight in five negative
static Shell random_shell(int l, const double *c)
{
    Shell s;
    memcpy(s.c, c, sizeof(s.c));
    const int n = 1 + (int)uni(0, l == 2 ? 2.99 : 5.99);
    for (int i = 0; i < n; i++) {
        const double e = 0.1 * pow(300.0, uni(0, 1));
        s.e.push_back(e);
        s.w.push_back(pow(2 * e / M_PI, 0.75) * pow(4 * e, l / 2.0) / (l == 2 ? sqrt(3.0) : 1.0) * uni(0.1, 1) *
                      (uni(0, 1) < 0.2 ? -1 : 1));
    }
    return s;
}

// the engine's records of a shell pair, FP64 and FP32, appended; and the same values in 113 bits
static void make_pair(const Shell &a, const Shell &b, PairRec &r, std::vector<double> &pp, std::vector<float> &pp32,
                      std::vector<Prim> &q)
{
    double r2 = 0;
    for (int d = 0; d < 3; d++) r2 += (a.c[d] - b.c[d]) * (a.c[d] - b.c[d]);
    r.Ax = a.c[0];
    r.Ay = a.c[1];
    r.Az = a.c[2];
    r.ABx = a.c[0] - b.c[0];
    r.ABy = a.c[1] - b.c[1];
    r.ABz = a.c[2] - b.c[2];
    r.off = (int)(pp.size() / (2 * GTF_PPREC_D2));
    r.n = 0;
    for (size_t i = 0; i < a.e.size(); i++)
        for (size_t j = 0; j < b.e.size(); j++) {
            const double p = a.e[i] + b.e[j], ip = 1.0 / p;
            const double K = GTF_PAIR_PREF * a.w[i] * b.w[j] * exp(-a.e[i] * b.e[j] * ip * r2) * ip;
            if (fabs(K) < GTF_PRIM_EPS) continue;
            double P[3];
            Prim x;
            for (int d = 0; d < 3; d++) x.P[d] = P[d] = (a.e[i] * a.c[d] + b.e[j] * b.c[d]) * ip;
            x.p = p;
            x.K = K;
            x.h = (Q)0.5 / x.p;
            q.push_back(x);
            pp.insert(pp.end(), {p, K, P[0], P[1], P[2], 0.5 * ip});
            pp32.insert(pp32.end(), {(float)p, (float)K, (float)(P[0] - a.c[0]), (float)(P[1] - a.c[1]),
                                     (float)(P[2] - a.c[2]), (float)(0.5 * ip), 0.0f, 0.0f});
            r.n++;
        }
}

template <int LA, int LB, int LC, int LD>
static void eri_class(int n)
{
    constexpr int NQ = ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD), NCD = ncart(LC) * ncart(LD);
    constexpr int LT = LA + LB + LC + LD, NR = LT / 2 + 1;
    double lg[3] = {0, 0, 0};
    for (int it = 0; it < n;) {
        // half of the quartets within 4 bohr a side, half up to 12 apart; some share centres
        double c[4][3];
        const double side = uni(0, 1) < 0.5 ? 12.0 / sqrt(3.0) : 4.0;
        for (auto &x : c)
            for (double &v : x) v = uni(0, side);
        if (uni(0, 1) < 0.15) memcpy(c[1], c[0], sizeof(c[0]));
        if (uni(0, 1) < 0.15) memcpy(c[3], c[2], sizeof(c[0]));
        if (uni(0, 1) < 0.1) memcpy(c[2], c[0], sizeof(c[0]));
        const Shell a = random_shell(LA, c[0]), b = random_shell(LB, c[1]);
        const Shell s = random_shell(LC, c[2]), t = random_shell(LD, c[3]);
        PairRec pb, pk;
        std::vector<double> pp;
        std::vector<float> pp32;
        std::vector<Prim> qb, qk;
        make_pair(a, b, pb, pp, pp32, qb);
        make_pair(s, t, pk, pp, pp32, qk);
        if (qb.empty() || qk.empty()) continue;
        std::vector<Q> ref;
        const int l[4] = {LA, LB, LC, LD};
        reference(l, pb, pk, qb, qk, ref);
        double mx = 0;
        for (Q v : ref) mx = std::max(mx, (double)fabsq(v));
        if (mx < 1e-11) continue;
        it++;
        std::vector<double2> r64(pp.size() / 2);
        std::vector<float4> r32(pp32.size() / 4);
        memcpy(r64.data(), pp.data(), sizeof(double) * pp.size());
        memcpy(r32.data(), pp32.data(), sizeof(float) * pp32.size());
        const PPRec src{r64.data()};
        const PPRec32 src32{r32.data()};
        double o[2][NQ] = {};
        float q[NQ] = {};
        eri_accumulate_cd<LA, LB, LC, LD, 0, NCD, false, false, false>(src, pb, src, pk, o[0], RysTab<double>::ptr(NR));
        eri_accumulate_cd<LA, LB, LC, LD, 0, NCD, false, false, true>(src, pb, src, pk, o[1], BoysTab<double>::ptr(LT));
        eri_accumulate_cd32<LA, LB, LC, LD, 0, NCD, false, false, true>(src32, pb, pk, q, BoysTab<float>::ptr(LT));
        double e[3] = {1e-17, 1e-17, 1e-10};
        for (int k = 0; k < NQ; k++) {
            e[0] = std::max(e[0], (double)fabsq(o[0][k] - ref[k]) / mx);
            e[1] = std::max(e[1], (double)fabsq(o[1][k] - ref[k]) / mx);
            e[2] = std::max(e[2], (double)fabsq(q[k] - ref[k]) / mx);
        }
        for (int f = 0; f < 3; f++) lg[f] += log(e[f]);
    }
    printf("%d %d %d %d", LA, LB, LC, LD);
    for (double v : lg) printf(" %.4e", exp(v / n));
    printf("\n");
}

template <int M, class R>
static void boys_errors(double (&err)[2][BOYS_MMAX + 1])
{
    for (int i = 0; i < 20000; i++) {
        double T = i < 12000 ? uni(0, BOYS_TMAX) : BOYS_TMAX * pow(10.0, uni(0, 1.5));
        if (i % 10 == 0) T = BOYS_H * (i / 10 % (BOYS_NINT + 8));                              // interval edges
        if (i % 10 == 1) T = nextafter((float)(BOYS_H * (1 + i / 10 % BOYS_NINT)), 0.0f);   // just below them
        if (i % 10 == 2) T = BOYS_H * (0.5 + i / 10 % BOYS_NINT);                             // midpoints
        const R t = (R)T;
        R F[M + 1];
        Q f[M + 1];
        boys<M>(t, F, BoysTab<R>::ptr(M));
        boys_ref(M, (Q)t, f);
        for (int m = 0; m <= M; m++) {
            double &e = err[t >= (R)BOYS_TMAX][m];
            e = std::max(e, (double)(fabsq(F[m] - f[m]) / f[m]) / (sizeof(R) == 4 ? 0x1p-24 : 0x1p-53));
        }
    }
}

template <class R>
static void boys_report()
{
    double err[2][BOYS_MMAX + 1] = {};
    boys_errors<0, R>(err);
    boys_errors<1, R>(err);
    boys_errors<2, R>(err);
    boys_errors<3, R>(err);
    boys_errors<4, R>(err);
    for (int m = 0; m <= BOYS_MMAX; m++) printf("%d %d %.3f %.3f\n", m, 8 * (int)sizeof(R), err[0][m], err[1][m]);
}

int main(int argc, char **argv)
{
    if (argc > 1 && !strcmp(argv[1], "boys")) {
        boys_report<double>();
        boys_report<float>();
        return 0;
    }
    if (argc < 4) return 2;
    const int c = atoi(argv[2]), n = atoi(argv[3]);
    rng.seed(777 + c);
    switch (c) {
        case 0: eri_class<0, 0, 0, 0>(n); break;
        case 1: eri_class<1, 0, 0, 0>(n); break;
        case 2: eri_class<1, 0, 1, 0>(n); break;
        case 3: eri_class<1, 1, 0, 0>(n); break;
        case 4: eri_class<2, 0, 0, 0>(n); break;
        case 5: eri_class<2, 0, 1, 0>(n); break;
        case 6: eri_class<1, 1, 1, 0>(n); break;
        case 7: eri_class<2, 1, 0, 0>(n); break;
        case 8: eri_class<2, 1, 1, 0>(n); break;
        case 9: eri_class<2, 0, 1, 1>(n); break;
        case 10: eri_class<2, 0, 2, 0>(n); break;
        case 11: eri_class<2, 2, 0, 0>(n); break;
        default: return 2;
    }
    return 0;
}
