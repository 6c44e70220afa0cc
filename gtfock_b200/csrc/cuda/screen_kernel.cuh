// screen_kernel.cuh -- diagonal quartets (MN|MN) of the Schwarz screening
// (pfock/screening.c:59-90); included by screen.cu and screen_dd.cu.
#pragma once

#include "gtf_dev.cuh"
#include "sph_dev.cuh"

#define SCREEN_THREADS 64

// Screening slices: the ket components cd = CD0 .. CD0+N-1 (cd = k + NA*l)
// of the diagonal quartet (MN|MN) at a time, folded into the sums
// s[m][n] = sum_{i,j,k,l} T[m][i] T[n][j] T[m][k] T[n][l] (ij|kl), so that no
// thread holds all NA*NB*NA*NB integrals (1296 for (dd|dd)).
__host__ __device__ constexpr int screen_slice_n(int LA, int LB)
{
    // whole quartets up to 81 integrals; else slices of at most 72
    return ncart(LA) * ncart(LB) * ncart(LA) * ncart(LB) <= 81 ? ncart(LA) * ncart(LB)
           : ncart(LA) * ncart(LB) * 3 <= 54                   ? 3
                                                               : 2;
}

// Lanes per pair: the pair's ket primitives are dealt out to G neighbouring
// lanes, whose partial integrals are summed by shuffles.  A pair has up to 64
// primitive pairs of s shells but a single one of d shells; one lane walking
// all 64 x 64 primitive quartets of an (ss|ss) diagonal took 4 ms however
// small the molecule.
__host__ __device__ constexpr int screen_lanes(int LA, int LB)
{
    return LA + LB == 0 ? 32 : LA + LB == 1 ? 16 : LA + LB == 2 ? 8 : LA + LB == 3 ? 4 : 1;
}

template <int LA, int LB, int CD0, int N>
__global__ void __launch_bounds__(SCREEN_THREADS) k_screen(const PairRec *__restrict__ pairs, PrimPairs pp, int n,
                                                           int pure, double *__restrict__ sums)
{
    constexpr int NA = ncart(LA), NB = ncart(LB), NR = LA + LB + 1, G = screen_lanes(LA, LB);
    const int x = blockIdx.x * SCREEN_THREADS + threadIdx.x;
    const int t = x / G, sub = x % G;
    const bool active = t < n;
    double acc[NA * NB * N];
#pragma unroll
    for (int k = 0; k < NA * NB * N; k++) acc[k] = 0.0;
    if (active) {
        const PairRec pr = pairs[t];
        const PPStored src{pp};
        eri_accumulate_cd<LA, LB, LA, LB, CD0, N, false>(src, pr, src, pr, acc, RysTab<double>::ptr(NR),
                                                         prim_split(G, sub, 1, 0));
    }
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) {
#pragma unroll
        for (int k = 0; k < NA * NB * N; k++) acc[k] += __shfl_xor_sync(GTF_FULL_MASK, acc[k], o);
    }
    if (!active || sub != 0) return;
    const int sa = nsph_of(LA, pure), sb = nsph_of(LB, pure);
    double *s = sums + (size_t)t * (NA * NB);
#pragma unroll
    for (int m = 0; m < NA; m++) {
#pragma unroll
        for (int q = 0; q < NB; q++) {
            if (m >= sa || q >= sb) continue;
            double v = 0.0;
#pragma unroll
            for (int u = 0; u < N; u++) {
                const int k = (CD0 + u) % NA, l = (CD0 + u) / NA;
                const double tk = sph_coef(LA, pure, m, k), tl = sph_coef(LB, pure, q, l);
                if (tk == 0.0 || tl == 0.0) continue;
#pragma unroll
                for (int i = 0; i < NA; i++) {
                    const double ti = sph_coef(LA, pure, m, i);
                    if (ti == 0.0) continue;
#pragma unroll
                    for (int j = 0; j < NB; j++) {
                        const double tj = sph_coef(LB, pure, q, j);
                        if (tj == 0.0) continue;
                        v += ti * tj * tk * tl * acc[i + NA * (j + NB * u)];
                    }
                }
            }
            // the slices of a class run one after another on one stream
            s[m * NB + q] = CD0 == 0 ? v : s[m * NB + q] + v;
        }
    }
}

// one launch per slice; returns 0, or -1 on a launch error
template <int LA, int LB, int CD0 = 0>
int launch_screen_slices(const PairRec *pairs, PrimPairs pp, int n, int pure, double *sums, cudaStream_t st)
{
    if constexpr (CD0 < ncart(LA) * ncart(LB)) {
        constexpr int N = screen_slice_n(LA, LB), G = screen_lanes(LA, LB);
        static_assert(ncart(LA) * ncart(LB) % N == 0, "whole slices");
        const unsigned g = (unsigned)(((long long)n * G + SCREEN_THREADS - 1) / SCREEN_THREADS);
        k_screen<LA, LB, CD0, N><<<g, SCREEN_THREADS, 0, st>>>(pairs, pp, n, pure, sums);
        if (cudaGetLastError() != cudaSuccess) return -1;
        return launch_screen_slices<LA, LB, CD0 + N>(pairs, pp, n, pure, sums, st);
    }
    return 0;
}
