// screen.cu -- Schwarz screening launches of the shell-pair classes; the
// (dd) diagonals, most of the code, compile apart (screen_dd.cu).
#include "screen_kernel.cuh"

int launch_screen_dd(const PairRec *pairs, PrimPairs pp, int n, int pure, double *sums, cudaStream_t st);

// max |(mn|mn)| over the diagonal of (MN|MN) in the basis's own functions
__global__ void k_screen_max(const double *__restrict__ sums, const int2 *__restrict__ mn, int n, int ns, int la,
                             int lb, int pure, double *__restrict__ sq, unsigned long long *__restrict__ gmax)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int na = ncart(la), nb = ncart(lb), sa = nsph_of(la, pure), sb = nsph_of(lb, pure);
    const double *s = sums + (size_t)t * na * nb;
    double mx = 0.0;
    for (int m = 0; m < sa; m++)
        for (int q = 0; q < sb; q++) {
            const double v = fabs(s[m * nb + q]);
            if (v > mx) mx = v;
        }
    const int M = mn[t].x, N = mn[t].y;
    sq[(size_t)M * ns + N] = mx;
    sq[(size_t)N * ns + M] = mx;
    atomicMax(gmax, (unsigned long long)__double_as_longlong(mx));
}

// sums: [n][ncart(la) * ncart(lb)] scratch
int gtf_launch_screen(int la, int lb, const PairRec *pairs, PrimPairs pp, const int2 *mn, int n, int ns, int pure,
                      double *sums, double *sq, unsigned long long *gmax, cudaStream_t st)
{
    int r = -1;
    switch (la * (la + 1) / 2 + lb) {
        case 0: r = launch_screen_slices<0, 0>(pairs, pp, n, pure, sums, st); break;
        case 1: r = launch_screen_slices<1, 0>(pairs, pp, n, pure, sums, st); break;
        case 2: r = launch_screen_slices<1, 1>(pairs, pp, n, pure, sums, st); break;
        case 3: r = launch_screen_slices<2, 0>(pairs, pp, n, pure, sums, st); break;
        case 4: r = launch_screen_slices<2, 1>(pairs, pp, n, pure, sums, st); break;
        case 5: r = launch_screen_dd(pairs, pp, n, pure, sums, st); break;
    }
    if (r != 0) return r;
    k_screen_max<<<(n + 127) / 128, 128, 0, st>>>(sums, mn, n, ns, la, lb, pure, sq, gmax);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
