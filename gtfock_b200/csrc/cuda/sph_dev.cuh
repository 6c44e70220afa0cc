// sph_dev.cuh -- the d-shell spherical transform shared by the Fock and the
// screening kernels.
#pragma once

#include "gtf_dev.cuh"

// rows m = -2..2, cols xx, xy, xz, yy, yz, zz
static __constant__ double c_sph_d[5][6] = {
    {0.0, 1.7320508075688772, 0.0, 0.0, 0.0, 0.0},
    {0.0, 0.0, 0.0, 0.0, 1.7320508075688772, 0.0},
    {-0.5, 0.0, 0.0, -0.5, 0.0, 1.0},
    {0.0, 0.0, 1.7320508075688772, 0.0, 0.0, 0.0},
    {0.8660254037844386, 0.0, 0.0, -0.8660254037844386, 0.0, 0.0}};

__device__ __forceinline__ double sph_coef(int L, int pure, int m, int c)
{
    if (pure && L == 2) return c_sph_d[m][c];
    return (m == c) ? 1.0 : 0.0;
}

__device__ __forceinline__ int nsph_of(int L, int pure) { return (pure && L == 2) ? 5 : ncart(L); }
