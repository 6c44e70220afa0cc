// Host stand-in for cuda_runtime.h: lets g++ compile the device building
// blocks (gtf_dev.cuh, eri_low.cuh) for the CPU tests of their arithmetic.
// The warp functions are never called there.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>

using std::max;
using std::min;
#define __device__
#define __host__
#define __global__
#define __constant__
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))
struct double2 { double x, y; };
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct int2 { int x, y; };
struct Idx { unsigned x, y, z; };
static Idx threadIdx, blockIdx, blockDim, gridDim;
template <class T> inline T __ldg(const T *p) { return *p; }
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
inline float rsqrtf(float x) { return (float)(1.0 / std::sqrt((double)x)); }
inline unsigned __ballot_sync(unsigned, bool) { return 0; }
template <class T> inline T __shfl_xor_sync(unsigned, T v, int) { return v; }
inline void __syncthreads() {}
inline void __syncwarp() {}
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int __clz(int x) { return __builtin_clz(x); }
template <class T> inline T atomicAdd(T *p, T v) { T o = *p; *p += v; return o; }
inline size_t __cvta_generic_to_shared(const void *p) { return (size_t)p; }
