// purif.cu -- canonical density purification and Pulay DIIS on one GPU
// (pscf/purif.c:257-641; the 3-D pdgemm of pscf/pdgemm.c becomes one product:
// k_abt for D D^T and D D^2, cuBLAS DGEMM for the others).
//
// Purification (pscf/purif.c:301-476): Gershgorin bounds and tr F give the
// initial D; each iteration forms D2 = D D^T and D3 = D D2, reduces
// ||D - D2||_F, tr(D2 - D3) and tr(D - D2) deterministically (fixed block
// partials summed in order), updates D with the trace-conserving polynomial,
// and stops once ||D - D2||_F < 1e-11.  D_AO = X D X at the end.
// DIIS (pscf/purif.c:491-641): error X (F D S - S D F) X, dot products into
// the bordered B matrix, (m+1)^2 solve, F = sum c_i F_i.
#include <cublas_v2.h>
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include "devmem.cuh"
#include "diis_dev.cuh"
#include "gtf_cuda.h"

#define PUR_MAX_ITERS 200
#define PUR_MAX_DIIS GTF_MAX_DIIS
#define RED_BLOCKS 148
#define RED_THREADS 256

#define CKP(call)                                                                       \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) {                                                        \
            fprintf(stderr, "gtfock_b200 %s:%d %s\n", __FILE__, __LINE__, cudaGetErrorString(e_)); \
            return GTF_ERR_CUDA;                                                        \
        }                                                                               \
    } while (0)
#define CKB(call)                                                       \
    do {                                                                \
        if ((call) != CUBLAS_STATUS_SUCCESS) {                          \
            fprintf(stderr, "gtfock_b200 %s:%d cuBLAS failure\n", __FILE__, __LINE__); \
            return GTF_ERR_CUDA;                                        \
        }                                                               \
    } while (0)

extern "C" void gtf_note_launches(int n);

struct gtf_purif_dev {
    int n, nocc;
    cudaStream_t st;
    int own_st;               // the stream was created here
    cublasHandle_t blas;      // leased for the duration of one call (BlasLease)
    double *S, *X, *D, *D2, *D3, *F, *W, *W2;
    double *vecs, *Fvecs;
    double *part;     // [part_len(n)] block partials
    double *scal;     // device scalars
    double *h_scal;   // pinned mirror
    double *E;        // this iteration's DIIS error vector, before it enters its slot
    struct DiisState *ds;   // device: DIIS bookkeeping and coefficients
    int sx_set;
    cudaEvent_t e0, e1;
    double ms_gemm, ms_total, errnorm, idem, trerr;
    int mode;                 // 0 FP64, 1 split-BF16 then FP64
    gtf_bf16x3_t *bx;
    int it_bf16, it_fp64;
};

#define GERSH_COLS 32
#define GERSH_ROWS 8
// block partials: 16 per reduction block, or 3 per block of the Gershgorin pass
static size_t part_len(int n)
{
    const size_t a = (size_t)RED_BLOCKS * 16, b = 3 * (size_t)((n + GERSH_COLS - 1) / GERSH_COLS);
    return a > b ? a : b;
}

// row-major C = A B^T (pdgemm3D_2), via column-major cuBLAS
static int gemm_abt(gtf_purif_dev *p, const double *A, const double *B, double *C)
{
    const double one = 1.0, zero = 0.0;
    CKB(cublasDgemm(p->blas, CUBLAS_OP_T, CUBLAS_OP_N, p->n, p->n, p->n, &one, B, p->n, A, p->n, &zero, C, p->n));
    return GTF_OK;
}

// ---------------------------------------------------------------------------
// C = A B^T, row-major n x n.  SYM: for products that are symmetric (D D^T;
// D D^2 of a symmetric D), the tiles on and below the diagonal, mirrored.
//
// One block per 32 x 32 tile; its four warps share the K loop (each takes 8 of
// a slab's 32) and hold the whole tile in FP64 tensor-core accumulators
// (m8n8k4: 16 products per 8 fragment loads), summed through shared memory at
// the end.  Bound by the FP64 pipe; at 846 functions the 378 tiles are one
// wave of three blocks per SM.  cuBLAS's full product in 729 such tiles took
// 57 us there.
// ---------------------------------------------------------------------------
#define ST_TILE 32
#define ST_LD 36   // row stride in doubles: the 4 x 4 elements a half warp reads are in different banks

__device__ __forceinline__ void cp_async8(double *dst, const double *src, bool ok)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
}

// tile (ti, tj), tj <= ti, of the linear index ti (ti + 1) / 2 + tj
__device__ __forceinline__ void tri_tile(int x, int &ti, int &tj)
{
    ti = (int)((sqrtf(8.0f * (float)x + 1.0f) - 1.0f) * 0.5f);
    while (ti * (ti + 1) / 2 > x) ti--;
    while ((ti + 1) * (ti + 2) / 2 <= x) ti++;
    tj = x - ti * (ti + 1) / 2;
}

template <bool SYM>
__global__ void __launch_bounds__(128) k_abt(const double *__restrict__ A, const double *__restrict__ B,
                                             double *__restrict__ C, int n)
{
    __shared__ __align__(16) double buf[2][2][ST_TILE * ST_LD];   // [stage][A or B]
    int ti, tj;
    if constexpr (SYM) {
        tri_tile((int)blockIdx.x, ti, tj);
    } else {
        const int nt = (n + ST_TILE - 1) / ST_TILE;
        ti = (int)blockIdx.x / nt;
        tj = (int)blockIdx.x - ti * nt;
    }
    const int r0 = ti * ST_TILE, c0 = tj * ST_TILE;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    auto load = [&](int stage, int k0) {
#pragma unroll
        for (int q = 0; q < ST_TILE * ST_TILE / 128; q++) {
            const int e = threadIdx.x + 128 * q, r = e / ST_TILE, k = e % ST_TILE;
            const bool ka = k0 + k < n, oa = ka && r0 + r < n, ob = ka && c0 + r < n;
            cp_async8(&buf[stage][0][r * ST_LD + k], oa ? A + (size_t)(r0 + r) * n + k0 + k : A, oa);
            cp_async8(&buf[stage][1][r * ST_LD + k], ob ? B + (size_t)(c0 + r) * n + k0 + k : B, ob);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
    load(0, 0);
    int st = 0;
    for (int k0 = 0; k0 < n; k0 += ST_TILE, st ^= 1) {
        if (k0 + ST_TILE < n) {
            load(st ^ 1, k0 + ST_TILE);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        // fragments: A row lane / 4, k lane % 4; B column lane / 4, k lane % 4
        const int o = (lane >> 2) * ST_LD + 8 * w + (lane & 3);
#pragma unroll
        for (int k = 0; k < 8; k += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                a[i] = buf[st][0][o + 8 * i * ST_LD + k];
                b[i] = buf[st][1][o + 8 * i * ST_LD + k];
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                                 : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
                                 : "d"(a[i]), "d"(b[j]));
        }
        __syncthreads();
    }
    // the four warps' sums: 32 x 32 each, row stride 33
    double *part = &buf[0][0][0];
    static_assert(4 * ST_TILE * 33 <= 4 * ST_TILE * ST_LD, "partial tiles fit the stages");
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 2; q++)
                part[w * ST_TILE * 33 + (8 * i + (lane >> 2)) * 33 + 8 * j + 2 * (lane & 3) + q] = acc[i][j][q];
    __syncthreads();
    for (int e = threadIdx.x; e < ST_TILE * ST_TILE; e += 128) {
        const int r = e / ST_TILE, c = e % ST_TILE;
        double *p = part + r * 33 + c;
        p[0] = (p[0] + p[ST_TILE * 33]) + (p[2 * ST_TILE * 33] + p[3 * ST_TILE * 33]);
        if (r0 + r < n && (SYM ? c0 + c <= r0 + r : c0 + c < n)) C[(size_t)(r0 + r) * n + c0 + c] = p[0];
    }
    if constexpr (!SYM) return;
    __syncthreads();
    for (int e = threadIdx.x; e < ST_TILE * ST_TILE; e += 128) {
        const int c = e / ST_TILE, r = e % ST_TILE;
        if (r0 + r < n && c0 + c < r0 + r) C[(size_t)(c0 + c) * n + r0 + r] = part[r * 33 + c];
    }
}

static int sym_abt(gtf_purif_dev *p, const double *A, const double *B, double *C)
{
    const int nt = (p->n + ST_TILE - 1) / ST_TILE;
    k_abt<true><<<nt * (nt + 1) / 2, 128, 0, p->st>>>(A, B, C, p->n);
    CKP(cudaGetLastError());
    gtf_note_launches(1);
    return GTF_OK;
}

static int full_abt(gtf_purif_dev_t *p, const double *A, const double *B, double *C)
{
    const int nt = (p->n + ST_TILE - 1) / ST_TILE;
    k_abt<false><<<nt * nt, 128, 0, p->st>>>(A, B, C, p->n);
    CKP(cudaGetLastError());
    gtf_note_launches(1);
    return GTF_OK;
}

// Largest |F - F^T|, as the bits of a double, into scal[12] (zeroed before)
__global__ void __launch_bounds__(256) k_asymmetry(const double *__restrict__ F, int n, double *__restrict__ scal)
{
    __shared__ double t[ST_TILE][ST_TILE + 1];
    int ti, tj;
    tri_tile((int)blockIdx.x, ti, tj);
    const int r0 = ti * ST_TILE, c0 = tj * ST_TILE, x = threadIdx.x % ST_TILE;
    for (int y = threadIdx.x / ST_TILE; y < ST_TILE; y += 256 / ST_TILE)
        if (r0 + y < n && c0 + x < n) t[y][x] = F[(size_t)(r0 + y) * n + c0 + x];
    __syncthreads();
    unsigned long long m = 0;
    for (int y = threadIdx.x / ST_TILE; y < ST_TILE; y += 256 / ST_TILE)
        if (c0 + y < n && r0 + x < n) {
            const double d = fabs(F[(size_t)(c0 + y) * n + r0 + x] - t[x][y]);
            const unsigned long long b = (unsigned long long)__double_as_longlong(d);
            m = b > m ? b : m;
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long b = __shfl_xor_sync(0xffffffffu, m, o);
        m = b > m ? b : m;
    }
    if ((threadIdx.x & 31) == 0 && m != 0) atomicMax((unsigned long long *)(scal + 12), m);
}

// sums over the 32 lanes, the same total in every lane
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// per column i: Gershgorin interval [diag - off, diag + off], off = sum_j |F[j][i]| - |diag|
// (pscf/purif.c:309-322); block partials of min, max and the trace.  A block
// takes 32 columns, its 8 rows of threads every 8th matrix row: one thread
// walking a whole column kept 4 blocks busy for 360 us at 846 functions.
static_assert(GERSH_COLS * GERSH_ROWS == RED_THREADS, "block shape");
__global__ void k_gersh(const double *__restrict__ F, int n, double *__restrict__ part)
{
    __shared__ double soff[GERSH_ROWS][GERSH_COLS];
    const int c = threadIdx.x % GERSH_COLS, r = threadIdx.x / GERSH_COLS, i = blockIdx.x * GERSH_COLS + c;
    double off = 0.0;
    if (i < n) {
#pragma unroll 4
        for (int j = r; j < n; j += GERSH_ROWS) off += fabs(F[(size_t)j * n + i]);
    }
    soff[r][c] = off;
    __syncthreads();
    if (r != 0) return;
    double lmin = DBL_MAX, lmax = -DBL_MAX, ltr = 0.0;
    if (i < n) {
        off = 0.0;
#pragma unroll
        for (int k = 0; k < GERSH_ROWS; k++) off += soff[k][c];
        const double dg = F[(size_t)i * n + i];
        off -= fabs(dg);
        lmin = dg - off;
        lmax = dg + off;
        ltr = dg;
    }
    ltr = warp_sum(ltr);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lmin = fmin(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
        lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
    }
    if (c == 0) {
        part[3 * blockIdx.x] = lmin;
        part[3 * blockIdx.x + 1] = lmax;
        part[3 * blockIdx.x + 2] = ltr;
    }
}

// scal[0] = -lambda/n, scal[1] = lambda mu_bar / n + nocc / n (pscf/purif.c:355-373)
__global__ void k_purif_init(const double *__restrict__ part, int nblk, int n, int nocc, double *scal)
{
    double hmin = DBL_MAX, hmax = -DBL_MAX, trF = 0.0;
    for (int b = threadIdx.x; b < nblk; b += 32) {
        hmin = fmin(hmin, part[3 * b]);
        hmax = fmax(hmax, part[3 * b + 1]);
        trF += part[3 * b + 2];
    }
    trF = warp_sum(trF);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        hmin = fmin(hmin, __shfl_xor_sync(0xffffffffu, hmin, o));
        hmax = fmax(hmax, __shfl_xor_sync(0xffffffffu, hmax, o));
    }
    if (threadIdx.x != 0) return;
    const double mu_bar = trF / (double)n;
    const double lambda = fmin((double)nocc / (hmax - mu_bar), (double)(n - nocc) / (mu_bar - hmin));
    scal[0] = -lambda / n;
    scal[1] = lambda * mu_bar / (double)n + (double)nocc / n;
    scal[2] = hmin;
    scal[3] = hmax;
    scal[4] = mu_bar;
    scal[5] = lambda;
}

__global__ void k_purif_d0(const double *__restrict__ F, double *__restrict__ D, int n, const double *scal)
{
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (size_t)n * n) return;
    double v = F[k] * scal[0];
    if (k / n == k % n) v += scal[1];
    D[k] = v;
}

// block partials of ||D - D2||^2, tr(D2 - D3), tr(D - D2)
__global__ void k_purif_stats(const double *__restrict__ D, const double *__restrict__ D2,
                              const double *__restrict__ D3, int n, double *__restrict__ part)
{
    __shared__ double sh[3][RED_THREADS / 32];
    const size_t nn = (size_t)n * n;
    double e = 0.0, t = 0.0, t2 = 0.0;
#pragma unroll 4
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += (size_t)gridDim.x * blockDim.x) {
        const double d = D[k] - D2[k];
        e += d * d;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const size_t k = (size_t)i * n + i;
        t += D2[k] - D3[k];
        t2 += D[k] - D2[k];
    }
    e = warp_sum(e);
    t = warp_sum(t);
    t2 = warp_sum(t2);
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = e;
        sh[1][threadIdx.x >> 5] = t;
        sh[2][threadIdx.x >> 5] = t2;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < RED_THREADS / 32; w++) v += sh[threadIdx.x][w];
        part[3 * blockIdx.x + threadIdx.x] = v;
    }
}

// scal[6] = errnorm, scal[7] = c = tr(D2-D3)/tr(D-D2) (pscf/purif.c:394-440).
// Where the reference would divide 0/0 (an exactly idempotent D) and write NaN
// into D, the iteration stops instead: errnorm is reported as 0 and the
// update below is skipped (c set to NaN).  It stops the same way when c is
// far outside [0, 1]: with every eigenvalue of D in [0, 1], c lies in [0, 1];
// far outside it the eigenvalues have left that interval and the cubic
// update diverges (in the reference, to Inf and NaN within a few steps).
// The loop's stop is kept on the device, so the host need not wait for every
// step: scal[8] != 0 once a step found ||D - D2||_F < 1e-11 (that step's
// update still applies, as in pscf/purif.c:394-455) or stopped as above;
// later steps then change nothing.  scal[9] counts the steps that ran.
// It also stops once the error, already below PURIF_FLOOR, has not fallen by
// 1% in PURIF_STALL steps (scal[10] the best error so far, 0 before the first
// step; scal[11] the steps since): rounding that holds the error just above
// the 1e-11 tolerance keeps the reference's loop running to its cap without
// changing D.  Above the floor the early steps of a purification can move
// the error by less than 1% for many steps, so no such stop applies there.
#define PURIF_C_LO (-0.25)
#define PURIF_C_HI 1.25
#define PURIF_TOL 1e-11
#define PURIF_STALL 8
#define PURIF_FLOOR 1e-8
// One warp: a single thread reading the 148 partials took 20 us of a step.
__global__ void k_purif_finish(const double *__restrict__ part, int nblk, double *scal)
{
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    if (scal[8] != 0.0) {
        if (threadIdx.x == 0) scal[7] = nan;   // stopped: no update
        return;
    }
    double e = 0.0, t = 0.0, t2 = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x; b < nblk; b += 32) {
        e += part[3 * b];
        t += part[3 * b + 1];
        t2 += part[3 * b + 2];
    }
    e = warp_sum(e);
    t = warp_sum(t);
    t2 = warp_sum(t2);
    if (threadIdx.x != 0) return;
    const double c = t / t2;
    const bool ok = isfinite(c) && c >= PURIF_C_LO && c <= PURIF_C_HI;
    scal[6] = ok ? sqrt(e) : 0.0;
    scal[7] = ok ? c : nan;
    scal[9] += 1.0;
    if (ok) {
        if (scal[10] == 0.0 || scal[6] < 0.99 * scal[10]) {
            scal[10] = scal[6];
            scal[11] = 0.0;
        } else {
            scal[11] += 1.0;
        }
    }
    if (!ok || scal[6] < PURIF_TOL || (scal[10] < PURIF_FLOOR && scal[11] >= PURIF_STALL)) scal[8] = 1.0;
}

// steps between two host reads of the stop flag (FP64 phase)
#define PURIF_CHECK 4

// D update (pscf/purif.c:441-455)
__global__ void k_purif_update(double *__restrict__ D, const double *__restrict__ D2, const double *__restrict__ D3,
                               size_t nn, const double *scal)
{
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nn) return;
    const double c = scal[7];
    if (!isfinite(c)) return;
    if (c < 0.5) D[k] = ((1.0 - 2.0 * c) * D[k] + (1.0 + c) * D2[k] - D3[k]) / (1.0 - c);
    else D[k] = ((1.0 + c) * D2[k] - D3[k]) / c;
}

// D = (D + D^T) / 2 (the split-BF16 products are symmetric only to FP32
// rounding; the FP64 steps assume a symmetric D, as D D^T = D^2)
__global__ void k_symmetrize(double *__restrict__ D, int n)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= n || j <= i) return;
    const double v = 0.5 * (D[(size_t)i * n + j] + D[(size_t)j * n + i]);
    D[(size_t)i * n + j] = v;
    D[(size_t)j * n + i] = v;
}

// cur = W - W^T (F D S - (F D S)^T, pscf/purif.c:553-558)
__global__ void k_antisym(const double *__restrict__ W, double *__restrict__ cur, int n)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= n) return;
    cur[(size_t)i * n + j] = W[(size_t)i * n + j] - W[(size_t)j * n + i];
}

__global__ void k_diis_reset(DiisState *ds) { diis_reset(ds, threadIdx.x, blockDim.x); }

// slot of this iteration: the next free one, else the largest-error one
__global__ void k_diis_slot(DiisState *ds) { diis_slot(ds); }

// block partials of <e, e_k> for the stored vectors k < len, slot `cur`
// standing for e itself, which is stored into it on the way
__global__ void k_dots(const double *__restrict__ e, double *__restrict__ vecs, size_t nn, const DiisState *ds,
                       double *__restrict__ part)
{
    __shared__ double s[RED_THREADS];
    const int m = ds->len, cur = ds->cur;
    for (int k = 0; k < m; k++) {
        double *b = vecs + nn * k;
        double v = 0.0;
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += (size_t)gridDim.x * blockDim.x) {
            const double a = e[i];
            if (k == cur) {
                b[i] = a;
                v += a * a;
            } else {
                v += a * b[i];
            }
        }
        s[threadIdx.x] = v;
        __syncthreads();
        for (int st = RED_THREADS / 2; st > 0; st >>= 1) {
            if (threadIdx.x < st) s[threadIdx.x] += s[threadIdx.x + st];
            __syncthreads();
        }
        if (threadIdx.x == 0) part[blockIdx.x * PUR_MAX_DIIS + k] = s[0];
        __syncthreads();
    }
}

// New row and column of b from the block partials, then the largest-error
// slot and the coefficients (diis_coefficients).  One warp: lane i sums the
// partials of column i in block order.
__global__ void k_diis_solve(const double *__restrict__ part, DiisState *ds)
{
    __shared__ double dots[PUR_MAX_DIIS];
    const int lane = threadIdx.x;
    if (lane < ds->len) {
        double v = 0.0;
#pragma unroll 8
        for (int bk = 0; bk < RED_BLOCKS; bk++) v += part[bk * PUR_MAX_DIIS + lane];
        dots[lane] = v;
    }
    __syncwarp();
    diis_update_solve(ds, dots, lane);
}

// F = sum_i c_i F_i over the stored Fock matrices, slot `cur` standing for
// this iteration's X F X (Fx), which is stored into it on the way
__global__ void k_combine(double *__restrict__ F, double *__restrict__ Fvecs, const double *__restrict__ Fx, size_t nn,
                          const DiisState *ds)
{
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nn) return;
    const int m = ds->len, cur = ds->cur;
    const double fx = Fx[k];
    Fvecs[nn * cur + k] = fx;
    double v = 0.0;
    for (int i = 0; i < m; i++) v += ds->co[i] * (i == cur ? fx : Fvecs[nn * i + k]);
    F[k] = v;
}

extern "C" int gtf_purif_create(int nbf, int nocc, void *stream, gtf_purif_dev_t **out)
{
    *out = nullptr;
    if (nbf <= 0 || nocc < 0 || nocc > nbf) return GTF_ERR_INVALID;
    gtf_purif_dev *p = new gtf_purif_dev();
    memset(p, 0, sizeof(*p));
    p->n = nbf;
    p->nocc = nocc;
    p->st = (cudaStream_t)stream;
    if (!p->st) {
        CKP(cudaStreamCreateWithFlags(&p->st, cudaStreamNonBlocking));
        p->own_st = 1;
    }
    // device buffers from the stream-ordered pool on the object's stream,
    // pinned host scalars from the pinned pool (devmem.cu): creating and
    // destroying this object synchronizes nothing else
    const size_t nn = (size_t)nbf * nbf;
    double **bufs[] = {&p->S, &p->X, &p->D, &p->D2, &p->D3, &p->F, &p->W, &p->W2, &p->E};
    for (double **b : bufs) CKP(gtf_dmalloc((void **)b, sizeof(double) * nn, p->st));
    CKP(gtf_dmalloc((void **)&p->vecs, sizeof(double) * nn * PUR_MAX_DIIS, p->st));
    CKP(gtf_dmalloc((void **)&p->Fvecs, sizeof(double) * nn * PUR_MAX_DIIS, p->st));
    CKP(gtf_dmalloc((void **)&p->part, sizeof(double) * part_len(p->n), p->st));
    CKP(gtf_dmalloc((void **)&p->scal, sizeof(double) * 16, p->st));
    p->h_scal = (double *)gtf_pinned_alloc(sizeof(double) * 16);
    if (!p->h_scal) return GTF_ERR_ALLOC;
    CKP(gtf_dmalloc((void **)&p->ds, sizeof(DiisState), p->st));
    CKP(cudaEventCreate(&p->e0));
    CKP(cudaEventCreate(&p->e1));
    k_diis_reset<<<1, 128, 0, p->st>>>(p->ds);
    CKP(cudaGetLastError());
    *out = p;
    return GTF_OK;
}

extern "C" int gtf_purif_set_mode(gtf_purif_dev_t *p, int mode)
{
    if (mode != 0 && mode != 1) return GTF_ERR_INVALID;
    if (mode == 1 && !p->bx) {
        const int r = gtf_bf16x3_create(p->n, p->st, &p->bx);
        if (r != GTF_OK) return r;
    }
    p->mode = mode;
    return GTF_OK;
}

extern "C" void gtf_purif_last_iters(gtf_purif_dev_t *p, int *bf16_iters, int *fp64_iters)
{
    if (bf16_iters) *bf16_iters = p->it_bf16;
    if (fp64_iters) *fp64_iters = p->it_fp64;
}

extern "C" void gtf_purif_destroy(gtf_purif_dev_t *p)
{
    if (!p) return;
    cudaStreamSynchronize(p->st);
    if (p->bx) gtf_bf16x3_destroy(p->bx);
    double *bufs[] = {p->S, p->X, p->D, p->D2, p->D3, p->F, p->W, p->W2, p->E, p->vecs, p->Fvecs, p->part, p->scal};
    for (double *b : bufs) gtf_dfree(b, p->st);
    gtf_dfree(p->ds, p->st);
    gtf_pinned_free(p->h_scal);
    if (p->e0) cudaEventDestroy(p->e0);
    if (p->e1) cudaEventDestroy(p->e1);
    if (p->own_st) cudaStreamDestroy(p->st);
    delete p;
}

// forget the DIIS history (a new SCF solve starts); stream-ordered
extern "C" void gtf_purif_reset(gtf_purif_dev_t *p)
{
    k_diis_reset<<<1, 128, 0, p->st>>>(p->ds);
    gtf_note_launches(1);
}

extern "C" int gtf_purif_set_sx(gtf_purif_dev_t *p, const double *S_host, const double *X_host)
{
    const size_t nn = (size_t)p->n * p->n;
    CKP(cudaMemcpyAsync(p->S, S_host, sizeof(double) * nn, cudaMemcpyHostToDevice, p->st));
    CKP(cudaMemcpyAsync(p->X, X_host, sizeof(double) * nn, cudaMemcpyHostToDevice, p->st));
    CKP(cudaStreamSynchronize(p->st));
    p->sx_set = 1;
    return GTF_OK;
}

extern "C" int gtf_purif_set_sx_dev(gtf_purif_dev_t *p, const double *S_dev, const double *X_dev)
{
    const size_t nn = (size_t)p->n * p->n;
    CKP(cudaMemcpyAsync(p->S, S_dev, sizeof(double) * nn, cudaMemcpyDeviceToDevice, p->st));
    CKP(cudaMemcpyAsync(p->X, X_dev, sizeof(double) * nn, cudaMemcpyDeviceToDevice, p->st));
    p->sx_set = 1;
    return GTF_OK;
}

extern "C" int gtf_purif_run_dev(gtf_purif_dev_t *p, const double *F_dev, double *D_dev, int *iters)
{
    BlasLease lease(p->st);
    if (!lease.h) return GTF_ERR_CUDA;
    p->blas = lease.h;
    const int n = p->n;
    const size_t nn = (size_t)n * n;
    const unsigned ge = (unsigned)((nn + 255) / 256);
    cudaStream_t st = p->st;
    CKP(cudaEventRecord(p->e0, st));
    const int gb = (n + GERSH_COLS - 1) / GERSH_COLS;
    k_gersh<<<gb, RED_THREADS, 0, st>>>(F_dev, n, p->part);
    k_purif_init<<<1, 32, 0, st>>>(p->part, gb, n, p->nocc, p->scal);
    k_purif_d0<<<ge, 256, 0, st>>>(F_dev, p->D, n, p->scal);
    CKP(cudaGetLastError());
    gtf_note_launches(3);
    int it;
    double err = 0.0;
    // split-BF16 phase: tensor-core products until the error stops falling
    // (their rounding sets a floor near 2^-16 relative), then FP64 steps
    p->it_bf16 = 0;
    if (p->mode == 1 && p->bx) {
        CKP(cudaMemsetAsync(p->scal + 8, 0, sizeof(double) * 4, st));
        double best = 1e300;
        int stall = 0;
        for (int k = 0; k < PUR_MAX_ITERS; k++) {
            if (gtf_bf16x3_abt(p->bx, p->D, p->D, p->D2, st)) return GTF_ERR_CUDA;
            if (gtf_bf16x3_abt(p->bx, p->D, p->D2, p->D3, st)) return GTF_ERR_CUDA;
            k_purif_stats<<<RED_BLOCKS, RED_THREADS, 0, st>>>(p->D, p->D2, p->D3, n, p->part);
            k_purif_finish<<<1, 32, 0, st>>>(p->part, RED_BLOCKS, p->scal);
            k_purif_update<<<ge, 256, 0, st>>>(p->D, p->D2, p->D3, nn, p->scal);
            k_symmetrize<<<dim3((n + 127) / 128, n), 128, 0, st>>>(p->D, n);
            CKP(cudaGetLastError());
            gtf_note_launches(4);
            CKP(cudaMemcpyAsync(p->h_scal + 6, p->scal + 6, sizeof(double) * 2, cudaMemcpyDeviceToHost, st));
            CKP(cudaStreamSynchronize(st));
            p->it_bf16++;
            const double e = p->h_scal[6];
            // hand over to FP64 once the error is small or stops falling
            // (BF16 rounding floor)
            if (!(e == e) || e < 1e-2) break;
            if (e < 0.99 * best) {
                best = e;
                stall = 0;
            } else if (++stall >= 3) {
                break;
            }
        }
    }
    // FP64 canonical steps (from the split-BF16 state in mode 1, which is
    // symmetrised), PURIF_CHECK launched per host read of the device-side stop
    // flag.  The first read also tells whether F was symmetric but for rounding
    // (1e-11 of its Gershgorin bound; X F X leaves 1e-14 to 1e-12).  If not, D D^2
    // is not symmetric either, and the loop starts again with it in full.
    CKP(cudaMemsetAsync(p->scal + 8, 0, sizeof(double) * 5, st));
    bool known = p->it_bf16 > 0, symmetric = true;
    if (!known) {
        const int nt = (n + ST_TILE - 1) / ST_TILE;
        k_asymmetry<<<nt * (nt + 1) / 2, 256, 0, st>>>(F_dev, n, p->scal);
        CKP(cudaGetLastError());
        gtf_note_launches(1);
    }
    int steps = 0;
    bool stopped = false;
    for (it = 0; it < PUR_MAX_ITERS && !stopped;) {
        for (int k = 0; k < PURIF_CHECK && it < PUR_MAX_ITERS; k++, it++) {
            if (sym_abt(p, p->D, p->D, p->D2)) return GTF_ERR_CUDA;
            if (symmetric ? sym_abt(p, p->D, p->D2, p->D3) : full_abt(p, p->D, p->D2, p->D3)) return GTF_ERR_CUDA;
            k_purif_stats<<<RED_BLOCKS, RED_THREADS, 0, st>>>(p->D, p->D2, p->D3, n, p->part);
            k_purif_finish<<<1, 32, 0, st>>>(p->part, RED_BLOCKS, p->scal);
            k_purif_update<<<ge, 256, 0, st>>>(p->D, p->D2, p->D3, nn, p->scal);
            CKP(cudaGetLastError());
            gtf_note_launches(3);
        }
        CKP(cudaMemcpyAsync(p->h_scal + 2, p->scal + 2, sizeof(double) * 11, cudaMemcpyDeviceToHost, st));
        CKP(cudaStreamSynchronize(st));
        err = p->h_scal[6];
        steps = (int)p->h_scal[9];
        stopped = p->h_scal[8] != 0.0;
        if (!known) {
            known = true;
            symmetric = p->h_scal[12] <= 1e-11 * fmax(fabs(p->h_scal[2]), fabs(p->h_scal[3]));   // false for a NaN
            if (!symmetric) {
                k_purif_d0<<<ge, 256, 0, st>>>(F_dev, p->D, n, p->scal);
                CKP(cudaGetLastError());
                gtf_note_launches(1);
                CKP(cudaMemsetAsync(p->scal + 8, 0, sizeof(double) * 4, st));
                it = 0;
                stopped = false;
            }
        }
    }
    p->errnorm = err;
    // the counts of the reference's loop: steps run, and the index of the
    // step that met the tolerance
    p->it_fp64 = stopped ? steps : PUR_MAX_ITERS;
    it = (stopped ? steps - 1 : PUR_MAX_ITERS) + p->it_bf16;
    // D_AO = X D X (pscf/purif.c:469-476)
    if (gemm_abt(p, p->X, p->D, p->W)) return GTF_ERR_CUDA;
    if (gemm_abt(p, p->W, p->X, D_dev)) return GTF_ERR_CUDA;
    CKP(cudaEventRecord(p->e1, st));
    CKP(cudaEventSynchronize(p->e1));
    float ms = 0.0f;
    CKP(cudaEventElapsedTime(&ms, p->e0, p->e1));
    p->ms_total = ms;
    if (iters) *iters = (it < PUR_MAX_ITERS) ? it : PUR_MAX_ITERS;
    return GTF_OK;
}

extern "C" int gtf_purif_run(gtf_purif_dev_t *p, const double *F_host, double *D_host, int *iters)
{
    const size_t nn = (size_t)p->n * p->n;
    CKP(cudaMemcpyAsync(p->F, F_host, sizeof(double) * nn, cudaMemcpyHostToDevice, p->st));
    int r = gtf_purif_run_dev(p, p->F, p->D2, iters);
    if (r) return r;
    CKP(cudaMemcpyAsync(D_host, p->D2, sizeof(double) * nn, cudaMemcpyDeviceToHost, p->st));
    CKP(cudaStreamSynchronize(p->st));
    return GTF_OK;
}

// One DIIS step (pscf/purif.c:491-641) with its bookkeeping on the device:
// no host synchronisation.  iter <= 1: F = X F X only.
extern "C" int gtf_diis_step_dev(gtf_purif_dev_t *p, const double *D_dev, double *F_dev, int iter)
{
    BlasLease lease(p->st);
    if (!lease.h) return GTF_ERR_CUDA;
    p->blas = lease.h;
    const int n = p->n;
    const size_t nn = (size_t)n * n;
    cudaStream_t st = p->st;
    if (iter <= 1) {
        // F = X F X
        if (gemm_abt(p, p->X, F_dev, p->W)) return GTF_ERR_CUDA;
        if (gemm_abt(p, p->W, p->X, F_dev)) return GTF_ERR_CUDA;
        return GTF_OK;
    }
    k_diis_slot<<<1, 1, 0, st>>>(p->ds);
    // error vector e = X (F D S - S D F) X (pscf/purif.c:540-566)
    if (gemm_abt(p, F_dev, D_dev, p->W)) return GTF_ERR_CUDA;
    if (gemm_abt(p, p->W, p->S, p->W2)) return GTF_ERR_CUDA;
    dim3 g((n + 127) / 128, n);
    k_antisym<<<g, 128, 0, st>>>(p->W2, p->E, n);
    if (gemm_abt(p, p->X, p->E, p->W)) return GTF_ERR_CUDA;
    if (gemm_abt(p, p->W, p->X, p->E)) return GTF_ERR_CUDA;
    k_dots<<<RED_BLOCKS, RED_THREADS, 0, st>>>(p->E, p->vecs, nn, p->ds, p->part);
    k_diis_solve<<<1, 32, 0, st>>>(p->part, p->ds);
    // this iteration's X F X, then the extrapolation
    if (gemm_abt(p, p->X, F_dev, p->W)) return GTF_ERR_CUDA;
    if (gemm_abt(p, p->W, p->X, p->W2)) return GTF_ERR_CUDA;
    k_combine<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(F_dev, p->Fvecs, p->W2, nn, p->ds);
    CKP(cudaGetLastError());
    gtf_note_launches(5);
    return GTF_OK;
}

extern "C" int gtf_diis_step(gtf_purif_dev_t *p, const double *D_host, double *F_host, int iter)
{
    const size_t nn = (size_t)p->n * p->n;
    CKP(cudaMemcpyAsync(p->F, F_host, sizeof(double) * nn, cudaMemcpyHostToDevice, p->st));
    CKP(cudaMemcpyAsync(p->D3, D_host, sizeof(double) * nn, cudaMemcpyHostToDevice, p->st));
    int r = gtf_diis_step_dev(p, p->D3, p->F, iter);
    if (r) return r;
    CKP(cudaMemcpyAsync(F_host, p->F, sizeof(double) * nn, cudaMemcpyDeviceToHost, p->st));
    CKP(cudaStreamSynchronize(p->st));
    return GTF_OK;
}

extern "C" int gtf_purif_stats(gtf_purif_dev_t *p, double *ms_gemm, double *ms_total, double *errnorm,
                               double *idem_err, double *tr_err)
{
    if (ms_gemm) *ms_gemm = p->ms_gemm;
    if (ms_total) *ms_total = p->ms_total;
    if (errnorm) *errnorm = p->errnorm;
    if (idem_err) *idem_err = p->idem;
    if (tr_err) *tr_err = p->trerr;
    return GTF_OK;
}
