// Device-resident flexible PCG for K u = b with the bilinear-FEM
// preconditioner (include/iga_solve.h).
//
// Reference loop (matrix_free/iteration_number_fempc_mf.cpp:193-233): PETSc
// KSPSolve on the MATSHELL operator, PCSHELL apply = inner KSPCG + PCJACOBI on
// the FEM matrix to rtol = abstol = 1e-10 (:210-224). Here every vector, every
// scalar (alpha, beta, dot products) and every convergence test lives on the
// device; the host only reads one flag per outer iteration. All reductions
// are deterministic (fixed-order block partials, summed by the last block).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <random>
#include <cmath>
#include <cstring>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include "../../include/iga_solve.h"
#include "iga_fastdiag.hpp"
#include "iga_fem.hpp"
#include "iga_gemm.hpp"
#include "iga_plan.hpp"

namespace iga {

constexpr int kRedBlocks = 592;   // fixed grid of every reduction kernel (4 x 148 SMs)
constexpr int kThreads = 256;
constexpr int kChunk = 16;        // inner CG iterations per captured graph

struct DevScalars {
    double alpha, beta, rz, rzo, rr, rr0, tol2, bb; // outer PCG (rzo = r_new . z_old)
    double ialpha, ibeta, irz, irr, itol2;          // inner FEM-CG
    int done, breakdown, idone, iiters, ibreak, imax;
    int err;                                        // a bounded wait in a kernel gave up
    int it, maxit;                                  // outer PCG in a device-side loop
    long long ipc;                                  // inner iterations of one call's cluster FEM-CG solves
    double rzv[2];                                  // r.z of the PCG loop's even / odd iterations
};

}  // namespace iga

#include "iga_femcg.cuh"

namespace iga {

// ------------------------------------------------------------ reductions
// Block sums of K values; the last block to finish sums the per-block
// partials in block order and returns true (thread 0 holds the totals).
template <int K>
__device__ bool reduce_last(double (&v)[K], double *partials, unsigned *counter, double (&tot)[K])
{
    __shared__ double sh[K][kThreads / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = v[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) sh[k][wid] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double s = 0.0;
            for (int w = 0; w < kThreads / 32; ++w) s += sh[k][w];
            partials[blockIdx.x * K + k] = s;
        }
        __threadfence();
        const unsigned t = atomicAdd(counter, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    // Last block: every thread sums a fixed subset of the partials in block
    // order, then a fixed-shape tree (warp shuffles, then warp 0) combines them.
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads) s += ((volatile double *)partials)[b * K + k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) sh[k][wid] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double s = 0.0;
            for (int w = 0; w < kThreads / 32; ++w) s += sh[k][w];
            tot[k] = s;
        }
        *counter = 0u;
    }
    return true;
}

// Blocks of a loop kernel over N entries: 16 bytes a thread, at most
// kRedBlocks (a 64^2 patch's 592 mostly empty blocks cost 0.5 us a launch and
// 0.9 us a reduction more than its 9).
template <typename T>
static int vec_blocks(long long N)
{
    const long long per = (long long)kThreads * (16 / (long long)sizeof(T));
    return (int)std::max(1LL, std::min<long long>(kRedBlocks, (N + per - 1) / per));
}

// One partial sum per block, v summed over the block in a fixed order.
__device__ __forceinline__ void put_partial(double v, double *part)
{
    __shared__ double sh[kThreads / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) s += sh[w];
        part[blockIdx.x] = s;
    }
}

// The sum of an earlier kernel's np block partials, in every thread of every
// block, in the same order. The kernel that needs a dot product sums its
// partials itself instead of the producer's last block (whose fence, counter
// and second pass are serial: a producer and consumer 4.0 us apart with 592
// blocks against 5.3, 2.8 against 3.8 with 16).
__device__ __forceinline__ double sum_partials(const double *part, int np)
{
    __shared__ double sh[kThreads / 32];
    double v = 0.0;
    for (int b = threadIdx.x; b < np; b += kThreads) v += __ldcg(part + b);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) v += sh[w];
    return v;
}

__device__ __forceinline__ bool bnd(int i, int j, int m, int n) { return i == 0 || j == 0 || i == m - 1 || j == n - 1; }

// ------------------------------------------------------------ FEM stencil
// K_fem = Kx (x) My + Mx (x) Ky on the free nodes (1-D linear-element
// stiffness K and mass M from the node coordinates; the 2x2-Gauss bilinear
// element matrices of matrix_free/src/ElementFEM.cpp:3-117 are exactly these
// tensor products), identity rows on the boundary.
template <typename T>
struct FemCoef {
    const T *kd, *ko, *md, *mo;   // x: diag / off-diagonal (i,i+1)
    const T *ld, *lo, *nd, *no;   // y: stiffness diag / off, mass diag / off
    int m, n;
};

template <typename T>
__device__ __forceinline__ T fem_row(const T *__restrict__ p, int i, int j, const FemCoef<T> &c)
{
    const T kx[3] = {c.ko[i - 1], c.kd[i], c.ko[i]}, mx[3] = {c.mo[i - 1], c.md[i], c.mo[i]};
    const T ky[3] = {c.lo[j - 1], c.ld[j], c.lo[j]}, my[3] = {c.no[j - 1], c.nd[j], c.no[j]};
    const bool xl = i - 1 >= 1, xr = i + 1 <= c.m - 2, yl = j - 1 >= 1, yr = j + 1 <= c.n - 2;
    T s = 0;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        if ((b == 0 && !yl) || (b == 2 && !yr)) continue;
        const T *row = p + (size_t)(j + b - 1) * c.m;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if ((a == 0 && !xl) || (a == 2 && !xr)) continue;
            s += (kx[a] * my[b] + mx[a] * ky[b]) * row[i + a - 1];
        }
    }
    return s;
}

template <typename T>
__device__ __forceinline__ T fem_diag(int i, int j, const FemCoef<T> &c)
{
    return c.kd[i] * c.nd[j] + c.md[i] * c.ld[j];
}

template <typename T>
__global__ void fem_apply_kernel(const T *__restrict__ x, T *__restrict__ y, FemCoef<T> c)
{
    const long long N = (long long)c.m * c.n;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % c.m), j = (int)(t / c.m);
        y[t] = bnd(i, j, c.m, c.n) ? x[t] : fem_row(x, i, j, c);
    }
}

// CSR rows of the FEM matrix (sorted columns); rowptr precomputed on the host.
__global__ void fem_csr_kernel(const int32_t *__restrict__ rowptr, int32_t *__restrict__ col, double *__restrict__ val,
                               FemCoef<double> c, double sign)
{
    const long long N = (long long)c.m * c.n;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % c.m), j = (int)(t / c.m);
        int k = rowptr[t];
        if (bnd(i, j, c.m, c.n)) {
            col[k] = (int32_t)t;
            val[k] = 1.0;
            continue;
        }
        const double kx[3] = {c.ko[i - 1], c.kd[i], c.ko[i]}, mx[3] = {c.mo[i - 1], c.md[i], c.mo[i]};
        const double ky[3] = {c.lo[j - 1], c.ld[j], c.lo[j]}, my[3] = {c.no[j - 1], c.nd[j], c.no[j]};
        for (int b = 0; b < 3; ++b) {
            const int jj = j + b - 1;
            if (jj < 1 || jj > c.n - 2) continue;
            for (int a = 0; a < 3; ++a) {
                const int ii = i + a - 1;
                if (ii < 1 || ii > c.m - 2) continue;
                col[k] = (int32_t)((long long)jj * c.m + ii);
                val[k] = sign * (kx[a] * my[b] + mx[a] * ky[b]);
                ++k;
            }
        }
    }
}

// ------------------------------------------------------------ inner FEM-CG (the PC apply)
// Jacobi-preconditioned CG on K_fem z = r_in to ||r|| <= pc_rtol ||r_in||.
template <typename T>
struct InnerCG {
    T *z, *r, *p, *q;
    const T *rhs;
    FemCoef<T> c;
    DevScalars *s;
    double *partials;
    unsigned *counter;
};

template <typename T>
__global__ void icg_init_kernel(InnerCG<T> a, const T *__restrict__ rhs, double rtol, int maxit)
{
    const long long N = (long long)a.c.m * a.c.n;
    double v[2] = {0.0, 0.0};
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % a.c.m), j = (int)(t / a.c.m);
        const T r = rhs[t];
        const T d = bnd(i, j, a.c.m, a.c.n) ? T(1) : fem_diag(i, j, a.c);
        const T zz = r / d;
        a.z[t] = 0;
        a.r[t] = r;
        a.p[t] = zz;
        v[0] += (double)r * (double)zz;
        v[1] += (double)r * (double)r;
    }
    double tot[2];
    if (reduce_last<2>(v, a.partials, a.counter, tot) && threadIdx.x == 0) {
        a.s->irz = tot[0];
        a.s->irr = tot[1];
        a.s->itol2 = rtol * rtol * tot[1];
        a.s->iiters = 0;
        a.s->imax = maxit;
        a.s->ibreak = 0;
        a.s->idone = (tot[1] == 0.0) ? 1 : 0;
    }
}

template <typename T>
__global__ void icg_q_kernel(InnerCG<T> a)
{
    if (a.s->idone) return;
    const long long N = (long long)a.c.m * a.c.n;
    double v[1] = {0.0};
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % a.c.m), j = (int)(t / a.c.m);
        const T pv = a.p[t];
        const T qv = bnd(i, j, a.c.m, a.c.n) ? pv : fem_row(a.p, i, j, a.c);
        a.q[t] = qv;
        v[0] += (double)pv * (double)qv;
    }
    double tot[1];
    if (reduce_last<1>(v, a.partials, a.counter, tot) && threadIdx.x == 0) {
        if (!(tot[0] > 0.0)) {
            a.s->ibreak = 1;
            a.s->idone = 1;
        } else {
            a.s->ialpha = a.s->irz / tot[0];
        }
    }
}

template <typename T>
__global__ void icg_update_kernel(InnerCG<T> a)
{
    if (a.s->idone) return;
    const long long N = (long long)a.c.m * a.c.n;
    const T al = (T)a.s->ialpha;
    double v[2] = {0.0, 0.0};
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % a.c.m), j = (int)(t / a.c.m);
        a.z[t] += al * a.p[t];
        const T r = a.r[t] - al * a.q[t];
        a.r[t] = r;
        const T d = bnd(i, j, a.c.m, a.c.n) ? T(1) : fem_diag(i, j, a.c);
        v[0] += (double)r * (double)(r / d);
        v[1] += (double)r * (double)r;
    }
    double tot[2];
    if (reduce_last<2>(v, a.partials, a.counter, tot) && threadIdx.x == 0) {
        a.s->ibeta = tot[0] / a.s->irz;
        a.s->irz = tot[0];
        a.s->irr = tot[1];
        a.s->iiters += 1;
        if (tot[1] <= a.s->itol2 || a.s->iiters >= a.s->imax || !(tot[1] == tot[1])) a.s->idone = 1;
    }
}

template <typename T>
__global__ void icg_p_kernel(InnerCG<T> a)
{
    if (a.s->idone) return;
    const long long N = (long long)a.c.m * a.c.n;
    const T be = (T)a.s->ibeta;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % a.c.m), j = (int)(t / a.c.m);
        const T d = bnd(i, j, a.c.m, a.c.n) ? T(1) : fem_diag(i, j, a.c);
        a.p[t] = a.r[t] / d + be * a.p[t];
    }
}

// ------------------------------------------------------------ outer PCG vector kernels
// Elementwise loops move 16 bytes per access (4 floats / 2 doubles) when every
// array of the kernel starts on a 16-byte boundary; the last N % VN entries
// (or all of them, for unaligned arrays) take scalar accesses. The thread that
// handles an entry depends only on N and the grid, so the reductions stay
// deterministic.
template <typename T>
struct alignas(16) Pk {
    static constexpr int n = 16 / sizeof(T);
    T v[n];
};

template <typename T>
__device__ __forceinline__ Pk<T> ldp(const T *a, long long i)
{
    return *reinterpret_cast<const Pk<T> *>(a + i);
}

template <typename T>
__device__ __forceinline__ void stp(T *a, long long i, const Pk<T> &v)
{
    *reinterpret_cast<Pk<T> *>(a + i) = v;
}

__device__ __forceinline__ bool al16(const void *a) { return ((uintptr_t)a & 15u) == 0; }

// Calls f(i, c) for the first entry i and count c of every pack this thread
// owns, then f(i, 1) for its scalar tail entries.
template <typename T, typename F>
__device__ __forceinline__ void vloop(long long N, bool vec, F &&f)
{
    constexpr int VN = Pk<T>::n;
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x, st = (long long)gridDim.x * blockDim.x;
    const long long nv = vec ? N / VN : 0;
    for (long long k = g; k < nv; k += st) f(k * VN, VN);
    for (long long i = nv * VN + g; i < N; i += st) f(i, 1);
}

// Loads c entries (a pack or one scalar) starting at i.
template <typename T>
__device__ __forceinline__ Pk<T> ldc(const T *a, long long i, int c)
{
    if (c > 1) return ldp(a, i);
    Pk<T> v;
    v.v[0] = a[i];
    return v;
}

template <typename T>
__device__ __forceinline__ void stc(T *a, long long i, int c, const Pk<T> &v)
{
    if (c > 1) stp(a, i, v);
    else a[i] = v.v[0];
}

template <typename T>
__global__ void dot_kernel(const T *__restrict__ a, const T *__restrict__ b, long long N, double *out, double *partials,
                           unsigned *counter)
{
    double v[1] = {0.0};
    vloop<T>(N, al16(a) && al16(b), [&](long long i, int c) {
        const Pk<T> x = ldc(a, i, c), y = ldc(b, i, c);
#pragma unroll
        for (int k = 0; k < Pk<T>::n; ++k)
            if (k < c) v[0] += (double)x.v[k] * (double)y.v[k];
    });
    double tot[1];
    if (reduce_last<1>(v, partials, counter, tot) && threadIdx.x == 0) *out = tot[0];
}

// ---- the Lanczos process's kernels (iga_spectrum_estimate: the host reads each
// dot product's total from S)
// alpha = rz / (p.q) from the device scalars
template <typename T>
__global__ void pcg_pq_kernel(const T *__restrict__ p, const T *__restrict__ q, long long N, DevScalars *s,
                              double *partials, unsigned *counter)
{
    pdl_begin();
    double v[1] = {0.0};
    vloop<T>(N, al16(p) && al16(q), [&](long long i, int c) {
        const Pk<T> a = ldc(p, i, c), b = ldc(q, i, c);
#pragma unroll
        for (int k = 0; k < Pk<T>::n; ++k)
            if (k < c) v[0] += (double)a.v[k] * (double)b.v[k];
    });
    double tot[1];
    if (reduce_last<1>(v, partials, counter, tot) && threadIdx.x == 0) {
        if (!(tot[0] > 0.0) || s->breakdown) {   // breakdown already set: by the preconditioner
            s->breakdown = 1;
            s->alpha = 0.0;
        } else {
            s->alpha = s->rz / tot[0];
        }
    }
}

// x += alpha p, r -= alpha q; rr = r.r and rzo = r.z with the previous
// preconditioned residual z (the flexible beta's correction term, taken here
// so that z need not be kept). Returns the totals to the last block.
template <typename T>
__device__ __forceinline__ bool xr_update(T *__restrict__ x, T *__restrict__ r, const T *__restrict__ p,
                                          const T *__restrict__ q, const T *__restrict__ z, long long N, T al,
                                          double *partials, unsigned *counter, double (&tot)[2])
{
    double v[2] = {0.0, 0.0};
    vloop<T>(N, al16(x) && al16(r) && al16(p) && al16(q) && al16(z), [&](long long i, int c) {
        Pk<T> xv = ldc(x, i, c), rv = ldc(r, i, c);
        const Pk<T> pv = ldc(p, i, c), qv = ldc(q, i, c), zv = ldc(z, i, c);
#pragma unroll
        for (int k = 0; k < Pk<T>::n; ++k) {
            if (k < c) {
                xv.v[k] += al * pv.v[k];
                rv.v[k] -= al * qv.v[k];
                v[0] += (double)rv.v[k] * (double)rv.v[k];
                v[1] += (double)rv.v[k] * (double)zv.v[k];
            }
        }
        stc(x, i, c, xv);
        stc(r, i, c, rv);
    });
    return reduce_last<2>(v, partials, counter, tot);
}

template <typename T>
__global__ void pcg_xr_kernel(T *__restrict__ x, T *__restrict__ r, const T *__restrict__ p, const T *__restrict__ q,
                              const T *__restrict__ z, long long N, DevScalars *s, double *partials, unsigned *counter)
{
    double tot[2];
    if (xr_update(x, r, p, q, z, N, (T)s->alpha, partials, counter, tot) && threadIdx.x == 0) {
        s->rr = tot[0];
        s->rzo = tot[1];
    }
}

// ---- the PCG loop's kernels: dot products as block partials, summed
// by the kernel that uses them (sum_partials); r.z of iteration `it` in
// rzv[it & 1], so that no block reads a scalar another block has replaced
template <typename T>
__global__ void __launch_bounds__(kThreads) loop_dot_kernel(const T *__restrict__ a, const T *__restrict__ b, long long N,
                                                            double *part)
{
    pdl_begin();
    double v = 0.0;
    vloop<T>(N, al16(a) && al16(b), [&](long long i, int c) {
        const Pk<T> x = ldc(a, i, c), y = ldc(b, i, c);
#pragma unroll
        for (int k = 0; k < Pk<T>::n; ++k)
            if (k < c) v += (double)x.v[k] * (double)y.v[k];
    });
    put_partial(v, part);
}

// Flexible (Polak-Ribiere) beta = r.(z - z_old) / rz_old with r.z_old = rzo
// from the last update, zero in the first iteration; p = z + beta p.
template <typename T>
__global__ void __launch_bounds__(kThreads) loop_p_kernel(T *__restrict__ p, const T *__restrict__ z, long long N,
                                                          DevScalars *s, const double *part, int np)
{
    pdl_begin();
    const double rz = sum_partials(part, np);
    const int it = s->it;
    const T be = it == 0 ? T(0) : (T)((rz - s->rzo) / s->rzv[(it & 1) ^ 1]);
    if (blockIdx.x == 0 && threadIdx.x == 0) s->rzv[it & 1] = rz;
    vloop<T>(N, al16(p) && al16(z), [&](long long i, int c) {
        const Pk<T> zv = ldc(z, i, c);
        if (it == 0) {   // the first direction never reads stale p
            stc(p, i, c, zv);
            return;
        }
        Pk<T> pv = ldc(p, i, c);
#pragma unroll
        for (int k = 0; k < Pk<T>::n; ++k) pv.v[k] = zv.v[k] + be * pv.v[k];
        stc(p, i, c, pv);
    });
}

// The device-side loop's condition (on = 0: the host drives the loop).
struct LoopCond {
    cudaGraphConditionalHandle h = 0;
    int on = 0;
};

// alpha = rz / p.q (zero, and a breakdown, unless p.q > 0); the update; counts
// the iteration (unless the preconditioner broke down) and sets the loop's
// condition (continue while rr > tol2, it < maxit, no breakdown, finite) where
// the loop runs on the device.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    loop_xr_kernel(T *__restrict__ x, T *__restrict__ r, const T *__restrict__ p, const T *__restrict__ q,
                   const T *__restrict__ z, long long N, DevScalars *s, const double *part, int np, double *partials,
                   unsigned *counter, LoopCond cond)
{
    pdl_begin();
    const double pq = sum_partials(part, np);
    const bool pc_bad = s->breakdown;   // set by the preconditioner
    const bool bad = !(pq > 0.0) || pc_bad;
    const double alpha = bad ? 0.0 : s->rzv[s->it & 1] / pq;
    double tot[2];
    if (xr_update(x, r, p, q, z, N, (T)alpha, partials, counter, tot) && threadIdx.x == 0) {
        s->alpha = alpha;
        if (bad) s->breakdown = 1;
        s->rr = tot[0];
        s->rzo = tot[1];
        if (!pc_bad) s->it += 1;
        const bool go = tot[0] > s->tol2 && s->it < s->maxit && !bad && tot[0] == tot[0];
        if (cond.on) cudaGraphSetConditional(cond.h, go ? 1u : 0u);
    }
}

__global__ void loop_init_kernel(DevScalars *s, double tol2, int maxit)
{
    s->tol2 = tol2;
    s->maxit = maxit;
    s->it = 0;
    s->breakdown = 0;
}

// p = z + beta p (first: p = z)
template <typename T>
__global__ void pcg_p_kernel(T *__restrict__ p, const T *__restrict__ z, long long N, const DevScalars *s, int first)
{
    pdl_begin();
    const T be = first ? T(0) : (T)s->beta;
    vloop<T>(N, al16(p) && al16(z), [&](long long i, int c) {
        const Pk<T> zv = ldc(z, i, c);
        if (first) {   // the first direction never reads stale p
            stc(p, i, c, zv);
            return;
        }
        Pk<T> pv = ldc(p, i, c);
#pragma unroll
        for (int k = 0; k < Pk<T>::n; ++k) pv.v[k] = zv.v[k] + be * pv.v[k];
        stc(p, i, c, pv);
    });
}

// r = b - Ax (FP64), rr = r.r, bb = b.b
__global__ void residual_kernel(const double *__restrict__ b, const double *__restrict__ Ax, double *__restrict__ r,
                                long long N, DevScalars *s, double *partials, unsigned *counter)
{
    double v[2] = {0.0, 0.0};
    vloop<double>(N, al16(b) && al16(Ax) && al16(r), [&](long long i, int c) {
        const Pk<double> bv = ldc(b, i, c), av = ldc(Ax, i, c);
        Pk<double> rv;
#pragma unroll
        for (int k = 0; k < Pk<double>::n; ++k) {
            rv.v[k] = bv.v[k] - av.v[k];
            if (k < c) {
                v[0] += rv.v[k] * rv.v[k];
                v[1] += bv.v[k] * bv.v[k];
            }
        }
        stc(r, i, c, rv);
    });
    double tot[2];
    if (reduce_last<2>(v, partials, counter, tot) && threadIdx.x == 0) {
        s->rr = tot[0];
        s->bb = tot[1];
    }
}

// r = b - q, rr = r.r
template <typename T>
__global__ void sub_kernel(const T *__restrict__ b, const T *__restrict__ q, T *__restrict__ r, long long N,
                           DevScalars *s, double *partials, unsigned *counter)
{
    double v[1] = {0.0};
    vloop<T>(N, al16(b) && al16(q) && al16(r), [&](long long i, int c) {
        const Pk<T> bv = ldc(b, i, c), qv = ldc(q, i, c);
        Pk<T> rv;
#pragma unroll
        for (int k = 0; k < Pk<T>::n; ++k) {
            rv.v[k] = bv.v[k] - qv.v[k];
            if (k < c) v[0] += (double)rv.v[k] * (double)rv.v[k];
        }
        stc(r, i, c, rv);
    });
    double tot[1];
    if (reduce_last<1>(v, partials, counter, tot) && threadIdx.x == 0) s->rr = tot[0];
}

template <typename T>
__global__ void copy_kernel(T *__restrict__ dst, const T *__restrict__ src, long long N)
{
    pdl_begin();
    vloop<T>(N, al16(dst) && al16(src), [&](long long i, int c) { stc(dst, i, c, ldc(src, i, c)); });
}

template <typename T>
__global__ void zero_kernel(T *__restrict__ dst, long long N)
{
    Pk<T> zv;
#pragma unroll
    for (int k = 0; k < Pk<T>::n; ++k) zv.v[k] = T(0);
    vloop<T>(N, al16(dst), [&](long long i, int c) { stc(dst, i, c, zv); });
}

// FP32 sweep right-hand side r32 = r64 / scale.
__global__ void scale_down_kernel(const double *__restrict__ r, float *__restrict__ r32, long long N, const DevScalars *s)
{
    const double inv = s->rr > 0.0 ? 1.0 / sqrt(s->rr) : 0.0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x)
        r32[t] = (float)(r[t] * inv);
}

// Refinement update x64 += scale * d32 (scale = ||r64|| of the sweep's rhs).
__global__ void refine_update_kernel(double *__restrict__ x, const float *__restrict__ d, long long N, double scale)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x)
        x[t] += scale * (double)d[t];
}

// Scale of an FP64 vector carried through an FP32 preconditioner: the input
// is divided by ||r|| (rr = r.r of the current residual) on the way down and
// the output multiplied by it on the way up, so FP32's exponent range holds
// any residual size. 1 when rr is zero or not finite.
__device__ __forceinline__ double pc_scale(const DevScalars *s)
{
    const double rr = s->rr;
    return (rr > 0.0 && rr < 1e300) ? sqrt(rr) : 1.0;
}

__global__ void to_fp32_kernel(const double *__restrict__ r, float *__restrict__ r32, long long N, const DevScalars *s)
{
    pdl_begin();
    const double inv = 1.0 / pc_scale(s);
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x)
        r32[t] = (float)(r[t] * inv);
}

__global__ void from_fp32_kernel(const float *__restrict__ z32, double *__restrict__ z, long long N, const DevScalars *s)
{
    pdl_begin();
    const double sc = pc_scale(s);
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x)
        z[t] = sc * (double)z32[t];
}

// ------------------------------------------------------------ exact FEM inverse (fast diagonalisation)
// ---- tridiagonal solves along y of the x-diagonalised FEM system
// For every x mode a < nx: (lx[a] My + Ky) t = w, w = column a of the nyp x nxp
// matrix Wt (y contiguous: element (b, a) at b + a nyp), in place. The LDL^T
// factors are precomputed per mode in the same layout: Lf_b = e_{b-1} / d_{b-1}
// (the unit lower factor's subdiagonal, Lf_0 = 0) and Dv_b = 1 / d_b, so
//   forward  u_b = w_b - Lf_b u_{b-1},       v_b = Dv_b u_b,
//   backward x_b = v_b - Lf_{b+1} x_{b+1}    (no term past the last free row).
// One CTA of NW warps per mode: thread t owns rows [t s, t s + s) with s odd,
// so that a warp's shared-memory accesses fall in distinct banks. Each
// recurrence is composed per thread into an affine map c -> E + P c, the maps
// are combined by a warp shuffle scan and across the warps through shared
// memory, and each thread then runs its rows from its carry-in. Arithmetic in
// T. STAGED: the mode's column and factors are brought into shared memory by
// the bulk-copy engine and the result is written back with 16-byte stores;
// else (columns too long for shared memory) the kernel works on them in place.
// Bound: the recurrences' latency, then bytes. A warp per mode with all of an
// SM's modes in one CTA had every warp load, then solve, then store at the
// same time (2048^2: FP32 25 us, FP64 50 us; two buffers per warp, half the
// warps: 30 and 67 us); CTAs of their own overlap these phases, and up to four
// warps shorten the chains in FP64: 22.7 and 31 us.

// inclusive scan of affine maps over lanes, lane order (forward) or reverse lane order
template <typename R>
__device__ __forceinline__ void affine_scan(R &E, R &P, int lane, bool reverse)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const R pe = reverse ? __shfl_down_sync(0xffffffffu, E, o) : __shfl_up_sync(0xffffffffu, E, o);
        const R pp = reverse ? __shfl_down_sync(0xffffffffu, P, o) : __shfl_up_sync(0xffffffffu, P, o);
        if (reverse ? lane + o < 32 : lane >= o) {
            E = E + P * pe;
            P = P * pp;
        }
    }
}

template <typename T, bool STAGED, int NW>
__global__ void __launch_bounds__(NW * 32)
fd_tri_kernel(T *__restrict__ W, const T *__restrict__ Lf, const T *__restrict__ Dv, int ny, int nyp, int seg,
              DevScalars *sc)
{
    pdl_launch();
    extern __shared__ __align__(16) unsigned char tri_smem[];
    __shared__ uint64_t bar;
    __shared__ T fE[NW], fP[NW], rE[NW], rP[NW];   // the warps' maps, forward and backward
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const size_t a = blockIdx.x;
    T *wg = W + a * nyp, *wp = wg;
    const T *lp = Lf + a * nyp, *dp = Dv + a * nyp;
    const uint32_t bytes = (uint32_t)nyp * (uint32_t)sizeof(T);
    if constexpr (STAGED) {
        T *wb = reinterpret_cast<T *>(tri_smem);
        if (t == 0) {   // the factors (constant) before the wait for the preceding grid, the column after it
            mbar_init(&bar, 1);
            fence_mbar_init();
            mbar_arrive_expect_tx(&bar, 3u * bytes);
            bulk_g2s(wb + nyp, lp, bytes, &bar);
            bulk_g2s(wb + 2 * nyp, dp, bytes, &bar);
        }
        wp = wb;
        lp = wb + nyp;
        dp = wb + 2 * nyp;
    }
    pdl_wait();
    if constexpr (STAGED) {
        if (t == 0) bulk_g2s(wp, wg, bytes, &bar);
        __syncthreads();   // the barrier is set up
        if (!__syncthreads_and(mbar_wait_bounded(&bar, 0))) {
            if (t == 0) sc->err = 1;
            mbar_wait_bounded(&bar, 0);   // let the copies land before leaving
            return;
        }
    }
    const int b0 = t * seg, b1 = min(b0 + seg, ny);
    // forward: this thread's map, the scan, then its rows from the carry-in
    T E = 0, P = 1;
#pragma unroll 4
    for (int b = b0; b < b1; ++b) {
        const T l = lp[b];
        E = wp[b] - l * E;
        P = -l * P;
    }
    affine_scan(E, P, lane, false);
    T c = 0;   // the carry into this warp
    if constexpr (NW > 1) {
        if (lane == 31) {
            fE[wid] = E;
            fP[wid] = P;
        }
        __syncthreads();
        for (int w = 0; w < wid; ++w) c = fE[w] + fP[w] * c;
    }
    const T pe = __shfl_up_sync(0xffffffffu, E, 1), pp = __shfl_up_sync(0xffffffffu, P, 1);
    T u = lane == 0 ? c : pe + pp * c;
#pragma unroll 4
    for (int b = b0; b < b1; ++b) {
        u = wp[b] - lp[b] * u;
        wp[b] = u * dp[b];
    }
    // backward over the same rows, threads in reverse order
    E = 0;
    P = 1;
#pragma unroll 4
    for (int b = b1 - 1; b >= b0; --b) {
        const T l = b + 1 < ny ? lp[b + 1] : T(0);
        E = wp[b] - l * E;
        P = -l * P;
    }
    affine_scan(E, P, lane, true);
    c = 0;
    if constexpr (NW > 1) {
        if (lane == 0) {
            rE[wid] = E;
            rP[wid] = P;
        }
        __syncthreads();
        for (int w = NW - 1; w > wid; --w) c = rE[w] + rP[w] * c;
    }
    const T ne = __shfl_down_sync(0xffffffffu, E, 1), np = __shfl_down_sync(0xffffffffu, P, 1);
    T x = lane == 31 ? c : ne + np * c;
#pragma unroll 4
    for (int b = b1 - 1; b >= b0; --b) {
        const T l = b + 1 < ny ? lp[b + 1] : T(0);
        x = wp[b] - l * x;
        wp[b] = x;
    }
    if constexpr (STAGED) {
        __syncthreads();
        const int nv = (int)((size_t)nyp * sizeof(T) / 16);
        const uint4 *src = reinterpret_cast<const uint4 *>(wp);
        uint4 *dst = reinterpret_cast<uint4 *>(wg);
        for (int i = t; i < nv; i += NW * 32) dst[i] = src[i];
    }
}

// Warps per mode: FP64, enough that a thread has few rows, no more than keep
// most threads busy. FP32 one: where a recurrence is cut moves its rounding, and
// in the smoothest modes (condition ~ 1e6) that is worth up to 4e-5 of z, more
// than FP32 results should depend on a launch shape (2048^2 with four warps: 17
// us).
template <typename T>
constexpr int tri_warps(int ny)
{
    return sizeof(T) == 4 || ny <= 96 ? 1 : ny <= 384 ? 2 : 4;
}
constexpr size_t kTriSmem = 226 * 1024;   // most shared memory of a staged mode (leaves room for the static part)

template <typename T, int NW>
static cudaError_t launch_tri(T *W, const T *Lf, const T *Dv, int nmodes, int ny, int nyp, cudaStream_t s, DevScalars *sc)
{
    const size_t smem = 3 * (size_t)nyp * sizeof(T);
    int seg = (ny + 32 * NW - 1) / (32 * NW);
    seg |= 1;   // odd: conflict-free shared-memory rows
    if (smem > kTriSmem)
        return launch_k(fd_tri_kernel<T, false, NW>, dim3(nmodes), dim3(NW * 32), 0, s, W, Lf, Dv, ny, nyp, seg, sc);
    return launch_k(fd_tri_kernel<T, true, NW>, dim3(nmodes), dim3(NW * 32), smem, s, W, Lf, Dv, ny, nyp, seg, sc);
}

template <typename T>
static cudaError_t tri_prepare()   // the staged kernels' shared-memory limit
{
    auto set = [](auto k) { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTriSmem); };
    cudaError_t e = set(fd_tri_kernel<T, true, 1>);
    if constexpr (sizeof(T) == 8) {
        if (e == cudaSuccess) e = set(fd_tri_kernel<T, true, 2>);
        if (e == cudaSuccess) e = set(fd_tri_kernel<T, true, 4>);
    }
    return e;
}

// Entry t of the boundary ring of the m x n grid (2 m + 2 (n - 2) entries).
__device__ __forceinline__ long long ring_index(long long t, int m, int n)
{
    if (t < m) return t;
    if (t < 2LL * m) return (long long)(n - 1) * m + (t - m);
    const long long u = t - 2LL * m;
    return (1 + u / 2) * m + ((u % 2) ? (m - 1) : 0);
}

// z = r on the boundary ring (identity rows of K_fem; ks r ks with a scaling
// ks), ring entries t0, t0 + stride, ...
template <typename T>
__device__ __forceinline__ void ring_copy(T *__restrict__ z, const T *__restrict__ r, const T *__restrict__ ks, int m,
                                          int n, long long t0, long long stride)
{
    const long long nb = 2LL * m + 2LL * (n - 2);
    for (long long t = t0; t < nb; t += stride) {
        const long long i = ring_index(t, m, n);
        z[i] = ks ? ks[i] * r[i] * ks[i] : r[i];
    }
}

// The exact inverse's gather and unfold move a row's 32 kFoldN columns per
// warp and step, lane by lane, so that every access is a whole line although
// the rows of r and z start anywhere, with kFoldN loads of each array in
// flight per lane (bound: bytes; 2048^2 FP32: gather 15 -> 11 us against 16-byte
// stores with scalar loads of their own, unfold 20.5 -> 9.4 us against one column).
constexpr int kFoldN = 4;

// Interior block of r (m x n grid, x fastest) into the zero-padded GEMM
// operand U [nyp][nxp], and the boundary ring of r into z (one launch fewer),
// both times the kappa scaling ks (or null). With sc (FP64 vectors, FP32
// transform) the values are divided by pc_scale. With the parity split (kb >
// 0) column c of U is, for c < kb, the even fold r[c] + r[nx-1-c] (c < fo; the
// middle entry r[fo] alone when nx is odd) and, for c >= kb, the odd fold
// r[j] - r[nx-1-j] with j = c - kb < fo.
template <typename T, typename V>
__global__ void __launch_bounds__(kThreads)
    fd_gather_kernel(const V *__restrict__ r, const V *__restrict__ ks, T *__restrict__ U, V *__restrict__ z, int m, int n,
                     int nx, int ny, int nxp, int nyp, int kb, int fo, const DevScalars *sc)
{
    pdl_begin();
    ring_copy(z, r, ks, m, n, blockIdx.x * (long long)kThreads + threadIdx.x, (long long)gridDim.x * kThreads);
    const double inv = sc ? 1.0 / pc_scale(sc) : 1.0;
    const int lane = threadIdx.x & 31, half = kb > 0 ? kb : nxp, cb = (half + 32 * kFoldN - 1) / (32 * kFoldN);
    const int w0 = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), ws = gridDim.x * (kThreads / 32);
    for (long long u = w0; u < (long long)cb * nyp; u += ws) {
        const int b = (int)(u / cb), a0 = (int)(u - (long long)b * cb) * 32 * kFoldN + lane;
        const size_t o = (size_t)(b + 1) * m + 1;
        V f[kFoldN], g[kFoldN];
#pragma unroll
        for (int k = 0; k < kFoldN; ++k) {
            const int a = a0 + 32 * k, e = nx - 1 - a;
            // kb > 0: a pairs with e for a < fo; the middle entry (odd nx) has none
            f[k] = b < ny && (kb > 0 ? a < nx - fo : a < nx) ? r[o + a] : V(0);
            g[k] = b < ny && kb > 0 && a < fo ? r[o + e] : V(0);
            if (ks) {
                if (b < ny && (kb > 0 ? a < nx - fo : a < nx)) f[k] *= ks[o + a];
                if (b < ny && kb > 0 && a < fo) g[k] *= ks[o + e];
            }
        }
        T *ub = U + (size_t)b * nxp;
#pragma unroll
        for (int k = 0; k < kFoldN; ++k) {
            const int a = a0 + 32 * k;
            if (a >= half) continue;
            ub[a] = (T)(((double)f[k] + (double)g[k]) * inv);
            if (kb > 0 && kb + a < nxp) ub[kb + a] = (T)((a < fo ? (double)f[k] - (double)g[k] : 0.0) * inv);
        }
    }
}

// z's interior from the parity-split transform W [nyp][nxp] (even block
// Ze = columns 0 .. fe-1, odd block Zo = columns kb .. kb+fo-1):
// z[j] = Ze[j] + Zo[j], z[nx-1-j] = Ze[j] - Zo[j] (j < fo), and the middle
// entry z[fo] = Ze[fo] when nx is odd; times sqrt(*rr) when rr is set and times
// the kappa scaling ks (or null). With part it also takes the solver's next
// dot product, r . z over the whole grid, as block partials while z is in
// registers (one launch and two passes fewer an iteration).
template <typename T, typename V>
__global__ void __launch_bounds__(kThreads)
    fd_unfold_kernel(const T *__restrict__ W, const V *__restrict__ r, const V *__restrict__ ks, V *__restrict__ z, int m,
                     int n, int nx, int ny, int nxp, int kb, int fe, int fo, const double *rr, double *part)
{
    pdl_begin();
    double f = 1.0;
    if (rr) {
        const double v = *rr;
        f = (v > 0.0 && v < 1e300) ? sqrt(v) : 1.0;
    }
    const int lane = threadIdx.x & 31, cb = (fe + 32 * kFoldN - 1) / (32 * kFoldN);
    const int w0 = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), ws = gridDim.x * (kThreads / 32);
    double dot = 0.0;
    for (long long u = w0; u < (long long)cb * ny; u += ws) {
        const int b = (int)(u / cb), j0 = (int)(u - (long long)b * cb) * 32 * kFoldN + lane;
        const T *wb = W + (size_t)b * nxp;
        const size_t o = (size_t)(b + 1) * m + 1;
        T e[kFoldN], d[kFoldN];
        V r0[kFoldN], r1[kFoldN], k0[kFoldN], k1[kFoldN];
#pragma unroll
        for (int k = 0; k < kFoldN; ++k) {
            const int j = j0 + 32 * k, jm = nx - 1 - j;
            e[k] = j < fe ? wb[j] : T(0);
            d[k] = j < fo ? wb[kb + j] : T(0);
            if (part) {
                r0[k] = j < fe ? r[o + j] : V(0);
                r1[k] = j < fo ? r[o + jm] : V(0);
            }
            if (ks) {
                k0[k] = j < fe ? ks[o + j] : V(0);
                k1[k] = j < fo ? ks[o + jm] : V(0);
            }
        }
#pragma unroll
        for (int k = 0; k < kFoldN; ++k) {
            const int j = j0 + 32 * k;
            if (j >= fe) continue;
            V z0 = (V)(f * ((double)e[k] + (double)d[k]));
            if (ks) z0 *= k0[k];
            z[o + j] = z0;
            if (part) dot += (double)r0[k] * (double)z0;
            if (j >= fo) continue;   // the middle entry (d = 0)
            V z1 = (V)(f * ((double)e[k] - (double)d[k]));
            if (ks) z1 *= k1[k];
            z[o + nx - 1 - j] = z1;
            if (part) dot += (double)r1[k] * (double)z1;
        }
    }
    if (!part) return;
    for (long long t = blockIdx.x * (long long)kThreads + threadIdx.x; t < 2LL * m + 2LL * (n - 2);
         t += (long long)gridDim.x * kThreads) {
        const long long i = ring_index(t, m, n);
        const V rv = r[i], zv = ks ? ks[i] * rv * ks[i] : rv;
        dot += (double)rv * (double)zv;
    }
    put_partial(dot, part);
}

// z = r on the boundary ring (identity rows of K_fem).
template <typename T>
__global__ void boundary_copy_kernel(T *__restrict__ z, const T *__restrict__ r, const T *__restrict__ ks, int m, int n)
{
    pdl_begin();
    ring_copy(z, r, ks, m, n, blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

// ------------------------------------------------------------ kappa scaling of the preconditioner
// s_i = 1 / sqrt(mean of kappa over the quadrature points of the elements
// supporting control point i); the preconditioner becomes S M^-1 S, which
// keeps the FEM matrix's shape and adds the coefficient's local magnitude.
// A CTA sums kappa over each element of its tile's supports once (kKsX x kKsY
// control points and a halo of P elements; one thread per element and
// quadrature row, then the rows) and the control points sum those. Bound: the
// bytes of kappa (p=3 512^2: 17 us; every control point summing all points of
// its elements: 262 us).
constexpr int kKsX = 32, kKsY = 8;

__global__ void __launch_bounds__(kKsX *kKsY) kappa_scale_kernel(const double *__restrict__ kappa, double *__restrict__ s64,
                                                                 float *__restrict__ s32, StripGrid g)
{
    __shared__ double part[(kKsX + 5) * (kKsY + 5) * 6];
    __shared__ double sum[(kKsX + 5) * (kKsY + 5)];
    const int P = g.P, NQ = P + 1, EX = kKsX + P, EY = kKsY + P;
    const int cols = (g.m + kKsX - 1) / kKsX, by = blockIdx.x / cols;
    const int C0 = kKsX * (blockIdx.x - by * cols), R0 = kKsY * by;
    for (int u = threadIdx.x; u < EX * EY * NQ; u += blockDim.x) {
        const int qy = u % NQ, k = u / NQ, ex = C0 - P + k % EX, ey = R0 - P + k / EX;
        double v = 0.0;
        if (ex >= 0 && ex < g.nex && ey >= 0 && ey < g.ney) {
            const double *q = kappa + (((size_t)ey * g.nex + ex) * NQ + qy) * NQ;
            for (int a = 0; a < NQ; ++a) v += q[a];
        }
        part[u] = v;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < EX * EY; k += blockDim.x) {
        double v = 0.0;
        for (int a = 0; a < NQ; ++a) v += part[k * NQ + a];
        sum[k] = v;
    }
    __syncthreads();
    const int cl = threadIdx.x % kKsX, rl = threadIdx.x / kKsX, C = C0 + cl, R = R0 + rl;
    if (C >= g.m || R >= g.n) return;
    double v = 0.0;
    for (int b = 0; b <= P; ++b)
        for (int a = 0; a <= P; ++a) v += sum[(rl + b) * EX + cl + a];
    const int nx = min(C, g.nex - 1) - max(0, C - P) + 1, ny = min(R, g.ney - 1) - max(0, R - P) + 1;
    v = v > 0.0 ? 1.0 / sqrt(v / ((double)nx * ny * NQ * NQ)) : 1.0;
    s64[(size_t)R * g.m + C] = v;
    s32[(size_t)R * g.m + C] = (float)v;
}

// out = a b on `rows` rows of `cols` entries, ld apart; ld > 0: the interior of
// an m = ld wide grid (the boundary ring is left alone).
template <typename T>
__global__ void mul_kernel(T *__restrict__ out, const T *__restrict__ a, const T *__restrict__ b, int rows, int cols,
                           int ld)
{
    pdl_begin();
    const long long N = (long long)rows * cols;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x) {
        const long long i = ld > 0 ? (t / cols + 1) * ld + 1 + t % cols : t;
        out[i] = a[i] * b[i];
    }
}

// ------------------------------------------------------------ host state
template <typename T>
struct PrecState {
    bool ready = false;
    T *kd = nullptr, *ko = nullptr, *md = nullptr, *mo = nullptr;
    T *ld = nullptr, *lo = nullptr, *nd = nullptr, *no = nullptr;
    T *x = nullptr, *r = nullptr, *z = nullptr, *p = nullptr, *q = nullptr, *b = nullptr;
    T *tz = nullptr;   // FP32 state: the preconditioner's output inside an FP64 (IGA_MIXED_PC) solve
    T *sc = nullptr;   // kappa-scaled preconditioner input
    T *iz = nullptr, *ir = nullptr, *ip = nullptr, *iq = nullptr;
    cudaGraphExec_t chunk = nullptr;
    // exact FEM inverse: x eigenvectors (column-major), eigenvalues, two work
    // matrices, and the LDL^T factors of the y systems of every x mode
    T *Vx = nullptr, *lx = nullptr, *W1 = nullptr, *W2 = nullptr, *Dv = nullptr;
    T *Lf = nullptr;   // LDL^T unit lower factor's subdiagonal per x mode (layout of Dv)
    int nxp = 0, nyp = 0;   // transform sizes padded to multiples of 16
    // parity split of the x transform (centrosymmetric x pencil): kb = the
    // padded even block (0: no split), fe / fo the even / odd mode counts;
    // nmodes = rows of the mode-major work matrix the y solves walk
    int kb = 0, fe = 0, fo = 0, nmodes = 0;
    GemmTF32 g1, g2;        // FP32: the two transforms' prepared tensor-core GEMMs
    int nsm = 148;          // SMs of the plan's device
    // device-side PCG loop: a CUDA graph whose conditional WHILE node runs one
    // iteration per pass (built for one preconditioner / kappa-scaling choice)
    cudaGraphExec_t loop = nullptr;
    int loop_pc = -1, loop_scaled = -1, loop_prec = -1;
    long long loop_wait_polls = -1;   // the plan's limit on the kernels' waits
    double loop_pc_rtol = 0.0;   // IGA_PC_FEM_CG: the inner solve's parameters in the loop
    int loop_pc_max_it = 0;
    IcgShape icg;                // IGA_PC_FEM_CG in one cluster (C = 0: the grid does not fit)
    bool loop_failed = false;   // the loop graph could not be instantiated: host-driven loop
    FemCoef<T> coef() const
    {
        FemCoef<T> c;
        c.kd = kd; c.ko = ko; c.md = md; c.mo = mo;
        c.ld = ld; c.lo = lo; c.nd = nd; c.no = no;
        return c;
    }
};

struct SolverState {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev = nullptr;   // orders a call's work on `stream` after and before the caller's stream
    bool pc_chain = false;  // a call outside any capture: the exact preconditioner's kernels as programmatic dependents
    bool pc_sync = false;   // IGA_PC_FEM_CG: the call wants the inner solve's status at once
    bool fd_host = false;
    // host x eigenpairs (built once). Split by parity (fold): even modes
    // 0 .. fe-1 then odd modes, Vx = the fe x fe even block followed by the
    // fo x fo odd block, each row one mode's half vector; else n x n.
    bool fold = false;
    int fe = 0, fo = 0;
    std::vector<double> lamx, Vx;
    std::vector<double> Dv, Lf;               // host LDL^T factors of the y systems, [a][b]
    double *ks64 = nullptr;                   // kappa scaling of the preconditioner
    float *ks32 = nullptr;
    int kappa_version = 0;
    DevScalars *s = nullptr;
    DevScalars *h = nullptr;   // pinned mirror
    double *partials = nullptr;   // of reduce_last; then the loop's p.q and r.z partials (kRedBlocks each)
    double *part_pq() const { return partials + 4 * kRedBlocks; }
    double *part_rz() const { return partials + 5 * kRedBlocks; }
    unsigned *counter = nullptr;
    double *r64 = nullptr, *q64 = nullptr;   // refinement residual / operator output
    PrecState<double> d;
    PrecState<float> f;
    std::vector<double> gx, gy;
};

}  // namespace iga

using namespace iga;

namespace iga {

void fem_1d(const std::vector<double> &g, std::vector<double> &kd, std::vector<double> &ko,
                   std::vector<double> &md, std::vector<double> &mo)
{
    const int n = (int)g.size();
    kd.assign(n, 0.0);
    md.assign(n, 0.0);
    ko.assign(n, 0.0);
    mo.assign(n, 0.0);
    for (int e = 0; e + 1 < n; ++e) {   // linear element [g_e, g_e+1], 2-point Gauss is exact
        const double h = g[e + 1] - g[e];
        kd[e] += 1.0 / h;
        kd[e + 1] += 1.0 / h;
        ko[e] = -1.0 / h;
        md[e] += h / 3.0;
        md[e + 1] += h / 3.0;
        mo[e] = h / 6.0;
    }
}

std::vector<double> fem_nodes_1d(int p, int ne, double L)
{
    if (p >= 3) {   // matrix_free/preprocess_fem.cpp:38-60
        std::vector<double> S;
        const double h = L / (ne + 2);
        for (int i = 0; i < p - 1; ++i) S.push_back(0.0);
        for (int i = 1; i < ne + 2; ++i) S.push_back(i * h);
        for (int i = 0; i < p - 1; ++i) S.push_back(L);
        return greville(p - 2, S);
    }
    return greville(p, open_knots(p, ne, L));
}

// Lengths of the FEM grid: mean polyline length of the control-net rows
// (x direction) and columns (y direction); 1 x 1 on the unit square.
// Segment lengths as sqrt(dx^2 + dy^2): control-net coordinates are far from
// the overflow range, and std::hypot's scaling made this loop a third of a
// 256-problem batch's preconditioner set-up.
void net_lengths(const Patch &P, double &Lx, double &Ly)
{
    double sx = 0.0, sy = 0.0;
    auto seg = [](double dx, double dy) { return std::sqrt(dx * dx + dy * dy); };
    for (int j = 0; j < P.n; ++j)
        for (int i = 0; i + 1 < P.m; ++i) {
            const size_t a = (size_t)j * P.m + i;
            sx += seg(P.CP[2 * (a + 1)] - P.CP[2 * a], P.CP[2 * (a + 1) + 1] - P.CP[2 * a + 1]);
        }
    for (int j = 0; j + 1 < P.n; ++j)
        for (int i = 0; i < P.m; ++i) {
            const size_t a = (size_t)j * P.m + i, b = a + P.m;
            sy += seg(P.CP[2 * b] - P.CP[2 * a], P.CP[2 * b + 1] - P.CP[2 * a + 1]);
        }
    Lx = sx / P.n;
    Ly = sy / P.m;
}

}  // namespace iga

#define SOLVE_TRY(call)                                                              \
    do {                                                                             \
        cudaError_t e_ = (call);                                                     \
        if (e_ != cudaSuccess) {                                                     \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));          \
            return e_ == cudaErrorMemoryAllocation ? IGA_ERR_NOMEM : IGA_ERR_CUDA;   \
        }                                                                            \
    } while (0)

template <typename T, bool LIMITED>
static void (*icg_kernel(int L))(IcgArgs<T>)
{
    return L == 1   ? icg_cluster_kernel<T, 1, LIMITED>
           : L == 2 ? icg_cluster_kernel<T, 2, LIMITED>
           : L == 4 ? icg_cluster_kernel<T, 4, LIMITED>
                    : icg_cluster_kernel<T, 8, LIMITED>;
}

// The kernel for a plan with or without a limit of its own on the waits.
template <typename T>
static auto icg_kernel(int L, bool limited)
{
    return limited ? icg_kernel<T, true>(L) : icg_kernel<T, false>(L);
}

// The cluster shape of the inner FEM-CG for this plan's grid: the first one
// that fits and that the device can place. The kernel's shared-memory limit
// belongs to the function, which all plans launch: it is set to the most any
// shape may take, never to this plan's own size.
template <typename T>
static int icg_prepare(PrecState<T> &ps, const iga_plan *pl)
{
    for (int k = 0; k < 4; ++k) {
        const IcgShape sh = icg_shape<T>(pl->m, pl->n, k);
        if (!sh.C) continue;
        auto kern = icg_kernel<T>(sh.L, false);
        bool wide = true;
        for (bool limited : {false, true}) {
            auto k2 = icg_kernel<T>(sh.L, limited);
            if (sh.C > 8) wide &= cudaFuncSetAttribute(k2, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
            SOLVE_TRY(cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kIcgMaxSmem));
        }
        if (!wide) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(sh.C);
        cfg.blockDim = dim3(sh.threads);
        cfg.dynamicSmemBytes = sh.smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = sh.C;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess || fit < 1) {
            cudaGetLastError();
            continue;
        }
        ps.icg = sh;
        break;
    }
    return IGA_OK;
}

template <typename T>
static int alloc_prec(PrecState<T> &ps, const iga_plan *pl, const SolverState &S)
{
    if (ps.ready) return IGA_OK;
    const size_t N = (size_t)pl->nfunc;
    std::vector<double> kd, ko, md, mo, ld, lo, nd, no;
    fem_1d(S.gx, kd, ko, md, mo);
    fem_1d(S.gy, ld, lo, nd, no);
    auto up = [&](T **dst, const std::vector<double> &v) -> int {
        std::vector<T> h(v.begin(), v.end());
        SOLVE_TRY(cudaMalloc((void **)dst, sizeof(T) * h.size()));
        SOLVE_TRY(cudaMemcpy(*dst, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
        return IGA_OK;
    };
    int st;
    if ((st = up(&ps.kd, kd)) || (st = up(&ps.ko, ko)) || (st = up(&ps.md, md)) || (st = up(&ps.mo, mo)) ||
        (st = up(&ps.ld, ld)) || (st = up(&ps.lo, lo)) || (st = up(&ps.nd, nd)) || (st = up(&ps.no, no)))
        return st;
    for (T **v : {&ps.x, &ps.r, &ps.z, &ps.tz, &ps.p, &ps.q, &ps.b, &ps.sc, &ps.iz, &ps.ir, &ps.ip, &ps.iq})
        SOLVE_TRY(cudaMalloc((void **)v, sizeof(T) * N));
    if ((st = icg_prepare(ps, pl))) return st;
    ps.ready = true;
    return IGA_OK;
}

static int ensure_state(iga_plan *pl, SolverState **out)
{
    if (pl->solver) {
        *out = pl->solver;
        return IGA_OK;
    }
    SolverState *S = new SolverState();
    pl->solver = S;
    S->device = pl->device;
    SOLVE_TRY(cudaSetDevice(pl->device));
    SOLVE_TRY(cudaStreamCreateWithFlags(&S->stream, cudaStreamNonBlocking));
    SOLVE_TRY(cudaMalloc((void **)&S->s, sizeof(DevScalars)));
    SOLVE_TRY(cudaMemset(S->s, 0, sizeof(DevScalars)));
    SOLVE_TRY(cudaEventCreateWithFlags(&S->ev, cudaEventDisableTiming));
    SOLVE_TRY(cudaMallocHost((void **)&S->h, sizeof(DevScalars)));
    SOLVE_TRY(cudaMalloc((void **)&S->partials, sizeof(double) * kRedBlocks * 6));
    SOLVE_TRY(cudaMalloc((void **)&S->counter, sizeof(unsigned)));
    SOLVE_TRY(cudaMemset(S->counter, 0, sizeof(unsigned)));
    SOLVE_TRY(cudaMalloc((void **)&S->r64, sizeof(double) * pl->nfunc));
    SOLVE_TRY(cudaMalloc((void **)&S->q64, sizeof(double) * pl->nfunc));
    double Lx, Ly;
    net_lengths(pl->patch, Lx, Ly);
    S->gx = fem_nodes_1d(pl->p, pl->nex, Lx);
    S->gy = fem_nodes_1d(pl->p, pl->ney, Ly);
    *out = S;
    return IGA_OK;
}

template <typename T>
static void free_prec(PrecState<T> &ps)
{
    T *bufs[] = {ps.kd, ps.ko, ps.md, ps.mo, ps.ld, ps.lo, ps.nd, ps.no, ps.x, ps.r, ps.z, ps.tz, ps.p,
                 ps.q, ps.b, ps.sc, ps.iz, ps.ir, ps.ip, ps.iq, ps.Vx, ps.lx, ps.W1, ps.W2, ps.Dv, ps.Lf};
    for (T *v : bufs)
        if (v) cudaFree(v);
    if (ps.chunk) cudaGraphExecDestroy(ps.chunk);
    if (ps.loop) cudaGraphExecDestroy(ps.loop);
    ps = PrecState<T>{};
}

void iga_solver_release(iga_plan *pl)
{
    SolverState *S = pl->solver;
    if (!S) return;
    cudaSetDevice(S->device);
    free_prec(S->d);
    free_prec(S->f);
    for (void *v : {(void *)S->s, (void *)S->partials, (void *)S->counter, (void *)S->r64, (void *)S->q64,
                    (void *)S->ks64, (void *)S->ks32})
        if (v) cudaFree(v);
    if (S->h) cudaFreeHost(S->h);
    if (S->ev) cudaEventDestroy(S->ev);
    if (S->stream) cudaStreamDestroy(S->stream);
    delete S;
    pl->solver = nullptr;
}

template <typename T>
static FemCoef<T> coef_of(const PrecState<T> &ps, const iga_plan *pl)
{
    FemCoef<T> c = ps.coef();
    c.m = pl->m;
    c.n = pl->n;
    return c;
}

template <typename T>
static InnerCG<T> inner_of(PrecState<T> &ps, const iga_plan *pl, SolverState *S)
{
    InnerCG<T> a;
    a.z = ps.iz;
    a.r = ps.ir;
    a.p = ps.ip;
    a.q = ps.iq;
    a.rhs = nullptr;
    a.c = coef_of(ps, pl);
    a.s = S->s;
    a.partials = S->partials;
    a.counter = S->counter;
    return a;
}

// One captured graph of kChunk inner iterations (3 kernels each, no-ops once done).
template <typename T>
static int inner_chunk_graph(PrecState<T> &ps, const iga_plan *pl, SolverState *S)
{
    if (ps.chunk) return IGA_OK;
    InnerCG<T> a = inner_of(ps, pl, S);
    cudaGraph_t g;
    SOLVE_TRY(cudaStreamBeginCapture(S->stream, cudaStreamCaptureModeThreadLocal));
    for (int k = 0; k < kChunk; ++k) {
        icg_q_kernel<T><<<kRedBlocks, kThreads, 0, S->stream>>>(a);
        icg_update_kernel<T><<<kRedBlocks, kThreads, 0, S->stream>>>(a);
        icg_p_kernel<T><<<kRedBlocks, kThreads, 0, S->stream>>>(a);
    }
    SOLVE_TRY(cudaStreamEndCapture(S->stream, &g));
    SOLVE_TRY(cudaGraphInstantiate(&ps.chunk, g, 0));
    cudaGraphDestroy(g);
    return IGA_OK;
}

namespace iga {
void interior_pencil(const std::vector<double> &g, std::vector<double> &Kd, std::vector<double> &Ko,
                            std::vector<double> &Md, std::vector<double> &Mo)
{
    std::vector<double> kd, ko, md, mo;
    fem_1d(g, kd, ko, md, mo);
    const int n = (int)g.size() - 2;
    Kd.assign(kd.begin() + 1, kd.begin() + 1 + n);
    Md.assign(md.begin() + 1, md.begin() + 1 + n);
    Ko.assign(ko.begin() + 1, ko.begin() + 1 + n);
    Mo.assign(mo.begin() + 1, mo.begin() + 1 + n);
}
}  // namespace iga

// Eigenpairs of the x pencil split by parity (pencil_fold): even modes
// 0 .. fe-1 then odd modes, each a half vector. v . r = u . (r[i] + r[nx-1-i])_i
// (the middle entry taken once) for an even mode and u . (r[i] - r[nx-1-i])_i
// for an odd one, which halves the flops of both transforms (the even-odd
// decomposition of spectral and fast-diagonalisation methods). Eigenpairs
// computed on the device (bisection, inverse iteration).
static int fold_eig(const std::vector<double> &Kd, const std::vector<double> &Ko, const std::vector<double> &Md,
                    const std::vector<double> &Mo, SolverState *S)
{
    const int n = (int)Kd.size(), fo = n / 2, fe = n - fo;
    std::vector<double> hk[2][4];
    std::vector<PencilRef> refs(2);
    for (int parity = 0; parity < 2; ++parity) {
        pencil_fold(n, Kd.data(), Ko.data(), Md.data(), Mo.data(), parity, hk[parity][0], hk[parity][1],
                    hk[parity][2], hk[parity][3]);
        refs[parity] = PencilRef{parity == 0 ? fe : fo, hk[parity][0].data(), hk[parity][1].data(),
                                 hk[parity][2].data(), hk[parity][3].data()};
    }
    std::vector<std::vector<double>> lam, vec;
    int st = pencil_eig_device(S->device, refs, lam, &vec);
    if (st) return st;
    S->fold = true;
    S->fe = fe;
    S->fo = fo;
    S->lamx.assign(n, 0.0);
    S->Vx.assign((size_t)fe * fe + (size_t)fo * fo, 0.0);
    for (int parity = 0; parity < 2; ++parity) {
        const int h = refs[parity].n;
        if (h == 0) continue;
        double *L = S->lamx.data() + (parity == 0 ? 0 : fe);
        double *V = S->Vx.data() + (parity == 0 ? 0 : (size_t)fe * fe);
        std::copy(lam[parity].begin(), lam[parity].end(), L);
        const double sc = 1.0 / std::sqrt(2.0);
        for (size_t i = 0; i < (size_t)h * h; ++i) V[i] = sc * vec[parity][i];
    }
    return IGA_OK;
}

// The x pencil's eigenpairs and, for every x mode a, the LDL^T factors of the
// y system lx[a] My + Ky on the free nodes, built once per plan on the host.
static int fd_setup(PrecState<double> &, const iga_plan *pl, SolverState *S)
{
    if (S->fd_host) return IGA_OK;
    std::vector<double> Kd, Ko, Md, Mo;
    interior_pencil(S->gx, Kd, Ko, Md, Mo);
    const int nx = (int)Kd.size();
    if (pl->pc_split && pencil_centrosymmetric(nx, Kd.data(), Ko.data(), Md.data(), Mo.data())) {
        const int st = fold_eig(Kd, Ko, Md, Mo, S);
        if (st) return st;
    } else {
        S->fold = false;
        std::vector<std::vector<double>> lam, vec;
        const int st = pencil_eig_device(S->device, {PencilRef{nx, Kd.data(), Ko.data(), Md.data(), Mo.data()}}, lam, &vec);
        if (st) return st;
        S->lamx = lam[0];
        S->Vx = vec[0];
    }
    interior_pencil(S->gy, Kd, Ko, Md, Mo);
    const int ny = (int)Kd.size();
    S->Dv.assign((size_t)nx * ny, 0.0);
    S->Lf.assign((size_t)nx * ny, 0.0);
    for (int a = 0; a < nx; ++a) {
        const double lam = S->lamx[a];
        double cprev = 0.0, eprev = 0.0;   // e_{b-1} / d_{b-1} and e_{b-1}
        for (int b = 0; b < ny; ++b) {
            const double den = lam * Md[b] + Kd[b] - eprev * cprev;
            const double e = b + 1 < ny ? lam * Mo[b] + Ko[b] : 0.0;
            S->Dv[(size_t)a * ny + b] = 1.0 / den;
            S->Lf[(size_t)a * ny + b] = cprev;
            cprev = e / den;
            eprev = e;
        }
    }
    S->fd_host = true;
    return IGA_OK;
}

static int prepare_gemms(PrecState<double> &) { return IGA_OK; }
static int prepare_gemms(PrecState<float> &ps)
{
    const int nxp = ps.nxp, nyp = ps.nyp;
    int st = gemm_tf32_prepare(ps.g1, GemmOperand{ps.Vx, nxp, false}, GemmOperand{ps.W2, nxp, false}, ps.W1, nyp, nxp,
                               nyp, nxp, nxp, nyp, GemmSplit{ps.kb, false});
    if (st) return st;
    ps.g1.const_op = 1;   // Vx
    st = gemm_tf32_prepare(ps.g2, GemmOperand{ps.W1, nyp, true}, GemmOperand{ps.Vx, nxp, true}, ps.W2, nxp, nyp, nxp,
                           nxp, nyp, nxp, GemmSplit{ps.kb, true});
    ps.g2.const_op = 2;   // Vx
    return st;
}

template <typename T>
static int fd_upload(PrecState<T> &ps, const iga_plan *pl, SolverState *S)
{
    if (ps.Vx) return IGA_OK;
    PrecState<double> dummy;
    if (const int st0 = fd_setup(dummy, pl, S)) return st0;
    const int nx = pl->m - 2, ny = pl->n - 2;
    // multiples of 16: aligned rows for the GEMMs and 16-byte moves; the
    // DGEMMs do no more flops than they must (2112 -> 2064 at 2048^2: FP64
    // PCG 114 -> 111 ms; TF32 GEMMs inside the solver's graph unchanged).
    // With the parity split the x index runs over the even block (fe values,
    // padded to kb) and then the odd block (fo values, padded).
    const int fe = S->fold ? S->fe : nx, fo = S->fold ? S->fo : 0;
    const int kb = (fe + 15) / 16 * 16, kob = (fo + 15) / 16 * 16;
    const int nxp = S->fold ? kb + kob : kb, nyp = (ny + 15) / 16 * 16;
    ps.nxp = nxp;
    ps.nyp = nyp;
    ps.kb = S->fold ? kb : 0;
    ps.fe = fe;
    ps.fo = fo;
    ps.nmodes = S->fold ? nxp : nx;
    // device row of host mode a (even modes, then odd ones from row kb)
    auto row_of = [&](int a) { return a < fe ? a : kb + (a - fe); };
    // zero-padded eigenvector matrix, block diagonal with the split: row
    // row_of(a) holds mode a's (half) vector from column 0 (even) or kb (odd)
    auto up_mat = [&](T **dst) -> int {
        std::vector<T> h((size_t)nxp * nxp, T(0));
        for (int a = 0; a < fe; ++a)
            for (int i = 0; i < fe; ++i) h[(size_t)a * nxp + i] = (T)S->Vx[(size_t)a * fe + i];
        const double *Vo = S->Vx.data() + (size_t)fe * fe;
        for (int a = 0; a < fo; ++a)
            for (int i = 0; i < fo; ++i) h[(size_t)(kb + a) * nxp + kb + i] = (T)Vo[(size_t)a * fo + i];
        SOLVE_TRY(cudaMalloc((void **)dst, sizeof(T) * h.size()));
        SOLVE_TRY(cudaMemcpy(*dst, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
        return IGA_OK;
    };
    // padded eigenvalues 1 keep the scaling finite
    auto up_vec = [&](T **dst, const std::vector<double> &v, int np) -> int {
        std::vector<T> h(np, T(1));
        for (size_t i = 0; i < v.size(); ++i) h[row_of((int)i)] = (T)v[i];
        SOLVE_TRY(cudaMalloc((void **)dst, sizeof(T) * h.size()));
        SOLVE_TRY(cudaMemcpy(*dst, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
        return IGA_OK;
    };
    // y factors in the layout of Wt: element (b, row_of(a)) at b + row_of(a) nyp
    // (padded modes: zero factors, so their solves return zeros)
    auto up_fac = [&](T **dst, const std::vector<double> &F) -> int {
        std::vector<T> h((size_t)nxp * nyp, T(0));
        for (int a = 0; a < nx; ++a)
            for (int b = 0; b < ny; ++b) h[(size_t)row_of(a) * nyp + b] = (T)F[(size_t)a * ny + b];
        SOLVE_TRY(cudaMalloc((void **)dst, sizeof(T) * h.size()));
        SOLVE_TRY(cudaMemcpy(*dst, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
        return IGA_OK;
    };
    int st;
    if ((st = up_mat(&ps.Vx)) || (st = up_vec(&ps.lx, S->lamx, nxp)) || (st = up_fac(&ps.Dv, S->Dv)) ||
        (st = up_fac(&ps.Lf, S->Lf)))
        return st;
    SOLVE_TRY(cudaDeviceGetAttribute(&ps.nsm, cudaDevAttrMultiProcessorCount, pl->device));
    SOLVE_TRY(tri_prepare<T>());
    SOLVE_TRY(cudaMalloc((void **)&ps.W1, sizeof(T) * (size_t)nxp * nyp));
    SOLVE_TRY(cudaMalloc((void **)&ps.W2, sizeof(T) * (size_t)nxp * nyp));
    return prepare_gemms(ps);
}

// The transforms' GEMMs in the row-major views of the work matrices:
//   W1[a][b] = sum_k Vx[a][k] W2[b][k]   (both operands K-major),
//   W2[b][i] = sum_a W1[a][b] Vx[a][i]   (both operands MN-major),
// with Vx[a][k] = component k of eigenvector a (ld nxp), W1 [nxp][nyp],
// W2 [nyp][nxp]. With the parity split, W2's columns (the GEMMs' k for the
// first, their n for the second) are the even folds then the odd folds, and
// Vx is block diagonal at kb (even modes' half vectors, odd modes' half
// vectors): each output tile runs over its own block's k range only, half
// the flops of the full transforms. FP32: tcgen05 TF32 tiles fed by tensor maps built here once
// (the preconditioner only has to be a close SPD approximation of K_fem^-1;
// the flexible PCG and the FP64 refinement absorb the difference); FP64:
// DMMA tiles.
static int transform_gemm(PrecState<double> &ps, const iga_plan *, int which, cudaStream_t s,
                          const GemmScatter &sc = GemmScatter())
{
    const int nxp = ps.nxp, nyp = ps.nyp;
    if (which == 1)
        return gemm_f64_launch(GemmOperand{ps.Vx, nxp, false}, GemmOperand{ps.W2, nxp, false}, ps.W1, nyp, nxp, nyp,
                               nxp, nxp, nyp, s, GemmScatter(), GemmSplit{ps.kb, false});
    return gemm_f64_launch(GemmOperand{ps.W1, nyp, true}, GemmOperand{ps.Vx, nxp, true}, ps.W2, nxp, nyp, nxp, nxp, nyp,
                           nxp, s, sc, GemmSplit{ps.kb, true});
}

static int transform_gemm(PrecState<float> &ps, const iga_plan *pl, int which, cudaStream_t s,
                          const GemmScatter &sc = GemmScatter())
{
    return gemm_tf32_launch(which == 1 ? ps.g1 : ps.g2, s, pl->d_err, sc);
}

// z = K_fem^-1 r on the free nodes (R, Z: the interior blocks of r, z,
// zero-padded to multiples of 16 so the GEMMs run with aligned leading
// dimensions). With Kx V = Mx V diag(lx) (V Mx-orthonormal), K_fem =
// Kx (x) My + Mx (x) Ky becomes, mode by mode in x, the tridiagonal y system
// lx[a] My + Ky: Wt = R^T Vx (so that each mode's y values are contiguous),
// column a of Wt solved along y, Z = Vx Wt^T. Two GEMMs and one pass of
// tridiagonal solves (the fast diagonalisation in both directions would take
// four GEMMs). With the parity split the gather folds r (r[i] +- r[nx-1-i]),
// the GEMMs work on the two half blocks, and the unfold kernel forms z.
// ks: the kappa scaling of r and z, or null. rz (or null): where the r . z
// partials go; its n stays 0 when this path does not take them.
// V is the vectors' type; an FP32 transform of FP64 vectors (T = float,
// V = double) passes sc, the device scalars whose rr scales the data.
struct DotPart {
    double *part = nullptr;
    int n = 0;
};

template <typename T, typename V>
static int fd_apply(PrecState<T> &ps, const iga_plan *pl, SolverState *S, const V *r, V *z, const DevScalars *sc,
                    const V *ks, DotPart *rz)
{
    const int m = pl->m, n = pl->n, nx = m - 2, ny = n - 2;
    if (nx <= 0 || ny <= 0) {   // no free nodes: the ring is everything
        SOLVE_TRY(launch_k(boundary_copy_kernel<V>, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, z, r, ks, m, n));
        return IGA_OK;
    }
    const int nxp = ps.nxp, nyp = ps.nyp;
    // warp steps of `cols` columns by `rows` rows, in at most `most` blocks
    auto blocks = [](int cols, int rows, int most) {
        const long long steps = (long long)((cols + 32 * kFoldN - 1) / (32 * kFoldN)) * rows;
        return (int)std::max(1LL, std::min<long long>(most, (steps + kThreads / 32 - 1) / (kThreads / 32)));
    };
    SOLVE_TRY(launch_k(fd_gather_kernel<T, V>, dim3(blocks(ps.kb > 0 ? ps.kb : nxp, nyp, 8 * ps.nsm)), dim3(kThreads), 0,
                       S->stream, r, ks, ps.W2, z, m, n, nx, ny, nxp, nyp, ps.kb, ps.fo, sc));
    // the gather follows whatever the stream holds (a wait for the caller's
    // stream, say); its successors follow this call's own kernels
    struct Chain {
        bool was = pdl_capture();
        ~Chain() { pdl_capture() = was; }
    } chain;
    if (S->pc_chain) pdl_capture() = true;
    int e = transform_gemm(ps, pl, 1, S->stream);
    if (e == IGA_OK) {
        const T *lf = ps.Lf, *dv = ps.Dv;
        const int nw = tri_warps<T>(ny);
        if constexpr (sizeof(T) == 8) {
            if (nw == 4) SOLVE_TRY((launch_tri<T, 4>(ps.W1, lf, dv, ps.nmodes, ny, nyp, S->stream, S->s)));
            if (nw == 2) SOLVE_TRY((launch_tri<T, 2>(ps.W1, lf, dv, ps.nmodes, ny, nyp, S->stream, S->s)));
        }
        if (nw == 1) SOLVE_TRY((launch_tri<T, 1>(ps.W1, lf, dv, ps.nmodes, ny, nyp, S->stream, S->s)));
        if (ps.kb > 0) {
            // parity split: the second GEMM writes both halves' products, the
            // unfold kernel combines them into z's interior
            e = transform_gemm(ps, pl, 2, S->stream);
            if (e == IGA_OK) {
                const int nu = blocks(ps.fe, ny, kRedBlocks);
                SOLVE_TRY(launch_k(fd_unfold_kernel<T, V>, dim3(nu), dim3(kThreads), 0, S->stream,
                                   (const T *)ps.W2, r, ks, z, m, n, nx, ny, nxp, ps.kb, ps.fe, ps.fo,
                                   sc ? &sc->rr : (const double *)nullptr, rz ? rz->part : (double *)nullptr));
                if (rz) rz->n = nu;
            }
        } else {
            // the second GEMM's epilogue writes z's interior itself
            GemmScatter gs;
            gs.out = z;
            gs.f64 = std::is_same<V, double>::value;
            gs.ld = m;
            gs.rows = ny;
            gs.cols = nx;
            gs.rr = sc ? &sc->rr : nullptr;
            e = transform_gemm(ps, pl, 2, S->stream, gs);
            if (e == IGA_OK && ks)
                SOLVE_TRY(launch_k(mul_kernel<V>, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, z, (const V *)z, ks, ny, nx,
                                   m));
        }
    }
    if (e != IGA_OK) {
        set_error("GEMM launch failed in the FEM preconditioner: " + last_error());
        return e;
    }
    return IGA_OK;
}

static int sync_scalars(SolverState *S)
{
    SOLVE_TRY(cudaMemcpyAsync(S->h, S->s, sizeof(DevScalars), cudaMemcpyDeviceToHost, S->stream));
    SOLVE_TRY(cudaStreamSynchronize(S->stream));
    return IGA_OK;
}

template <typename T>
static int pc_apply_core(PrecState<T> &ps, const iga_plan *pl, SolverState *S, const iga_solve_opts &o, const T *r,
                         T *z, double pc_rtol, int64_t &pc_iters, const T *ks = nullptr, DotPart *rz = nullptr);

static const double *kscale(SolverState *S, double *) { return S->ks64; }
static const float *kscale(SolverState *S, float *) { return S->ks32; }

// Scaling vector of the current kappa (null when the plan has none).
static int update_kscale(const iga_plan *pl, SolverState *S)
{
    if (!pl->kappa_dev || S->kappa_version == pl->kappa_version) return IGA_OK;
    if (!S->ks64) {
        SOLVE_TRY(cudaMalloc((void **)&S->ks64, sizeof(double) * pl->nfunc));
        SOLVE_TRY(cudaMalloc((void **)&S->ks32, sizeof(float) * pl->nfunc));
    }
    const StripGrid &g = pl->grid;
    const long long tiles = (long long)((g.m + kKsX - 1) / kKsX) * ((g.n + kKsY - 1) / kKsY);
    kappa_scale_kernel<<<(unsigned)tiles, kKsX * kKsY, 0, S->stream>>>(pl->kappa_dev, S->ks64, S->ks32, g);
    S->kappa_version = pl->kappa_version;
    SOLVE_TRY(cudaGetLastError());
    return IGA_OK;
}

// z = M^-1 r for FP64 vectors with the preconditioner evaluated in FP32
// (IGA_MIXED_PC): the input divided by ||r|| into FP32 (inside the
// transform's gather for the exact inverse), the FP32 preconditioner, the
// output multiplied back into FP64. The outer flexible PCG absorbs the FP32
// (TF32 GEMM) rounding of the preconditioner.
static int pc_apply_fp32(const iga_plan *pl, SolverState *S, const iga_solve_opts &o, const double *r, double *z,
                         double pc_rtol, int64_t &pc_iters, DotPart *rz)
{
    const long long N = pl->nfunc;
    PrecState<float> &f = S->f;
    int st;
    if (pl->kappa_dev && (st = update_kscale(pl, S))) return st;
    const double *ks = pl->kappa_dev ? S->ks64 : nullptr;
    if (o.pc == IGA_PC_FEM_EXACT) {
        if ((st = fd_upload(f, pl, S))) return st;
        return fd_apply<float, double>(f, pl, S, r, z, S->s, ks, rz);
    }
    const double *rin = r;
    if (ks) {
        SOLVE_TRY(launch_k(mul_kernel<double>, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, S->d.sc, r, ks, 1, (int)N, 0));
        rin = S->d.sc;
    }
    {
        SOLVE_TRY(launch_k(to_fp32_kernel, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, rin, f.sc, N,
                           (const DevScalars *)S->s));
        if ((st = pc_apply_core<float>(f, pl, S, o, f.sc, f.tz, pc_rtol, pc_iters))) return st;
        SOLVE_TRY(launch_k(from_fp32_kernel, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, (const float *)f.tz, z, N,
                           (const DevScalars *)S->s));
    }
    if (ks)
        SOLVE_TRY(launch_k(mul_kernel<double>, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, z, (const double *)z, ks, 1,
                           (int)N, 0));
    return IGA_OK;
}

// z = M^-1 r for the configured preconditioner; with a coefficient kappa,
// z = S M^-1 (S r) with the local scaling S.
template <typename T>
static int pc_apply(PrecState<T> &ps, const iga_plan *pl, SolverState *S, const iga_solve_opts &o, const T *r, T *z,
                    double pc_rtol, int64_t &pc_iters, DotPart *rz = nullptr)
{
    const int N = (int)pl->nfunc;
    if constexpr (std::is_same<T, double>::value) {
        if (o.precision == IGA_MIXED_PC && o.pc != IGA_PC_NONE)
            return pc_apply_fp32(pl, S, o, r, z, pc_rtol, pc_iters, rz);
    }
    if (o.pc == IGA_PC_NONE || !pl->kappa_dev)
        return pc_apply_core(ps, pl, S, o, r, z, pc_rtol, pc_iters, (const T *)nullptr, rz);
    int st;
    if ((st = update_kscale(pl, S))) return st;
    const T *sv = kscale(S, (T *)nullptr);
    if (o.pc == IGA_PC_FEM_EXACT) return pc_apply_core(ps, pl, S, o, r, z, pc_rtol, pc_iters, sv, rz);
    SOLVE_TRY(launch_k(mul_kernel<T>, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, ps.sc, r, sv, 1, N, 0));
    if ((st = pc_apply_core(ps, pl, S, o, ps.sc, z, pc_rtol, pc_iters))) return st;
    SOLVE_TRY(launch_k(mul_kernel<T>, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, z, (const T *)z, sv, 1, N, 0));
    return IGA_OK;
}

template <typename T>
static int pc_apply_core(PrecState<T> &ps, const iga_plan *pl, SolverState *S, const iga_solve_opts &o, const T *r,
                         T *z, double pc_rtol, int64_t &pc_iters, const T *ks, DotPart *rz)
{
    const long long N = pl->nfunc;
    if (o.pc == IGA_PC_NONE) {
        SOLVE_TRY(launch_k(copy_kernel<T>, dim3(kRedBlocks), dim3(kThreads), 0, S->stream, z, r, N));
        return IGA_OK;
    }
    int st;
    if (o.pc == IGA_PC_FEM_EXACT) {
        if ((st = fd_upload(ps, pl, S))) return st;
        return fd_apply<T, T>(ps, pl, S, r, z, nullptr, ks, rz);
    }
    if (ps.icg.C) {   // one cluster runs the whole inner solve
        IcgArgs<T> a;
        a.kd = ps.kd; a.ko = ps.ko; a.md = ps.md; a.mo = ps.mo;
        a.ld = ps.ld; a.lo = ps.lo; a.nd = ps.nd; a.no = ps.no;
        a.m = pl->m;
        a.n = pl->n;
        a.rows = ps.icg.rows;
        a.rhs = r;
        a.z = z;
        a.rtol = pc_rtol;
        a.maxit = o.pc_max_it;
        a.zero_on_break = !S->pc_sync;
        a.wait_polls = pl->wait_polls;
        a.s = S->s;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ps.icg.C);
        cfg.blockDim = dim3(ps.icg.threads);
        cfg.dynamicSmemBytes = ps.icg.smem;
        cfg.stream = S->stream;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = ps.icg.C;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = pdl_capture() ? 2 : 1;
        if (S->pc_sync) {
            SOLVE_TRY(cudaMemsetAsync(&S->s->ibreak, 0, sizeof(int), S->stream));
            SOLVE_TRY(cudaMemsetAsync(&S->s->err, 0, sizeof(int), S->stream));
        }
        SOLVE_TRY(cudaLaunchKernelEx(&cfg, icg_kernel<T>(ps.icg.L, pl->wait_polls >= 0), a));
        if (S->pc_sync) {
            if ((st = sync_scalars(S))) return st;
            if (S->h->err) {
                set_error("a bounded device wait gave up in the preconditioner");
                return IGA_ERR_TIMEOUT;
            }
            if (S->h->ibreak) return IGA_ERR_BREAKDOWN;
        }
        return IGA_OK;
    }
    if ((st = inner_chunk_graph(ps, pl, S))) return st;
    InnerCG<T> a = inner_of(ps, pl, S);
    icg_init_kernel<T><<<kRedBlocks, kThreads, 0, S->stream>>>(a, r, pc_rtol, o.pc_max_it);
    // Keep one chunk in flight ahead of the completion check.
    SOLVE_TRY(cudaGraphLaunch(ps.chunk, S->stream));
    int launched = 1;
    for (;;) {
        SOLVE_TRY(cudaMemcpyAsync(S->h, S->s, sizeof(DevScalars), cudaMemcpyDeviceToHost, S->stream));
        cudaEvent_t ev;
        SOLVE_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        SOLVE_TRY(cudaEventRecord(ev, S->stream));
        if ((long long)launched * kChunk < (long long)o.pc_max_it + kChunk) {
            SOLVE_TRY(cudaGraphLaunch(ps.chunk, S->stream));
            ++launched;
        }
        SOLVE_TRY(cudaEventSynchronize(ev));
        cudaEventDestroy(ev);
        if (S->h->idone) break;
        if ((long long)launched * kChunk >= (long long)o.pc_max_it + 2 * kChunk) break;
    }
    SOLVE_TRY(cudaStreamSynchronize(S->stream));
    pc_iters += S->h->iiters;
    if (S->h->ibreak) return IGA_ERR_BREAKDOWN;
    copy_kernel<T><<<kRedBlocks, kThreads, 0, S->stream>>>(z, ps.iz, N);
    return IGA_OK;
}

// One iteration of the flexible PCG on the fixed buffers of ps: z = M^-1 r;
// beta; p = z + beta p (p = z in the first); q = K p; alpha; x += alpha p, r -=
// alpha q, r.z. With the preconditioner first no iteration ends on one whose
// result nobody reads (a 12-iteration solve of four sweeps otherwise applies it
// 16 times). Both loops, the device's and the host's, are made of it.
template <typename T>
static int pcg_step(iga_plan *pl, SolverState *S, PrecState<T> &ps, const iga_solve_opts &o, int prec, LoopCond cond,
                    int64_t &pc_iters)
{
    const long long N = pl->nfunc;
    const cudaStream_t s = S->stream;
    DotPart rz;
    rz.part = S->part_rz();
    int st = pc_apply(ps, pl, S, o, ps.r, ps.z, o.pc_rtol, pc_iters, &rz);
    if (st) return st;
    const int nb = vec_blocks<T>(N);
    // the vector kernels of vectors of 4 MB or more get ordinary edges: their
    // blocks run long enough for an uneven start to cost more than a launch
    // gap (1024^2 mixed 118.8 -> 117 us an iteration, 2048^2 FP64 1111 -> 1100;
    // 512^2 FP64 97.7 -> 99.5)
    const bool even = N * (long long)sizeof(T) >= (4LL << 20);
    auto launch_vec = [&](auto kern, auto... args) {
        return even ? launch_even(kern, dim3(nb), dim3(kThreads), 0, s, args...)
                    : launch_k(kern, dim3(nb), dim3(kThreads), 0, s, args...);
    };
    if (rz.n == 0) {   // no preconditioner that took r . z itself
        SOLVE_TRY(launch_vec(loop_dot_kernel<T>, (const T *)ps.r, (const T *)ps.z, N, rz.part));
        rz.n = nb;
    }
    SOLVE_TRY(launch_vec(loop_p_kernel<T>, ps.p, (const T *)ps.z, N, S->s, (const double *)rz.part, rz.n));
    if ((st = iga_apply_internal_sb(pl, prec, ps.p, ps.q, s, IGA_SIGN_SPD, IGA_BC_IDENTITY))) return st;
    SOLVE_TRY(launch_vec(loop_dot_kernel<T>, (const T *)ps.p, (const T *)ps.q, N, S->part_pq()));
    SOLVE_TRY(launch_vec(loop_xr_kernel<T>, ps.x, ps.r, (const T *)ps.p, (const T *)ps.q, (const T *)ps.z, N, S->s,
                         (const double *)S->part_pq(), nb, S->partials, S->counter, cond));
    return IGA_OK;
}

// Builds the device-side loop for the current preconditioner choice: its body
// is one pcg_step().
template <typename T>
static int build_loop(iga_plan *pl, SolverState *S, PrecState<T> &ps, const iga_solve_opts &o, int prec)
{
    const int scaled = pl->kappa_dev ? 1 : 0;
    const bool same_pc = ps.loop_pc == o.pc && (o.pc != IGA_PC_FEM_CG || (ps.loop_pc_rtol == o.pc_rtol &&
                                                                         ps.loop_pc_max_it == o.pc_max_it));
    if (same_pc && ps.loop_scaled == scaled && ps.loop_prec == o.precision && ps.loop_wait_polls == pl->wait_polls &&
        (ps.loop || ps.loop_failed))
        return ps.loop ? IGA_OK : IGA_ERR_UNSUPPORTED;
    if (ps.loop) {
        cudaGraphExecDestroy(ps.loop);
        ps.loop = nullptr;
    }
    const cudaStream_t s = S->stream;
    cudaGraph_t g;
    SOLVE_TRY(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle h;
    SOLVE_TRY(cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node;
    SOLVE_TRY(cudaGraphAddNode(&node, g, nullptr, 0, &np));
    cudaGraph_t body = np.conditional.phGraph_out[0];
    SOLVE_TRY(cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    int64_t dummy = 0;
    // Programmatic dependencies between the body's kernels.
    pdl_capture() = true;
    LoopCond cond;
    cond.h = h;
    cond.on = 1;
    const int st = pcg_step(pl, S, ps, o, prec, cond, dummy);
    pdl_capture() = false;
    cudaGraph_t captured = body;
    const cudaError_t ce = cudaStreamEndCapture(s, &captured);
    if (st || ce != cudaSuccess) {
        cudaGraphDestroy(g);
        if (!st) set_error(std::string("PCG loop capture: ") + cudaGetErrorString(ce));
        return st ? st : IGA_ERR_CUDA;
    }
    cudaGraphInstantiateParams ip = {};
    const cudaError_t ie = cudaGraphInstantiateWithParams(&ps.loop, g, &ip);
    if (ie != cudaSuccess) {
        cudaGraphNodeType t = cudaGraphNodeTypeEmpty;
        if (ip.errNode_out) cudaGraphNodeGetType(ip.errNode_out, &t);
        set_error(std::string("PCG loop instantiation: ") + cudaGetErrorString(ie) + " (result " +
                  std::to_string((int)ip.result_out) + ", node type " + std::to_string((int)t) + ")");
        cudaGetLastError();
        cudaGraphDestroy(g);
        ps.loop = nullptr;
        ps.loop_pc = o.pc;
        ps.loop_scaled = scaled;
        ps.loop_prec = o.precision;
        ps.loop_wait_polls = pl->wait_polls;
        ps.loop_pc_rtol = o.pc_rtol;
        ps.loop_pc_max_it = o.pc_max_it;
        ps.loop_failed = true;
        return IGA_ERR_UNSUPPORTED;
    }
    cudaGraphDestroy(g);
    ps.loop_failed = false;
    ps.loop_pc = o.pc;
    ps.loop_scaled = scaled;
    ps.loop_prec = o.precision;
    ps.loop_wait_polls = pl->wait_polls;
    ps.loop_pc_rtol = o.pc_rtol;
    ps.loop_pc_max_it = o.pc_max_it;
    return IGA_OK;
}

// Flexible PCG on K x = b in precision T, from the current x; stops when the
// recurrence residual satisfies ||r|| <= rtol bnorm. Its iterations run on the
// device, in one graph launch, or (host, and where a plan asks for it or the
// graph cannot be had) one by one from the host, which reads the scalars after
// each. x_zero: x is known to be zero and b nonzero (a refinement sweep on the
// normalised residual): r = b without the operator and no host check before
// the loop.
template <typename T>
static int pcg(iga_plan *pl, SolverState *S, PrecState<T> &ps, const iga_solve_opts &o, const T *b, T *x, double rtol,
               double bnorm, int prec, int &its, int64_t &pc_iters, bool host, bool x_zero = false)
{
    const long long N = pl->nfunc;
    const cudaStream_t s = S->stream;
    int st;
    if ((st = update_kscale(pl, S))) return st;
    if (o.pc == IGA_PC_FEM_EXACT) {   // device set-up before any capture
        if (std::is_same<T, double>::value && o.precision == IGA_MIXED_PC) st = fd_upload(S->f, pl, S);
        else st = fd_upload(ps, pl, S);
        if (st) return st;
    }
    if (b != ps.b) copy_kernel<T><<<kRedBlocks, kThreads, 0, s>>>(ps.b, b, N);
    if (x != ps.x) copy_kernel<T><<<kRedBlocks, kThreads, 0, s>>>(ps.x, x, N);
    if (x_zero) {
        copy_kernel<T><<<kRedBlocks, kThreads, 0, s>>>(ps.r, ps.b, N);
        dot_kernel<T><<<kRedBlocks, kThreads, 0, s>>>(ps.r, ps.r, N, &S->s->rr, S->partials, S->counter);
    } else {
        if ((st = iga_apply_internal_sb(pl, prec, ps.x, ps.q, s, IGA_SIGN_SPD, IGA_BC_IDENTITY))) return st;
        sub_kernel<T><<<kRedBlocks, kThreads, 0, s>>>(ps.b, ps.q, ps.r, N, S->s, S->partials, S->counter);
        if ((st = sync_scalars(S))) return st;
        if (std::sqrt(S->h->rr) <= rtol * bnorm) return IGA_OK;
    }
    if (!host) {
        st = pl->solver_graph ? build_loop(pl, S, ps, o, prec) : IGA_ERR_UNSUPPORTED;
        if (st && st != IGA_ERR_UNSUPPORTED) return st;
        host = st != IGA_OK;   // e.g. a library kernel not allowed in a conditional body
    }
    // the graph's body runs at least once; a solve from the host or with the
    // inner FEM-CG that is asked for no iteration does none
    if ((host || o.pc == IGA_PC_FEM_CG) && o.max_it <= 0) return IGA_ERR_NOT_CONVERGED;
    loop_init_kernel<<<1, 1, 0, s>>>(S->s, rtol * rtol * bnorm * bnorm, o.max_it);
    st = IGA_OK;
    if (host) {
        const DevScalars &h = *S->h;
        do {
            if ((st = pcg_step(pl, S, ps, o, prec, LoopCond(), pc_iters))) break;
            if ((st = sync_scalars(S))) return st;
        } while (h.rr > h.tol2 && h.it < h.maxit && !h.breakdown && std::isfinite(h.rr));
    } else {
        SOLVE_TRY(cudaGraphLaunch(ps.loop, s));
    }
    if (x != ps.x) copy_kernel<T><<<kRedBlocks, kThreads, 0, s>>>(x, ps.x, N);
    if (st && st != IGA_ERR_BREAKDOWN) return st;
    const int pc_st = st;   // IGA_ERR_BREAKDOWN: of an inner solve that the host drives
    if ((st = sync_scalars(S))) return st;
    its += S->h->it;
    if (pc_st) return pc_st;
    if (S->h->breakdown) return IGA_ERR_BREAKDOWN;
    if (!std::isfinite(S->h->rr)) return IGA_ERR_NONFINITE;
    return std::sqrt(S->h->rr) <= rtol * bnorm ? IGA_OK : IGA_ERR_NOT_CONVERGED;
}

// ||b - K x|| (FP64 operator), into S->h->rr and S->h->bb.
static int true_residual(iga_plan *pl, SolverState *S, const double *b, const double *x)
{
    int st;
    if ((st = iga_apply_internal_sb(pl, IGA_FP64, x, S->q64, S->stream, IGA_SIGN_SPD, IGA_BC_IDENTITY))) return st;
    residual_kernel<<<kRedBlocks, kThreads, 0, S->stream>>>(b, S->q64, S->r64, pl->nfunc, S->s, S->partials,
                                                          S->counter);
    return sync_scalars(S);
}

extern "C" {

void iga_solve_opts_default(iga_solve_opts *o)
{
    if (!o) return;
    o->precision = IGA_FP64;
    o->pc = IGA_PC_FEM_CG;
    o->rtol = 1e-10;
    o->max_it = 10000;
    o->pc_rtol = 1e-10;
    o->pc_max_it = 10000;
    o->sweep_rtol = 1e-3;
    o->max_sweeps = 10;
    o->x0_nonzero = 0;
}

int iga_fem_nodes(const iga_plan *pl, double *gx, double *gy)
{
    if (!pl || !gx || !gy) return IGA_ERR_ARG;
    double Lx, Ly;
    net_lengths(pl->patch, Lx, Ly);
    const std::vector<double> a = fem_nodes_1d(pl->p, pl->nex, Lx), b = fem_nodes_1d(pl->p, pl->ney, Ly);
    std::memcpy(gx, a.data(), a.size() * sizeof(double));
    std::memcpy(gy, b.data(), b.size() * sizeof(double));
    return IGA_OK;
}

int iga_fem_nodes_1d(int p, int ne, double L, double *g)
{
    if (!g || p < 1 || p > 5 || ne < 1 || !(L > 0.0)) return IGA_ERR_ARG;
    const std::vector<double> a = fem_nodes_1d(p, ne, L);
    std::memcpy(g, a.data(), a.size() * sizeof(double));
    return IGA_OK;
}

int iga_pc_apply(iga_plan *pl, int pc, int prec, const void *r, void *z, double pc_rtol, int pc_max_it,
                 void *stream)
{
    if (!pl || !r || !z || (prec != IGA_FP64 && prec != IGA_FP32)) return IGA_ERR_ARG;
    if (pc != IGA_PC_NONE && pc != IGA_PC_FEM_CG && pc != IGA_PC_FEM_EXACT) return IGA_ERR_ARG;
    SolverState *S;
    int st;
    if ((st = ensure_state(pl, &S))) return st;
    SOLVE_TRY(cudaEventRecord(S->ev, (cudaStream_t)stream));
    SOLVE_TRY(cudaStreamWaitEvent(S->stream, S->ev, 0));
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    SOLVE_TRY(cudaStreamIsCapturing(S->stream, &cap));
    S->pc_chain = cap == cudaStreamCaptureStatusNone;
    iga_solve_opts o;
    iga_solve_opts_default(&o);
    o.pc = pc;
    o.pc_max_it = pc_max_it;
    int64_t its = 0;
    S->pc_sync = true;
    if (prec == IGA_FP64) {
        if (!(st = alloc_prec(S->d, pl, *S)))
            st = pc_apply<double>(S->d, pl, S, o, (const double *)r, (double *)z, pc_rtol, its);
    } else {
        if (!(st = alloc_prec(S->f, pl, *S)))
            st = pc_apply<float>(S->f, pl, S, o, (const float *)r, (float *)z, pc_rtol, its);
    }
    S->pc_sync = S->pc_chain = false;
    SOLVE_TRY(cudaEventRecord(S->ev, S->stream));
    SOLVE_TRY(cudaStreamWaitEvent((cudaStream_t)stream, S->ev, 0));
    return st;
}

int iga_plan_set_pc_split(iga_plan *pl, int enable)
{
    if (!pl || (enable != 0 && enable != 1)) return IGA_ERR_ARG;
    if (pl->solver) {
        cudaSetDevice(pl->device);
        cudaDeviceSynchronize();
        iga_solver_release(pl);
    }
    pl->pc_split = enable != 0;
    return IGA_OK;
}

int iga_plan_set_solver_graph(iga_plan *pl, int enable)
{
    if (!pl || (enable != 0 && enable != 1)) return IGA_ERR_ARG;
    pl->solver_graph = enable != 0;
    return IGA_OK;
}

int iga_fem_apply(iga_plan *pl, int prec, const void *x, void *y, void *stream)
{
    if (!pl || !x || !y) return IGA_ERR_ARG;
    SolverState *S;
    int st;
    if ((st = ensure_state(pl, &S))) return st;
    if (prec == IGA_FP64) {
        if ((st = alloc_prec(S->d, pl, *S))) return st;
        fem_apply_kernel<double><<<kRedBlocks, kThreads, 0, (cudaStream_t)stream>>>(
            (const double *)x, (double *)y, coef_of(S->d, pl));
    } else if (prec == IGA_FP32) {
        if ((st = alloc_prec(S->f, pl, *S))) return st;
        fem_apply_kernel<float><<<kRedBlocks, kThreads, 0, (cudaStream_t)stream>>>((const float *)x, (float *)y,
                                                                                 coef_of(S->f, pl));
    } else {
        return IGA_ERR_ARG;
    }
    SOLVE_TRY(cudaGetLastError());
    return IGA_OK;
}

int iga_fem_assemble_csr(iga_plan *pl, int sign, int32_t *rowptr, int32_t *col, double *val, int64_t *nnz,
                         void *stream)
{
    if (!pl || (sign != 1 && sign != -1)) return IGA_ERR_ARG;
    const int m = pl->m, n = pl->n;
    // Row lengths: 1 on the boundary, (free neighbours in x) * (free neighbours in y) inside.
    auto cnt = [](int i, int mm) { return 1 + (i - 1 >= 1) + (i + 1 <= mm - 2); };
    std::vector<int32_t> rp((size_t)m * n + 1);
    long long acc = 0;
    for (int j = 0; j < n; ++j)
        for (int i = 0; i < m; ++i) {
            rp[(size_t)j * m + i] = (int32_t)acc;
            const bool b = i == 0 || j == 0 || i == m - 1 || j == n - 1;
            acc += b ? 1 : cnt(i, m) * cnt(j, n);
        }
    rp[(size_t)m * n] = (int32_t)acc;
    if (acc > INT32_MAX) return IGA_ERR_UNSUPPORTED;
    if (nnz) *nnz = acc;
    if (!rowptr && !col && !val) return IGA_OK;
    if (!rowptr || !col || !val) return IGA_ERR_ARG;
    SolverState *S;
    int st;
    if ((st = ensure_state(pl, &S))) return st;
    if ((st = alloc_prec(S->d, pl, *S))) return st;
    cudaStream_t s = (cudaStream_t)stream;
    SOLVE_TRY(cudaMemcpyAsync(rowptr, rp.data(), rp.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s));
    fem_csr_kernel<<<kRedBlocks, kThreads, 0, s>>>(rowptr, col, val, coef_of(S->d, pl), (double)sign);
    SOLVE_TRY(cudaStreamSynchronize(s));
    return IGA_OK;
}

int iga_solve(iga_plan *pl, const double *b, double *x, const iga_solve_opts *o_in, iga_solve_stats *stats,
              void *stream)
{
    if (!pl || !b || !x) return IGA_ERR_ARG;
    iga_solve_opts o;
    iga_solve_opts_default(&o);
    if (o_in) o = *o_in;
    if (o.pc != IGA_PC_NONE && o.pc != IGA_PC_FEM_CG && o.pc != IGA_PC_FEM_EXACT) {
        set_error("unknown preconditioner");
        return IGA_ERR_ARG;
    }
    if (!pl->op64.ready) {
        set_error("iga_solve needs the FP64 operator (plan precision IGA_FP64 or IGA_MIXED)");
        return IGA_ERR_ARG;
    }
    if (o.precision != IGA_FP64 && o.precision != IGA_MIXED && o.precision != IGA_MIXED_PC) {
        set_error("iga_solve precision is IGA_FP64, IGA_MIXED or IGA_MIXED_PC");
        return IGA_ERR_ARG;
    }
    if (o.precision == IGA_MIXED && !pl->op32.ready) {
        set_error("IGA_MIXED solves need a plan created with precision IGA_MIXED");
        return IGA_ERR_ARG;
    }
    SolverState *S;
    int st;
    if ((st = ensure_state(pl, &S))) return st;
    SOLVE_TRY(cudaSetDevice(pl->device));
    const auto t0 = std::chrono::steady_clock::now();
    // Order the solve after the caller's stream and the caller's stream after the solve.
    cudaEvent_t ev;
    SOLVE_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    SOLVE_TRY(cudaEventRecord(ev, (cudaStream_t)stream));
    SOLVE_TRY(cudaStreamWaitEvent(S->stream, ev, 0));
    const long long N = pl->nfunc;
    iga_solve_stats stt{};
    SOLVE_TRY(cudaMemsetAsync(&S->s->err, 0, sizeof(int), S->stream));
    SOLVE_TRY(cudaMemsetAsync(&S->s->ibreak, 0, sizeof(int), S->stream));
    SOLVE_TRY(cudaMemsetAsync(&S->s->ipc, 0, sizeof(long long), S->stream));
    if (!o.x0_nonzero) zero_kernel<double><<<kRedBlocks, kThreads, 0, S->stream>>>(x, N);
    if ((st = true_residual(pl, S, b, x))) return st;
    if (!std::isfinite(S->h->bb) || !std::isfinite(S->h->rr)) {
        cudaEventDestroy(ev);
        if (stats) {
            *stats = iga_solve_stats{};
            stats->status = IGA_ERR_NONFINITE;
            stats->relres = NAN;
        }
        set_error("non-finite value in b or in the initial residual");
        return IGA_ERR_NONFINITE;
    }
    const double bnorm = std::sqrt(S->h->bb);
    double rel = bnorm > 0 ? std::sqrt(S->h->rr) / bnorm : 0.0;
    int result = IGA_OK;
    if (o.precision != IGA_MIXED) {
        if ((st = alloc_prec(S->d, pl, *S))) return st;
        if (o.precision == IGA_MIXED_PC && o.pc != IGA_PC_NONE && (st = alloc_prec(S->f, pl, *S))) return st;
        // Restart from the true residual until it meets rtol (recurrence drift).
        for (int restart = 0; restart < 4 && rel > o.rtol; ++restart) {
            // the inner FEM-CG of grids past one cluster is driven by the host
            const bool host = o.pc == IGA_PC_FEM_CG && !(o.precision == IGA_MIXED_PC ? S->f.icg.C : S->d.icg.C);
            st = pcg<double>(pl, S, S->d, o, b, x, o.rtol, bnorm, IGA_FP64, stt.iterations, stt.pc_iterations, host);
            if (st && st != IGA_ERR_NOT_CONVERGED) {
                result = st;
                break;
            }
            if ((st = true_residual(pl, S, b, x))) return st;
            rel = std::sqrt(S->h->rr) / bnorm;
            if (!std::isfinite(rel)) {
                result = IGA_ERR_NONFINITE;
                break;
            }
        }
    } else {
        if ((st = alloc_prec(S->f, pl, *S))) return st;
        for (int sw = 0; sw < o.max_sweeps && rel > o.rtol; ++sw) {
            // rhs of the sweep: r64 / ||r64|| in FP32; correction d solves K d = r / ||r||.
            const double scale = std::sqrt(S->h->rr);
            // A sweep asks for sweep_rtol, or for less when less is left to do:
            // a fifth of the reduction that would reach rtol (margin for the
            // FP32 recurrence residual drifting from the FP64 one).
            const double need = o.rtol * bnorm / scale;
            const double srtol = std::max(o.sweep_rtol, std::min(0.2 * need, 0.5));
            scale_down_kernel<<<kRedBlocks, kThreads, 0, S->stream>>>(S->r64, S->f.b, N, S->s);
            zero_kernel<float><<<kRedBlocks, kThreads, 0, S->stream>>>(S->f.x, N);
            const bool host = o.pc == IGA_PC_FEM_CG && !S->f.icg.C;
            st = pcg<float>(pl, S, S->f, o, S->f.b, S->f.x, srtol, 1.0, IGA_FP32, stt.iterations, stt.pc_iterations, host,
                            true);
            if (st && st != IGA_ERR_NOT_CONVERGED) {
                result = st;
                break;
            }
            refine_update_kernel<<<kRedBlocks, kThreads, 0, S->stream>>>(x, S->f.x, N, scale);
            ++stt.sweeps;
            if ((st = true_residual(pl, S, b, x))) return st;
            rel = std::sqrt(S->h->rr) / bnorm;
            if (!std::isfinite(rel)) {
                result = IGA_ERR_NONFINITE;
                break;
            }
        }
    }
    SOLVE_TRY(cudaEventRecord(ev, S->stream));
    SOLVE_TRY(cudaStreamWaitEvent((cudaStream_t)stream, ev, 0));
    SOLVE_TRY(cudaStreamSynchronize(S->stream));
    cudaEventDestroy(ev);
    stt.relres = rel;
    stt.pc_iterations += S->h->ipc;
    if (S->h->err) {   // host copy current as of the last true residual
        set_error("a bounded device wait gave up in the preconditioner");
        result = IGA_ERR_TIMEOUT;
    }
    if (result == IGA_OK && !(rel <= o.rtol)) result = IGA_ERR_NOT_CONVERGED;
    stt.status = result;
    stt.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (stats) *stats = stt;
    return result;
}

int iga_spectrum_estimate(iga_plan *pl, int pc, int steps, uint64_t seed, double *lam_min, double *lam_max,
                          int *steps_done)
{
    if (!pl || !lam_min || !lam_max || steps < 1) return IGA_ERR_ARG;
    if (pc != IGA_PC_NONE && pc != IGA_PC_FEM_CG && pc != IGA_PC_FEM_EXACT) return IGA_ERR_ARG;
    if (!pl->op64.ready) {
        set_error("iga_spectrum_estimate needs the FP64 operator");
        return IGA_ERR_ARG;
    }
    SolverState *S;
    int st;
    if ((st = ensure_state(pl, &S))) return st;
    SOLVE_TRY(cudaSetDevice(pl->device));
    if ((st = alloc_prec(S->d, pl, *S))) return st;
    PrecState<double> &ps = S->d;
    const long long N = pl->nfunc;
    const cudaStream_t s = S->stream;
    iga_solve_opts o;
    iga_solve_opts_default(&o);
    o.pc = pc;
    o.pc_rtol = 1e-13;
    // seeded random start vector, zero on the boundary ring (the Krylov space
    // stays on the free control points: identity rows and identity PC rows)
    std::vector<double> h((size_t)N);
    std::mt19937_64 gen(seed);
    std::normal_distribution<double> nd(0.0, 1.0);
    for (int j = 0; j < pl->n; ++j)
        for (int i = 0; i < pl->m; ++i)
            h[(size_t)j * pl->m + i] = (i == 0 || j == 0 || i == pl->m - 1 || j == pl->n - 1) ? 0.0 : nd(gen);
    SOLVE_TRY(cudaMemcpyAsync(ps.r, h.data(), sizeof(double) * N, cudaMemcpyHostToDevice, s));
    zero_kernel<double><<<kRedBlocks, kThreads, 0, s>>>(ps.x, N);
    int64_t pcits = 0;
    SOLVE_TRY(cudaMemsetAsync(&S->s->breakdown, 0, sizeof(int), s));
    SOLVE_TRY(cudaMemsetAsync(&S->s->ibreak, 0, sizeof(int), s));
    SOLVE_TRY(cudaMemsetAsync(&S->s->err, 0, sizeof(int), s));
    auto pc_status = [&] {   // of the preconditioner's kernels up to the last sync_scalars
        if (S->h->err) set_error("a bounded device wait gave up in the preconditioner");
        return S->h->err ? IGA_ERR_TIMEOUT : S->h->ibreak ? IGA_ERR_BREAKDOWN : IGA_OK;
    };
    if ((st = pc_apply(ps, pl, S, o, ps.r, ps.z, o.pc_rtol, pcits))) return st;
    dot_kernel<double><<<kRedBlocks, kThreads, 0, s>>>(ps.r, ps.z, N, &S->s->rz, S->partials, S->counter);
    pcg_p_kernel<double><<<kRedBlocks, kThreads, 0, s>>>(ps.p, ps.z, N, S->s, 1);
    if ((st = sync_scalars(S))) return st;
    if ((st = pc_status())) return st;
    const double rr0 = S->h->rz;
    std::vector<double> alpha, beta;
    for (int k = 0; k < steps; ++k) {
        const double rz_old = S->h->rz;
        if ((st = iga_apply_internal_sb(pl, IGA_FP64, ps.p, ps.q, s, IGA_SIGN_SPD, IGA_BC_IDENTITY))) return st;
        pcg_pq_kernel<double><<<kRedBlocks, kThreads, 0, s>>>(ps.p, ps.q, N, S->s, S->partials, S->counter);
        pcg_xr_kernel<double><<<kRedBlocks, kThreads, 0, s>>>(ps.x, ps.r, ps.p, ps.q, ps.z, N, S->s, S->partials,
                                                             S->counter);
        if ((st = pc_apply(ps, pl, S, o, ps.r, ps.z, o.pc_rtol, pcits))) return st;
        dot_kernel<double><<<kRedBlocks, kThreads, 0, s>>>(ps.r, ps.z, N, &S->s->rz, S->partials, S->counter);
        if ((st = sync_scalars(S))) return st;
        if ((st = pc_status())) return st;
        if (S->h->breakdown || !(S->h->alpha > 0.0)) break;
        alpha.push_back(S->h->alpha);
        const double rz_new = S->h->rz;
        if (!(rz_new > 1e-28 * rr0)) break;   // the Krylov space is exhausted
        beta.push_back(rz_new / rz_old);
        S->h->beta = beta.back();
        SOLVE_TRY(cudaMemcpyAsync(&S->s->beta, &S->h->beta, sizeof(double), cudaMemcpyHostToDevice, s));
        pcg_p_kernel<double><<<kRedBlocks, kThreads, 0, s>>>(ps.p, ps.z, N, S->s, 0);
    }
    const int K = (int)alpha.size();
    if (K < 1) {
        set_error("iga_spectrum_estimate: no Lanczos step completed");
        return IGA_ERR_BREAKDOWN;
    }
    // Lanczos matrix of the PCG coefficients: T_kk = 1/a_k + b_{k-1}/a_{k-1},
    // T_k,k+1 = sqrt(b_k) / a_k (M^-1 K in the M-inner product)
    std::vector<double> Td(K), To(K, 0.0), Md(K, 1.0), Mo(K, 0.0), lam(K), V((size_t)K * K);
    for (int k = 0; k < K; ++k) {
        Td[k] = 1.0 / alpha[k] + (k > 0 ? beta[k - 1] / alpha[k - 1] : 0.0);
        if (k + 1 < K) To[k] = -std::sqrt(beta[k]) / alpha[k];
    }
    pencil_eig(K, Td.data(), To.data(), Md.data(), Mo.data(), lam.data(), V.data());
    *lam_min = lam[0];
    *lam_max = lam[K - 1];
    if (steps_done) *steps_done = K;
    return IGA_OK;
}

}  // extern "C"
