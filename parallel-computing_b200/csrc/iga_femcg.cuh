// The reference's preconditioner apply, one launch: Jacobi-preconditioned CG
// on the bilinear FEM matrix (MyPCApply: an inner KSPCG + PCJACOBI,
// matrix_free/iteration_number_fempc_mf.cpp:11-17,210-224) for grids that fit
// one thread-block cluster.
//
// What bounds it: latency. A 66 x 66 grid has 4356 unknowns; as three
// launches per iteration (stencil + p.q, update, direction; 16 launches'
// worth captured per graph) an iteration took 16 us, nearly all of it launch
// gaps and grid-wide reductions. Here one cluster of up to 16 CTAs runs every
// iteration: CTA k owns a band of grid rows, thread (i, g) the L consecutive
// rows of column i in group g, with r, z and 1 / diag in registers and p in
// shared memory (one halo row on either side). Per iteration two cluster
// barriers: the warps' partial sums go straight into every CTA's slots
// through distributed shared memory, and after the barrier every warp sums
// all slots in the same order, so all threads hold the same totals without a
// broadcast (deterministic; sums in FP64). The direction's halo rows are
// recomputed locally: the neighbours send r / diag of their edge rows with
// the second reduction, which saves a third barrier.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "iga_device.cuh"

namespace iga {

constexpr int kIcgMaxCluster = 16;

// Launch shape of icg_cluster_kernel for an m x n grid: cluster CTAs (0: the
// grid does not fit), rows per CTA, rows per thread, threads, shared bytes.
struct IcgShape {
    int C = 0, rows = 0, L = 0, threads = 0;
    size_t smem = 0;
};

// Threads a CTA of L rows per thread may have (the kernel's launch bounds).
__host__ __device__ constexpr int icg_max_threads(int L) { return L <= 2 ? 1024 : 512; }

template <typename T>
inline size_t icg_smem(int m, int rows, int C, int nw)
{
    // reduction slots (p.q; r.z and r.r), p with halo rows (one entry of
    // slack at both ends), the neighbours' r / diag, the y coefficients
    return sizeof(double) * 3 * (size_t)C * nw +
           sizeof(T) * ((size_t)m * (rows + 2) + 2 + 2 * (size_t)m + 6 * (size_t)rows);
}

// The fewest rows per thread whose CTAs fit, with as many CTAs as cmax (a
// power of two) allows but no more than the rows: an iteration's time is its
// barriers plus one thread's rows.
template <typename T>
inline IcgShape icg_shape(int m, int n, int cmax)
{
    IcgShape s;
    int C = 1;
    while (2 * C <= cmax && 2 * C <= n) C *= 2;
    const int rows = (n + C - 1) / C;
    for (int L = 1; L <= 8; L *= 2) {
        const long long threads = (long long)m * ((rows + L - 1) / L);
        if (threads > icg_max_threads(L)) continue;
        s.C = C;
        s.rows = rows;
        s.L = L;
        s.threads = (int)((threads + 31) / 32 * 32);
        s.smem = icg_smem<T>(m, rows, C, s.threads / 32);
        return s;
    }
    return s;
}

template <typename T>
struct IcgArgs {
    const T *kd, *ko, *md, *mo;   // x: stiffness diag / off-diagonal (i, i+1), mass diag / off
    const T *ld, *lo, *nd, *no;   // y
    int m, n, rows;
    const T *rhs;
    T *z;
    double rtol;
    int maxit;
    int zero_on_break;   // z = 0 on a breakdown (a solver's own buffer), else z is left as it is
    DevScalars *s;
};

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Address of shared-memory location p in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void *p, int rank)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_store(uint32_t a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename T, int L>
__global__ void __launch_bounds__(icg_max_threads(L), 1) icg_cluster_kernel(IcgArgs<T> a)
{
    pdl_begin();
    extern __shared__ __align__(16) unsigned char icg_smem_raw[];
    uint32_t rank_u, C_u;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank_u));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(C_u));
    const int rank = (int)rank_u, C = (int)C_u, t = threadIdx.x, nt = blockDim.x;
    const int lane = t & 31, wid = t >> 5, nw = nt >> 5;
    const int m = a.m, n = a.n, rows = a.rows;
    double *red1 = reinterpret_cast<double *>(icg_smem_raw);   // p.q slots [C][nw]
    double *red2 = red1 + C * nw;                                // r.z and r.r slots [2][C][nw]
    T *ps = reinterpret_cast<T *>(red2 + 2 * C * nw) + 1;        // p: rows -1 .. rows, m per row
    T *hz = ps + (size_t)m * (rows + 2) + 1;                     // r / diag of the halo rows [2][m]
    T *yc = hz + 2 * m;                                          // y coefficients [rows][ky -1,0,1, my -1,0,1]
    const int j0 = rank * rows, nr = max(0, min(rows, n - j0));  // this CTA's rows

    // couplings of row j: none across the boundary ring
    for (int k = t; k < nr; k += nt) {
        const int j = j0 + k;
        const bool in = j > 0 && j < n - 1, lo = in && j - 1 >= 1, hi = in && j + 1 <= n - 2;
        yc[6 * k + 0] = lo ? a.lo[j - 1] : T(0);
        yc[6 * k + 1] = in ? a.ld[j] : T(0);
        yc[6 * k + 2] = hi ? a.lo[j] : T(0);
        yc[6 * k + 3] = lo ? a.no[j - 1] : T(0);
        yc[6 * k + 4] = in ? a.nd[j] : T(0);
        yc[6 * k + 5] = hi ? a.no[j] : T(0);
    }
    const int i = t % m, k0 = (t / m) * L;   // this thread's column and first row of the band
    const int cnt = min(L, nr - k0);         // its rows (may be <= 0)
    const bool xin = i > 0 && i < m - 1, xlo = xin && i - 1 >= 1, xhi = xin && i + 1 <= m - 2;
    const T kxl = xlo ? a.ko[i - 1] : T(0), kxd = xin ? a.kd[i] : T(0), kxr = xhi ? a.ko[i] : T(0);
    const T mxl = xlo ? a.mo[i - 1] : T(0), mxd = xin ? a.md[i] : T(0), mxr = xhi ? a.mo[i] : T(0);
    auto inv_diag = [&](int ii, int j) -> T {
        const bool in = ii > 0 && ii < m - 1 && j > 0 && j < n - 1;
        return in ? T(1) / (a.kd[ii] * a.nd[j] + a.md[ii] * a.ld[j]) : T(1);
    };

    T r[L], z[L], di[L];
    double v0 = 0.0, v1 = 0.0;
#pragma unroll
    for (int l = 0; l < L; ++l) {
        r[l] = z[l] = T(0);
        di[l] = T(1);
        if (l < cnt) {
            const int j = j0 + k0 + l;
            r[l] = a.rhs[(size_t)j * m + i];
            di[l] = inv_diag(i, j);
            const T p = r[l] * di[l];
            ps[(size_t)(k0 + l + 1) * m + i] = p;
            v0 += (double)r[l] * (double)p;
            v1 += (double)r[l] * (double)r[l];
        }
    }
    // halo rows of the first direction (zero past the grid's ends)
    for (int u = t; u < 2 * m; u += nt) {
        const int up = u >= m, ii = up ? u - m : u, j = up ? j0 + nr : j0 - 1;
        T p = T(0);
        if (nr > 0 && j >= 0 && j < n) p = a.rhs[(size_t)j * m + ii] * inv_diag(ii, j);
        ps[(size_t)(up ? nr + 1 : 0) * m + ii] = p;
    }
    if (t == 0) ps[-1] = ps[(size_t)m * (rows + 2)] = T(0);

    // sum over the cluster of v (slot array red, its K-th part)
    auto post = [&](double *red, double v) {
        v = warp_sum(v);
        if (lane < C) cluster_store(cluster_addr(red + rank * nw + wid, lane), v);
    };
    auto total = [&](const double *red) -> double {
        double v = 0.0;
        for (int u = lane; u < C * nw; u += 32) v += red[u];
        return warp_sum(v);
    };

    cluster_barrier();   // every CTA of the cluster runs: its slots may be written
    post(red2, v0);
    post(red2 + C * nw, v1);
    cluster_barrier();
    double rz = total(red2), rr = total(red2 + C * nw);
    const double tol2 = a.rtol * a.rtol * rr;
    int its = 0, brk = 0;
    if (rr != 0.0) {
        for (;;) {
            // q = K p: p's row contracted with the x stiffness and mass, then
            // combined along y (three rows of contractions roll through)
            T q[L];
            double pq = 0.0;
            if (cnt > 0) {
                auto rowk = [&](int k, T &s, T &c) {   // band row k (-1 .. rows)
                    const T *pp = ps + (size_t)(k + 1) * m + i;
                    const T pl = pp[-1], pc = pp[0], pr = pp[1];
                    s = kxl * pl + kxd * pc + kxr * pr;
                    c = mxl * pl + mxd * pc + mxr * pr;
                };
                T s0, c0, s1, c1, s2, c2;
                rowk(k0 - 1, s0, c0);
                rowk(k0, s1, c1);
#pragma unroll
                for (int l = 0; l < L; ++l) {
                    if (l < cnt) {
                        rowk(k0 + l + 1, s2, c2);
                        const T *y = yc + 6 * (k0 + l);
                        const T p = ps[(size_t)(k0 + l + 1) * m + i];
                        const int j = j0 + k0 + l;
                        const T w = (y[3] * s0 + y[0] * c0) + (y[4] * s1 + y[1] * c1) + (y[5] * s2 + y[2] * c2);
                        q[l] = xin && j > 0 && j < n - 1 ? w : p;
                        pq += (double)p * (double)q[l];
                        s0 = s1;
                        c0 = c1;
                        s1 = s2;
                        c1 = c2;
                    }
                }
            }
            post(red1, pq);
            cluster_barrier();
            pq = total(red1);
            if (!(pq > 0.0)) {
                brk = 1;
                break;
            }
            const T al = (T)(rz / pq);
            v0 = v1 = 0.0;
#pragma unroll
            for (int l = 0; l < L; ++l) {
                if (l < cnt) {
                    const T p = ps[(size_t)(k0 + l + 1) * m + i];
                    z[l] += al * p;
                    r[l] -= al * q[l];
                    const T rd = r[l] * di[l];
                    v0 += (double)r[l] * (double)rd;
                    v1 += (double)r[l] * (double)r[l];
                    const int k = k0 + l;
                    if (k == 0 && rank > 0) cluster_store(cluster_addr(hz + m + i, rank - 1), rd);
                    if (k == nr - 1 && j0 + nr < n) cluster_store(cluster_addr(hz + i, rank + 1), rd);
                }
            }
            post(red2, v0);
            post(red2 + C * nw, v1);
            cluster_barrier();
            const double rzn = total(red2);
            rr = total(red2 + C * nw);
            const T be = (T)(rzn / rz);
            rz = rzn;
            ++its;
            if (rr <= tol2 || its >= a.maxit || !(rr == rr)) break;
#pragma unroll
            for (int l = 0; l < L; ++l) {
                if (l < cnt) {
                    T *pp = ps + (size_t)(k0 + l + 1) * m + i;
                    *pp = fma(be, *pp, r[l] * di[l]);
                }
            }
            for (int u = t; u < 2 * m; u += nt) {
                const int up = u >= m, ii = up ? u - m : u, j = up ? j0 + nr : j0 - 1;
                if (nr > 0 && j >= 0 && j < n) {
                    T *pp = ps + (size_t)(up ? nr + 1 : 0) * m + ii;
                    *pp = fma(be, *pp, hz[u]);
                }
            }
            __syncthreads();
        }
    }
    if (!brk || a.zero_on_break) {
#pragma unroll
        for (int l = 0; l < L; ++l)
            if (l < cnt) a.z[(size_t)(j0 + k0 + l) * m + i] = brk ? T(0) : z[l];
    }
    if (rank == 0 && t == 0) {
        a.s->iiters = its;
        a.s->ipc += its;
        if (brk) a.s->ibreak = a.s->breakdown = 1;
    }
    // no CTA leaves while another may still store into its shared memory: the
    // last stores come before the barrier every CTA has just passed
}

}  // namespace iga
