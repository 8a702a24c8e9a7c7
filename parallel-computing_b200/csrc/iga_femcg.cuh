// The reference's preconditioner apply, one launch: Jacobi-preconditioned CG
// on the bilinear FEM matrix (MyPCApply: an inner KSPCG + PCJACOBI,
// matrix_free/iteration_number_fempc_mf.cpp:11-17,210-224) for grids that fit
// one thread-block cluster.
//
// What bounds it: latency. A 66 x 66 grid has 4356 unknowns; as three
// launches per iteration (stencil + p.q, update, direction) an iteration took
// 16.4 us, nearly all of it launch gaps and grid-wide reductions. Here one
// cluster of CTAs runs every iteration: CTA k owns a band of grid rows, thread
// (i, g) the L consecutive rows of column i in group g, with r, z and 1 / diag
// in registers and p in shared memory (one halo row on either side). The
// warps' partial sums go straight into every CTA's slots (st.async through
// distributed shared memory, counted by the receiver's mbarrier), and every
// warp sums all slots in the same order, so all threads hold the same totals
// without a broadcast (deterministic; sums in FP64). The direction's halo
// rows are recomputed locally: the neighbours send r / diag of their edge rows
// with the second sum, which saves a third exchange. So an iteration has two
// exchanges and one CTA barrier but no cluster barrier: with two cluster
// barriers (arrive.release / wait.acquire) in their place an iteration at 64^2
// took 2.9 us, 22% of the stalls on the release fence, against 2.2 us (128^2:
// 4.1 against 2.9).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "iga_device.cuh"

namespace iga {

// Launch shape of icg_cluster_kernel for an m x n grid: cluster CTAs (0: the
// grid does not fit), rows per CTA, rows per thread, threads, shared bytes.
struct IcgShape {
    int C = 0, rows = 0, L = 0, threads = 0;
    size_t smem = 0;
};

constexpr int kIcgMaxThreads = 512;         // of a CTA (the kernel's launch bounds)
constexpr size_t kIcgMaxSmem = 226 * 1024;   // of a CTA (the limit set for every instance of the kernel)

template <typename T>
inline size_t icg_smem(int m, int rows, int C, int nw)
{
    // three mbarriers, the slots (r.z and r.r; p.q), p with halo rows (one entry
    // of slack at both ends), the neighbours' r / diag, the y coefficients
    return 32 + sizeof(double) * 3 * (size_t)C * nw +
           sizeof(T) * ((size_t)m * (rows + 2) + 2 + 2 * (size_t)m + 6 * (size_t)rows);
}

// Shape k = 0 .. 3 in the order of preference (C = 0: does not fit, or no
// further shape). Four rows per thread before eight, whose own rows dominate
// an iteration, and eight CTAs (the portable cluster size) before sixteen,
// whose sums have twice the slots. FP64, us an iteration, in CTAs x rows per
// thread: 64^2 8 x 4 2.25, 16 x 4 2.22, 8 x 8 3.65, 16 x 8 3.23; 128^2 16 x 4 2.85,
// 8 x 8 4.35. Other shapes would be a little faster where they fit (64^2 8 x 2
// 2.00, 16^2 8 x 1 1.05 against 1.14, 96^2 16 x 4 2.42 against 2.71): fewer rows
// per thread lost only with the cluster barriers that the mbarriers replaced.
template <typename T>
inline IcgShape icg_shape(int m, int n, int k)
{
    const int cmax = k == 0 || k == 2 ? 8 : 16, L = k < 2 ? 4 : 8;
    IcgShape s;
    int C = 1;
    while (2 * C <= cmax && 2 * C <= n) C *= 2;
    const int rows = (n + C - 1) / C;
    const long long threads = (long long)m * ((rows + L - 1) / L);
    if (threads > kIcgMaxThreads) return s;
    s.rows = rows;
    s.L = L == 4 && rows < 4 ? (rows >= 2 ? 2 : 1) : L;
    s.threads = (int)(((long long)m * ((rows + s.L - 1) / s.L) + 31) / 32 * 32);
    if (s.threads > kIcgMaxThreads) {
        s.L = L;
        s.threads = (int)((threads + 31) / 32 * 32);
    }
    s.smem = icg_smem<T>(m, rows, C, s.threads / 32);
    s.C = s.smem <= kIcgMaxSmem ? C : 0;
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
    long long wait_polls;   // LIMITED: polls of each wait before the solve gives up (IGA_ERR_TIMEOUT)
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
// Store into a CTA of the cluster, counted in bytes by the mbarrier there.
__device__ __forceinline__ void cluster_store(uint32_t a, double v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(a), "d"(v),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t a, float v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t a, double2 v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(a),
                 "d"(v.x), "d"(v.y), "r"(bar)
                 : "memory");
}
// Bounded wait of a whole warp: the same answer in every lane.
__device__ __forceinline__ bool cluster_wait(uint64_t *bar, uint32_t parity, long long limit = kWaitLimit)
{
    bool done = false;
    for (long long it = 0; it < limit; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) {
            done = true;
            break;
        }
    }
    return __all_sync(0xffffffffu, done);
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// LIMITED: with a limit of the caller's on each wait, in place of kWaitLimit (a
// limit the compiler does not know costs 0.1 us an iteration).
template <typename T, int L, bool LIMITED>
__global__ void __launch_bounds__(kIcgMaxThreads, 1) icg_cluster_kernel(IcgArgs<T> a)
{
    pdl_begin();
    extern __shared__ __align__(16) unsigned char icg_smem_raw[];
    uint32_t rank_u, C_u;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank_u));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(C_u));
    const int rank = (int)rank_u, C = (int)C_u, t = threadIdx.x, nt = blockDim.x;
    const int lane = t & 31, wid = t >> 5, nw = nt >> 5;
    const int m = a.m, n = a.n, rows = a.rows;
    uint64_t *bar = reinterpret_cast<uint64_t *>(icg_smem_raw);         // p.q; r.z, r.r and halo rows; CTA
    double2 *red2 = reinterpret_cast<double2 *>(icg_smem_raw + 32);     // (r.z, r.r) slots [C][nw]
    double *red1 = reinterpret_cast<double *>(red2 + C * nw);           // p.q slots [C][nw]
    T *ps = reinterpret_cast<T *>(red1 + C * nw) + 1;                   // p: rows -1 .. rows, m per row
    T *hz = ps + (size_t)m * (rows + 2) + 1;                     // r / diag of the halo rows [2][m]
    T *yc = hz + 2 * m;                                          // y coefficients [rows][ky -1,0,1, my -1,0,1]
    const int j0 = rank * rows, nr = max(0, min(rows, n - j0));         // this CTA's rows
    // bytes an exchange brings: every warp's partial sums, and the halo rows
    const uint32_t tx1 = (uint32_t)(C * nw * 8), tx2 = (uint32_t)(C * nw * 16);
    const uint32_t txh = (uint32_t)(m * sizeof(T)) * ((nr > 0 && rank > 0 ? 1u : 0u) + (nr > 0 && j0 + nr < n ? 1u : 0u));
    if (t == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_init(&bar[2], nw);
        fence_mbar_init();
        mbar_arrive_expect_tx(&bar[0], tx1);
        mbar_arrive_expect_tx(&bar[1], tx2);
    }

    // The x stiffness and mass go in scaled to about 1 by powers of two, which
    // the y factors undo (exactly): K's products of the two are about 1 whatever
    // the mesh width, so its rows overflow and underflow no earlier than p does.
    auto scale = [](T v) { return v > T(0) && isfinite(v) ? (T)scalbn(T(1), -ilogb(v)) : T(1); };
    const T sk = scale(a.kd[m / 2]), sm = scale(a.md[m / 2]), uk = T(1) / sk, um = T(1) / sm;

    // couplings of row j: none across the boundary ring
    for (int k = t; k < nr; k += nt) {
        const int j = j0 + k;
        const bool in = j > 0 && j < n - 1, lo = in && j - 1 >= 1, hi = in && j + 1 <= n - 2;
        yc[6 * k + 0] = lo ? um * a.lo[j - 1] : T(0);
        yc[6 * k + 1] = in ? um * a.ld[j] : T(0);
        yc[6 * k + 2] = hi ? um * a.lo[j] : T(0);
        yc[6 * k + 3] = lo ? uk * a.no[j - 1] : T(0);
        yc[6 * k + 4] = in ? uk * a.nd[j] : T(0);
        yc[6 * k + 5] = hi ? uk * a.no[j] : T(0);
    }
    const int i = t % m, k0 = (t / m) * L;   // this thread's column and first row of the band
    const int cnt = min(L, nr - k0);         // its rows (may be <= 0)
    const bool xin = i > 0 && i < m - 1, xlo = xin && i - 1 >= 1, xhi = xin && i + 1 <= m - 2;
    const T kxl = xlo ? sk * a.ko[i - 1] : T(0), kxd = xin ? sk * a.kd[i] : T(0), kxr = xhi ? sk * a.ko[i] : T(0);
    const T mxl = xlo ? sm * a.mo[i - 1] : T(0), mxd = xin ? sm * a.md[i] : T(0), mxr = xhi ? sm * a.mo[i] : T(0);
    auto inv_diag = [&](int ii, int j) -> T {
        const bool in = ii > 0 && ii < m - 1 && j > 0 && j < n - 1;
        return in ? T(1) / (a.kd[ii] * a.nd[j] + a.md[ii] * a.ld[j]) : T(1);
    };

    // An infinite entry of the boundary ring is no neighbour of an interior one,
    // but its zero coupling would make NaN of it there: the first direction holds
    // 1 in its place, and r.z is NaN, which makes NaN of z and ends the solve
    // after one iteration.
    auto ring_inf = [&](int ii, int j, T p) { return isinf(p) && (ii == 0 || j == 0 || ii == m - 1 || j == n - 1); };

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
            const bool inf = ring_inf(i, j, p);
            ps[(size_t)(k0 + l + 1) * m + i] = inf ? T(1) : p;
            v0 += inf ? nan("") : (double)r[l] * (double)p;
            v1 += (double)r[l] * (double)r[l];
        }
    }
    // halo rows of the first direction (zero past the grid's ends)
    for (int u = t; u < 2 * m; u += nt) {
        const int up = u >= m, ii = up ? u - m : u, j = up ? j0 + nr : j0 - 1;
        T p = T(0);
        if (nr > 0 && j >= 0 && j < n) p = a.rhs[(size_t)j * m + ii] * inv_diag(ii, j);
        if (ring_inf(ii, j, p)) p = T(1);
        ps[(size_t)(up ? nr + 1 : 0) * m + ii] = p;
    }
    if (t == 0) ps[-1] = ps[(size_t)m * (rows + 2)] = T(0);

    // Exchanges: every warp stores its sum into each CTA's slots, then each
    // warp sums all slots. A slot array is written again only after its
    // readers have taken part in the other exchange, so one copy is enough.
    uint32_t ph1 = 0, ph2 = 0, ph3 = 0;
    auto post1 = [&](double v) {
        v = warp_sum(v);
        if (lane < C) cluster_store(cluster_addr(red1 + rank * nw + wid, lane), v, cluster_addr(&bar[0], lane));
    };
    auto post2 = [&](double va, double vb) {
        const double2 v = make_double2(warp_sum(va), warp_sum(vb));
        if (lane < C) cluster_store(cluster_addr(red2 + rank * nw + wid, lane), v, cluster_addr(&bar[1], lane));
    };
    const long long limit = LIMITED ? a.wait_polls : kWaitLimit;
    bool ok = true;
    auto sum1 = [&]() -> double {
        double v = 0.0;
        for (int u = lane; u < C * nw; u += 32) v += red1[u];
        return warp_sum(v);
    };
    auto total1 = [&]() -> double {
        ok = cluster_wait(&bar[0], ph1, limit);
        ph1 ^= 1u;
        if (t == 0 && ok) mbar_arrive_expect_tx(&bar[0], tx1);
        return sum1();
    };
    auto sum2 = [&](double &va, double &vb) {
        va = vb = 0.0;
        for (int u = lane; u < C * nw; u += 32) {
            const double2 w = red2[u];
            va += w.x;
            vb += w.y;
        }
        va = warp_sum(va);
        vb = warp_sum(vb);
    };
    auto total2 = [&](double &va, double &vb) {
        ok = cluster_wait(&bar[1], ph2, limit);
        ph2 ^= 1u;
        if (t == 0 && ok) mbar_arrive_expect_tx(&bar[1], tx2 + txh);
        sum2(va, vb);
    };
    // the CTA's warps meet on an mbarrier too, so that a warp whose wait gave
    // up cannot leave the others at a barrier
    auto arrive3 = [&] {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar[2])) : "memory");
    };

    cluster_barrier();   // every CTA of the cluster has set up its mbarriers; p is in place
    post2(v0, v1);
    double rz, rr;
    total2(rz, rr);
    const double tol2 = a.rtol * a.rtol * rr;
    int its = 0, brk = 0, gave = ok ? -1 : 1;   // gave: the mbarrier this warp gave up at
    if (ok && rr != 0.0) {
        double inv_rz = 1.0 / rz;
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
            post1(pq);
            pq = total1();
            if (!ok || !(pq > 0.0)) {
                brk = 1;
                gave = 0;
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
                    if (k == 0 && rank > 0) cluster_store(cluster_addr(hz + m + i, rank - 1), rd, cluster_addr(&bar[1], rank - 1));
                    if (k == nr - 1 && j0 + nr < n) cluster_store(cluster_addr(hz + i, rank + 1), rd, cluster_addr(&bar[1], rank + 1));
                }
            }
            post2(v0, v1);
            const double inv_old = inv_rz;
            total2(rz, rr);
            const T be = (T)(rz * inv_old);
            inv_rz = 1.0 / rz;   // next iteration's, off the critical path
            ++its;
            if (!ok || rr <= tol2 || its >= a.maxit || !(rr == rr)) {
                gave = 1;
                break;
            }
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
            arrive3();
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bar[2], ph3, limit));
            ph3 ^= 1u;
            if (!ok) {
                gave = 2;
                break;
            }
        }
    }
    // No CTA may leave while stores are on their way into its shared memory. So
    // a warp that gave up lets that exchange land, with the full limit, and
    // unless its totals end the solve anyway sends NaN in the next one and lets
    // that land too: the NaN ends the solve in every CTA there, with every
    // exchange complete.
    if (!ok) {
        bool landed = gave == 2 ? __all_sync(0xffffffffu, mbar_wait_bounded(&bar[2], ph3 ^ 1u)) != 0
                                : cluster_wait(&bar[gave], (gave == 0 ? ph1 : ph2) ^ 1u);
        if (gave == 0 && landed && sum1() > 0.0) {
#pragma unroll
            for (int l = 0; l < L; ++l) {
                if (l >= cnt) continue;
                const int k = k0 + l;
                if (k == 0 && rank > 0) cluster_store(cluster_addr(hz + m + i, rank - 1), T(0), cluster_addr(&bar[1], rank - 1));
                if (k == nr - 1 && j0 + nr < n) cluster_store(cluster_addr(hz + i, rank + 1), T(0), cluster_addr(&bar[1], rank + 1));
            }
            post2(nan(""), nan(""));
            cluster_wait(&bar[1], ph2);
        }
        if (gave == 1 && landed) {
            sum2(rz, rr);
            if (its == 0) landed = rr != 0.0;
            else landed = !(rr <= tol2 || its >= a.maxit || !(rr == rr));
            if (landed && its > 0) arrive3();
        }
        if (gave > 0 && landed) {
            post1(nan(""));
            cluster_wait(&bar[0], ph1);
        }
    }
    if ((!brk && ok) || a.zero_on_break) {
#pragma unroll
        for (int l = 0; l < L; ++l)
            if (l < cnt) a.z[(size_t)(j0 + k0 + l) * m + i] = brk || !ok ? T(0) : z[l];
    }
    if (!ok) a.s->err = a.s->breakdown = 1;
    if (rank == 0 && t == 0) {
        a.s->iiters = its;
        a.s->ipc += its;
        if (brk && ok) a.s->ibreak = a.s->breakdown = 1;
    }
    // no CTA leaves while another may still store into its shared memory
    cluster_barrier();
}

}  // namespace iga
