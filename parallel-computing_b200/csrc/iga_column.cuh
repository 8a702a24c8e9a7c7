// Quadrature-point fields by sum factorisation, one thread per (element
// column, x quadrature point): the precomputed geometry G, the adjoint
// gradient and the load vector.
//
// A thread contracts each control-point row along x once (value and
// derivative) into a rolling window of P + 1 rows and walks up its column of
// elements; at every quadrature row the window is contracted along y. That is
// 4 (P + 1) multiply-adds per field and point where the point's full double
// sum takes 4 (P + 1)^2, and no lane idles (the point-per-thread kernels this
// replaced spent their time on the tables' and control points' loads: every
// term of the double sum read both).
#pragma once
#include <cuda_runtime.h>

#include "iga_plan.hpp"

namespace iga {

// Element rows a thread walks: up to 8, over which its P prologue rows are
// spread; fewer on patches that would leave SMs without a unit (64^2 p=3, one
// row: adjoint gradient 5.8 us, eight rows 18.7 us).
inline int column_rows(int NSX, int ney, int nsm)
{
    int r = 8;
    while (r > 1 && (long long)NSX * ((ney + r - 1) / r) < 4LL * nsm) r /= 2;
    return r;
}

// Basis of one x quadrature point of one element column.
template <int P>
struct ColumnBasis {
    static constexpr int NB = P + 1, NQ = P + 1;
    double n[NB], d[NB];
    __device__ __forceinline__ void load(const double *__restrict__ tabX, int ex, int qx)
    {
        const double *v = tabX + ((size_t)ex * 2 * NQ + qx) * NB;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            n[i] = v[i];
            d[i] = v[NQ * NB + i];
        }
    }
};

// The rolling window of one scalar field: rows ey .. ey + P contracted along x.
template <int P>
struct ColumnField {
    static constexpr int NB = P + 1;
    double v[NB], d[NB];
    __device__ __forceinline__ void shift()
    {
#pragma unroll
        for (int k = 0; k < P; ++k) {
            v[k] = v[k + 1];
            d[k] = d[k + 1];
        }
    }
    // row `slot` from the field's values at the element's columns, stride
    // apart (explicit multiply-adds: every kernel rounds alike)
    __device__ __forceinline__ void row(int slot, const ColumnBasis<P> &b, const double *__restrict__ f, int stride)
    {
        double a = 0.0, c = 0.0;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const double x = f[(size_t)i * stride];
            a = fma(b.n[i], x, a);
            c = fma(b.d[i], x, c);
        }
        v[slot] = a;
        d[slot] = c;
    }
    // d/dxi and d/deta at a quadrature row with y values ny and derivatives dy
    __device__ __forceinline__ void grad(const double *ny, const double *dy, double &xi, double &eta) const
    {
        double a = 0.0, c = 0.0;
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            a = fma(ny[k], d[k], a);
            c = fma(dy[k], v[k], c);
        }
        xi = a;
        eta = c;
    }
    __device__ __forceinline__ double value(const double *ny) const
    {
        double a = 0.0;
#pragma unroll
        for (int k = 0; k < NB; ++k) a = fma(ny[k], v[k], a);
        return a;
    }
};

// Both coordinates of the control net (x, y interleaved).
template <int P>
struct ColumnNet {
    static constexpr int NB = P + 1;
    ColumnField<P> x, y;
    __device__ __forceinline__ void shift()
    {
        x.shift();
        y.shift();
    }
    __device__ __forceinline__ void row(int slot, const ColumnBasis<P> &b, const double *__restrict__ CP, size_t A)
    {
        double xa = 0.0, xc = 0.0, ya = 0.0, yc = 0.0;
        const double2 *p = reinterpret_cast<const double2 *>(CP) + A;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const double2 q = p[i];
            xa = fma(b.n[i], q.x, xa);
            xc = fma(b.d[i], q.x, xc);
            ya = fma(b.n[i], q.y, ya);
            yc = fma(b.d[i], q.y, yc);
        }
        x.v[slot] = xa;
        x.d[slot] = xc;
        y.v[slot] = ya;
        y.d[slot] = yc;
    }
};

// y basis of quadrature row qy of element row ey (the same for every thread
// of a column walk: cached loads).
template <int P>
__device__ __forceinline__ void load_y_basis(const double *__restrict__ tabY, int ey, int qy, double (&n)[P + 1],
                                             double (&d)[P + 1])
{
    constexpr int NB = P + 1, NQ = P + 1;
    const double *v = tabY + ((size_t)ey * 2 * NQ + qy) * NB;
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        n[k] = v[k];
        d[k] = v[NQ * NB + k];
    }
}

// ------------------------------------------------------------ geometry
// Units of a job: one column strip (16 element columns x NQ quadrature
// points: one thread each) by `rows` element rows.
__host__ __device__ __forceinline__ int column_chunks(int ney, int rows) { return (ney + rows - 1) / rows; }
__host__ __device__ __forceinline__ long long geom_units(const GeomJob &j)
{
    return (long long)j.g.NSX * column_chunks(j.g.ney, j.rows);
}

// G = w kappa det(J) J^-1 J^-T of one unit, in the order the apply kernel
// streams it, for either precision's strips; kappa_out (or null) receives a
// copy of the unit's kappa. Thread t of 16 NQ: where a quadrature row of G is
// lane-major (even NQ) column t / NQ, point t % NQ, so that a warp's 96 values
// are one contiguous run, written through shared memory (stage: 96 values per
// warp) as whole lines; else point t / 16, column t % 16, whose 16 columns are
// contiguous. Padding columns get G = 0; padding rows past the patch are
// never read. The unit's kappa comes a row ahead of its use. Bound: latency of
// FP64 chains and loads at 20 warps per SM, then the bytes of G and kappa
// (168 MB, 26 us at p=3 512^2). set_kappa, FP64: p=3 512^2 217 -> 52 us (64
// us with kappa loaded at its use), 1024^2 848 -> 174 us, p=2 2048^2 1364 ->
// 490 us against one point per thread with the full double sum; holding the
// registers to more CTAs per SM was slower (p=3 512^2 72 us at 12).
template <int P>
__device__ __forceinline__ void geom_unit(const GeomJob &j, int gx, int chunk, int t, double *stage)
{
    constexpr int NB = P + 1, NQ = P + 1, NQ2 = NQ * NQ;
    constexpr bool LM = g_lane_major(NQ);
    const StripGrid &g = j.g;
    const int c = LM ? t / NQ : t % kSW, qx = LM ? t % NQ : t / kSW;
    const int ex = kSW * gx + c;
    const bool in = ex < g.nex;
    const int e0 = chunk * j.rows, e1 = min(e0 + j.rows, g.ney);
    const int lane = threadIdx.x & 31;
    ColumnBasis<P> b;
    ColumnNet<P> net;
    double wx = 0.0;
    if (in) {
        b.load(j.tx, ex, qx);
        wx = j.qw[qx];
#pragma unroll
        for (int r = 0; r < P; ++r) net.row(r, b, j.cp, (size_t)(e0 + r) * g.m + ex);
    }
    bool bad = false;
    // kappa of the next element row, requested a row ahead
    double kn[NQ];
    const double *__restrict__ kin = j.kappa;
    auto fetch = [&](int e) {
#pragma unroll
        for (int qy = 0; qy < NQ; ++qy)
            kn[qy] = __ldg(kin + ((size_t)e * g.nex + ex) * NQ2 + qy * NQ + qx);
    };
    if (in && kin) fetch(e0);
    for (int e = e0; e < e1; ++e) {
        double kq[NQ];
        if (in) {
            net.row(P, b, j.cp, (size_t)(e + P) * g.m + ex);
#pragma unroll
            for (int qy = 0; qy < NQ; ++qy) kq[qy] = kin ? kn[qy] : 1.0;
            if (kin && e + 1 < e1) fetch(e + 1);
            if (j.kappa_out)
#pragma unroll
                for (int qy = 0; qy < NQ; ++qy) j.kappa_out[((size_t)e * g.nex + ex) * NQ2 + qy * NQ + qx] = kq[qy];
        }
        double *G64 = j.G64 ? j.G64 + (((size_t)gx * j.NSY64 + e / j.TY64) * j.TY64 + e % j.TY64) * NQ2 * 3 * kSW : nullptr;
        float *G32 = j.G32 ? j.G32 + (((size_t)gx * j.NSY32 + e / j.TY32) * j.TY32 + e % j.TY32) * NQ2 * 3 * kSW : nullptr;
#pragma unroll
        for (int qy = 0; qy < NQ; ++qy) {
            double g3[3] = {0.0, 0.0, 0.0};
            if (in) {
                double ny[NB], dy[NB], x_xi, x_eta, y_xi, y_eta;
                load_y_basis<P>(j.ty, e, qy, ny, dy);
                net.x.grad(ny, dy, x_xi, x_eta);
                net.y.grad(ny, dy, y_xi, y_eta);
                const double det = fma(x_xi, y_eta, -(x_eta * y_xi));
                if (!(det > 0.0)) bad = true;
                const double f = wx * j.qw[qy] * kq[qy] / det;
                g3[0] = f * fma(x_eta, x_eta, y_eta * y_eta);
                g3[1] = -f * fma(x_xi, x_eta, y_xi * y_eta);
                g3[2] = f * fma(x_xi, x_xi, y_xi * y_xi);
            }
            if constexpr (LM) {
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 3; ++k) stage[3 * lane + k] = g3[k];
                __syncwarp();
                const size_t o = (size_t)qy * NQ * 3 * kSW + 3 * (t - lane) + lane;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double v = stage[32 * k + lane];
                    if (G64) G64[o + 32 * k] = v;
                    if (G32) G32[o + 32 * k] = (float)v;
                }
            } else {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if (G64) G64[g_index(NQ, 8, qy, qx, k, c)] = g3[k];
                    if (G32) G32[g_index(NQ, 4, qy, qx, k, c)] = (float)g3[k];
                }
            }
        }
        net.shift();
    }
    if (bad) atomicExch(j.err, 1 /* IGA_ERR_ARG: non-positive Jacobian */);
}

template <int P>
__global__ void __launch_bounds__(kSW *(P + 1)) geom_kernel(const GeomJob j)
{
    __shared__ double stage[kSW * (P + 1) * 3];
    const int nc = column_chunks(j.g.ney, j.rows), gx = blockIdx.x / nc;
    geom_unit<P>(j, gx, blockIdx.x - gx * nc, threadIdx.x, stage + (threadIdx.x >> 5) * 96);
}

// ------------------------------------------------------------ adjoint gradient
// g_q = -(grad lambda . grad u)(x_q) JxW_q. Thread t of a unit: column t / NQ,
// point t % NQ (a thread row of one element is contiguous in g). Bound: FP64
// and load latency (p=3 512^2 187 -> 36 us, floor 5 us for g's bytes; p=4 411
// -> 70 us against one point per thread).
template <int P>
__global__ void __launch_bounds__(kSW *(P + 1)) adjoint_kernel(const double *__restrict__ u, const double *__restrict__ lam,
                                                               double *__restrict__ out, const double *__restrict__ tabX,
                                                               const double *__restrict__ tabY,
                                                               const double *__restrict__ CP,
                                                               const double *__restrict__ qw, StripGrid g, int nrows)
{
    constexpr int NB = P + 1, NQ = P + 1, NQ2 = NQ * NQ;
    const int nc = column_chunks(g.ney, nrows), gx = blockIdx.x / nc;
    const int ex = kSW * gx + threadIdx.x / NQ, qx = threadIdx.x % NQ;
    if (ex >= g.nex) return;
    const int e0 = (blockIdx.x - gx * nc) * nrows, e1 = min(e0 + nrows, g.ney);
    ColumnBasis<P> b;
    b.load(tabX, ex, qx);
    ColumnNet<P> net;
    ColumnField<P> fu, fl;
    auto rows = [&](int slot, int R) {
        const size_t A = (size_t)R * g.m + ex;
        net.row(slot, b, CP, A);
        fu.row(slot, b, u + A, 1);
        fl.row(slot, b, lam + A, 1);
    };
#pragma unroll
    for (int r = 0; r < P; ++r) rows(r, e0 + r);
    const double wx = qw[qx];
    for (int e = e0; e < e1; ++e) {
        rows(P, e + P);
        double *o = out + ((size_t)e * g.nex + ex) * NQ2 + qx;
#pragma unroll
        for (int qy = 0; qy < NQ; ++qy) {
            double ny[NB], dy[NB], x_xi, x_eta, y_xi, y_eta, u_xi, u_eta, l_xi, l_eta;
            load_y_basis<P>(tabY, e, qy, ny, dy);
            net.x.grad(ny, dy, x_xi, x_eta);
            net.y.grad(ny, dy, y_xi, y_eta);
            fu.grad(ny, dy, u_xi, u_eta);
            fl.grad(ny, dy, l_xi, l_eta);
            const double f = wx * qw[qy] / fma(x_xi, y_eta, -(x_eta * y_xi));
            // w det (J^-T grad lambda) . (J^-T grad u), J^-T = adj / det
            const double ux = fma(y_eta, u_xi, -(y_xi * u_eta)), uy = fma(x_xi, u_eta, -(x_eta * u_xi));
            const double lx = fma(y_eta, l_xi, -(y_xi * l_eta)), ly = fma(x_xi, l_eta, -(x_eta * l_xi));
            o[qy * NQ] = -f * fma(ux, lx, uy * ly);
        }
        net.shift();
        fu.shift();
        fl.shift();
    }
}

// ------------------------------------------------------------ load vector
// F = int R f (LocalAssemblyMF::AssemLocalLoad, matrix_free/src/
// LocalAssemblyMF.cpp:3-29), zero on the boundary ring, without atomics: a
// CTA owns kRhsCols control-point columns by `rows` rows and evaluates f at
// every quadrature point of the elements that support them (a halo of P
// columns and rows). Each (element column, point) thread walks up its
// column, sums f w det times the y values into a rolling window of P + 1
// rows, and puts every finished row in shared memory; after kRhsBlock rows
// all threads contract those with the x values of the P + 1 elements under
// each control-point column.
// Bound: FP64 arithmetic of f (a sine, an arctangent, a square root a point).
// With one control point per thread, f and the geometry evaluated at every
// point of its (P + 1)^2 elements, the annulus load took 16.2 ms at p=4 512^2
// (now 0.21 ms), f = x(1-x)y(1-y) 35 ms at p=3 1024^2 (now 0.19 ms).
constexpr int kRhsCols = 32, kRhsBlock = 8;

__device__ inline double load_f(int fkind, double x, double y)
{
    const double pi = 3.141592653589793238462643383279;
    if (fkind == 0) return x * (1 - x) * y * (1 - y);
    if (fkind == 1) return 2.0 * pi * pi * sin(pi * x) * sin(pi * y);
    const double r = sqrt(x * x + y * y), th = atan2(y, x);
    double s, c;
    sincos(pi * r, &s, &c);
    return (pi * pi * s - pi * c / r + 4.0 * s / (r * r)) * sin(2.0 * th);
}

constexpr int rhs_threads(int P) { return ((kRhsCols + P) * (P + 1) + 31) / 32 * 32; }
// CTAs an SM holds (registers): the launch makes one wave of them.
constexpr int rhs_ctas(int P) { return P <= 2 ? 4 : P == 3 ? 3 : P == 4 ? 2 : 1; }

template <int P>
__global__ void __launch_bounds__(rhs_threads(P), rhs_ctas(P)) rhs_kernel(double *__restrict__ F, const double *__restrict__ tabX,
                                                             const double *__restrict__ tabY,
                                                             const double *__restrict__ CP,
                                                             const double *__restrict__ qw, int fkind, StripGrid g,
                                                             int rows)
{
    constexpr int NB = P + 1, NQ = P + 1, EC = kRhsCols + P;   // element columns of the CTA
    __shared__ double sh[kRhsBlock][EC * NQ];
    const int cols = (g.m + kRhsCols - 1) / kRhsCols, by = blockIdx.x / cols;
    const int C0 = kRhsCols * (blockIdx.x - by * cols), R0 = rows * by, R1 = min(R0 + rows, g.n);
    const int t = threadIdx.x, ex = C0 - P + t / NQ, qx = t % NQ;
    const bool in = t < EC * NQ && ex >= 0 && ex < g.nex;
    ColumnBasis<P> b;
    ColumnNet<P> net;
    double acc[NB], wx = 0.0;
#pragma unroll
    for (int k = 0; k < NB; ++k) acc[k] = 0.0;
    int e = max(R0 - P, 0);   // the first element row that touches R0
    if (in) {
        b.load(tabX, ex, qx);
        wx = qw[qx];
        if (e < g.ney)
#pragma unroll
            for (int r = 0; r < P; ++r) net.row(r, b, CP, (size_t)(e + r) * g.m + ex);
    }
    for (int B0 = R0; B0 < R1; B0 += kRhsBlock) {
        const int B1 = min(B0 + kRhsBlock, R1);
        for (; e < B1; ++e) {   // element row e finishes control-point row e
            if (in && e < g.ney) {
                net.row(P, b, CP, (size_t)(e + P) * g.m + ex);
#pragma unroll
                for (int qy = 0; qy < NQ; ++qy) {
                    double ny[NB], dy[NB], x_xi, x_eta, y_xi, y_eta;
                    load_y_basis<P>(tabY, e, qy, ny, dy);
                    net.x.grad(ny, dy, x_xi, x_eta);
                    net.y.grad(ny, dy, y_xi, y_eta);
                    const double det = fma(x_xi, y_eta, -(x_eta * y_xi));
                    const double s = load_f(fkind, net.x.value(ny), net.y.value(ny)) * (wx * qw[qy]) * det;
#pragma unroll
                    for (int k = 0; k < NB; ++k) acc[k] = fma(ny[k], s, acc[k]);
                }
                net.shift();
            }
            if (e >= B0 && t < EC * NQ) sh[e - B0][t] = in ? acc[0] : 0.0;
#pragma unroll
            for (int k = 0; k < P; ++k) acc[k] = acc[k + 1];
            acc[P] = 0.0;
        }
        __syncthreads();
        for (int o = t; o < (B1 - B0) * kRhsCols; o += blockDim.x) {
            const int k = o / kRhsCols, cl = o % kRhsCols, C = C0 + cl, R = B0 + k;
            if (C >= g.m) continue;
            double v = 0.0;
            if (R > 0 && C > 0 && R < g.n - 1 && C < g.m - 1) {
                // element C - il holds control-point column C as its function il
                for (int il = 0; il < NB; ++il) {
                    const int x = C - il;
                    if (x < 0 || x >= g.nex) continue;
                    const double *N = tabX + (size_t)x * 2 * NQ * NB + il;
                    const double *q = sh[k] + (cl + P - il) * NQ;
                    for (int a = 0; a < NQ; ++a) v = fma(N[a * NB], q[a], v);
                }
            }
            F[(size_t)R * g.m + C] = v;
        }
        __syncthreads();
    }
}

}  // namespace iga
