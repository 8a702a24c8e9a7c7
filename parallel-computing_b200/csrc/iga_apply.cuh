// Matrix-free IGA Poisson operator y = sign * K x for sm_100a.
//
// Maths (reference: LocalAssemblyMF::LocalMatMulMF, matrix_free/src/LocalAssemblyMF.cpp:31-67,
// and ElementMF, matrix_free/src/ElementMF.cpp:106-296): per element e and
// quadrature point q,
//     y_e += sign * sum_q  grad_xi N^T  G_q  grad_xi u,
//     G_q  = w_q kappa_q det(J) J^-1 J^-T   (symmetric 2x2, 3 values),
// with N the tensor product of the element's 1-D B-spline (or 1-D rational)
// bases, derivatives in reference-element coordinates. The element operator
// is applied by sum factorisation: two 1-D contractions in, a 2x2 multiply per
// quadrature point, two 1-D contractions out.
//
// Work decomposition: a WARP owns a strip of SW = 16 element columns and
// marches over TY element rows. Two lanes share an element column: lane
// 2c + h handles column c and the quadrature columns qx = h*QH + j, j < QH
// (QH = ceil((p+1)/2)). Per row step every lane
//   1. contracts the new control-point row along x for its qx (rolling xs),
//   2. contracts along y with the row's tables (warp-uniform loads),
//   3. applies G: streamed into shared memory by the bulk-copy (TMA) engine
//      (GEOM = 0, the mult_sf path) or computed in registers from the control
//      points by the same rolling sum factorisation (GEOM = 1, the mult_mf path),
//   4. accumulates the y-transposed contraction into rolling row buffers acc,
//   5. finalises the control-point row no later element touches: sums its qx
//      half with the partner lane, then the p+1 neighbouring columns' values
//      with rotate-shuffles.
// Values a strip completes alone are stored to y; values other strips also
// touch (p-wide seams) go to a per-strip frame and are summed in a fixed order
// by seam_fixup_kernel. No atomics: bitwise reproducible.
#pragma once
#include <type_traits>
#include "iga_device.cuh"

namespace iga {

template <typename T>
struct ApplyParams {
    const T *x;
    T *y;
    const T *G;       // GEOM 0: [strip][TY][NQ][NQ][3][SW]
    const T *tabX;    // [NSX][2][QH][NB][32]  (kind 0: value, 1: d/dxi)
    const T *tabY;    // [ney][2][NQ][NBP] (NB values, zero-padded to 16-byte rows)
    const T *CP;      // GEOM 1: (x, y) per control point, in T
    const T *wq;      // GEOM 1: w_qx * w_qy, [NQ*NQ] (qx fastest)
    const T *kappa;   // GEOM 1: per quadrature point or null
    T *frame;         // [NSX*NSY][FS]
    StripGrid g;
    T sign;
    int bc;
    int *err;
    // apply_kernel's window of strip rows: gy0 .. gy0 + gyn - 1 (default: all;
    // a host-buffer MatMult applies the patch slab by slab to overlap copies)
    int gy0 = 0, gyn = 1 << 30;
    // Equation numbers (the reference's ID array, matrix_free_gpu/src/mult.cu:
    // 455-460): when set, control point A's value goes to y[ID[A]] if
    // 0 <= ID[A] < m n and nowhere otherwise (use with bc = 2: every row the
    // full element sum, x read everywhere).
    const int *ID = nullptr;
    // Polls of each wait for a G stage before it reports IGA_ERR_TIMEOUT.
    long long wait_polls = kWaitLimit;
};

// Stores sign * v for control point i = R m + C under boundary rule bc
// (0: y[boundary] = 0, 1: y[boundary] = x[boundary], 2: none) or, when ID is
// set, at equation ID[i] (skipped for ID[i] < 0 or out of range).
template <typename T>
__device__ __forceinline__ void store_point(const StripGrid &g, const T *__restrict__ x, T *__restrict__ y,
                                            const int *__restrict__ ID, T sign, int bc, int R, int C, T v)
{
    const size_t i = (size_t)R * g.m + C;
    if (ID) {
        const int e = ID[i];
        if (e >= 0 && (long long)e < (long long)g.m * g.n) y[e] = sign * v;
        return;
    }
    const bool bnd = bc != 2 && (R == 0 || C == 0 || R == g.n - 1 || C == g.m - 1);
    y[i] = bnd ? (bc == 1 ? x[i] : T(0)) : sign * v;
}

template <int P, typename T>
struct ApplyShape {
    static constexpr int NB = P + 1;
    static constexpr int NQ = P + 1;
    static constexpr int QH = (NQ + 1) / 2;
    static constexpr int NQ2 = NQ * NQ;
    static constexpr int GE = NQ2 * 3 * kSW;            // one row step of G for a warp
    static constexpr int GBYTES = GE * (int)sizeof(T);
    static constexpr int TABX = 2 * QH * NB * 32;       // x tables of a column strip
    static constexpr int XR = 8;                        // x / CP rows in flight per warp
    static constexpr int XW = 24;                       // >= SW + P, padded
    static constexpr int NBP = tab_nbp(NB, (int)sizeof(T));   // y-table row length
    static constexpr int TYW = tab_row_len(NB, NQ, (int)sizeof(T));   // one element row's y tables
    static_assert(GBYTES % 16 == 0, "bulk copy size must be a multiple of 16 bytes");
    static_assert(kSW + P <= XW, "row buffer too narrow");
};

// Stages of each warp's G ring: about 12 KiB per warp (at least 2, at most 8),
// except FP32 at p = 3, where 2 stages (6 KiB) leave room for 16 instead of
// 15 warps per SM (measured 1.13x faster at 2048^2).
template <int P, typename T>
__host__ __device__ constexpr int apply_stages()
{
    return (P == 3 && sizeof(T) == 4) ? 2 : 12288 / ApplyShape<P, T>::GBYTES < 2 ? 2
                                                 : (12288 / ApplyShape<P, T>::GBYTES > 8 ? 8 : 12288 / ApplyShape<P, T>::GBYTES);
}

// Warps that share a strip. One, except for the FP64 on-the-fly kernels of p >=
// 4, whose state (u's and both coordinates' contracted rows for every
// quadrature column of a lane, 120 doubles at p = 4) did not fit the 255
// registers a thread can have and spilled. There each of K = ceil(NQ / 2) = 3
// warps takes two quadrature columns of the strip, one per lane: a third of
// the state, and 12 instead of 8 warps per SM. The warps run independently
// but for one exchange per finished row, where warp 0 adds the others' sums,
// in order. Measured (MatMult): p=5 800^2 470 -> 240 us, 512^2 227 -> 105, p=4
// 1024^2 288 -> 266, 512^2 80 -> 74. At p = 2, 3, which do not spill, the rows'
// work that every warp repeats costs more than the warps gain (p=3 1024^2 127
// -> 142 us without a spill, p=2 94 -> 96).
template <int P, typename T, int GEOM>
__host__ __device__ constexpr int apply_split()
{
    return GEOM == 1 && sizeof(T) == 8 && P >= 4 ? (P + 2) / 2 : 1;
}

// Whether a lane keeps its x-direction tables in registers (16 values at
// p = 3) or reads them from shared memory: registers except where they are
// the scarcer resource (FP64 precomputed p >= 4, FP64 on-the-fly p <= 2). In
// registers they save 32 shared loads per element row of a p=3 FP64 strip
// (12 instead of 13 warps per SM: 1.12x faster), and the warps of a CTA need
// not share a column strip, so strips are dealt to warps one by one and every
// SM gets work. The FP64 on-the-fly kernel at p = 3 keeps them in registers
// at 8 warps per SM (254 registers, no spills; shared tables: 10 warps with
// spills): 2048^2 673 -> 536 us, 1024^2 208 -> 149 us. At p = 2 the same
// change was slower (2048^2 392 -> 435 us).
template <int P, typename T, int GEOM>
__host__ __device__ constexpr bool apply_txreg()
{
    return sizeof(T) == 4 || apply_split<P, T, GEOM>() > 1 || (GEOM == 0 ? P <= 3 : P == 3);
}

// Where the tables are not in registers they are copied to shared memory by a
// CTA whose strips lie in at most two column strips. (Read by each lane from
// global memory instead: FP64 p=4 precomputed 152.6 -> 164.8 us, p=5 249 -> 278
// us at 1024^2.)
template <int P, typename T, int GEOM>
__host__ __device__ constexpr bool apply_txshared()
{
    return !apply_txreg<P, T, GEOM>();
}

// Shared memory of a CTA of W warps: barriers, then each warp's G ring, x
// (and control-point) rows and y-table rows, then (apply_split) the strips'
// exchange slots, two rows of K - 1 warps' values, then (apply_txshared) ntab
// slots of column-strip x tables, 128-byte aligned.
template <int P, typename T, int GEOM>
__host__ __device__ constexpr size_t apply_exchange(int W)
{
    constexpr int K = apply_split<P, T, GEOM>();
    return (size_t)(W / K) * 2 * (K - 1) * 32 * sizeof(T);
}

template <int P, typename T, int GEOM, int NST>
__host__ __device__ constexpr size_t apply_tab_offset(int W)
{
    using S = ApplyShape<P, T>;
    return (((256 + (size_t)W * NST * 8 + 127) & ~size_t(127)) + (GEOM == 0 ? (size_t)W * NST * S::GBYTES : 0) +
            (size_t)W * S::XR * S::XW * sizeof(T) * (GEOM == 1 ? 3 : 1) + (size_t)W * S::XR * S::TYW * sizeof(T) +
            apply_exchange<P, T, GEOM>(W) + 127) &
           ~size_t(127);
}

template <int P, typename T, int GEOM, int NST>
__host__ __device__ constexpr size_t apply_smem_bytes(int W, int ntab = 1)
{
    return apply_tab_offset<P, T, GEOM, NST>(W) +
           (apply_txshared<P, T, GEOM>() ? (size_t)ntab * ApplyShape<P, T>::TABX * sizeof(T) : 0);
}

// The CTA's x-table slots in shared memory (apply_txshared kernels).
template <int P, typename T, int GEOM, int NST>
__device__ __forceinline__ T *apply_tab_slots()
{
    extern __shared__ __align__(128) unsigned char smem[];
    return reinterpret_cast<T *>(smem + apply_tab_offset<P, T, GEOM, NST>(blockDim.y));
}

// Copies the x tables of column strips gx0 .. gx0 + n - 1 into the slots (all
// threads of the CTA; the caller synchronises).
template <int P, typename T, int GEOM, int NST>
__device__ __forceinline__ void apply_load_tabs(const T *__restrict__ tabX, int gx0, int n, T *slots)
{
    constexpr int TABX = ApplyShape<P, T>::TABX;
    const int t = threadIdx.y * 32 + threadIdx.x, nt = 32 * blockDim.y;
    for (int k = 0; k < n; ++k) {
        const T *src = tabX + (size_t)(gx0 + k) * TABX;
        for (int i = t; i < TABX; i += nt) slots[(size_t)k * TABX + i] = src[i];
    }
}

template <typename T>
__device__ __forceinline__ T shfl_idx(T v, int src)
{
    return __shfl_sync(0xffffffffu, v, src);
}

// 1 / v for the Jacobian determinant of the on-the-fly geometry (v > 0 and
// far from the extremes of the exponent range). FP64: the hardware's
// approximate reciprocal (rcp.approx.ftz.f64) refined by two Newton-Raphson
// steps y <- y + y (1 - v y), each of which squares the relative error, so
// the result is within a few units in the last place of 1 / v; five FP64
// instructions in place of the correctly rounded reciprocal's longer
// sequence with its special-case branch. The operator is checked against
// the oracle at 1e-12 relative.
template <typename T>
__device__ __forceinline__ T recip(T v);
template <>
__device__ __forceinline__ double recip<double>(double v)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    double e = fma(-v, y, 1.0);
    y = fma(y, e, y);
    e = fma(-v, y, 1.0);
    return fma(y, e, y);
}
template <>
__device__ __forceinline__ float recip<float>(float v) { return __frcp_rn(v); }

// Threads per CTA the register budget allows (one CTA per SM): the kernel's
// per-thread state grows with p and doubles in FP64. FP64 precomputed p >= 4
// runs 8 warps without register spills (at 10 warps it spilled and ran 1.8x
// slower at p = 4), and p = 1 on the fly 16 (12: 1024^2 41 -> 37 us).
template <int P, typename T, int GEOM>
__host__ __device__ constexpr int apply_max_threads()
{
    return sizeof(T) == 4 ? (P <= 3 ? 512 : (GEOM ? 384 : 512))
           : GEOM         ? (P == 1 ? 512 : P == 3 ? 256 : 384)
                          : (P <= 2 ? 512 : P == 3 ? 384 : 256);
}

// One warp: strip (gx, gy), or its share of it (apply_split: quadrature columns
// 2 k and 2 k + 1 for warp k = threadIdx.y % K). tab_slot: the slot of the CTA's shared memory
// holding the column strip's x tables (apply_txshared), loaded by the caller.
template <int P, typename T, int GEOM, int NST>
__device__ __forceinline__ void apply_tile(const ApplyParams<T> &a, const T *__restrict__ x, T *__restrict__ y, const int gx,
                                           const int gy, const int tab_slot)
{
    using S = ApplyShape<P, T>;
    constexpr int K = apply_split<P, T, GEOM>();
    constexpr int NB = S::NB, NQ = S::NQ, QH = K > 1 ? 1 : S::QH;   // QH: quadrature columns of a lane
    constexpr bool TXREG = apply_txreg<P, T, GEOM>();
    const StripGrid &g = a.g;
    const int lane = threadIdx.x, w = threadIdx.y, W = blockDim.y;
    const int c = lane >> 1, h = lane & 1;
    const int kw = K > 1 ? w % K : 0;

    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    size_t off = 256 + (size_t)W * NST * 8;
    off = (off + 127) & ~size_t(127);
    T *Gs = reinterpret_cast<T *>(smem + off) + (size_t)w * NST * S::GE;
    if (GEOM == 0) off += (size_t)W * NST * S::GBYTES;
    T *xr = reinterpret_cast<T *>(smem + off) + (size_t)w * S::XR * S::XW;
    off += (size_t)W * S::XR * S::XW * sizeof(T);
    T *cr = reinterpret_cast<T *>(smem + off) + (size_t)w * S::XR * S::XW * 2;   // GEOM 1: CP rows (x, y)
    if (GEOM == 1) off += (size_t)W * S::XR * S::XW * 2 * sizeof(T);
    T *yr = reinterpret_cast<T *>(smem + off) + (size_t)w * S::XR * S::TYW;     // y tables of upcoming rows
    off += (size_t)W * S::XR * S::TYW * sizeof(T);
    T *xch = reinterpret_cast<T *>(smem + off) + (size_t)(w / K) * 2 * (K - 1) * 32;   // apply_split: exchange slots
    uint64_t *wbar = bars + w * NST;
    // (addressed from the shared array itself, so that the compiler emits shared loads)
    const T *tabXs = reinterpret_cast<const T *>(smem + apply_tab_offset<P, T, GEOM, NST>(W)) + (size_t)tab_slot * S::TABX;

    if (gx >= g.NSX || gy >= g.NSY) return;
    const int ex0 = kSW * gx, ey0 = g.TY * gy;
    const int nsteps = min(g.TY, g.ney - ey0);
    if (nsteps <= 0) return;
    const int ex = ex0 + c;
    const T *Gstrip = GEOM == 0 ? a.G + (size_t)(gx * g.NSY + gy) * g.TY * S::GE : nullptr;

    // The policy is held in registers, except where those two make the kernel
    // spill more (FP32 p = 5, 800^2: 86 -> 93 us): made at each use there.
    constexpr bool HOLD = !(sizeof(T) == 4 && P == 5);
    const uint64_t pol = GEOM == 0 && HOLD ? policy_once() : 0;
    auto fetch_g = [&](T *dst, const T *src, uint64_t *bar) {
        bulk_g2s(dst, src, S::GBYTES, bar, HOLD ? pol : policy_once());
    };
    if (GEOM == 0) {
        if (lane == 0) {
            for (int i = 0; i < NST; ++i) mbar_init(&wbar[i], 1);
            fence_mbar_init();
        }
        __syncwarp();
        if (lane == 0)
            for (int s = 0; s < NST && s < nsteps; ++s) {
                mbar_arrive_expect_tx(&wbar[s], S::GBYTES);
                fetch_g(Gs + (size_t)s * S::GE, Gstrip + (size_t)s * S::GE, &wbar[s]);
            }
    }

    // Control-point rows consumed in order k = 0, 1, ... (row ey0 + k); lanes
    // 0 .. SW+P-1 each fetch one column (zero outside the patch). The same
    // group brings the y tables of element row ey0 + k - P, used at step k - P.
    const int nrows = nsteps + P;
    auto fetch_row = [&](int k) {
        if (k < nrows && lane < kSW + P) {
            const int R = ey0 + k, C = ex0 + lane;
            const bool v = R < g.n && C < g.m;
            // IGA_BC_IDENTITY: boundary entries of x enter the operator as zero
            const bool xb = a.bc == 1 && (R == 0 || C == 0 || R == g.n - 1 || C == g.m - 1);
            const size_t gi = v ? (size_t)R * g.m + C : 0;
            cp_async_zfill<sizeof(T)>(xr + (k % S::XR) * S::XW + lane, x + gi, v && !xb);
            if (GEOM == 1) cp_async_zfill<2 * sizeof(T)>(cr + ((k % S::XR) * S::XW + lane) * 2, a.CP + 2 * gi, v);
        }
        if (k >= P && k < nrows) {   // 16-byte copies (rows are whole 16-byte words)
            constexpr int CH = S::TYW * (int)sizeof(T) / 16;
            const unsigned char *src = reinterpret_cast<const unsigned char *>(a.tabY + (size_t)(ey0 + k - P) * S::TYW);
            unsigned char *dst = reinterpret_cast<unsigned char *>(yr + (k % S::XR) * S::TYW);
            for (int t = lane; t < CH; t += 32) cp_async_zfill<16>(dst + 16 * t, src + 16 * t, true);
        }
        cp_async_commit();
    };
    constexpr int D = S::XR - 1;

    // This lane's x-direction tables, [kind][j][il][lane] per column strip
    // (apply_txreg: registers, loaded straight from global memory; else the
    // CTA's shared copy). The FP32 precomputed-geometry kernel at p <= 3
    // (PAIR) keeps them as (derivative, value) pairs and forms both kinds of
    // every 1-D contraction with one packed f32x2 FMA (sm_100). Measured
    // (B200, FP32, cold L2): p=2 2048^2 157 -> 146 us, p=3 181 -> 175 us; at
    // p = 4, 5 the pairs' registers spill (83 -> 97 us, 144 -> 216 us), and
    // the on-the-fly kernels were slower too (p=3 1024^2 87 -> 101 us), so
    // those keep scalar FMAs (reading paired y tables up to p = 4: on-the-fly
    // p=3 1024^2 87 -> 85 us, p=2 62.4 -> 60.4 us).
    constexpr bool TPAIR = tab_paired(NB, (int)sizeof(T));
    constexpr bool PAIR = TPAIR && GEOM == 0 && P <= 3;
    static_assert(!PAIR || TXREG, "FP32 x tables live in registers");
    T txr[TXREG && !PAIR ? 2 : 1][TXREG && !PAIR ? QH : 1][TXREG && !PAIR ? NB : 1];
    float2 tpr[PAIR ? QH : 1][PAIR ? NB : 1];
    if constexpr (PAIR) {
        const T *src = a.tabX + (size_t)gx * S::TABX;
#pragma unroll
        for (int j = 0; j < QH; ++j)
#pragma unroll
            for (int il = 0; il < NB; ++il)
                tpr[j][il] = make_float2(src[((QH + j) * NB + il) * 32 + lane], src[(j * NB + il) * 32 + lane]);
    } else if constexpr (K > 1) {
        // entry of quadrature column qx in the one-warp layout (lane_qx): its
        // lane half and slot there
        constexpr int Q0 = S::QH;
        const int qx = 2 * kw + h;
        const bool mid = mid_shared(NQ, (int)sizeof(T)) && qx == Q0 - 1;
        const int h0 = mid ? 0 : qx / Q0, j0 = mid ? Q0 - 1 : qx - h0 * Q0;
        const T *src = a.tabX + (size_t)gx * S::TABX + 2 * c + h0;
#pragma unroll
        for (int kind = 0; kind < 2; ++kind)
#pragma unroll
            for (int il = 0; il < NB; ++il) txr[kind][0][il] = qx < NQ ? src[((kind * Q0 + j0) * NB + il) * 32] : T(0);
    } else if constexpr (TXREG) {
        const T *src = a.tabX + (size_t)gx * S::TABX;
#pragma unroll
        for (int kind = 0; kind < 2; ++kind)
#pragma unroll
            for (int j = 0; j < QH; ++j)
#pragma unroll
                for (int il = 0; il < NB; ++il) txr[kind][j][il] = src[((kind * QH + j) * NB + il) * 32 + lane];
    }
    auto tx = [&](int kind, int j, int il) -> T {
        if constexpr (PAIR) return kind ? tpr[j][il].x : tpr[j][il].y;
        else if constexpr (TXREG) return txr[kind][j][il];
        else return tabXs[((kind * QH + j) * NB + il) * 32 + lane];
    };
    // Everything above reads only the plan's constant tables and geometry;
    // x (an earlier grid's output) and every write come after the wait.
    pdl_wait();
    for (int k = 0; k < D; ++k) fetch_row(k);

    constexpr int NR = PAIR ? 1 : NB;
    T xs0[NR][QH], xs1[NR][QH];     // x contracted with value / derivative tables, rows ey..ey+P
    T acc0[NR][QH], acc1[NR][QH];   // y-transposed partial sums for control-point rows ey..ey+P
    T cs[2][2][GEOM == 1 && !PAIR ? NB : 1][QH];   // GEOM 1: CP coordinates contracted likewise
    // PAIR: X = (xs1, xs0), A = (acc0, acc1), CX = (cs[0][1], cs[0][0]), CY = (cs[1][1], cs[1][0])
    float2 X[PAIR ? NB : 1][QH], A[PAIR ? NB : 1][QH];
    float2 CX[PAIR && GEOM == 1 ? NB : 1][QH], CY[PAIR && GEOM == 1 ? NB : 1][QH];

    // x contraction of control-point row k into state row `slot` (0 .. P)
    auto contract_row = [&](int k, int slot) {
        cp_async_wait<D - 1>();
        __syncwarp();
        const T *src = xr + (k % S::XR) * S::XW;
        T xv[NB];
#pragma unroll
        for (int il = 0; il < NB; ++il) xv[il] = src[c + il];
        T px[NB], py[NB];
        if constexpr (GEOM == 1) {
            const T *cp = cr + (k % S::XR) * S::XW * 2;
#pragma unroll
            for (int il = 0; il < NB; ++il) {
                px[il] = cp[2 * (c + il)];
                py[il] = cp[2 * (c + il) + 1];
            }
        }
        __syncwarp();
        fetch_row(k + D);
        if constexpr (PAIR) {
#pragma unroll
            for (int j = 0; j < QH; ++j) {
                float2 s2 = __fmul2_rn(tpr[j][0], make_float2(xv[0], xv[0]));
#pragma unroll
                for (int il = 1; il < NB; ++il) s2 = __ffma2_rn(tpr[j][il], make_float2(xv[il], xv[il]), s2);
                X[slot][j] = s2;
            }
            if constexpr (GEOM == 1) {
#pragma unroll
                for (int j = 0; j < QH; ++j) {
                    float2 ax = __fmul2_rn(tpr[j][0], make_float2(px[0], px[0]));
                    float2 ay = __fmul2_rn(tpr[j][0], make_float2(py[0], py[0]));
#pragma unroll
                    for (int il = 1; il < NB; ++il) {
                        ax = __ffma2_rn(tpr[j][il], make_float2(px[il], px[il]), ax);
                        ay = __ffma2_rn(tpr[j][il], make_float2(py[il], py[il]), ay);
                    }
                    CX[slot][j] = ax;
                    CY[slot][j] = ay;
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < QH; ++j) {
                T s0 = 0, s1 = 0;
#pragma unroll
                for (int il = 0; il < NB; ++il) {
                    s0 = fma(tx(0, j, il), xv[il], s0);
                    s1 = fma(tx(1, j, il), xv[il], s1);
                }
                xs0[slot][j] = s0;
                xs1[slot][j] = s1;
            }
            if constexpr (GEOM == 1) {
#pragma unroll
                for (int j = 0; j < QH; ++j) {
                    T a0 = 0, a1 = 0, b0 = 0, b1 = 0;
#pragma unroll
                    for (int il = 0; il < NB; ++il) {
                        a0 = fma(tx(0, j, il), px[il], a0);
                        a1 = fma(tx(1, j, il), px[il], a1);
                        b0 = fma(tx(0, j, il), py[il], b0);
                        b1 = fma(tx(1, j, il), py[il], b1);
                    }
                    cs[0][0][slot][j] = a0;
                    cs[0][1][slot][j] = a1;
                    cs[1][0][slot][j] = b0;
                    cs[1][1][slot][j] = b1;
                }
            }
        }
    };

    auto store = [&](int R, int C, T v) { store_point<T>(g, x, y, a.ID, a.sign, a.bc, R, C, v); };
    T *frame = a.frame + (size_t)(gx * g.NSY + gy) * g.FS;
    // finishes control-point row ey0 + lr from state row 0 of the partial sums
    auto write_row = [&](int lr) {
        T out[NB];
#pragma unroll
        for (int il = 0; il < NB; ++il) {
            T s = 0;
            if constexpr (PAIR) {   // the derivative-table and value-table sums, then their total
                float2 s2 = __fmul2_rn(tpr[0][il], A[0][0]);
#pragma unroll
                for (int j = 1; j < QH; ++j) s2 = __ffma2_rn(tpr[j][il], A[0][j], s2);
                s = s2.x + s2.y;
            } else {
#pragma unroll
                for (int j = 0; j < QH; ++j) {
                    s = fma(tx(1, j, il), acc0[0][j], s);
                    s = fma(tx(0, j, il), acc1[0][j], s);
                }
            }
            out[il] = s + __shfl_xor_sync(0xffffffffu, s, 1);   // both qx halves, same order on both lanes
        }
        // Column c collects out[il] from column c-il (lane - 2 il); lanes of
        // columns c < il receive the wrapped value, which belongs to column SW+c.
        T tot = out[0], spill = 0;
#pragma unroll
        for (int il = 1; il < NB; ++il) {
            const T v = shfl_idx(out[il], (lane - 2 * il) & 31);
            if (c >= il) tot += v;
            else spill += v;
        }
        // Always inside the patch (ey0 + nsteps + P <= n), but the exit changes
        // how the stores below are scheduled: with it p=5 precomputed FP64 141 ->
        // 138 us at 800^2, on-the-fly p=2 75.0 -> 73.9; without it on-the-fly
        // FP64 p=3 377 -> 371, p=4 213 -> 207.
        const int R = ey0 + lr;
        if constexpr (!(GEOM == 1 && sizeof(T) == 8 && P >= 3))
            if (R >= g.n) return;
        // Strips covering row R / column C: the
        // first P rows/columns of a strip are shared with the strip before
        // it (if any), the P rows/columns past its end with the one after it.
        const bool row_single = lr < g.TY ? (lr >= P || gy == 0) : (gy + 1 >= g.NSY);
        const int lc = h ? kSW + c : c;
        const int C = ex0 + lc;
        T v = h ? spill : tot;
        if constexpr (K > 1) {   // the other warps' shares, in order (two slots: row lr + 1 may be on its way)
            T *x0 = xch + (lr & 1) * (K - 1) * 32 + lane;
            if (kw > 0) x0[(kw - 1) * 32] = v;
            asm volatile("bar.sync %0, %1;" ::"r"(1 + w / K), "n"(32 * K) : "memory");
            if (kw > 0) return;
#pragma unroll
            for (int k = 0; k < K - 1; ++k) v += x0[k * 32];
        }
        if ((h == 0 || c < P) && C < g.m) {
            const bool col_single = h ? (gx + 1 >= g.NSX) : (c >= P || gx == 0);
            if (row_single && col_single) store(R, C, v);
            else frame[frame_index(lr, lc, P, g.TY)] = v;
        }
    };

    // Prologue: rows ey0 .. ey0+P-1.
#pragma unroll
    for (int r = 0; r < P; ++r) contract_row(r, r);
#pragma unroll
    for (int r = 0; r < NB; ++r)
#pragma unroll
        for (int q = 0; q < QH; ++q) {
            if constexpr (PAIR) A[r][q] = make_float2(0.f, 0.f);
            else acc0[r][q] = acc1[r][q] = 0;
        }
    // state rows r+1 -> r (the next element row); the partial sums of row P restart
    auto shift_rows = [&](bool inputs) {
#pragma unroll
        for (int r = 0; r < P; ++r)
#pragma unroll
            for (int q = 0; q < QH; ++q) {
                if constexpr (PAIR) {
                    A[r][q] = A[r + 1][q];
                    if (inputs) {
                        X[r][q] = X[r + 1][q];
                        if constexpr (GEOM == 1) {
                            CX[r][q] = CX[r + 1][q];
                            CY[r][q] = CY[r + 1][q];
                        }
                    }
                } else {
                    acc0[r][q] = acc0[r + 1][q];
                    acc1[r][q] = acc1[r + 1][q];
                    if (inputs) {
                        xs0[r][q] = xs0[r + 1][q];
                        xs1[r][q] = xs1[r + 1][q];
                        if constexpr (GEOM == 1) {
                            cs[0][0][r][q] = cs[0][0][r + 1][q];
                            cs[0][1][r][q] = cs[0][1][r + 1][q];
                            cs[1][0][r][q] = cs[1][0][r + 1][q];
                            cs[1][1][r][q] = cs[1][1][r + 1][q];
                        }
                    }
                }
            }
#pragma unroll
        for (int q = 0; q < QH; ++q) {
            if constexpr (PAIR) A[P][q] = make_float2(0.f, 0.f);
            else acc0[P][q] = acc1[P][q] = 0;
        }
    };

    bool ok = true;
    int failed_step = 0;
    for (int s = 0; s < nsteps; ++s) {
        const int ey = ey0 + s;
        contract_row(s + P, P);
        const int slot = s % NST;
        const T *Gst = Gs + (size_t)slot * S::GE;
        if (GEOM == 0) {
            if (!mbar_wait_bounded(&wbar[slot], (uint32_t)((s / NST) & 1), a.wait_polls)) {
                ok = false;
                failed_step = s;
                break;
            }
        }
        const T *ty = yr + ((s + P) % S::XR) * S::TYW;   // landed with x row s + P
        constexpr bool MID = K == 1 && mid_shared(NQ, (int)sizeof(T));
        constexpr int QJ = MID ? QH - 1 : QH;   // slots of this lane half's own columns
        // y tables of quadrature row qy: value n2 and derivative d2, or their
        // pairs nd (PAIR)
        struct YRow {
            T n2[PAIR ? 1 : NB], d2[PAIR ? 1 : NB];
            float2 nd[PAIR ? NB : 1];
        };
        auto load_tab = [&](int qy, YRow &t) {
            if constexpr (PAIR) {   // rows of NB pairs padded to 16 bytes: two pairs per vector load
                const float4 *v = reinterpret_cast<const float4 *>(ty + qy * tab_nbp2(NB));
#pragma unroll
                for (int u = 0; 2 * u < NB; ++u) {
                    const float4 q = v[u];
                    t.nd[2 * u] = make_float2(q.x, q.y);
                    if (2 * u + 1 < NB) t.nd[2 * u + 1] = make_float2(q.z, q.w);
                }
            } else if constexpr (TPAIR) {   // the same rows, split into the two kinds
                const float4 *v = reinterpret_cast<const float4 *>(ty + qy * tab_nbp2(NB));
#pragma unroll
                for (int u = 0; 2 * u < NB; ++u) {
                    const float4 q = v[u];
                    t.n2[2 * u] = q.x;
                    t.d2[2 * u] = q.y;
                    if (2 * u + 1 < NB) {
                        t.n2[2 * u + 1] = q.z;
                        t.d2[2 * u + 1] = q.w;
                    }
                }
            } else {
                // rows of NBP entries, 16-byte aligned in the ring: vector loads
                constexpr int V = 16 / sizeof(T), NBP = S::NBP;
                using VT = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
                const VT *va = reinterpret_cast<const VT *>(ty + qy * NBP);
                const VT *vb = reinterpret_cast<const VT *>(ty + (NQ + qy) * NBP);
#pragma unroll
                for (int v = 0; v < NBP / V; ++v) {
                    const VT ua = va[v], ub = vb[v];
                    const T *pa = reinterpret_cast<const T *>(&ua), *pb = reinterpret_cast<const T *>(&ub);
#pragma unroll
                    for (int e = 0; e < V; ++e) {
                        if (v * V + e < NB) {
                            t.n2[v * V + e] = pa[e];
                            t.d2[v * V + e] = pb[e];
                        }
                    }
                }
            }
        };
        // quadrature point (qy, qx) in slot j: gradient of u, times G, back
        // onto the slot's y-transposed partial sums (valid false: adds zero)
        // gv: this lane's G values of row qy (lane-major G), else read here
        auto qpoint = [&](int qy, int qx, int j, bool valid, const YRow &t, const T *gv) {
            T uxi = 0, ueta = 0;
            if constexpr (PAIR) {   // (n2 . xs1, d2 . xs0) together
                float2 u2 = __fmul2_rn(t.nd[0], X[0][j]);
#pragma unroll
                for (int jl = 1; jl < NB; ++jl) u2 = __ffma2_rn(t.nd[jl], X[jl][j], u2);
                uxi = u2.x;
                ueta = u2.y;
            } else {
#pragma unroll
                for (int jl = 0; jl < NB; ++jl) {
                    uxi = fma(t.n2[jl], xs1[jl][j], uxi);
                    ueta = fma(t.d2[jl], xs0[jl][j], ueta);
                }
            }
            T g00 = 0, g01 = 0, g11 = 0;
            T vxi, veta;
            if constexpr (GEOM == 0) {
                if constexpr (g_lane_major(NQ)) {
                    g00 = gv[3 * j];
                    g01 = gv[3 * j + 1];
                    g11 = gv[3 * j + 2];
                } else if constexpr (g_mid_lane_major(NQ, (int)sizeof(T))) {
                    if (j + 1 < QH) {   // a column of this lane half
                        g00 = gv[3 * j];
                        g01 = gv[3 * j + 1];
                        g11 = gv[3 * j + 2];
                    } else if (valid) {   // the middle column, row qy of this half
                        const T *gp = Gst + qy * (NQ * 3 * kSW) + 32 * (QH - 1) * 3 + c * 3;
                        g00 = gp[0];
                        g01 = gp[1];
                        g11 = gp[2];
                    }
                } else if (valid) {
                    const T *gp = Gst + ((qy * NQ + qx) * 3) * kSW + c;
                    g00 = gp[0];
                    g01 = gp[kSW];
                    g11 = gp[2 * kSW];
                }
            } else {
                T x_xi = 0, x_eta = 0, y_xi = 0, y_eta = 0;
                if constexpr (PAIR) {
                    float2 cx = __fmul2_rn(t.nd[0], CX[0][j]), cy = __fmul2_rn(t.nd[0], CY[0][j]);
#pragma unroll
                    for (int jl = 1; jl < NB; ++jl) {
                        cx = __ffma2_rn(t.nd[jl], CX[jl][j], cx);
                        cy = __ffma2_rn(t.nd[jl], CY[jl][j], cy);
                    }
                    x_xi = cx.x;
                    x_eta = cx.y;
                    y_xi = cy.x;
                    y_eta = cy.y;
                } else {
#pragma unroll
                    for (int jl = 0; jl < NB; ++jl) {
                        x_xi = fma(t.n2[jl], cs[0][1][jl][j], x_xi);
                        x_eta = fma(t.d2[jl], cs[0][0][jl][j], x_eta);
                        y_xi = fma(t.n2[jl], cs[1][1][jl][j], y_xi);
                        y_eta = fma(t.d2[jl], cs[1][0][jl][j], y_eta);
                    }
                }
                // G grad u = f adj(J) adj(J)^T grad u with adj(J) = [[y_eta,
                // -x_eta], [-y_xi, x_xi]] and f = w kappa / det J: ten
                // operations instead of forming G's three entries (thirteen)
                vxi = veta = 0;
                if (valid && ex < g.nex) {
                    T wgt = a.wq[qy * NQ + qx];
                    if (a.kappa) wgt *= a.kappa[((size_t)ey * g.nex + ex) * S::NQ2 + qy * NQ + qx];
                    const T f = wgt * recip(x_xi * y_eta - x_eta * y_xi);
                    const T t0 = f * fma(y_eta, uxi, -(y_xi * ueta));
                    const T t1 = f * fma(x_xi, ueta, -(x_eta * uxi));
                    vxi = fma(y_eta, t0, -(x_eta * t1));
                    veta = fma(x_xi, t1, -(y_xi * t0));
                }
            }
            if constexpr (GEOM == 0) {
                vxi = fma(g00, uxi, g01 * ueta);
                veta = fma(g01, uxi, g11 * ueta);
            }
            if constexpr (PAIR) {   // (acc0 += n2 vxi, acc1 += d2 veta) together
                const float2 v2 = make_float2(vxi, veta);
#pragma unroll
                for (int jl = 0; jl < NB; ++jl) A[jl][j] = __ffma2_rn(t.nd[jl], v2, A[jl][j]);
            } else {
#pragma unroll
                for (int jl = 0; jl < NB; ++jl) {
                    acc0[jl][j] = fma(t.n2[jl], vxi, acc0[jl][j]);
                    acc1[jl][j] = fma(t.d2[jl], veta, acc1[jl][j]);
                }
            }
        };

#pragma unroll
        for (int qy = 0; qy < NQ; ++qy) {
            YRow t;
            load_tab(qy, t);
            // this lane's G values of row qy for its own columns: 3 QJ contiguous
            // values (lane-major G rows), widest aligned loads
            constexpr int GVN = (g_lane_major(NQ) || g_mid_lane_major(NQ, (int)sizeof(T))) ? 3 * QJ : 1;
            T gv[GVN];
            if constexpr (GEOM == 0 && GVN > 1) {
                const T *src = Gst + (size_t)qy * (NQ * 3 * kSW) + (size_t)lane * GVN;
                constexpr int BYTES = GVN * (int)sizeof(T);
                constexpr int VB = BYTES % 16 == 0 ? 16 : BYTES % 8 == 0 ? 8 : (int)sizeof(T);
                using VT = typename std::conditional<VB == 16, float4, typename std::conditional<VB == 8, float2, T>::type>::type;
#pragma unroll
                for (int v = 0; v < BYTES / VB; ++v) {
                    const VT u = reinterpret_cast<const VT *>(src)[v];
                    const T *pu = reinterpret_cast<const T *>(&u);
#pragma unroll
                    for (int e = 0; e < VB / (int)sizeof(T); ++e) gv[v * (VB / (int)sizeof(T)) + e] = pu[e];
                }
            }
#pragma unroll
            for (int j = 0; j < QJ; ++j) {
                // only the last column can lie past NQ (h = 1's last slot, the last warp's h = 1)
                const int qx = K > 1 ? 2 * kw + h : h * QH + j;
                qpoint(qy, qx, j, NQ % 2 == 0 || (K == 1 && j + 1 < QH) || qx < NQ, t, gv);
            }
        }
        if constexpr (MID) {   // middle column QH - 1: half h takes rows qy = 2 t + h
#pragma unroll
            for (int tq = 0; tq < QH; ++tq) {
                const int qy = min(2 * tq + h, NQ - 1);
                YRow t;
                load_tab(qy, t);
                qpoint(qy, QH - 1, QH - 1, 2 * tq + h < NQ, t, nullptr);
            }
        }
        if (GEOM == 0) {
            __syncwarp();
            if (lane == 0 && s + NST < nsteps) {
                fence_proxy_async_smem();
                mbar_arrive_expect_tx(&wbar[slot], S::GBYTES);
                fetch_g(Gs + (size_t)slot * S::GE, Gstrip + (size_t)(s + NST) * S::GE, &wbar[slot]);
            }
        }
        write_row(s);
        shift_rows(true);
    }
    if (!ok) {
        if (lane == 0) atomicExch(a.err, 8 /* IGA_ERR_TIMEOUT */);
        // Let the copies already issued (steps failed_step .. failed_step+NST-1)
        // land before the CTA's shared memory is released; bounded as well,
        // always with the full poll limit.
        for (int t = failed_step; t < nsteps && t < failed_step + NST; ++t)
            mbar_wait_bounded(&wbar[t % NST], (uint32_t)((t / NST) & 1));
        cp_async_wait<0>();
        return;
    }
    // Rows above the last element row: partial sums for rows ey_last+1 .. ey_last+P.
#pragma unroll
    for (int r = 0; r < P; ++r) {
        write_row(nsteps + r);
        shift_rows(false);
    }
    cp_async_wait<0>();
}

// Strips to warps: warp k (apply_split: K warps) of the 1-D grid takes strip k in column-major
// order (gx outer), so the grid covers NSX * rows strips with no partly idle
// CTAs and the strip height can make the strip count fill the SMs. With the
// tables in shared memory (apply_txshared) the CTA copies the tables of the
// column strips its warps' strips lie in: two slots, as the launch keeps W - 1
// <= rows. (One CTA per column strip, W strips of it each, left 20 of 148
// SMs idle for the FP64 p=4 operator on a 1024-wide patch: 64 columns.)
template <int P, typename T, int GEOM, int NST>
__global__ void __launch_bounds__(apply_max_threads<P, T, GEOM>(), 1) apply_kernel(ApplyParams<T> a)
{
    pdl_launch();   // apply_tile waits for the preceding grid once its constant operands are in flight
    const int rows = min(a.gyn, a.g.NSY - a.gy0);   // strip rows of the window
    constexpr int K = apply_split<P, T, GEOM>();
    const int s0 = blockIdx.x * (blockDim.y / K), sid = s0 + threadIdx.y / K;   // strips: NSX * NSY < 2^31
    const int gx = sid / rows;
    int slot = 0;
    if constexpr (apply_txshared<P, T, GEOM>()) {
        const int total = a.g.NSX * rows;
        const int gx_lo = s0 / rows, gx_hi = (min(s0 + (int)blockDim.y, total) - 1) / rows;
        apply_load_tabs<P, T, GEOM, NST>(a.tabX, gx_lo, gx_hi - gx_lo + 1, apply_tab_slots<P, T, GEOM, NST>());
        __syncthreads();
        if (sid >= total) return;
        slot = gx - gx_lo;
    }
    apply_tile<P, T, GEOM, NST>(a, a.x, a.y, gx, a.gy0 + (sid - gx * rows), slot);
}

// Many independent patches in one launch, with that problem's parameters
// per work item, or nothing when the problem is marked inactive (converged)
// or the item is padding (problem -1). Tables in registers (apply_txreg):
// warp k of the grid runs strip items[k] = (problem, column strip, strip
// row), so the warps of a CTA may take strips of different problems and
// columns; else CTA b runs items[b] = (problem, column strip, block of W
// strips of that column).
template <int P, typename T, int NST>
__global__ void __launch_bounds__(apply_max_threads<P, T, 0>(), 1)
    apply_batch_kernel(const ApplyParams<T> *__restrict__ params, const int4 *__restrict__ items,
                       const int *__restrict__ active, const long long *__restrict__ offs, const T *__restrict__ xb,
                       T *__restrict__ yb)
{
    constexpr bool flat = !apply_txshared<P, T, 0>();
    const int4 it = items[flat ? blockIdx.x * blockDim.y + threadIdx.y : blockIdx.x];
    if (it.x < 0 || !active[it.x]) return;   // uniform over the CTA unless flat (no CTA barrier then)
    const long long o = offs[it.x];
    if constexpr (!flat) {   // the item's column strip, slot 0
        apply_load_tabs<P, T, 0, NST>(params[it.x].tabX, it.y, 1, apply_tab_slots<P, T, 0, NST>());
        __syncthreads();
    }
    // The item's parameters where stores to y cannot make the compiler fetch
    // them from global memory again at every element row: in FP32 registers
    // (256 problems of p = 2, 3: 285 -> 243 us; in shared memory 288), in FP64
    // and at p >= 4, whose registers are full, shared memory (FP64 403 -> 367;
    // in registers 385).
    const int gy = flat ? it.z : it.z * blockDim.y + threadIdx.y;
    if constexpr (sizeof(T) == 4 && P <= 3) {
        const ApplyParams<T> a = params[it.x];
        apply_tile<P, T, 0, NST>(a, xb + o, yb + o, it.y, gy, 0);
    } else {
        constexpr int NI = (int)sizeof(ApplyParams<T>) / 8;
        static_assert(sizeof(ApplyParams<T>) % 8 == 0, "copied in 8-byte words");
        __shared__ long long sp[apply_max_threads<P, T, 0>() / 32][NI];
        const long long *src = reinterpret_cast<const long long *>(params + it.x);
        for (int i = threadIdx.x; i < NI; i += 32) sp[threadIdx.y][i] = src[i];
        __syncwarp();
        apply_tile<P, T, 0, NST>(*reinterpret_cast<const ApplyParams<T> *>(sp[threadIdx.y]), xb + o, yb + o, it.y, gy, 0);
    }
}

// ------------------------------------------------------------ seams
// Sums the frames of the strips covering each seam control point, strip
// (row, then column) in ascending order, and stores sign * sum (boundary
// rules as in apply_kernel: bc 0 zero, 1 identity, 2 none).
//
// Work comes in blocks of kSeamBlock points of one seam: block k of the
// vertical seams (columns kSW c .. kSW c + P - 1, every row, the P columns
// fastest), then of the horizontal ones (rows TY s .. TY s + P - 1 outside
// those columns). So a thread finds its seam with one 32-bit division per
// block index and its strips without searching: a vertical seam's column
// strips are always c - 1 and c, a horizontal one's row strips s - 1 and s.
// Bound: the frames' L2 reads and the partial-sector writes of y; before, the
// 64-bit divisions and strip searches of a flat point index (p=3 2048^2 FP64
// 15.0 -> 11.5 us, FP32 12.9 -> 9.4 us; batch of 256 problems FP64 42.8 -> 33.4
// us, FP32 34.4 -> 30.3 us).
constexpr int kSeamBlock = 256;

// The seam blocks of control-point rows R0 .. R1 - 1 (vertical seams) and of
// the horizontal seams s0 .. s1 - 1.
struct SeamRange {
    int R0, R1, s0, s1, bv, bh, nv, total;
};

__host__ __device__ __forceinline__ SeamRange seam_range(const StripGrid &g, int R0, int R1)
{
    SeamRange r;
    r.R0 = R0;
    r.R1 = R1;
    r.s0 = R0 / g.TY > 1 ? R0 / g.TY : 1;
    const int s1 = (R1 + g.TY - 1) / g.TY;
    r.s1 = s1 < g.NSY ? s1 : g.NSY;
    r.bv = ((R1 - R0) * g.P + kSeamBlock - 1) / kSeamBlock;
    r.bh = (g.P * g.m + kSeamBlock - 1) / kSeamBlock;
    r.nv = (g.NSX - 1) * r.bv;
    r.total = r.nv + (r.s1 > r.s0 ? r.s1 - r.s0 : 0) * r.bh;
    return r;
}

__host__ __device__ __forceinline__ SeamRange seam_range(const StripGrid &g) { return seam_range(g, 0, g.n); }

template <int P, typename T>
__device__ __forceinline__ void seam_block(const T *__restrict__ frame, const T *__restrict__ x, T *__restrict__ y,
                                           const StripGrid &g, T sign, int bc, const int *__restrict__ ID,
                                           const SeamRange &r, int k)
{
    const int TY = g.TY;
    T v = 0;
    int R, C;
    if (k < r.nv) {
        const int c = k / r.bv, u = (k - c * r.bv) * kSeamBlock + threadIdx.x;   // seam of column strips c, c + 1
        if (u >= (r.R1 - r.R0) * P) return;
        R = r.R0 + u / P;
        const int lc = u % P;
        C = kSW * (c + 1) + lc;
        if (C >= g.m) return;
        const int b = R / TY, lr = R - b * TY;
        const T *f0 = frame + (size_t)(c * g.NSY) * g.FS + P * (TY + P) + lc;   // right edge of strip column c
        const T *f1 = frame + (size_t)((c + 1) * g.NSY) * g.FS + lc;            // left edge of strip column c + 1
        if (lr < P && b >= 1) {
            const size_t o = (size_t)(b - 1) * g.FS + (lr + TY) * P;
            v += f0[o];
            v += f1[o];
        }
        if (b < g.NSY) {
            const size_t o = (size_t)b * g.FS + lr * P;
            v += f0[o];
            v += f1[o];
        }
    } else {
        const int h = (k - r.nv) / r.bh, u = (k - r.nv - h * r.bh) * kSeamBlock + threadIdx.x;
        if (u >= P * g.m) return;
        const int lr = u / g.m, b = r.s0 + h;
        C = u - lr * g.m;
        R = b * TY + lr;
        if (R >= r.R1 || R >= g.n) return;
        const int s = C / kSW;
        if (C % kSW < P && s >= 1 && s < g.NSX) return;   // a vertical seam's point
        const int a = min(s, g.NSX - 1), lc = C - kSW * a;
        const T *f = frame + (size_t)(a * g.NSY + b - 1) * g.FS;
        v += f[frame_index(lr + TY, lc, P, TY)];
        v += f[g.FS + frame_index(lr, lc, P, TY)];
    }
    store_point<T>(g, x, y, ID, sign, bc, R, C, v);
}

// The seams of control-point rows R0 .. R1 - 1, where R0 = TY * s0 is a
// strip-row boundary. Valid once every strip covering those rows has written
// its frame. One block of points per CTA.
template <int P, typename T>
__global__ void __launch_bounds__(kSeamBlock) seam_fixup_kernel(const T *__restrict__ frame, const T *__restrict__ x,
                                                                T *__restrict__ y, StripGrid g, T sign, int bc,
                                                                int R0, int R1, const int *__restrict__ ID)
{
    pdl_begin();
    const SeamRange r = seam_range(g, R0, R1);
    seam_block<P, T>(frame, x, y, g, sign, bc, ID, r, blockIdx.x);
}

template <int P, typename T>
__device__ __forceinline__ void seam_loop(const ApplyParams<T> &a, const T *__restrict__ x, T *__restrict__ y)
{
    const SeamRange r = seam_range(a.g);
    for (int k = blockIdx.x; k < r.total; k += gridDim.x) seam_block<P, T>(a.frame, x, y, a.g, a.sign, a.bc, a.ID, r, k);
}

// Seams of every active problem of a batch: blockIdx.y = problem.
template <typename T>
__global__ void __launch_bounds__(kSeamBlock) seam_fixup_batch_kernel(const ApplyParams<T> *__restrict__ params,
                                                                      const int *__restrict__ active,
                                                                      const long long *__restrict__ offs,
                                                                      const T *__restrict__ xb, T *__restrict__ yb)
{
    const int pr = blockIdx.y;
    if (!active[pr]) return;
    const ApplyParams<T> a = params[pr];   // a copy: see apply_batch_kernel
    const long long o = offs[pr];
    switch (a.g.P) {
    case 1: seam_loop<1, T>(a, xb + o, yb + o); break;
    case 2: seam_loop<2, T>(a, xb + o, yb + o); break;
    case 3: seam_loop<3, T>(a, xb + o, yb + o); break;
    case 4: seam_loop<4, T>(a, xb + o, yb + o); break;
    default: seam_loop<5, T>(a, xb + o, yb + o); break;
    }
}

}  // namespace iga
