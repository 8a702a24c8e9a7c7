// Device-side building blocks shared by the IGA kernels: PTX wrappers for the
// bulk-copy engine (TMA, cp.async.bulk) with mbarrier completion, Ampere-style
// cp.async for small ragged rows, bounded waits, and strip geometry.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include <utility>

namespace iga {

// ---------------------------------------------------------------- dependent launches
// Kernels that run inside the solver's captured loop start with pdl_begin():
// griddepcontrol.wait blocks until the preceding grid has completed and its
// memory is visible (a no-op when the kernel was launched without a
// programmatic dependency), then launch_dependents lets the next grid be
// scheduled while this one runs. A kernel whose CTAs all passed pdl_begin()
// can therefore have its successor's CTAs resident and waiting, which hides
// the launch gap between graph nodes.
__device__ __forceinline__ void pdl_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The two halves of pdl_begin() for kernels that first fetch operands no
// earlier grid writes (tables, geometry, eigenvectors) and set up shared
// memory and tensor memory while the preceding grid drains: pdl_launch() at
// the start, pdl_wait() before the first read of data an earlier grid
// produced and before the first global write. pdl_wait() is per thread.
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Host side: while pdl_capture() is true on this thread (the solver's loop
// capture), launch_k() launches with a programmatic stream serialisation
// attribute, so that stream capture records programmatic edges; otherwise
// it is an ordinary launch. Only kernels that begin with pdl_begin() may be
// launched through it.
inline bool &pdl_capture()
{
    static thread_local bool on = false;
    return on;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                            Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (pdl_capture()) {
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// SMs of the current device.
inline int device_sms()
{
    int nsm = 148, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        nsm = 148;
    return nsm;
}

// launch_k() with an ordinary edge for grids of more than `most` CTAs: as
// programmatic dependents their CTAs start where the preceding grid's leave
// first, and those SMs fill up while others stay empty.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_upto(long long most, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                               Args &&...args)
{
    const bool was = pdl_capture();
    if ((long long)grid.x * grid.y * grid.z > most) pdl_capture() = false;
    const cudaError_t e = launch_k(kern, grid, block, smem, s, std::forward<Args>(args)...);
    pdl_capture() = was;
    return e;
}

// The line for the solver's other kernels, at one CTA an SM: bound by latency
// or bandwidth, they lose less to an uneven start than the launch gap is worth
// (TF32 GEMMs at 1024^2: 37.6 us as dependents, 42.2 with ordinary edges; the
// operator in an FP64 PCG iteration p=2 256^2 33.2 against 33.9, p=3 512^2, 147
// CTAs, 67.3 against 67.7).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_even(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                               Args &&...args)
{
    return launch_upto(pdl_capture() ? device_sms() : 0, kern, grid, block, smem, s, std::forward<Args>(args)...);
}

// Launches a kernel that follows this call's own preceding kernel on s and
// begins with pdl_begin(): as a programmatic dependent, so that its CTAs are
// set up while that one drains (with the seams' own change: MatMult p=2 64^2
// 10.2 -> 8.2 us, p=3 1024^2 86.6 -> 83.7 us, 2048^2 297.5 -> 292.3 us, where the
// ordinary edge gives 295.1). Outside the solver's capture only on streams
// that are not being captured: a caller's graph keeps ordinary edges.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_after(void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args &&...args)
{
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    const bool was = pdl_capture();
    if (!was) {
        if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
            (void)cudaGetLastError();
            st = cudaStreamCaptureStatusActive;
        }
        pdl_capture() = st == cudaStreamCaptureStatusNone;
    }
    const cudaError_t e = launch_k(kern, grid, block, 0, s, std::forward<Args>(args)...);
    pdl_capture() = was;
    return e;
}

// Upper bound on mbarrier polls before a wait gives up and reports
// IGA_ERR_TIMEOUT; each try_wait suspends for a hardware-defined interval, so
// this is seconds of wall time, far beyond any legitimate copy latency.
constexpr long long kWaitLimit = 1LL << 24;

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// 1-D bulk copy global -> shared through the async (TMA) proxy; completion is
// signalled on *bar as transaction bytes. dst, src 16-byte aligned, bytes % 16 == 0.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// The same with an L2 policy. policy_once() is for data one kernel reads once
// (a strip's geometry): its lines are the first to be replaced, so that a
// geometry larger than L2 does not push out the vectors the next kernels read,
// and one about as large as L2 keeps some of itself (an LRU of a cyclic stream
// keeps nothing). Measured: FP64 PCG an iteration, p=3 700^2 185 -> 172 us, 1024^2
// 225 -> 212, 1600^2 596 -> 573, 2048^2 1063 -> 1050, p=4 1024^2 287 -> 277; MatMult
// FP64 p=3 1024^2 80.9 -> 74.8 us, 1600^2 177 -> 165, 2048^2 298 -> 285, FP32 2048^2
// 157 -> 154, 2600^2 261 -> 255, p=5 1700^2 351 -> 338 (at the full clock; a GPU held
// at its power limit by a second of MatMults takes 309 and 305 us at FP64
// 2048^2). Marking a fixed part of it to stay instead gained half of that.
__device__ __forceinline__ uint64_t policy_once()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar, uint64_t policy)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for phase `parity` of *bar; returns false after `limit` polls
// (limit 0: gives up at once, which tests use to exercise the timeout path).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, long long limit = kWaitLimit)
{
    for (long long it = 0; it < limit; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// cp.async (LDGSTS) of 4, 8 or 16 bytes with zero fill when `valid` is false.
template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(void *dst, const void *src, bool valid)
{
    const int src_size = valid ? BYTES : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES),
                 "r"(src_size)
                 : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Entries per (kind, qy) row of the apply kernel's y tables: the NB basis
// values padded so that a row is a whole number of 16-byte words (vector
// loads, 16-byte copies).
__host__ __device__ constexpr int tab_nbp(int NB, int esz)
{
    return (NB * esz) % 16 == 0 ? NB : ((NB * esz + 15) / 16 * 16) / esz;
}

// FP32 y tables up to p = 4 hold (value, derivative) pairs side by side, one
// row of NB pairs per qy padded to whole 16-byte words: the operands of packed
// f32x2 FMAs where the apply kernel uses them, and no more vector loads per
// row than two padded rows elsewhere (p=4 unchanged; at p = 5 the paired rows
// were slower, 144 -> 157 us at 1024^2); the others keep separate rows per
// kind. Entries of one element row: tab_row_len(NB, NQ, esz).
__host__ __device__ constexpr bool tab_paired(int NB, int esz) { return esz == 4 && NB <= 5; }
__host__ __device__ constexpr int tab_nbp2(int NB) { return (2 * NB * 4 + 15) / 16 * 16 / 4; }
__host__ __device__ constexpr int tab_row_len(int NB, int NQ, int esz)
{
    return tab_paired(NB, esz) ? NQ * tab_nbp2(NB) : 2 * NQ * tab_nbp(NB, esz);
}
// Offset of entry (kind, qy, jl) within an element row of y tables.
__host__ __device__ constexpr int tab_y_index(int NB, int NQ, int esz, int kind, int qy, int jl)
{
    return tab_paired(NB, esz) ? qy * tab_nbp2(NB) + 2 * jl + kind : (kind * NQ + qy) * tab_nbp(NB, esz) + jl;
}

// ---------------------------------------------------------------- strips
// Element columns per warp strip (two lanes per element column).
constexpr int kSW = 16;

// Whether the two lane halves share the middle quadrature column (odd NQ;
// esz = bytes per value): at NQ = 5 it saves 2 of 15 quadrature points per
// lane and element row (p=4 FP32 82 -> 75 us at 1024^2); at NQ = 3 it pays in
// FP32 (p=2 2048^2 153 -> 150 us) but not in FP64, where the split's extra
// table loads cost more than the idle slot (185 -> 192 us).
__host__ __device__ constexpr bool mid_shared(int NQ, int esz) { return NQ % 2 == 1 && (NQ >= 5 || esz == 4); }


// Quadrature column of x-table slot j (j < QH = ceil(NQ / 2)) of the lane
// half h: h QH + j (past NQ: an idle slot); where mid_shared(NQ, esz) the last
// slot of both halves is the middle column QH - 1 instead, whose quadrature
// rows the two halves split (h takes qy = h, h + 2, ...).
__host__ __device__ constexpr int lane_qx(int NQ, int esz, int h, int j)
{
    return (mid_shared(NQ, esz) && j == (NQ + 1) / 2 - 1) ? j : h * ((NQ + 1) / 2) + j;
}

// Layout of one element-row step of a strip's G (NQ^2 points x 3 values x
// kSW columns), per quadrature row qy. Even NQ: [lane = 2c + h][j][3] with
// qx = h QH + j, a lane's values contiguous (vector loads). Where the lane
// halves share the middle column at NQ = 3 (g_mid_lane_major): [lane][3] for
// the column of its own (qx = 0 or 2), then [c][3] for the middle column
// (p=2 2048^2 FP32 148.8 -> 144.9 us; at NQ = 5 the vector-loaded values
// spill under the FP32 kernel's 128-register cap, 75.6 -> 81.3 us, so p = 4
// keeps the columns apart). Otherwise: [qx][3][c].
__host__ __device__ constexpr bool g_lane_major(int NQ) { return NQ % 2 == 0; }
__host__ __device__ constexpr bool g_mid_lane_major(int NQ, int esz) { return mid_shared(NQ, esz) && NQ < 5; }
__host__ __device__ inline int g_index(int NQ, int esz, int qy, int qx, int comp, int c)
{
    const int QH = (NQ + 1) / 2, QB = NQ * 3 * kSW;
    if (g_lane_major(NQ)) {
        const int h = qx / QH, j = qx - h * QH;
        return qy * QB + ((2 * c + h) * QH + j) * 3 + comp;
    }
    if (g_mid_lane_major(NQ, esz)) {
        if (qx == QH - 1) return qy * QB + 32 * (QH - 1) * 3 + c * 3 + comp;
        const int h = qx < QH - 1 ? 0 : 1, j = h ? qx - QH : qx;
        return qy * QB + ((2 * c + h) * (QH - 1) + j) * 3 + comp;
    }
    return ((qy * NQ + qx) * 3 + comp) * kSW + c;
}

// The element grid is cut into warp strips of kSW element columns by TY
// element rows (nominal sizes; strips that overhang the mesh are padded with
// empty elements). A control-point row R (or column C) is covered by the
// strips whose element range, widened by p to the right/top, contains it:
// strip R/TY (if it exists) and strip R/TY - 1 when R % TY < p.
struct StripGrid {
    int m, n;       // control points per direction
    int nex, ney;
    int TY;         // element rows per strip
    int NSX, NSY;   // strips per direction
    int P;
    int FS;         // frame slots per strip
};

__host__ __device__ __forceinline__ int frame_size(int P, int TY) { return 2 * P * (TY + P) + 2 * P * (kSW - P); }

// Slot of footprint position (lr, lc) in a strip's frame (only positions that
// can be covered by another strip: lc < P, lc >= kSW, lr < P or lr >= TY).
__host__ __device__ __forceinline__ int frame_index(int lr, int lc, int P, int TY)
{
    if (lc < P) return lr * P + lc;
    if (lc >= kSW) return P * (TY + P) + lr * P + (lc - kSW);
    if (lr < P) return 2 * P * (TY + P) + lr * (kSW - P) + (lc - P);
    return 2 * P * (TY + P) + P * (kSW - P) + (lr - TY) * (kSW - P) + (lc - P);
}

}  // namespace iga
