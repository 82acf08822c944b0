// GB300 (sm_103a) resident quantized H-matrix matvec and its C ABI.
//
// y = A x for a matrix held as dense FP64 diagonal blocks plus low-rank blocks
// whose balanced factors P (rows) and Q (columns) are stored as per-component
// signed integer codes of width w_j in [2, 32] (src/qhmat/core.cpp:235-282),
// with one FP64 scale per factor and component.  The resident layout
// (layout.hpp) keeps each code's bits, re-ordered into tensor-core fragment
// order as base-256 digit planes.
//
// FP64 throughput on GB300 is a small fraction of its tensor throughput, so
// every code product is an exact small-integer product on the f16 tensor
// cores (digits <= 255 times 8-bit limbs of a fixed-point operand, FP32 sums
// that stay integers below 2^24), and FP64 is used only per output row and for
// the dense diagonal blocks:
//
//   prep_x / x_limbs   x (source order) -> clustered order; one exponent per
//                      rhs column; X = round(x 2^(62-e)) as eight f16 limbs.
//   column_kernel      warp per task (<= 32 components sharing a column range
//                      and a width): t_j = sum_i c_ij X_i exactly, then
//                      u_j = (s^P s^Q) t_j 2^(e-1022-62) in fixed point on the
//                      component's own exponent (a layout-time bound; one
//                      64 x 64-bit integer product), then shifted to each
//                      consuming row tile's exponent as that tile's B rows
//                      (limbs);
//                      and warp per dense unit (16 columns of a dense
//                      diagonal block part, FP64 row sums).
//   row_kernel         warp per (row tile, 16 rows, k split): sum_j c_ij U_j
//                      exactly, stored as 128-bit partial sums.
//   combine_kernel     thread per row: dense row sums in column order plus
//                      the partials -> y (one conversion).
//
// Most applies of three columns and more take the column, row and combine
// kernels of tc.cu instead (the same integers on the 5th-generation tensor
// cores; KernelChoice in layout.hpp).
//
// The only rounding steps are the fixed-point conversions of x and u (2^-63
// of the column's largest |x|, ~2^-62 of the component's and of the tile's
// bound on |u|), the product s^P s^Q, and the final FP64 conversions: the
// result agrees with the reference's FP64 matmul (src/qhmat/core.cpp:360-390) to
// ~1e-15 in norm.  (Less for a tile that mixes very narrow and very wide codes of
// equal size, which an allocation of widths by singular value never makes: a
// 32-bit component's u is 2^-29 of a 3-bit one's there, and keeps 33 bits.)
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <type_traits>
#include <string>
#include <vector>

#include <unistd.h>

#include "../../include/qhmat_gb300.h"
#include "batch.hpp"
#include "errors.hpp"
#include "layout.hpp"
#include "pages.hpp"
#include "status.hpp"
#include "tc.hpp"

namespace qhg {
namespace {

// Pipeline depth and CTAs per SM of the two streaming kernels (measured:
// two stages per warp and two CTAs of 8 warps per SM; capping registers for a
// third CTA spills the accumulators).
#ifndef QH_COL_STAGES
#define QH_COL_STAGES 2
#define QH_COL_CTAS 2
#endif
#ifndef QH_ROW_STAGES
#define QH_ROW_STAGES 2
#define QH_ROW_CTAS 2
#endif
constexpr int kColStages = QH_COL_STAGES;
constexpr int kRowStages = QH_ROW_STAGES;
constexpr int kWarps = 8;
constexpr int kColPipeSmem = kWarps * kColStages * kColSlotBytes;
// Unit descriptors a column warp keeps in shared memory.
constexpr int kStagedUnits = 24;
constexpr int kRowPipeSmem = kWarps * kRowStages * kRowSlotBytes;

// Test aid for the bounded wait: one warp waits, `polls` tests at most, on an
// mbarrier that nothing ever completes (no copy is issued, so giving up
// leaves nothing in flight) and records the timeout in the status word
// exactly as the streaming kernels do.
__global__ void wait_timeout_kernel(int polls, int* status) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_init_fence();
    }
    __syncwarp();
    const bool ok = mbar_wait(&bar, 0, polls);
    if (!ok && threadIdx.x == 0) flag_timeout(status);
}

// ---------------------------------------------------------------- kernels

// Block (bx, p) of 8 warps: source entries 256bx .. 256bx+255 of rhs column
// p, read in order (coalesced; x may be the caller's host memory, read over
// the coherent host link) and stored at their clustered positions as the
// FP64 copy of x; the block's largest exponent field; nonfinite flag.  The
// grid also zeroes the apply's counters.
__device__ __forceinline__ void prep_block(const Arena& A, const Work& W, const double* __restrict__ x, int n,
                                           long long ld, int n_chunks, int* zero, int n_zero, int* status,
                                           int* s_m) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p = blockIdx.y;
    const int chunk = blockIdx.x * 8 + warp;
    const int src = chunk * kChunk + lane;
    const bool valid = chunk < n_chunks && src < n;
    const double v = valid ? x[(long long)src * ld + p] : 0.0;  // (plain load)
    const int e = exp_field(v);
    if (__any_sync(0xFFFFFFFFu, e == 0x7FF) && lane == 0 && status) atomicOr(status, kStatusNonfinite);
    const int em = __reduce_max_sync(0xFFFFFFFFu, e == 0x7FF ? 0 : e);
    if (valid) W.xc[(long long)p * n + __ldg(A.iperm + src)] = e == 0x7FF ? 0.0 : v;
    if (lane == 0) s_m[warp] = em;
    __syncthreads();
    if (threadIdx.x == 0) {
        int m = 0;
        for (int i = 0; i < 8; ++i) m = max(m, s_m[i]);
        W.xblk[(long long)p * gridDim.x + blockIdx.x] = m;
    }
    const long long tid = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
    const long long nthr = (long long)gridDim.x * gridDim.y * blockDim.x;
    for (long long i = tid; i < n_zero; i += nthr) zero[i] = 0;
}

__global__ void __launch_bounds__(256) prep_x_kernel(Arena A, Work W, const double* __restrict__ x, int n,
                                                     long long ld, int n_chunks, int* zero, int n_zero,
                                                     int* status) {
    __shared__ int s_m[8];
    pdl_trigger();
    prep_block(A, W, x, n, ld, n_chunks, zero, n_zero, status, s_m);
}

// Blocks bx = 0, nbx, ... of rhs column p: the column's exponent from the prep
// blocks' maxima, then the limbs of X for entries bx*256 .. (zero past n).
__device__ __forceinline__ void limbs_block(const Work& W, int n, int n_pad, int nblk, int p, int bx, int nbx,
                                            int* s_m) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int m = 0;
    for (int i = threadIdx.x; i < nblk; i += blockDim.x) m = max(m, __ldcg(W.xblk + (long long)p * nblk + i));
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    __syncthreads();  // (s_m reused)
    if (lane == 0) s_m[warp] = m;
    __syncthreads();
    int xe = 0;
    for (int i = 0; i < 8; ++i) xe = max(xe, s_m[i]);
    if (bx == 0 && threadIdx.x == 0) W.xe[p] = xe;
    for (int k = bx * blockDim.x + threadIdx.x; k < n_pad; k += nbx * blockDim.x) {
        const long long X = (k < n && xe) ? to_fixed(__ldcg(W.xc + (long long)p * n + k), xe) : 0;
        W.xq[(long long)p * n_pad + k] = to_limbs(X);
    }
}

__global__ void __launch_bounds__(256) x_limbs_kernel(Work W, int n, int n_pad, int nblk) {
    __shared__ int s_m[8];
    pdl_trigger();
    pdl_wait();
    limbs_block(W, n, n_pad, nblk, blockIdx.y, blockIdx.x, gridDim.x, s_m);
}

// prep_x and x_limbs in one cooperative launch (every block resident): the
// prep work, a grid-wide synchronisation, then the limbs.
__global__ void __launch_bounds__(256) prep_limbs_kernel(Arena A, Work W, const double* __restrict__ x, int n,
                                                         long long ld, int n_chunks, int* zero, int n_zero,
                                                         int* status, int n_pad) {
    __shared__ int s_m[8];
    pdl_trigger();
    prep_block(A, W, x, n, ld, n_chunks, zero, n_zero, status, s_m);
    cooperative_groups::this_grid().sync();
    limbs_block(W, n, n_pad, gridDim.x, blockIdx.y, blockIdx.x, gridDim.x, s_m);
}

// prep_x and x_limbs for an order of at most kPrepCluster * kPrepThreads: a
// cluster of blocks per column, a thread per clustered entry, which keeps it
// in a register until the column's exponent is known (block maxima exchanged
// through distributed shared memory).  Bound by latency: no grid-wide
// synchronisation, no second read, and it is launched while its predecessor
// ends, which a cooperative launch is not.
constexpr int kPrepCluster = 8, kPrepThreads = 1024;
__global__ void __cluster_dims__(kPrepCluster, 1, 1) __launch_bounds__(kPrepThreads)
    prep_cluster_kernel(Arena A, Work W, const double* __restrict__ x, int n, long long ld, int* zero, int n_zero,
                        int* status, int n_pad) {
    __shared__ int s_m[kPrepThreads / 32], s_all[kPrepCluster];
    auto cluster = cooperative_groups::this_cluster();
    cluster.barrier_arrive();
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = blockIdx.y;
    const int k = int(blockIdx.x) * kPrepThreads + int(threadIdx.x);
    const int src = k < n ? __ldg(A.perm + k) : -1;
    pdl_wait();
    double v = src >= 0 ? x[(long long)src * ld + p] : 0.0;  // (plain load)
    constexpr int kStep = kPrepCluster * kPrepThreads;
    for (long long i = (long long)p * kStep + k; i < n_zero; i += (long long)gridDim.y * kStep) zero[i] = 0;
    const int e = exp_field(v);
    if (e == 0x7FF) v = 0.0;
    if (__any_sync(0xFFFFFFFFu, e == 0x7FF) && lane == 0 && status) atomicOr(status, kStatusNonfinite);
    int m = __reduce_max_sync(0xFFFFFFFFu, e == 0x7FF ? 0 : e);
    if (lane == 0) s_m[warp] = m;
    __syncthreads();
    cluster.barrier_wait();  // every block runs
    if (warp == 0) {
        m = __reduce_max_sync(0xFFFFFFFFu, s_m[lane]);
        if (lane < kPrepCluster) *cluster.map_shared_rank(&s_all[blockIdx.x], unsigned(lane)) = m;
    }
    cluster.sync();
    int xe = 0;
#pragma unroll
    for (int i = 0; i < kPrepCluster; ++i) xe = max(xe, s_all[i]);
    if (k == 0) W.xe[p] = xe;
    if (k < n) W.xc[(long long)p * n + k] = v;
    if (k < n_pad) W.xq[(long long)p * n_pad + k] = to_limbs(xe ? to_fixed(v, xe) : 0);
}
static_assert(kPrepThreads == 32 * 32, "one warp reduces the warps' maxima");

// Bring a line into L1 ahead of its use (no register waits on it).
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// 8-byte asynchronous global -> shared copy (no register held while in flight).
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A column unit's descriptor from four 16-byte words (shared or global).
__device__ __forceinline__ ColTask load_task(const int4* q) {
    const int4 a = q[0], b = q[1], c = q[2], d = q[3];
    ColTask T;
    T.col0 = a.x, T.n = a.y, T.count = a.z, T.width = a.w;
    T.off = (long long)(((unsigned long long)(unsigned)b.y << 32) | (unsigned)b.x);
    T.stride = b.z, T.comp_idx = b.w;
    T.chunk0 = c.x, T.nchunks = c.y, T.part = c.z, T.nparts = c.w;
    T.split_id = d.x, T.cps = d.y;
    T.dest0 = d.z, T.ndest = d.w;
    return T;
}

// Column-side accumulators of one warp: FP32 MMA sums per M-tile and plane
// (exact below 2^24), their 64-bit folds, and the same for sum_i X_i.
struct ColAcc {
    float D[2][4][4];
    long long acc[2][4];
    int since;
};

// Fold the FP32 sums into the 64-bit per-limb sums: plane m < P-1 holds
// subnormal digits (sums in units of 2^-24), the top plane signed digits
// (units of 1); plane m weighs 2^(8m).
template <int P>
__device__ __forceinline__ void col_fold(ColAcc& a) {
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            long long v = 0;
#pragma unroll
            for (int m = 0; m < P; ++m) {
                const float d = m == P - 1 ? a.D[q][m][r] : a.D[q][m][r] * 16777216.0f;
                v += (long long)__float2int_rn(d) << (8 * m);
                a.D[q][m][r] = 0.f;
            }
            a.acc[q][r] += v;
        }
    a.since = 0;
}

// The chunks of a step of a task with P planes (nibble top plane if nibtop):
// per chunk, the x limbs' B fragments and two MMAs per (M-tile, plane) group.
template <int P>
__device__ __forceinline__ void col_step(ColAcc& a, const uint8_t* slot, int nc, int stride, int count, bool nibtop,
                                         uint32_t hb, int g, int t, int lane) {
    const int RB = (P - 1) * 32 + (nibtop ? 16 : 32);  // bytes of one row over all planes
    const uint32_t xrow = smem_u32(slot + nc * stride) + 16u * unsigned(lane);
    const int rows0 = count < 16 ? count : 16, rows1 = count - 16;
    for (int c = 0; c < nc; ++c) {
        const uint8_t* cb = slot + c * stride;
        uint32_t b[4];
        limb_frags(xrow + unsigned(c * kColChunk * 16), b);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int rows = q ? rows1 : rows0;
            if (rows <= 0) break;
            const uint8_t* off = cb + q * 16 * RB;
#pragma unroll
            for (int m = 0; m < P - 1; ++m) {
                group_mma(a.D[q][m], off, false, rows, g, t, b);
                off += rows * 32;
            }
            group_mma_top(a.D[q][P - 1], off, nibtop, rows, g, t, b, hb);
        }
        if (++a.since == 8) col_fold<P>(a);
    }
}

// A dense unit of the column side: columns [k0, k0 + nc) of a dense diagonal
// block part of one row tile for rhs column p, lane l owning tile rows l and
// l + 32 (columns in order, FP64; consecutive lanes read consecutive doubles),
// stored as the unit's row-sum slice.  The FP64 pipe is the scarce one on
// this GPU, so the blocks are cut into many short units that spread over all
// schedulers and run beside the other warps' integer and tensor-core work.
__device__ __forceinline__ void dense_unit(const Arena& A, const Work& W, const ColTask& u, int p, int n,
                                           int n_dslices, int lane) {
    const int rows = __ldg(&A.tiles[u.stride].rows);
    const TileDense D = A.tdense[u.col0];
    const bool r0 = lane < rows, r1 = lane + 32 < rows;
    const double* col = A.dense + D.off + (long long)u.chunk0 * D.ld + lane;
    const double* xv = W.xc + (long long)p * n + D.xcol + u.chunk0;
    double s0 = 0.0, s1 = 0.0;
    // batches of eight columns: every load of a batch is issued before its
    // FMAs (the dense data comes from HBM); rows past the tile read 0 and add
    // nothing (fma(0, x, s) = s for finite x)
    int k = 0;
    for (; k + 8 <= u.n; k += 8) {
        double c0[8], c1[8], xk[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            xk[i] = __ldcg(xv + k + i);
            c0[i] = r0 ? __ldg(col + (long long)(k + i) * D.ld) : 0.0;
            c1[i] = r1 ? __ldg(col + (long long)(k + i) * D.ld + 32) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            s0 = fma(c0[i], xk[i], s0);
            s1 = fma(c1[i], xk[i], s1);
        }
    }
    for (; k < u.n; ++k) {
        const double xk = __ldcg(xv + k);
        if (r0) s0 = fma(__ldg(col + (long long)k * D.ld), xk, s0);
        if (r1) s1 = fma(__ldg(col + (long long)k * D.ld + 32), xk, s1);
    }
    double* out = W.pdense + ((long long)p * n_dslices + u.comp_idx) * 64;
    out[lane] = s0;
    out[lane + 32] = s1;
}

// Column side.  Warp gw owns the units warp_off[gw] .. warp_off[gw + 1]
// (assigned longest first at upload by a per-unit cycle model, heaviest first
// per warp; the first kStagedUnits descriptors are kept in shared memory); its
// work is the sequence (unit, rhs column, chunk), streamed through a
// kColStages-deep pipeline of shared-memory slots filled by bulk copies (the
// chunks' code groups and the limbs of their x entries), kColStages - 1 steps
// ahead of their use.  Per chunk the warp runs, for each M-tile and digit
// plane, two 16x8x16 MMAs (digits x the eight x limbs; the top plane's digits
// signed); the FP32 sums are folded into 64-bit integers every 8 chunks
// (before any can reach 2^24).  At the unit's end the limbs and planes are
// combined into exact 128-bit sums t_j = sum_i c_ij X_i (lane j: component j,
// through shared memory), u_j in fixed point (comp_fixed: integer shifts and
// one 64 x 64-bit product instead of a 128-bit to FP64 conversion, an FP64
// product and a conversion back per destination -- 85.2 -> 82.9 us per apply
// at n = 32768), and the B rows of u_j on each consuming tile's exponent are
// written.  Dense
// units (width 0) are computed in FP64 by dense_unit.
__global__ void __launch_bounds__(kWarps * 32, QH_COL_CTAS) column_kernel(Arena A, Work W, const int* __restrict__ warp_off,
                                                                int n_pad, int rhs, int n_split, int n_slots,
                                                                int n, int n_dslices, int* status) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_bar[kWarps][kColStages];
    __shared__ int2 s_td[kWarps][32];  // each lane's first B row record of the current unit
    __shared__ int4 s_desc[kWarps][kStagedUnits * 4];  // the warp's first unit descriptors
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    uint8_t* slots = smem_raw + (size_t)warp * kColStages * kColSlotBytes;
    uint64_t* bar = s_bar[warp];
    if (lane == 0) {
        for (int i = 0; i < kColStages; ++i) mbar_init(bar + i, 1);
        mbar_init_fence();
    }
    __syncwarp();
    const int gw = blockIdx.x * kWarps + warp;
    const int u0 = __ldg(warp_off + gw), my_units = __ldg(warp_off + gw + 1) - u0;
    const ColTask* my_tasks = A.tasks + u0;
    // the warp's first kStagedUnits descriptors into shared memory (read-only
    // layout: before waiting for the preceding kernel)
    {
        const int4* src = reinterpret_cast<const int4*>(my_tasks);
        const int nst = min(my_units, kStagedUnits) * 4;
        for (int i = lane; i < nst; i += 32) s_desc[warp][i] = __ldg(src + i);
        __syncwarp();
    }
    auto unit = [&](int k) {
        if (k < kStagedUnits) return load_task(&s_desc[warp][4 * k]);
        const int4* q = reinterpret_cast<const int4*>(my_tasks + k);
        const int4 gq[4] = {__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3)};
        return load_task(gq);
    };
    if (my_units <= 0) pdl_wait();  // (every thread waits before exiting)
    unsigned issued = 0, computed = 0;  // running step counters (slot, phase)
    ColAcc a;
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int r = 0; r < 4; ++r) a.D[q][m][r] = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) a.acc[0][r] = a.acc[1][r] = 0;
    a.since = 0;
    pdl_trigger();
    if (my_units > 0) {
        const int nb = my_units;
        int ik = 0, ip = 0, ic = 0;  // issue cursor
        ColTask di = unit(0);
        // The first stages' code bytes come from the read-only arena, so they
        // are fetched while the preceding kernel finishes; their x limbs only
        // after it has (programmatic dependent launch): deferred copies.
        bool defer = true;
        int npend = 0;
        const void* pend_src[kColStages];
        uint8_t* pend_dst[kColStages];
        unsigned pend_bytes[kColStages], pend_slot[kColStages];
        auto issue = [&]() {
            while (ik < nb && di.width == 0) {  // dense units stream nothing
                if (++ik < nb) di = unit(ik);
            }
            if (ik >= nb) return;
            const int nc = min(di.cps, di.nchunks - ic);
            const unsigned slot_i = issued % kColStages;
            uint8_t* slot = slots + slot_i * kColSlotBytes;
            const unsigned wbytes = unsigned(nc * di.stride);
            const unsigned xbytes = unsigned(nc * kColChunk * 16);
            const long long k0 = (long long)(di.chunk0 + ic) * kColChunk;
            if (lane == 0) {
                fence_async_smem();
                mbar_arrive_expect(bar + slot_i, wbytes + xbytes);
                bulk_load(slot, A.qcodes + di.off + (long long)(di.chunk0 + ic) * di.stride, wbytes, bar + slot_i);
                const void* xsrc = W.xq + (long long)ip * n_pad + di.col0 + k0;
                if (defer) {
                    pend_src[npend] = xsrc, pend_dst[npend] = slot + wbytes;
                    pend_bytes[npend] = xbytes, pend_slot[npend] = slot_i;
                    ++npend;
                } else {
                    bulk_load(slot + wbytes, xsrc, xbytes, bar + slot_i);
                }
            }
            ++issued;
            ic += nc;
            if (ic == di.nchunks) {
                ic = 0;
                if (++ip == rhs) {
                    ip = 0;
                    if (++ik < nb) {
                        di = unit(ik);
                    }
                }
            }
        };
        __syncwarp();
        int ck = 0, cp = 0, cc = 0;  // compute cursor (first unit: before the issue cursor moves on)
        ColTask dc = di;
#pragma unroll 1
        for (int s = 0; s < kColStages - 1; ++s) issue();
        pdl_wait();  // x limbs and exponents of this apply
        defer = false;
        if (lane == 0)
            for (int i = 0; i < npend; ++i) bulk_load(pend_dst[i], pend_src[i], pend_bytes[i], bar + pend_slot[i]);
        // this lane's component record and first B row record, loaded when a
        // unit starts (the record by an asynchronous copy into shared
        // memory) and used at its end
        int shift = 1;
        unsigned long long kappa = 0;
        int2* my_td = &s_td[warp][lane];
        auto load_rec = [&]() {
            if (lane < dc.count) {
                const uint4 r = __ldg(reinterpret_cast<const uint4*>(A.task_rec + dc.comp_idx + lane));
                shift = int((r.y >> 8) & 255u);
                kappa = ((unsigned long long)r.w << 32) | r.z;
            }
            if (lane < dc.ndest) cp_async8(my_td, A.task_dest + dc.dest0 + lane);
        };
        load_rec();
        while (ck < nb) {
            if (dc.width == 0) {  // dense unit: no stage
                dense_unit(A, W, dc, cp, n, n_dslices, lane);
                if (++cp == rhs) {
                    cp = 0;
                    if (++ck < nb) {
                        dc = unit(ck);
                        load_rec();
                    }
                }
                continue;
            }
            issue();
            const unsigned slot_i = computed % kColStages;
            if (!mbar_wait(bar + slot_i, (computed / kColStages) & 1)) {
                flag_timeout(status);
                break;
            }
            const int nc = min(dc.cps, dc.nchunks - cc);
            const uint8_t* slot = slots + slot_i * kColSlotBytes;
            const int P = (dc.width + 7) >> 3;
            const int tb = dc.width - 8 * (P - 1);  // bits of the top digit
            const bool nibtop = tb <= 4;
            const uint32_t hb = (0x6400u | (1u << (tb - 1))) * 0x00010001u;
            switch (P) {
                case 1: col_step<1>(a, slot, nc, dc.stride, dc.count, nibtop, hb, g, t, lane); break;
                case 2: col_step<2>(a, slot, nc, dc.stride, dc.count, nibtop, hb, g, t, lane); break;
                case 3: col_step<3>(a, slot, nc, dc.stride, dc.count, nibtop, hb, g, t, lane); break;
                default: col_step<4>(a, slot, nc, dc.stride, dc.count, nibtop, hb, g, t, lane); break;
            }
            ++computed;
            cc += nc;
            if (cc == dc.nchunks) {
                switch ((dc.width + 7) >> 3) {
                    case 1: col_fold<1>(a); break;
                    case 2: col_fold<2>(a); break;
                    case 3: col_fold<3>(a); break;
                    default: col_fold<4>(a); break;
                }
                // this lane's per-limb sums: rows 16q + g + 8h, limbs 2t, 2t+1.
                // Unsplit task: stage all rows' sums in the consumed slot (not
                // refilled before the next issue) and let lane j finish row j;
                // a part of a split task adds its sums exactly with atomics and
                // the part that finishes last finishes the rows.
                long long* st = reinterpret_cast<long long*>(const_cast<uint8_t*>(slot));
                bool finish = true;
                if (dc.nparts == 1) {
#pragma unroll
                    for (int q = 0; q < 2; ++q)
#pragma unroll
                        for (int hh = 0; hh < 2; ++hh) {
                            const int row = 16 * q + 8 * hh + g;
                            *reinterpret_cast<longlong2*>(st + row * 8 + 2 * t) =
                                make_longlong2(a.acc[q][2 * hh], a.acc[q][2 * hh + 1]);
                        }
                } else {
                    long long* blk = W.lsplit + ((long long)cp * n_split * 33 + dc.split_id * 33) * 8;
#pragma unroll
                    for (int q = 0; q < 2; ++q)
#pragma unroll
                        for (int hh = 0; hh < 2; ++hh) {
                            const int row = 16 * q + 8 * hh + g;
                            if (row >= dc.count) continue;
                            unsigned long long* dst = reinterpret_cast<unsigned long long*>(blk + row * 8 + 2 * t);
                            atomicAdd(dst, (unsigned long long)a.acc[q][2 * hh]);
                            atomicAdd(dst + 1, (unsigned long long)a.acc[q][2 * hh + 1]);
                        }
                    __threadfence();
                    __syncwarp();
                    int done = 0;
                    if (lane == 0) done = atomicAdd(W.split_cnt + (long long)cp * n_split + dc.split_id, 1);
                    done = __shfl_sync(0xFFFFFFFFu, done, 0);
                    finish = done == dc.nparts - 1;
                    if (finish) {
                        __threadfence();
                        if (lane < dc.count) {
                            const longlong2* src = reinterpret_cast<const longlong2*>(blk + lane * 8);
#pragma unroll
                            for (int l = 0; l < 4; ++l)
                                *reinterpret_cast<longlong2*>(st + lane * 8 + 2 * l) = __ldcg(src + l);
                        }
                    }
                }
                if (finish) {
                    for (int l = 32 + 16 * lane; l < dc.ndest; l += 512)  // the rest of a long B row list
                        prefetch_l2(A.task_dest + dc.dest0 + l);
                    __syncwarp();
                    // lane j: u of component row j in fixed point
                    long long v = 0;
                    if (lane < dc.count) {
                        const longlong2* r2 = reinterpret_cast<const longlong2*>(st + lane * 8);
                        __int128 S = 0;
#pragma unroll
                        for (int l = 0; l < 4; ++l) {
                            const longlong2 w = r2[l];
                            S += ((__int128)w.x << (16 * l)) + ((__int128)w.y << (16 * l + 8));
                        }
                        v = comp_fixed(S, shift, kappa);
                    }
                    // the task's B rows, lanes over the (component, slot)
                    // pairs: U on the tile's exponent and its limbs
                    const int2* tdp = reinterpret_cast<const int2*>(A.task_dest + dc.dest0);
                    cp_async_wait_all();  // this lane's first record
                    for (int d0 = 0; d0 < dc.ndest; d0 += 128) {
                        int2 td[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int d = d0 + 32 * j + lane;
                            td[j] = d < dc.ndest ? (d0 + j == 0 ? *my_td : __ldg(tdp + d)) : make_int2(-1, 0);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (d0 + 32 * j >= dc.ndest) break;
                            const long long vd = __shfl_sync(0xFFFFFFFFu, v, (td[j].y >> 16) & 31);
                            if (td[j].x >= 0)
                                W.blimb[(long long)cp * n_slots + td[j].x] = to_limbs(tile_fixed(vd, td[j].y & 63));
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                    for (int r = 0; r < 4; ++r) a.acc[q][r] = 0;
                cc = 0;
                if (++cp == rhs) {
                    cp = 0;
                    if (++ck < nb) {
                        dc = unit(ck);
                        load_rec();
                    }
                }
            }
            __syncwarp();
        }
    }
    // copies still in flight (only after a failed wait): wait for them, bounded
    while (computed < issued) {
        mbar_wait(bar + computed % kColStages, (computed / kColStages) & 1);
        ++computed;
    }
}

// A row unit's descriptor (four 16-byte loads, cached in L1).
struct RowDesc {
    long long code_off, kp_off;
    int tile, q, h, H, nkps, K, slot0, nsteps, step0;
};

__device__ __forceinline__ RowDesc load_rdesc(const RowUnit* p) {
    const int4* q = reinterpret_cast<const int4*>(p);
    const int4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2), e = __ldg(q + 3);
    RowDesc d;
    d.tile = a.x, d.q = a.y, d.h = a.z, d.H = a.w;
    d.nkps = b.x, d.K = b.y, d.slot0 = b.z, d.nsteps = b.w;
    d.code_off = (long long)(((unsigned long long)(unsigned)c.y << 32) | (unsigned)c.x);
    d.kp_off = (long long)(((unsigned long long)(unsigned)c.w << 32) | (unsigned)c.z);
    d.step0 = e.x;
    return d;
}

// The digit groups of one k-pair with P planes (nibble top plane if NIBTOP),
// at compile-time offsets.
template <int P, bool NIBTOP>
__device__ __forceinline__ void kp_groups(float (&D)[4][4], const uint8_t* gp, int g, int t, const uint32_t (&b)[4],
                                          uint32_t hb) {
#pragma unroll
    for (int m = 0; m < P - 1; ++m) {
        group_mma(D[m], gp, false, 16, g, t, b);
        gp += 512;
    }
    group_mma_rtop(D[P - 1], gp, NIBTOP, g, t, b, hb);
}

// Row side.  Warp gw owns the units warp_off[gw] .. warp_off[gw + 1]
// (assigned longest first at upload).  A
// low-rank unit (rows 16q.. of a tile, k-pairs h, h + H, ...) streams its
// digit groups and B rows through a kRowStages-deep bulk-copy pipeline; per
// k-pair it runs, for each plane, two 16x8x16 MMAs of its 16 rows of digits by
// the components' U limbs, folding the FP32 sums into 64-bit integers every 8
// k-pairs (at most 16 k-blocks, below 2^24).  At the end the limbs and planes
// of each row are combined into an exact 128-bit sum and stored as the unit's
// partial.  combine_kernel adds the partials and the dense diagonal blocks.
__global__ void __launch_bounds__(kWarps * 32, QH_ROW_CTAS) row_kernel(Arena A, Work W, const int* __restrict__ warp_off,
                                                             int rhs, int n_slots, int n_tiles, int* status) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_bar[kWarps][kRowStages];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    uint8_t* slots = smem_raw + (size_t)warp * kRowStages * kRowSlotBytes;
    uint64_t* bar = s_bar[warp];
    if (lane == 0) {
        for (int i = 0; i < kRowStages; ++i) mbar_init(bar + i, 1);
        mbar_init_fence();
    }
    __syncwarp();
    const int gw = blockIdx.x * kWarps + warp;
    const int u0 = __ldg(warp_off + gw), my_units = __ldg(warp_off + gw + 1) - u0;
    const RowUnit* my_units_p = A.units + u0;
    unsigned issued = 0, computed = 0;
    pdl_trigger();
    if (my_units <= 0) pdl_wait();
    if (my_units > 0) {
        const int nb = my_units;
        // issue cursor: unit ik, rhs column ip, step is (k-pair index ii,
        // byte offset ioff); the unit's step words isb .. isb + 31, one per lane
        int ik = 0, ip = 0, is = 0, isb = 0, ii = 0;
        long long ioff = 0;
        RowDesc di = load_rdesc(my_units_p);
        if (lane < 2 && lane + 1 < nb) prefetch_l1(my_units_p + lane + 1);
        // The first stages' code bytes come from the read-only arena, so they
        // are fetched while the column kernel finishes; their B rows only
        // after it has (programmatic dependent launch): deferred copies.
        bool defer = true;
        int npend = 0;
        const void* pend_src[kRowStages];
        uint8_t* pend_dst[kRowStages];
        unsigned pend_bytes[kRowStages], pend_slot[kRowStages];
        auto load_steps = [&](const RowDesc& d, int base) {
            return base + lane < d.nsteps ? __ldg(A.row_steps + d.step0 + base + lane) : 0u;
        };
        auto load_info = [&](const RowDesc& d, int base) {
            return base + lane < d.nkps ? int(__ldg(A.kp_info + d.kp_off + d.h + (base + lane) * d.H)) : 0;
        };
        uint32_t isteps = load_steps(di, 0);
        auto issue = [&]() {
            if (ik >= nb) return;
            if (is - isb == 32) {
                isb = is;
                isteps = load_steps(di, isb);
            }
            const uint32_t sw = __shfl_sync(0xFFFFFFFFu, isteps, is - isb);
            const int c = int(sw & 255u);
            const int cbytes = int((sw >> 8) & 255u) * 256;
            const unsigned slot_i = issued % kRowStages;
            uint8_t* slot = slots + slot_i * kRowSlotBytes;
            const unsigned lbytes = unsigned(c * 512);
            if (lane == 0) {
                fence_async_smem();
                mbar_arrive_expect(bar + slot_i, unsigned(cbytes) + lbytes);
                bulk_load(slot, A.pcodes + di.code_off + ioff, unsigned(cbytes), bar + slot_i);
                const void* bsrc = W.blimb + (long long)ip * n_slots + di.slot0 + 32 * ii;
                if (defer) {
                    pend_src[npend] = bsrc, pend_dst[npend] = slot + cbytes;
                    pend_bytes[npend] = lbytes, pend_slot[npend] = slot_i;
                    ++npend;
                } else {
                    bulk_load(slot + cbytes, bsrc, lbytes, bar + slot_i);
                }
            }
            ++issued;
            ++is;
            ii += c;
            ioff += cbytes;
            if (is == di.nsteps) {
                is = isb = ii = 0;
                ioff = 0;
                if (++ip == rhs) {
                    ip = 0;
                    if (++ik < nb) {
                        di = load_rdesc(my_units_p + ik);
                        if (ik + 2 < nb && lane == 0) prefetch_l1(my_units_p + ik + 2);
                        // the next unit's step words and k-pair infos
                        if (ik + 1 < nb && lane == 0) {
                            const RowDesc dn = load_rdesc(my_units_p + ik + 1);
                            prefetch_l1(A.row_steps + dn.step0);
                            prefetch_l1(A.kp_info + dn.kp_off + dn.h);
                        }
                    }
                }
                isteps = load_steps(di, 0);
            }
        };
        __syncwarp();
        // compute cursor: unit ck, rhs column cp, step cs (words csb ..), k-pair
        // index ci (infos cib ..); first unit: before the issue cursor moves on
        int ck = 0, cp = 0, cs = 0, csb = 0, ci = 0, cib = 0;
        RowDesc dc = di;
#pragma unroll 1
        for (int s = 0; s < kRowStages - 1; ++s) issue();
        pdl_wait();  // B rows of this apply
        defer = false;
        if (lane == 0)
            for (int i = 0; i < npend; ++i) bulk_load(pend_dst[i], pend_src[i], pend_bytes[i], bar + pend_slot[i]);
        uint32_t csteps = load_steps(dc, 0);
        int cinfo = load_info(dc, 0);
        float D[4][4];
        long long acc[4];
        int since = 0;
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int r = 0; r < 4; ++r) D[m][r] = 0.f;
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] = 0;
        auto fold_row = [&]() {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                long long v = 0;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    v += fold(D[m][r], m);
                    D[m][r] = 0.f;
                }
                acc[r] += v;
            }
            since = 0;
        };
        auto advance = [&]() {
            if (++cp == rhs) {
                cp = 0;
                if (++ck < nb) dc = load_rdesc(my_units_p + ck);
            }
            cs = csb = ci = cib = 0;
            csteps = load_steps(dc, 0);
            cinfo = load_info(dc, 0);
        };
        while (ck < nb) {
            issue();
            const unsigned slot_i = computed % kRowStages;
            if (!mbar_wait(bar + slot_i, (computed / kRowStages) & 1)) {
                flag_timeout(status);
                break;
            }
            const uint8_t* slot = slots + slot_i * kRowSlotBytes;
            if (cs - csb == 32) {
                csb = cs;
                csteps = load_steps(dc, csb);
            }
            const uint32_t sw = __shfl_sync(0xFFFFFFFFu, csteps, cs - csb);
            const int c = int(sw & 255u);
            const int cbytes = int((sw >> 8) & 255u) * 256;
            const uint8_t* gp = slot;
            const uint32_t lrow = smem_u32(slot + cbytes) + 16u * unsigned(lane);
            // a uniform step: one digit pattern, no k slot past the k axis
            auto run = [&](auto P_, auto NIB_) {
                constexpr int P = decltype(P_)::value;
                constexpr bool NIB = decltype(NIB_)::value;
                const uint32_t hb = kp_hb(int((sw >> 16) & 255u));
                for (int k = 0; k < c; ++k) {
                    uint32_t b[4];
                    limb_frags(lrow + unsigned(k * 512), b);
                    kp_groups<P, NIB>(D, gp, g, t, b, hb);
                    gp += P * 512 - (NIB ? 256 : 0);
                    if (++since == 8) fold_row();
                }
            };
            using I1 = std::integral_constant<int, 1>;
            using I2 = std::integral_constant<int, 2>;
            using I3 = std::integral_constant<int, 3>;
            using I4 = std::integral_constant<int, 4>;
            if (sw >> 24) {
                switch ((sw >> 16) & 15u) {
                    case 4: run(I4{}, std::false_type{}); break;
                    case 4 | 8: run(I4{}, std::true_type{}); break;
                    case 3: run(I3{}, std::false_type{}); break;
                    case 3 | 8: run(I3{}, std::true_type{}); break;
                    case 2: run(I2{}, std::false_type{}); break;
                    case 2 | 8: run(I2{}, std::true_type{}); break;
                    case 1: run(I1{}, std::false_type{}); break;
                    default: run(I1{}, std::true_type{}); break;
                }
            } else
            for (int k = 0; k < c; ++k) {
                if (ci + k - cib >= 32) {
                    cib = ci + k;
                    cinfo = load_info(dc, cib);
                }
                const int kp = dc.h + (ci + k) * dc.H;
                const int info = __shfl_sync(0xFFFFFFFFu, cinfo, ci + k - cib);
                uint32_t b[4];
                limb_frags(lrow + unsigned(k * 512), b);
                const int kv = dc.K - 32 * kp;  // k slots of this k-pair inside the k axis
                if (kv < 32) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int e = 8 * i + 2 * t;
                        if (e >= kv) b[i] &= 0xFFFF0000u;
                        if (e + 1 >= kv) b[i] &= 0x0000FFFFu;
                    }
                }
                const uint32_t hb = kp_hb(info);
                switch (info & 15) {  // planes | nibble top << 3
                    case 4: kp_groups<4, false>(D, gp, g, t, b, hb); break;
                    case 4 | 8: kp_groups<4, true>(D, gp, g, t, b, hb); break;
                    case 3: kp_groups<3, false>(D, gp, g, t, b, hb); break;
                    case 3 | 8: kp_groups<3, true>(D, gp, g, t, b, hb); break;
                    case 2: kp_groups<2, false>(D, gp, g, t, b, hb); break;
                    case 2 | 8: kp_groups<2, true>(D, gp, g, t, b, hb); break;
                    case 1: kp_groups<1, false>(D, gp, g, t, b, hb); break;
                    default: kp_groups<1, true>(D, gp, g, t, b, hb); break;
                }
                gp += kp_bytes(info);
                if (++since == 8) fold_row();
            }
            ++computed;
            ci += c;
            if (++cs == dc.nsteps) {
                fold_row();
                // row g + 8(t&1): limbs over the row's four lanes
                __int128 v0 = ((__int128)acc[0] << (16 * t)) + ((__int128)acc[1] << (16 * t + 8));
                __int128 v1 = ((__int128)acc[2] << (16 * t)) + ((__int128)acc[3] << (16 * t + 8));
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[r] = 0;
                const bool hi = t & 1;
                __int128 R = hi ? v1 : v0;
                R += shfl_xor_i128(hi ? v0 : v1, 1);
                R += shfl_xor_i128(R, 2);
                const long long tb = ((long long)cp * n_tiles + dc.tile) * kTileUnits;
                if (t < 2) st_i128(W.plr + (tb + dc.q * dc.H + dc.h) * 16 + g + 8 * t, R);
                advance();
            }
            __syncwarp();
        }
    }
    // copies still in flight (only after a failed wait): wait for them, bounded
    while (computed < issued) {
        mbar_wait(bar + computed % kRowStages, (computed / kRowStages) & 1);
        ++computed;
    }
}

// One CTA of 64 threads per (row tile, rhs column), one thread per row: y =
// the tile's dense slices (column side) added in column order + the low-rank
// row sums of the tile's units, converted once.
__global__ void __launch_bounds__(64) combine_kernel(Arena A, Work W, double* __restrict__ y, int n_tiles,
                                                    int n_dslices, long long ld) {
    pdl_trigger();
    const int p = blockIdx.y, tile = blockIdx.x, r = threadIdx.x;
    const RowTile T = A.tiles[tile];
    if (r >= T.rows) {
        pdl_wait();
        return;
    }
    const int out = __ldg(A.perm + T.row0 + r);
    pdl_wait();
    const int xe = W.xe[p];
    const long long tb = ((long long)p * n_tiles + tile) * kTileUnits;
    __int128 R = 0;
    for (int h = 0; h < T.nh; ++h) R += ld_i128(W.plr + (tb + (r >> 4) * T.hsplit + h) * 16 + (r & 15));
    double d = 0.0;
    for (int i = 0; i < T.nds; ++i) d += __ldcg(W.pdense + ((long long)p * n_dslices + T.ds0 + i) * 64 + r);
    const double lr = (xe && T.c_exp != kNoExp) ? i128_ldexp(R, xe + T.c_exp - 1022 - kFixBits) : 0.0;
    y[(long long)out * ld + p] = d + lr;
}

// Decode every code from the resident layout through the same fragment
// routines the apply kernels feed to the MMA (group_digits uses the permutes
// and masks of group_mma).  out[comp_base[c] + i] = code i of component c
// (i: block column on the right side, clustered row on the left).

// Part y of gridDim.y: chunks of a task.
__device__ __forceinline__ void decode_col(const Arena& A, int n_tasks, int block, int blocks,
                                           const long long* __restrict__ comp_base, int* out) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int warps = blocks * (blockDim.x >> 5);
    for (int ti = block * (blockDim.x >> 5) + (threadIdx.x >> 5); ti < n_tasks; ti += warps) {
        const ColTask T = A.tasks[ti];
        if (T.width == 0) continue;  // dense unit
        const int P = (T.width + 7) / 8;
        const bool nibtop = T.width - 8 * (P - 1) <= 4;
        const int RB = (P - 1) * 32 + (nibtop ? 16 : 32);
        for (int ch = T.chunk0 + blockIdx.y; ch < T.chunk0 + T.nchunks; ch += gridDim.y) {
            const uint8_t* cb = A.qcodes + T.off + (long long)ch * T.stride;
            for (int q = 0; q < 2; ++q) {
                const int rows = min(16, T.count - 16 * q);
                if (rows <= 0) continue;
                uint32_t u[2][8] = {};
                int off = q * 16 * RB;
                for (int m = 0; m < P; ++m) {
                    const bool nib = nibtop && m == P - 1;
                    uint32_t d[2][8];
                    group_digits(cb + off, nib, rows, g, t, d);
                    for (int hh = 0; hh < 2; ++hh)
                        for (int k = 0; k < 8; ++k) u[hh][k] |= d[hh][k] << (8 * m);
                    off += rows * (nib ? 16 : 32);
                }
                for (int hh = 0; hh < 2; ++hh) {
                    const int j = 16 * q + 8 * hh + g;
                    if (j >= T.count) continue;
                    const int c = A.task_rec[T.comp_idx + j].comp;
                    for (int k = 0; k < 8; ++k) {
                        const int i = ch * kColChunk + slot_entry(k >> 2, k & 3, t);
                        if (i < T.n) out[comp_base[c] + i] = int(int64_t(u[hh][k]) - (int64_t(1) << (T.width - 1)));
                    }
                }
            }
        }
    }
}

// Part y of gridDim.y: a run of a unit's k-pairs (found by summing the bytes of
// those before it).
__device__ __forceinline__ void decode_row(const Arena& A, int n_units, int block, int blocks,
                                           const long long* __restrict__ comp_base, int* out) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int warps = blocks * (blockDim.x >> 5);
    for (int ui = block * (blockDim.x >> 5) + (threadIdx.x >> 5); ui < n_units; ui += warps) {
        const RowUnit U = A.units[ui];
        const RowTile T = A.tiles[U.tile];
        const int per = (U.nkps + int(gridDim.y) - 1) / int(gridDim.y);
        const int i0 = min(int(blockIdx.y) * per, U.nkps), i1 = min(i0 + per, U.nkps);
        long long skip = 0;
        for (int i = lane; i < i0; i += 32) skip += kp_bytes(A.kp_info[U.kp_off + U.h + i * U.H]);
#pragma unroll
        for (int o = 16; o; o >>= 1) skip += __shfl_xor_sync(0xFFFFFFFFu, skip, o);
        const uint8_t* gp = A.pcodes + U.code_off + skip;
        for (int i = i0; i < i1; ++i) {
            const int kp = U.h + i * U.H;
            const int info = A.kp_info[U.kp_off + kp];
            const int planes = info & 7, half = 1 << (info >> 4);
            long long u[2][8] = {};
            for (int m = 0; m < planes; ++m) {
                const bool nib = m == planes - 1 && ((info >> 3) & 1);
                uint32_t d[2][8];
                group_digits(gp, nib, 16, g, t, d);
                for (int hh = 0; hh < 2; ++hh)
                    for (int k = 0; k < 8; ++k)
                        u[hh][k] += (m == planes - 1 ? (long long)d[hh][k] - half : (long long)d[hh][k]) << (8 * m);
                gp += nib ? 256 : 512;
            }
            for (int hh = 0; hh < 2; ++hh) {
                const int tr = 16 * U.q + 8 * hh + g;
                if (tr >= T.rows) continue;
                for (int k = 0; k < 8; ++k) {
                    const int e = slot_entry(k >> 2, k & 3, t);
                    const int c = A.slot_rec[U.slot0 + 32 * i + e].comp;
                    if (c < 0) continue;
                    out[comp_base[c] + T.row0 + tr] = int(u[hh][k]);
                }
            }
        }
    }
}

// Blocks [0, col_blocks) of x decode the column side, the others the row side.
__global__ void decode_kernel(Arena A, int n_tasks, int col_blocks, const long long* rbase, int* rout, int n_units,
                              const long long* lbase, int* lout) {
    if (int(blockIdx.x) < col_blocks) decode_col(A, n_tasks, blockIdx.x, col_blocks, rbase, rout);
    else decode_row(A, n_units, int(blockIdx.x) - col_blocks, int(gridDim.x) - col_blocks, lbase, lout);
}
cudaError_t launch_decode(const Arena& A, int n_tasks, const long long* rbase, int* rout, int n_units,
                          const long long* lbase, int* lout) {
    const int cb = std::min((n_tasks + 7) / 8, 4096), rb = std::min((n_units + 7) / 8, 4096);
    if (cb + rb == 0) return cudaSuccess;
    decode_kernel<<<dim3(unsigned(cb + rb), 8), 256>>>(A, n_tasks, cb, rbase, rout, n_units, lbase, lout);
    return cudaGetLastError();
}

// A block of the matrix to reconstruct: its first tile, and where its factors
// start (component-major: column j of P at left + j m).
struct DenseOut {
    long long tile0, left, right;
};
// Per component: where its entries start (decode_kernel's comp_base).
__global__ void factor_base_kernel(Arena A, int n_lr, const DenseOut* blocks, long long* lbase, long long* rbase) {
    const int b = blockIdx.x;
    const LowRankDesc d = A.lr[b];
    for (int j = threadIdx.x; j < d.rank; j += blockDim.x) {
        lbase[d.comp0 + j] = blocks[b].left + (long long)j * d.m - d.row0;  // indexed by clustered row
        rbase[d.comp0 + j] = blocks[b].right + (long long)j * d.n;
    }
}

// Dense reconstruction (src/qhmat/core.cpp:392-410): value = the dense entry or
// 0, plus, per component in order, (c^P s^P)(c^Q s^Q) with separate IEEE
// multiplies and adds in the reference's order, written to
// out[perm[row] * n + perm[col]].
//
// Bound by the FP64 unit: one multiply and one add per component and entry (the
// codes are scaled as they enter a tile, 6 % of its operations; scaling them per
// entry took six each).  One block per 32 x 32 tile, factors 16 components at a
// time in shared memory, 2 x 4 entries a thread.  n = 2048, 2-D, 11587
// components: 657 -> 250 us (about 180 us by the rate of the FP64 unit).  Factors
// scaled by decode_kernel took the same time (device call 412 us, now 410; 5000
// unknowns 2150, now 2213) but twice the scratch.
constexpr int kDenseTile = 32, kDenseComps = 16;
// A code as a double: its bits below those of 1.5 2^52, minus that number (one
// exact FP64 operation, at twice the rate of a conversion).
__device__ __forceinline__ double code_value(int c) {
    return __dsub_rn(__longlong_as_double(0x4338000000000000LL + c), 6755399441055744.0);
}
__global__ void __launch_bounds__(128) reconstruct_kernel(Arena A, int n_lr, int nb, const DenseOut* __restrict__ blocks,
                                                          const int* __restrict__ left,
                                                          const int* __restrict__ right, int n,
                                                          double* __restrict__ out) {
    __shared__ double P[kDenseComps][kDenseTile], Q[kDenseComps][kDenseTile];
    int lo = 0, hi = nb - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (blocks[mid].tile0 <= (long long)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const DenseOut B = blocks[lo];
    const int tile = int(blockIdx.x - B.tile0), tid = threadIdx.x;
    LowRankDesc d = {};
    long long off = 0;
    if (lo < n_lr) {
        d = A.lr[lo];
    } else {
        const DenseDesc e = A.dd[lo - n_lr];
        d.row0 = e.row0, d.m = e.m, d.col0 = e.col0, d.n = e.n;
        off = e.off;
    }
    const int tcols = (d.n + kDenseTile - 1) / kDenseTile;
    const int i0 = tile / tcols * kDenseTile, k0 = tile % tcols * kDenseTile;
    const int ti = tid >> 3, tk = tid & 7;  // rows ti, ti + 16; columns tk, tk + 8, ..
    double v[2][4] = {};
    if (lo < n_lr) {
        const int tx = tid & 31, ty = tid >> 5;
        for (int j0 = 0; j0 < d.rank; j0 += kDenseComps) {
            const int jn = min(kDenseComps, d.rank - j0);
            for (int j = ty; j < jn; j += 4) {
                const int c = d.comp0 + j0 + j;
                P[j][tx] = i0 + tx < d.m ? __dmul_rn(code_value(left[B.left + (long long)(j0 + j) * d.m + i0 + tx]),
                                                     __ldg(A.comp_sl + c))
                                         : 0.0;
                Q[j][tx] = k0 + tx < d.n ? __dmul_rn(code_value(right[B.right + (long long)(j0 + j) * d.n + k0 + tx]),
                                                     __ldg(A.comp_sr + c))
                                         : 0.0;
            }
            __syncthreads();
            for (int j = 0; j < jn; ++j) {
                const double a[2] = {P[j][ti], P[j][ti + 16]};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const double q = Q[j][tk + 8 * k];
#pragma unroll
                    for (int i = 0; i < 2; ++i) v[i][k] = __dadd_rn(v[i][k], __dmul_rn(a[i], q));
                }
            }
            __syncthreads();
        }
    } else {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int row = i0 + ti + 16 * i, col = k0 + tk + 8 * k;
                if (row < d.m && col < d.n) v[i][k] = A.dense[off + (long long)col * d.m + row];
            }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = i0 + ti + 16 * i;
        if (row >= d.m) continue;
        double* dst = out + (long long)A.perm[d.row0 + row] * n;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int col = k0 + tk + 8 * k;
            if (col < d.n) dst[A.perm[d.col0 + col]] = v[i][k];
        }
    }
}

// ---------------------------------------------------------------- host side

thread_local std::string g_last_error;

int fail(int code, const std::string& msg) {
    g_last_error = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char* what) {
    return fail(QH_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

}  // namespace

// Shared with the other translation units of the library (errors.hpp).
int set_error(int code, const std::string& msg) { return fail(code, msg); }

}  // namespace qhg

using namespace qhg;

// Scratch of qh_matmul_device_static: one fixed array per device, loaded with
// the library and held until exit.  Host code must not use this symbol as an
// address (it names a host-side stand-in); static_scratch() returns the
// device address for the current device.
static __device__ __align__(256) unsigned char g_static_scratch[QH_STATIC_SCRATCH_BYTES];

struct qh_matrix {
    Layout L;
    int device = 0;
    int sms = 1;
    void* arena = nullptr;  // device copy of L.arena
    Arena A{};
    // unit schedules: warp w of the column (row) grid runs units
    // warp_off[w] .. warp_off[w + 1] of the (reordered) task (unit) array
    int* sched = nullptr;
    int col_grid = 0, row_grid = 0;
    KernelChoice choice;
    StatusWords words;  // of qh_matmul_device_checked
    std::vector<LowRankDesc> lr;  // host copies of the blocks (reconstruct)
    std::vector<DenseDesc> dd;
    // lazily allocated scratch for calls without a workspace, and host staging
    std::mutex mu;
    void* own_ws = nullptr;  // qh_matmul_host's device buffer
    size_t own_ws_bytes = 0;
    void* dev_ws = nullptr;  // the workspace of qh_matmul_device calls without one
    size_t dev_ws_bytes = 0;
    double* pinned = nullptr;
    size_t pinned_bytes = 0;
    int* d_status = nullptr;
    int* h_status = nullptr;
    cudaStream_t stream = nullptr;
    // the device reads and writes pageable host memory through the host's
    // page tables (coherent host link): host-buffer applies need no staging
    bool host_direct = false;
    // most blocks of prep_limbs_kernel the device holds at once (0: no
    // cooperative launch)
    int prep_coop_max = 0;
    ~qh_matrix() {
        int prev = 0;
        cudaGetDevice(&prev);
        cudaSetDevice(device);
        if (arena) cudaFree(arena);
        if (sched) cudaFree(sched);
        if (own_ws) cudaFree(own_ws);
        if (dev_ws) cudaFree(dev_ws);
        if (d_status) cudaFree(d_status);
        if (pinned) cudaFreeHost(pinned);
        if (h_status) cudaFreeHost(h_status);
        if (stream) cudaStreamDestroy(stream);
        cudaSetDevice(prev);
    }
};

namespace {

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

int check_device(int device) {
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDeviceCount");
    if (!count) return fail(QH_ERUNTIME, "no CUDA device is available");
    if (device < 0 || device >= count) return fail(QH_EINVAL, "invalid CUDA device ordinal");
    return QH_OK;
}

template <class T>
void permute(T* a, const std::vector<int32_t>& order) {
    std::vector<T> tmp(a, a + order.size());
    for (size_t i = 0; i < order.size(); ++i) a[i] = tmp[size_t(order[i])];
}

int upload(Layout&& L, int device, qh_matrix** out) {
    int rc = check_device(device);
    if (rc) return rc;
    DeviceGuard g(device);
    qh_matrix* m = new (std::nothrow) qh_matrix();
    if (!m) return fail(QH_ERUNTIME, "out of host memory");
    m->L = std::move(L);
    m->device = device;
    cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device);
    {
        int pageable = 0, host_tables = 0;
        cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, device);
        cudaDeviceGetAttribute(&host_tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device);
        m->host_direct = pageable == 1 && host_tables == 1;
        int coop = 0, per_sm = 0;
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
        if (coop && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, prep_limbs_kernel, 256, 0) == cudaSuccess)
            m->prep_coop_max = per_sm * m->sms;
        cudaGetLastError();
    }
    {
        // warp schedules for this device's grids: units longest first, each
        // to the warp with the least predicted time.
        Layout& Lm = m->L;
        m->col_grid = std::max(1, std::min((Lm.n_tasks + kWarps - 1) / kWarps, m->sms * 2));
        m->row_grid = std::max(1, std::min((Lm.n_units + kWarps - 1) / kWarps, m->sms * 2));
        auto* tasks = reinterpret_cast<ColTask*>(Lm.arena.data() + Lm.sec.tasks);
        auto* units = reinterpret_cast<RowUnit*>(Lm.arena.data() + Lm.sec.units);
        const Schedule col = schedule_units(column_costs(Lm), m->col_grid * kWarps);
        const Schedule row = schedule_units(row_costs(Lm), m->row_grid * kWarps);
        permute(tasks, col.order);
        permute(units, row.order);
        m->choice = kernel_choice(Lm, col, row, m->sms);
        std::vector<int32_t> sched(col.off);
        sched.insert(sched.end(), row.off.begin(), row.off.end());
        cudaError_t e2 = cudaMalloc(&m->sched, 4 * sched.size());
        if (e2 == cudaSuccess) e2 = cudaMemcpy(m->sched, sched.data(), 4 * sched.size(), cudaMemcpyHostToDevice);
        if (e2 != cudaSuccess) {
            delete m;
            return cuda_fail(e2, "cudaMalloc");
        }
    }
    cudaError_t e = cudaMalloc(&m->arena, m->L.sec.total);
    if (e != cudaSuccess) {
        delete m;
        return cuda_fail(e, "cudaMalloc");
    }
    e = cudaMemcpy(m->arena, m->L.arena.data(), m->L.sec.total, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        delete m;
        return cuda_fail(e, "cudaMemcpy host-to-device");
    }
    m->words.prepare();
    e = cudaFuncSetAttribute(row_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowPipeSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(column_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kColPipeSmem);
    if (e == cudaSuccess) e = tc_setup();
    if (e != cudaSuccess) {
        delete m;
        return cuda_fail(e, "cudaFuncSetAttribute");
    }
    {
        const auto* a = m->L.arena.data();
        const auto* lr = reinterpret_cast<const LowRankDesc*>(a + m->L.sec.lr);
        const auto* dd = reinterpret_cast<const DenseDesc*>(a + m->L.sec.dd);
        m->lr.assign(lr, lr + m->L.n_lr);
        m->dd.assign(dd, dd + m->L.n_dense);
    }
    // The host image is no longer needed once uploaded.
    std::vector<uint8_t>().swap(m->L.arena);
    const Sections& S = m->L.sec;
    auto* base = static_cast<const uint8_t*>(m->arena);
    m->A.perm = reinterpret_cast<const int32_t*>(base + S.perm);
    m->A.iperm = reinterpret_cast<const int32_t*>(base + S.iperm);
    m->A.lr = reinterpret_cast<const LowRankDesc*>(base + S.lr);
    m->A.dd = reinterpret_cast<const DenseDesc*>(base + S.dd);
    m->A.tasks = reinterpret_cast<const ColTask*>(base + S.tasks);
    m->A.task_rec = reinterpret_cast<const TaskRec*>(base + S.task_rec);
    m->A.qcodes = base + S.qcodes;
    m->A.pcodes = base + S.pcodes;
    m->A.dense = reinterpret_cast<const double*>(base + S.dense);
    m->A.tiles = reinterpret_cast<const RowTile*>(base + S.tiles);
    m->A.units = reinterpret_cast<const RowUnit*>(base + S.units);
    m->A.tdense = reinterpret_cast<const TileDense*>(base + S.tdense);
    m->A.kp_info = base + S.kp_info;
    m->A.slot_rec = reinterpret_cast<const SlotRec*>(base + S.slot_rec);
    m->A.task_dest = reinterpret_cast<const TaskDest*>(base + S.task_dest);
    m->A.row_steps = reinterpret_cast<const uint32_t*>(base + S.row_steps);
    m->A.comp_sl = reinterpret_cast<const double*>(base + S.comp_sl);
    m->A.comp_sr = reinterpret_cast<const double*>(base + S.comp_sr);
    m->A.tc_items = reinterpret_cast<const TcItem*>(base + S.tc_items);
    m->A.tc_tasks = reinterpret_cast<const TcTask*>(base + S.tc_tasks);
    m->A.dense_units = reinterpret_cast<const DenseUnit*>(base + S.dense_units);
    m->A.tc_row_items = reinterpret_cast<const TcRowItem*>(base + S.tc_row_items);
    m->A.tc_steps = reinterpret_cast<const TcStep*>(base + S.tc_steps);
    *out = m;
    return QH_OK;
}

template <class F>
int guarded(F&& f) {
    try {
        return f();
    } catch (const std::invalid_argument& e) {
        return fail(QH_EINVAL, e.what());
    } catch (const std::overflow_error& e) {
        return fail(QH_EOVERFLOW, e.what());
    } catch (const std::bad_alloc&) {
        return fail(QH_ERUNTIME, "out of host memory");
    } catch (const std::exception& e) {
        return fail(QH_ERUNTIME, e.what());
    }
}

// Right-hand-side columns one chain of launches handles at most (gridDim.y
// of the prep and combine launches); wider applies run column chunks in
// turn (every column is computed independently, so the result is the same).
constexpr size_t kMaxRhsChunk = 65535;

size_t rhs_chunk(size_t rhs) { return std::min(rhs, kMaxRhsChunk); }

struct WsPlan {
    size_t xc, xblk, xe, xq, lsplit, cnt, blimb, part, plr, pdense, total, zero0, zero_bytes;
    int nblk, pv;  // pv > 0: columns of a row of V, an even number (the tensor-memory kernels)
};

// x limbs are read by whole 32-entry chunks: pad past the last chunk.
size_t padded_order(const Layout& L) { return (L.order + kColChunk - 1) / kColChunk * kColChunk + kColChunk; }

WsPlan ws_plan(const Layout& L, size_t rhs, bool tc) {
    WsPlan w = {};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += align256(std::max<size_t>(bytes, 1));
        return o;
    };
    w.nblk = (L.n_chunks + 7) / 8;
    // zeroed by prep_x (contiguous): split partial sums and counters
    w.zero0 = off;
    w.lsplit = take(8 * 8 * 33 * size_t(L.n_split) * rhs);
    w.cnt = take(4 * size_t(L.n_split) * rhs);
    w.zero_bytes = off - w.zero0;
    w.xe = take(4 * rhs);
    w.xblk = take(4 * size_t(w.nblk) * rhs);
    w.xc = take(8 * L.order * rhs);
    w.xq = take(16 * padded_order(L) * rhs);
    if (tc) {  // V and the row items' sums
        w.pv = (int(rhs) + 1) & ~1;
        w.blimb = take(8 * size_t(L.n_comp) * size_t(w.pv));
        w.part = take(16 * 128 * size_t(L.n_parts) * rhs);
    } else {  // B rows and row sums of the column-by-column kernels
        w.blimb = take(16 * size_t(L.n_slots) * rhs);
        w.plr = take(16 * 16 * kTileUnits * size_t(L.n_tiles) * rhs);
    }
    w.pdense = take(8 * 64 * size_t(L.n_dslices) * rhs);
    w.total = off;
    return w;
}

// The kernels of an apply of rhs columns: the tensor-memory ones (tc.cu) where
// KernelChoice predicts less time for them than for the column-by-column ones
// below.  Their workspace must also fit the column-by-column kernels' (which
// sizes every workspace): V has a row for every component, B rows one for every
// slot, so it does unless the factor arrays hold many components of no block.
bool use_tc(const qh_matrix* m, size_t rhs) {
    return m->choice.tensor(rhs) && ws_plan(m->L, rhs, true).total <= ws_plan(m->L, rhs, false).total;
}

// Workspace of an apply with rhs columns (one column chunk's worth).
size_t ws_bytes(const Layout& L, size_t rhs) { return ws_plan(L, rhs_chunk(rhs), false).total; }

// One chain of launches for columns [c0, c0 + rhs) of x and y (leading
// dimension ld).
int launch_chunk(const qh_matrix* m, const double* x, double* y, size_t rhs, long long ld, void* ws,
                 cudaStream_t s, int* status, void* const* ev) {
    const Layout& L = m->L;
    const int n = int(L.order);
    auto* w = static_cast<uint8_t*>(ws);
    const bool tc = use_tc(m, rhs);
    const WsPlan P = ws_plan(L, rhs, tc);
    Work W;
    W.xc = reinterpret_cast<double*>(w + P.xc);
    W.xblk = reinterpret_cast<int*>(w + P.xblk);
    W.xe = reinterpret_cast<int*>(w + P.xe);
    W.xq = reinterpret_cast<uint4*>(w + P.xq);
    W.lsplit = reinterpret_cast<long long*>(w + P.lsplit);
    W.split_cnt = reinterpret_cast<int*>(w + P.cnt);
    W.blimb = reinterpret_cast<uint4*>(w + P.blimb);
    W.v = reinterpret_cast<long long*>(w + P.blimb);
    W.part = reinterpret_cast<uint4*>(w + P.part);
    W.plr = reinterpret_cast<uint4*>(w + P.plr);
    W.pdense = reinterpret_cast<double*>(w + P.pdense);
    auto mark = [&](int i) {
        if (ev) cudaEventRecord(static_cast<cudaEvent_t>(ev[i]), s);
    };
    const int irhs = int(rhs);
    mark(0);
    const int n_pad = int(padded_order(L));
    int* zero = reinterpret_cast<int*>(w + P.zero0);
    const int n_zero = int(P.zero_bytes / 4);
    cudaError_t e;
    // One cluster per column where its threads reach and all clusters fit at once
    // (two blocks per SM).  Whole applies, us, cooperative / cluster: 2048 x 1
    // 18.5 / 16.2, 2048 x 4 26.9 / 25.1, 8000 x 1 32.8 / 30.6, 8000 x 16 90.5 / 87.6;
    // two entries a thread, 12345 x 1 40.8 / 40.9; more clusters than fit,
    // 8000 x 64 309 / 313.
    if (n_pad <= kPrepCluster * kPrepThreads && kPrepCluster * irhs <= 2 * m->sms) {
        e = launch_pdl(prep_cluster_kernel, dim3(kPrepCluster, unsigned(rhs)), dim3(kPrepThreads), 0, s, m->A, W, x, n, ld,
                       zero, n_zero, status, n_pad);
    } else if (static_cast<long long>(P.nblk) * irhs <= m->prep_coop_max) {
        // one cooperative launch: prep, a grid-wide synchronisation, limbs
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(unsigned(P.nblk), unsigned(rhs));
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, prep_limbs_kernel, m->A, W, x, n, ld, L.n_chunks, zero, n_zero, status, n_pad);
    } else {
        prep_x_kernel<<<dim3(unsigned(P.nblk), unsigned(rhs)), 256, 0, s>>>(m->A, W, x, n, ld, L.n_chunks, zero,
                                                                            n_zero, status);
        e = launch_pdl(x_limbs_kernel, dim3(unsigned((n_pad + 255) / 256), unsigned(rhs)), dim3(256), 0, s, W, n,
                       n_pad, P.nblk);
    }
    mark(1);
    if (tc) {
        const TcArgs t{m->A, W, L.n_tc_items, L.n_tc_row_items, L.n_dense_units, L.n_parts, L.n_tiles, irhs, P.pv, n,
                       n_pad, L.n_split, L.n_dslices, m->sms, y, ld, status};
        struct Ctx {
            void* const* ev;
            cudaStream_t s;
        } ctx{ev, s};
        void (*record)(void*, int) = [](void* c, int i) {
            auto* x = static_cast<Ctx*>(c);
            cudaEventRecord(static_cast<cudaEvent_t>(x->ev[i]), x->s);
        };
        if (e == cudaSuccess) e = tc_launch(t, s, ev ? record : nullptr, &ctx);
    } else {
        if (e == cudaSuccess && L.n_tasks > 0)
            e = launch_pdl(column_kernel, dim3(unsigned(m->col_grid)), dim3(kWarps * 32), size_t(kColPipeSmem), s, m->A,
                           W, static_cast<const int*>(m->sched), n_pad, irhs, L.n_split, L.n_slots, n, L.n_dslices, status);
        mark(2);
        if (e == cudaSuccess && L.n_units > 0)
            e = launch_pdl(row_kernel, dim3(unsigned(m->row_grid)), dim3(kWarps * 32), size_t(kRowPipeSmem), s, m->A, W,
                           static_cast<const int*>(m->sched + m->col_grid * kWarps + 1), irhs, L.n_slots, L.n_tiles,
                           status);
        if (e == cudaSuccess)
            e = launch_pdl(combine_kernel, dim3(unsigned(L.n_tiles), unsigned(rhs)), dim3(64), 0, s, m->A, W, y,
                           L.n_tiles, L.n_dslices, ld);
    }
    if (e != cudaSuccess) return cuda_fail(e, "CUDA kernel launch");
    mark(3);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "CUDA kernel launch");
    return QH_OK;
}

// The apply: column chunks of at most kMaxRhsChunk, one chain each, in stream
// order on the same workspace (sized for one chunk).  Events (profiling) are
// recorded around the first chunk's kernels.
int launch(const qh_matrix* m, const double* x, double* y, size_t rhs, void* ws, cudaStream_t s,
           int* status, void* const* ev = nullptr) {
    for (size_t c0 = 0; c0 < rhs; c0 += kMaxRhsChunk) {
        const int rc = launch_chunk(m, x + c0, y + c0, std::min(kMaxRhsChunk, rhs - c0), (long long)rhs, ws, s,
                                    status, c0 == 0 ? ev : nullptr);
        if (rc) return rc;
    }
    return QH_OK;
}

// The reference's checks (src/qhmat/cuda.cu:108-112): a zero or
// overflowing column count is a shape mismatch; more than INT_MAX * 256
// entries is "CUDA launch grid too large".
int check_rhs(const qh_matrix* m, size_t rhs) {
    if (rhs == 0 || rhs > SIZE_MAX / m->L.order) return fail(QH_EINVAL, "right-hand-side shape mismatch");
    if (m->L.order * rhs > size_t(INT32_MAX) * 256) return fail(QH_EOVERFLOW, "CUDA launch grid too large");
    return QH_OK;
}

}  // namespace

extern "C" {

const char* qh_last_error(void) { return g_last_error.c_str(); }

int qh_cuda_built(void) { return 1; }

int qh_matrix_from_qhmat(const void* bytes, size_t len, int device, qh_matrix** out) {
    if (!out) return fail(QH_EINVAL, "output handle pointer is null");
    *out = nullptr;
    if (!bytes && len) return fail(QH_EINVAL, "image pointer is null");
    return guarded([&] {
        HostMatrix hm = parse_qhmat(static_cast<const uint8_t*>(bytes), len);
        Layout L = build_layout(hm);
        return upload(std::move(L), device, out);
    });
}

int qh_matrix_from_arrays(size_t order, const size_t* permutation, size_t block_count,
                          const qh_block_desc* blocks, const double* dense,
                          const uint32_t* left_words, const uint32_t* right_words,
                          const size_t* left_offsets, const size_t* right_offsets,
                          const double* left_scales, const double* right_scales, const int* widths,
                          int device, qh_matrix** out) {
    if (!out) return fail(QH_EINVAL, "output handle pointer is null");
    *out = nullptr;
    if (!order || !permutation || !block_count || !blocks)
        return fail(QH_EINVAL, "invalid matrix order/permutation");
    return guarded([&] {
        HostMatrix hm;
        hm.order = order;
        hm.permutation.assign(permutation, permutation + order);
        size_t n_comp = 0, n_dense = 0, lw_end = 0, rw_end = 0;
        for (size_t k = 0; k < block_count; ++k) {
            const auto& d = blocks[k];
            HostMatrix::Block b;
            b.row0 = d.row0;
            b.row1 = d.row1;
            b.col0 = d.col0;
            b.col1 = d.col1;
            b.admissible = false;
            b.dense = d.is_dense != 0;
            if (d.row1 < d.row0 || d.col1 < d.col0) throw std::invalid_argument("invalid block rectangle");
            if (b.dense) {
                b.dense_off = d.dense_offset;
                n_dense = std::max(n_dense, d.dense_offset + (d.row1 - d.row0) * (d.col1 - d.col0));
            } else {
                b.rank = d.rank;
                b.comp0 = d.factor_offset;
                n_comp = std::max(n_comp, d.factor_offset + d.rank);
                for (size_t j = 0; j < d.rank; ++j) {
                    const size_t c = d.factor_offset + j;
                    const int w = widths[c];
                    if (w < 2 || w > 32) throw std::invalid_argument("bit width must be in [2, 32]");
                    lw_end = std::max(lw_end, left_offsets[c] + ((d.row1 - d.row0) * size_t(w) + 31) / 32);
                    rw_end = std::max(rw_end, right_offsets[c] + ((d.col1 - d.col0) * size_t(w) + 31) / 32);
                }
            }
            hm.blocks.push_back(b);
        }
        if (n_dense && !dense) throw std::invalid_argument("dense values pointer is null");
        hm.dense.assign(dense, dense + n_dense);
        if (n_comp && (!widths || !left_scales || !right_scales || !left_offsets || !right_offsets ||
                       !left_words || !right_words))
            throw std::invalid_argument("factor arrays are null");
        hm.width.resize(n_comp);
        for (size_t c = 0; c < n_comp; ++c) hm.width[c] = uint8_t(widths[c]);
        hm.left_scale.assign(left_scales, left_scales + n_comp);
        hm.right_scale.assign(right_scales, right_scales + n_comp);
        hm.left_off.assign(left_offsets, left_offsets + n_comp);
        hm.right_off.assign(right_offsets, right_offsets + n_comp);
        hm.left_words.assign(left_words, left_words + lw_end);
        hm.right_words.assign(right_words, right_words + rw_end);
        validate(hm);
        Layout L = build_layout(hm);
        return upload(std::move(L), device, out);
    });
}

int qh_matrix_from_batch(const void* const* images, const size_t* lens, size_t count, int device, qh_matrix** out,
                         uint64_t* offsets) {
    if (!out) return fail(QH_EINVAL, "output handle pointer is null");
    *out = nullptr;
    if (!images || !lens || !count) return fail(QH_EINVAL, "empty batch");
    return guarded([&] {
        std::vector<HostMatrix> ms;
        ms.reserve(count);
        for (size_t k = 0; k < count; ++k) ms.push_back(parse_qhmat(static_cast<const uint8_t*>(images[k]), lens[k]));
        std::vector<uint64_t> off;
        // no padding rows: the plain layout's row tiles already stay inside
        // the row slabs of blocks (so inside one matrix), and every row of
        // the block-diagonal matrix must belong to some block
        HostMatrix S = concat_block_diagonal(ms, 1, off);
        std::vector<HostMatrix>().swap(ms);
        Layout L = build_layout(S);
        const int rc = upload(std::move(L), device, out);
        if (rc == QH_OK && offsets)
            for (size_t k = 0; k < count; ++k) offsets[k] = off[k];
        return rc;
    });
}

void qh_matrix_destroy(qh_matrix* m) { delete m; }

int qh_matrix_stats(const qh_matrix* m, qh_stats* out) {
    if (!m || !out) return fail(QH_EINVAL, "null argument");
    const Layout& L = m->L;
    out->order = L.order;
    out->block_count = uint64_t(L.n_lr) + uint64_t(L.n_dense);
    out->dense_blocks = uint64_t(L.n_dense);
    out->lowrank_blocks = uint64_t(L.n_lr);
    out->components = uint64_t(L.n_comp);
    out->code_bytes = L.code_bytes;
    out->scale_bytes = L.scale_bytes;
    out->dense_bytes = L.dense_bytes;
    out->model_bytes = L.code_bytes + L.scale_bytes + L.dense_bytes + 16 * L.order;
    out->device_bytes = L.sec.total;
    out->row_tiles = uint64_t(L.n_tiles);
    out->flops_per_rhs = L.flops;
    const WsPlan P1 = ws_plan(L, 1, false);
    out->launches_per_apply = (P1.nblk <= m->prep_coop_max ? 2 : 3) + (L.n_tasks > 0) + (L.n_units > 0);
    out->host_direct = m->host_direct ? 1 : 0;
    out->left_code_bytes = L.left_code_bytes;
    out->right_code_bytes = L.right_code_bytes;
    return QH_OK;
}

double qh_matrix_reconstruction_bound(const qh_matrix* m) { return m ? m->L.bound : 0.0; }

size_t qh_workspace_bytes(const qh_matrix* m, size_t rhs) { return m ? ws_bytes(m->L, rhs) : 0; }

int qh_matmul_device(const qh_matrix* m, const double* x, double* y, size_t rhs, void* workspace,
                     size_t workspace_bytes, void* stream, int* status) {
    return qh_matmul_device_profiled(m, x, y, rhs, workspace, workspace_bytes, stream, status, nullptr);
}

int qh_matmul_device_profiled(const qh_matrix* m, const double* x, double* y, size_t rhs, void* workspace,
                              size_t workspace_bytes, void* stream, int* status, void* const* events4) {
    if (!m) return fail(QH_EINVAL, "null matrix handle");
    int rc = check_rhs(m, rhs);
    if (rc) return rc;
    if (!x || !y) return fail(QH_EINVAL, "null right-hand side or result pointer");
    DeviceGuard g(m->device);
    const size_t need = ws_bytes(m->L, rhs);
    if (workspace) {
        if (workspace_bytes < need) return fail(QH_EINVAL, "workspace too small");
        if (reinterpret_cast<uintptr_t>(workspace) & 255) return fail(QH_EINVAL, "workspace must be 256-byte aligned");
        return launch(m, x, y, rhs, workspace, static_cast<cudaStream_t>(stream), status, events4);
    }
    auto* mm = const_cast<qh_matrix*>(m);
    std::lock_guard<std::mutex> lock(mm->mu);
    if (mm->dev_ws_bytes < need) {
        if (mm->dev_ws) cudaFree(mm->dev_ws);
        mm->dev_ws = nullptr;
        mm->dev_ws_bytes = 0;
        cudaError_t e = cudaMalloc(&mm->dev_ws, need);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc");
        mm->dev_ws_bytes = need;
    }
    return launch(m, x, y, rhs, mm->dev_ws, static_cast<cudaStream_t>(stream), status, events4);
}

int qh_matmul_device_checked(const qh_matrix* m, const double* x, double* y, size_t rhs, void* workspace,
                             size_t workspace_bytes, void* stream) {
    if (!m) return fail(QH_EINVAL, "null matrix handle");
    DeviceGuard g(m->device);
    return checked_call(
        const_cast<qh_matrix*>(m)->words, static_cast<cudaStream_t>(stream),
        [&](int* word) { return qh_matmul_device(m, x, y, rhs, workspace, workspace_bytes, stream, word); },
        [](cudaError_t e, int st, const char* what) {
            if (e != cudaSuccess) return cuda_fail(e, what);
            if (st & kStatusNonfinite) return fail(QH_EINVAL, "nonfinite right-hand side");
            return fail(QH_ERUNTIME, "device copy wait timed out");
        });
}

int qh_matmul_device_static(const qh_matrix* m, const double* x, double* y, size_t rhs, void* stream,
                            int* status) {
    if (!m) return fail(QH_EINVAL, "null matrix handle");
    int rc = check_rhs(m, rhs);
    if (rc) return rc;
    if (!x || !y) return fail(QH_EINVAL, "null right-hand side or result pointer");
    const size_t need = ws_bytes(m->L, rhs);
    if (need > size_t(QH_STATIC_SCRATCH_BYTES))
        return fail(QH_EINVAL, "qh_matmul_device_static: this apply needs " + std::to_string(need) +
                                   " bytes of scratch, more than the fixed " +
                                   std::to_string(size_t(QH_STATIC_SCRATCH_BYTES)) +
                                   " (QH_STATIC_SCRATCH_BYTES); use qh_matmul_device with a workspace");
    // Device address of the array, looked up once per device with that device
    // current (the first call on a device does this set-up; a table entry per
    // device the process sees).
    static std::mutex mu;
    static std::vector<void*> addr;
    void* ptr = nullptr;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (addr.empty()) {
            int count = 0;
            cudaError_t e = cudaGetDeviceCount(&count);
            if (e != cudaSuccess) return cuda_fail(e, "cudaGetDeviceCount");
            addr.assign(size_t(std::max(count, 0)), nullptr);
        }
        if (m->device < 0 || size_t(m->device) >= addr.size()) return fail(QH_EINVAL, "invalid CUDA device ordinal");
        DeviceGuard g(m->device);
        if (!addr[size_t(m->device)]) {
            void* p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
            if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress");
            addr[size_t(m->device)] = p;
        }
        ptr = addr[size_t(m->device)];
    }
    DeviceGuard g(m->device);
    return launch(m, x, y, rhs, ptr, static_cast<cudaStream_t>(stream), status);
}

int qh_matmul_host(const qh_matrix* m, const double* x, double* y, size_t rhs) {
    if (!m) return fail(QH_EINVAL, "null matrix handle");
    int rc = check_rhs(m, rhs);
    if (rc) return rc;
    rc = check_device(m->device);
    if (rc) return rc;
    if (!x || !y) return fail(QH_EINVAL, "null right-hand side or result pointer");
    auto* mm = const_cast<qh_matrix*>(m);
    DeviceGuard g(m->device);
    std::lock_guard<std::mutex> lock(mm->mu);
    cudaError_t e;
    if (!mm->stream) {
        e = cudaStreamCreateWithFlags(&mm->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) return cuda_fail(e, "cudaStreamCreate");
    }
    if (!mm->d_status) {
        e = cudaMalloc(&mm->d_status, sizeof(int));
        if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc");
        e = cudaMallocHost(&mm->h_status, sizeof(int));
        if (e != cudaSuccess) return cuda_fail(e, "cudaMallocHost");
    }
    const size_t vec = m->L.order * rhs * sizeof(double);
    const size_t need_ws = ws_bytes(m->L, rhs);
    const auto* xb = reinterpret_cast<const uint8_t*>(x);
    const auto* yb = reinterpret_cast<const uint8_t*>(y);
    if (m->host_direct && (xb + vec <= yb || yb + vec <= xb)) {
        // the kernels read x and write y in the caller's memory directly
        // (each page of y is written once here first, so that the device
        // never touches an unpopulated page)
        if (mm->own_ws_bytes < need_ws) {
            if (mm->own_ws) cudaFree(mm->own_ws);
            mm->own_ws = nullptr;
            mm->own_ws_bytes = 0;
            e = cudaMalloc(&mm->own_ws, need_ws);
            if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc");
            mm->own_ws_bytes = need_ws;
        }
        {
            // one write per page makes every page of y present and writable
            static const uintptr_t page = uintptr_t(sysconf(_SC_PAGESIZE) > 0 ? sysconf(_SC_PAGESIZE) : 4096);
            const uintptr_t y0 = reinterpret_cast<uintptr_t>(y), y1 = y0 + vec;
            for (uintptr_t a = y0; a < y1; a = (a & ~(page - 1)) + page) *reinterpret_cast<volatile uint8_t*>(a) = 0;
        }
        // the status word is the pinned host int itself (device-accessible at
        // the same address under unified addressing): no memset and no copy
        // back on the stream
        volatile int* hs = mm->h_status;
        *hs = 0;
        rc = launch(m, x, y, rhs, mm->own_ws, mm->stream, mm->h_status);
        if (rc) return rc;
        if ((e = cudaStreamSynchronize(mm->stream)) != cudaSuccess) return cuda_fail(e, "CUDA kernel execution");
        const int st = *hs;
        if (st & kStatusNonfinite) return fail(QH_EINVAL, "nonfinite right-hand side");
        if (st & kStatusTimeout) return fail(QH_ERUNTIME, "device copy wait timed out");
        return QH_OK;
    }
    // one device buffer: workspace | x | y
    const size_t need = align256(need_ws) + 2 * align256(vec);
    if (mm->own_ws_bytes < need) {
        if (mm->own_ws) cudaFree(mm->own_ws);
        mm->own_ws = nullptr;
        mm->own_ws_bytes = 0;
        e = cudaMalloc(&mm->own_ws, need);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc");
        mm->own_ws_bytes = need;
    }
    if (mm->pinned_bytes < vec) {
        if (mm->pinned) cudaFreeHost(mm->pinned);
        mm->pinned = nullptr;
        mm->pinned_bytes = 0;
        e = cudaMallocHost(&mm->pinned, vec);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMallocHost");
        mm->pinned_bytes = vec;
    }
    auto* base = static_cast<uint8_t*>(mm->own_ws);
    double* dx = reinterpret_cast<double*>(base + align256(need_ws));
    double* dy = reinterpret_cast<double*>(base + align256(need_ws) + align256(vec));
    std::memcpy(mm->pinned, x, vec);
    if ((e = cudaMemsetAsync(mm->d_status, 0, sizeof(int), mm->stream)) != cudaSuccess)
        return cuda_fail(e, "cudaMemsetAsync");
    if ((e = cudaMemcpyAsync(dx, mm->pinned, vec, cudaMemcpyHostToDevice, mm->stream)) != cudaSuccess)
        return cuda_fail(e, "cudaMemcpy host-to-device");
    rc = launch(m, dx, dy, rhs, base, mm->stream, mm->d_status);
    if (rc) return rc;
    if ((e = cudaMemcpyAsync(mm->pinned, dy, vec, cudaMemcpyDeviceToHost, mm->stream)) != cudaSuccess)
        return cuda_fail(e, "cudaMemcpy device-to-host");
    if ((e = cudaMemcpyAsync(mm->h_status, mm->d_status, sizeof(int), cudaMemcpyDeviceToHost, mm->stream)) !=
        cudaSuccess)
        return cuda_fail(e, "cudaMemcpy device-to-host");
    if ((e = cudaStreamSynchronize(mm->stream)) != cudaSuccess) return cuda_fail(e, "CUDA kernel execution");
    if (*mm->h_status & kStatusNonfinite) return fail(QH_EINVAL, "nonfinite right-hand side");
    if (*mm->h_status & kStatusTimeout) return fail(QH_ERUNTIME, "device copy wait timed out");
    std::memcpy(y, mm->pinned, vec);
    return QH_OK;
}

int qh_debug_wait_timeout(int device, int polls) {
    if (polls < 1 || polls > (1 << 20)) return fail(QH_EINVAL, "polls must be in [1, 2^20]");
    int rc = check_device(device);
    if (rc) return rc;
    DeviceGuard g(device);
    // status words: the streaming kernels' wait, the two warps of the
    // tensor-memory kernels'; then which lanes of those gave up
    constexpr int kWords = 3 + 64;
    int* d = nullptr;
    cudaError_t e = cudaMalloc(&d, kWords * sizeof(int));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc");
    int h[kWords] = {};
    e = cudaMemset(d, 0, kWords * sizeof(int));
    if (e == cudaSuccess) {
        wait_timeout_kernel<<<1, 32>>>(polls, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = tc_debug_give_up(polls, d + 1, d + 3);
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return cuda_fail(e, "debug wait");
    // (the warp that was told to give up has not run out of its own tests)
    if (std::count(h + 3, h + kWords, 1) != 64 || h[1] != kStatusTimeout || h[2] != 0)
        return fail(QH_ECUDA, "a block did not give up as a whole");
    if (h[0] & kStatusTimeout) return fail(QH_ERUNTIME, "device copy wait timed out");
    return QH_OK;
}

int qh_matrix_reconstruct(const qh_matrix* m, double* out, size_t out_count, int out_on_device) {
    if (!m) return fail(QH_EINVAL, "null matrix handle");
    const size_t n = m->L.order;
    if (n > SIZE_MAX / n / sizeof(double)) return fail(QH_EOVERFLOW, "dense output size overflow");
    if (!out || out_count != n * n) return fail(QH_EINVAL, "output size does not match order * order");
    return guarded([&] {
        DeviceGuard g(m->device);
        const int n_lr = m->L.n_lr, nb = n_lr + m->L.n_dense;
        // blocks' tiles and factors (component-major)
        std::vector<DenseOut> blocks(static_cast<size_t>(nb));
        long long tiles = 0, ltotal = 0, rtotal = 0;
        size_t area = 0;  // entries inside the blocks, which do not overlap
        auto tiles_of = [](long long rows, long long cols) {
            return ((rows + kDenseTile - 1) / kDenseTile) * ((cols + kDenseTile - 1) / kDenseTile);
        };
        for (int b = 0; b < nb; ++b) {
            blocks[size_t(b)] = {tiles, ltotal, rtotal};
            if (b < n_lr) {
                const LowRankDesc& d = m->lr[size_t(b)];
                ltotal += (long long)d.rank * d.m;
                rtotal += (long long)d.rank * d.n;
                tiles += tiles_of(d.m, d.n);
                area += size_t(d.m) * size_t(d.n);
            } else {
                const DenseDesc& d = m->dd[size_t(b - n_lr)];
                tiles += tiles_of(d.m, d.n);
                area += size_t(d.m) * size_t(d.n);
            }
        }
        if (tiles > INT32_MAX) return fail(QH_EOVERFLOW, "CUDA launch grid too large");
        // one allocation (separate ones were slower at every order): factors,
        // bases, blocks, and the output if on the host
        const size_t parts[5] = {4 * size_t(ltotal), 4 * size_t(rtotal), 16 * size_t(m->L.n_comp),
                                 sizeof(DenseOut) * size_t(nb), out_on_device ? 0 : 8 * n * n};
        size_t at[5], bytes = 0;
        for (int i = 0; i < 5; ++i) {
            at[i] = bytes;
            bytes += align256(std::max<size_t>(parts[i], 1));
        }
        struct Scratch {
            uint8_t* p = nullptr;
            ~Scratch() {
                if (p) cudaFree(p);
            }
        } buf;
        if (cudaMalloc(&buf.p, bytes) != cudaSuccess) return fail(QH_ERUNTIME, "cudaMalloc: out of device memory");
        auto* left = reinterpret_cast<int*>(buf.p + at[0]);
        auto* right = reinterpret_cast<int*>(buf.p + at[1]);
        auto* lb = reinterpret_cast<long long*>(buf.p + at[2]);
        auto* rb = lb + m->L.n_comp;
        auto* d_blocks = reinterpret_cast<DenseOut*>(buf.p + at[3]);
        double* d_out = out_on_device ? out : reinterpret_cast<double*>(buf.p + at[4]);
        cudaError_t e = cudaMemcpy(d_blocks, blocks.data(), sizeof(DenseOut) * blocks.size(), cudaMemcpyHostToDevice);
        // the blocks of one matrix cover it; those of a block-diagonal handle
        // (qh_matrix_from_batch) do not, and what lies outside them is zero
        if (e == cudaSuccess && area < n * n) e = cudaMemsetAsync(d_out, 0, 8 * n * n, nullptr);
        if (e == cudaSuccess && n_lr) {
            factor_base_kernel<<<unsigned(n_lr), 32>>>(m->A, n_lr, d_blocks, lb, rb);
            e = launch_decode(m->A, m->L.n_tasks, rb, right, m->L.n_units, lb, left);
        }
        if (e == cudaSuccess && tiles) {
            reconstruct_kernel<<<unsigned(tiles), 128>>>(m->A, n_lr, nb, d_blocks, left, right, int(n), d_out);
            e = cudaGetLastError();
        }
        // (while the device works.  Before the allocation, its mappings and the
        // page faults held each other up: 1.4 ms more.  Only pageable memory, whose
        // pages may be absent, and only if the copy will follow: a pointer that
        // the host may not touch is the copy's to judge.)
        if (e == cudaSuccess && !out_on_device) {
            cudaPointerAttributes at{};
            if (cudaPointerGetAttributes(&at, out) != cudaSuccess) cudaGetLastError();
            else if (at.type == cudaMemoryTypeUnregistered) PagePopulator(out, 8 * n * n).wait();
        }
        if (e == cudaSuccess)
            e = out_on_device ? cudaDeviceSynchronize() : cudaMemcpy(out, d_out, 8 * n * n, cudaMemcpyDeviceToHost);
        return e == cudaSuccess ? QH_OK : cuda_fail(e, "reconstruct");
    });
}

int qh_debug_decode(const qh_matrix* m, int side, int32_t* out, size_t out_count, size_t* needed) {
    if (!m) return fail(QH_EINVAL, "null matrix handle");
    if (side != 0 && side != 1) return fail(QH_EINVAL, "side must be 0 (left) or 1 (right)");
    return guarded([&] {
        // Block offsets into the output, from the host copy of the descriptors.
        DeviceGuard g(m->device);
        std::vector<LowRankDesc> lr(size_t(m->L.n_lr));
        cudaError_t e;
        if (!lr.empty()) {
            e = cudaMemcpy(lr.data(), m->A.lr, sizeof(LowRankDesc) * lr.size(), cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpy device-to-host");
        }
        // component-major output: component c's codes start at off[c]; the
        // kernels index left codes by clustered row (base off[c] - row0) and
        // right codes by block column (base off[c])
        std::vector<long long> off(size_t(m->L.n_comp) + 1, 0);
        for (const auto& d : lr)
            for (int j = 0; j < d.rank; ++j)
                off[size_t(d.comp0 + j) + 1] = side == 0 ? d.m : d.n;
        for (size_t c = 0; c + 1 < off.size(); ++c) off[c + 1] += off[c];
        const size_t total = size_t(off.back());
        if (side == 0)
            for (const auto& d : lr)
                for (int j = 0; j < d.rank; ++j) off[size_t(d.comp0 + j)] -= d.row0;
        if (needed) *needed = total;
        if (!out) return QH_OK;
        if (out_count != total) return fail(QH_EINVAL, "output size does not match the code count");
        if (!total) return QH_OK;
        long long* d_off = nullptr;
        int* d_out = nullptr;
        if ((e = cudaMalloc(&d_off, sizeof(long long) * off.size())) != cudaSuccess) return cuda_fail(e, "cudaMalloc");
        if ((e = cudaMalloc(&d_out, sizeof(int) * total)) != cudaSuccess) {
            cudaFree(d_off);
            return cuda_fail(e, "cudaMalloc");
        }
        int rc = QH_OK;
        e = cudaMemcpy(d_off, off.data(), sizeof(long long) * off.size(), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) {
            e = launch_decode(m->A, side == 1 ? m->L.n_tasks : 0, d_off, d_out, side == 0 ? m->L.n_units : 0, d_off,
                                   d_out);
        }
        if (e == cudaSuccess) e = cudaMemcpy(out, d_out, sizeof(int) * total, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) rc = cuda_fail(e, "debug decode");
        cudaFree(d_off);
        cudaFree(d_out);
        return rc;
    });
}

}  // extern "C"
