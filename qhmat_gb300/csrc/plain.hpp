// Device side shared by the kernels of the plain (exact integer) form: the
// resident arena and scratch views, bulk copies, bounded waits, the digit and
// limb operands of the f16 tensor-core products, and the fixed-point helpers.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/qhmat_gb300.h"
#include "layout.hpp"
#include "pdl.hpp"

namespace qhg {

struct Arena {
    const int32_t* perm;   // clustered position -> source index
    const int32_t* iperm;  // source index -> clustered position
    const LowRankDesc* lr;
    const DenseDesc* dd;
    const ColTask* tasks;
    const TaskRec* task_rec;
    const uint8_t* qcodes;
    const uint8_t* pcodes;
    const double* dense;
    const RowTile* tiles;
    const TileDense* tdense;
    const RowUnit* units;
    const uint8_t* kp_info;
    const SlotRec* slot_rec;
    const TaskDest* task_dest;
    const uint32_t* row_steps;
    const double* comp_sl;  // s^P per component
    const double* comp_sr;  // s^Q per component
    const TcItem* tc_items;
    const TcTask* tc_tasks;
    const DenseUnit* dense_units;
    const TcRowItem* tc_row_items;
    const TcStep* tc_steps;
};

struct Work {
    double* xc;        // [rhs][n]            x in clustered order (FP64)
    int* xblk;         // [rhs][nblk]         largest exponent field of x per prep block
    int* xe;           // [rhs]               largest exponent field of x
    uint4* xq;         // [rhs][n_pad]        limbs of X (zero past n)
    long long* lsplit; // [rhs][n_split*33][8] per-limb sums sum_i c_ij limb_l(X_i) of split tasks'
                       //                     components (rows split_id*33 + j; zeroed by prep)
    int* split_cnt;    // [rhs][n_split]      finished parts of each split task (zeroed by prep)
    uint4* blimb;      // [rhs][n_slots]      row-side B rows: limbs of U (column by column)
    long long* v;      // [n_comp][pv]        u in fixed point (tensor-memory kernels; the same memory)
    uint4* part;       // [rhs][n_parts][128] 128-bit row sums of each row item (tensor-memory kernels)
    uint4* plr;        // [rhs][n_tiles][kTileUnits][16] low-rank row sums of each row unit (128-bit)
    double* pdense;    // [rhs][n_dslices][64] dense diagonal row sums per dense slice
};

namespace {

// Fixed point: x (per rhs column) and u (per row tile) are held as integers
// X = round(v * 2^(kFixBits - (e - 1022))), |X| <= 2^kFixBits, on one exponent
// field e; the tensor-core operand is X's eight base-256 limbs, all signed (-128 ..
// 127, the top one -64 .. 64), each an exact f16.
constexpr int kFixBits = 62;


// ---------------------------------------------------------------- helpers

// Biased IEEE exponent field; 0 for zero/subnormal.  |v| < 2^(e - 1022).
__device__ __forceinline__ int exp_field(double v) {
    return int((__double_as_longlong(v) >> 52) & 0x7FF);
}

// round(v * 2^(kFixBits - (emax - 1022))) as an integer, computed with integer
// operations only (the FP64 pipe is the scarce one).  emax must be >= the
// exponent field of v; subnormals give 0.
__device__ __forceinline__ long long to_fixed(double v, int emax) {
    const long long bits = __double_as_longlong(v);
    const int e = int((bits >> 52) & 0x7FF);
    if (e == 0) return 0;
    const long long mant = (bits & 0xFFFFFFFFFFFFFLL) | 0x10000000000000LL;
    const int rs = emax - e + (1075 - 1022 - kFixBits);  // right shift, >= 53 - kFixBits
    long long q;
    if (rs <= 0) q = mant << (-rs);
    else q = rs >= 62 ? 0 : ((mant + (1LL << (rs - 1))) >> rs);
    return bits < 0 ? -q : q;
}

// V = round(t s 2^-beta) of a component (TaskRec), t its 128-bit sum.
__device__ __forceinline__ long long comp_fixed(__int128 t, int shift, unsigned long long kappa) {
    const __int128 r = t + (__int128)(1ull << (shift - 1));
    const unsigned long long a =
        ((unsigned long long)r >> shift) | ((unsigned long long)(long long)(r >> 64) << (64 - shift));
    // signed a times unsigned kappa: the high 64 bits, rounded
    const unsigned long long hi = __umul64hi(a, kappa) - ((long long)a < 0 ? kappa : 0ull);
    return (long long)(hi + ((a * kappa) >> 63));
}
// U = V on a tile's coarser fixed point: round(V 2^-shift), shift in 0 .. 63.
__device__ __forceinline__ long long tile_fixed(long long v, int shift) {
    return (v + (long long)((1ull << shift) >> 1)) >> shift;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ uint32_t hsub2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// The eight limbs of X (|X| <= 2^62) as f16 values, limb k in half k:
// X = sum_{k<7} l_k 2^(8k) + l_7 2^56 with l_0..l_6 in [-128, 127] and l_7 in
// [-64, 64].  The bytes of X + 2^62 + 128 (1 + 2^8 + .. + 2^48) are those
// limbs plus 128, the top one plus 64; byte b becomes the f16 1024 + b
// (exponent bits 0x64 above it) and then the limb by one exact subtraction per
// pair.
__device__ __forceinline__ uint4 to_limbs(long long X) {
    const unsigned long long Y = (unsigned long long)X + 0x4080808080808080ull;
    const uint32_t lo = uint32_t(Y), hi = uint32_t(Y >> 32);
    return make_uint4(hsub2(prmt(lo, 0x64646464u, 0x4140u), 0x64806480u),
                      hsub2(prmt(lo, 0x64646464u, 0x4342u), 0x64806480u),
                      hsub2(prmt(hi, 0x64646464u, 0x4140u), 0x64806480u),
                      hsub2(prmt(hi, 0x64646464u, 0x4342u), 0x64406480u));
}

// -------------------------------------------------- bulk copies (TMA)

__device__ __forceinline__ unsigned smem_u32(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
// Arrive once and expect `bytes` more bytes of transactions on this phase.
__device__ __forceinline__ void mbar_arrive_expect(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// Potentially blocking test of a phase: the thread waits until the phase
// completes or a system-dependent time limit passes (measured faster than an
// explicit suspend-time hint, which delays the wake-up).
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up (returns false) after `limit` tests (kWaitLimit: about
// 16 seconds) instead of hanging; callers record the failure in the
// status word, stop issuing copies, give the copies already issued one more
// bounded wait each and return (best effort: a copy still outstanding after
// that wait is abandoned with the block).  Of a whole warp, whose lanes agree at
// every test: a lane that gave up alone would leave the others waiting for it at
// their next warp-wide instruction, without a limit.
constexpr int kWaitLimit = 1 << 22;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, int limit = kWaitLimit) {
    for (int i = 0; i < limit; ++i)
        if (__all_sync(0xFFFFFFFFu, mbar_try_wait(bar, parity))) return true;
    return false;
}
// Order this thread's (and, after a warp barrier, its warp's) earlier generic
// accesses to shared memory before later asynchronous-proxy writes to it.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// One-dimensional bulk copy global -> shared (16-byte aligned, bytes % 16 == 0),
// completing on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Status bits written by the kernels (status word of the apply).
constexpr int kStatusNonfinite = QH_STATUS_NONFINITE;
constexpr int kStatusTimeout = QH_STATUS_TIMEOUT;

__device__ __forceinline__ void flag_timeout(int* status) {
    if (status) atomicOr(status, kStatusTimeout);
}

// round(v * 2^k) for a 128-bit integer v, as a double, with integer
// operations only (round to nearest even; results outside the normal range
// take the slow path).
__device__ __forceinline__ double i128_ldexp(__int128 v, int k) {
    if (v == 0) return 0.0;
    const bool neg = v < 0;
    const unsigned __int128 a = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
    const unsigned long long hi = (unsigned long long)(a >> 64), lo = (unsigned long long)a;
    const int nbits = hi ? 128 - __clzll(hi) : 64 - __clzll(lo);
    unsigned long long mant;
    int e;
    if (nbits <= 53) {
        mant = lo << (53 - nbits);
        e = nbits - 53;
    } else {
        const int sh = nbits - 53;
        const unsigned __int128 q = a >> sh;
        const unsigned __int128 rem = a - (q << sh);
        const unsigned __int128 half = (unsigned __int128)1 << (sh - 1);
        mant = (unsigned long long)q;
        if (rem > half || (rem == half && (mant & 1))) ++mant;
        e = sh;
        if (mant >> 53) {
            mant >>= 1;
            ++e;
        }
    }
    const int E = e + k + 52 + 1023;
    if (E <= 0 || E >= 2047) return scalbn(neg ? -double(mant) : double(mant), e + k);
    const unsigned long long bits =
        ((unsigned long long)neg << 63) | ((unsigned long long)E << 52) | (mant & 0xFFFFFFFFFFFFFULL);
    return __longlong_as_double((long long)bits);
}

__device__ __forceinline__ __int128 shfl_xor_i128(__int128 v, int m) {
    const long long lo = __shfl_xor_sync(0xFFFFFFFFu, (long long)v, m);
    const long long hi = __shfl_xor_sync(0xFFFFFFFFu, (long long)(v >> 64), m);
    return ((__int128)hi << 64) | (unsigned long long)lo;
}

// ------------------------------------------------- tensor-core fragments
//
// A digit d enters the MMA as the f16 bit pattern d, i.e. the subnormal
// d * 2^-24, so a byte or nibble becomes an operand with one permute (bytes)
// or one shift-and-mask (nibbles); products with the normal-f16 limbs are
// exact and every accumulator value is an integer times 2^-24 below 1, exact
// in FP32.

// Byte group word (digits of entries 2t, 2t+1, 2t+8, 2t+9): the f16 pairs of
// entries (2t, 2t+1) and (2t+8, 2t+9).
__device__ __forceinline__ uint32_t dig_lo(uint32_t w) { return prmt(w, 0u, 0x4140u); }
__device__ __forceinline__ uint32_t dig_hi(uint32_t w) { return prmt(w, 0u, 0x4342u); }
// Nibble group word: pair k = (nibble k, nibble k + 4); k = 0, 1 are k-block
// 0's pairs (2t, 2t+1) and (2t+8, 2t+9), k = 2, 3 k-block 1's.
__device__ __forceinline__ uint32_t nib_pair(uint32_t v, int k) { return (v >> (4 * k)) & 0x000F000Fu; }

// d += A * B for one 16x8x16 step (A: rows g, g+8 x k 2t.., 2t+8..).
__device__ __forceinline__ void mma_dig(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// B fragments of two k-blocks from 32 rows of 16 bytes (limbs of 32 entries
// or components) at a 16-byte-aligned shared address: lane l points at row l.
__device__ __forceinline__ void limb_frags(uint32_t row_addr, uint32_t (&b)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                 : "r"(row_addr)
                 : "memory");
}

// One group (rows g and g+8 of a 16-row fragment pair of k-blocks, in
// shared memory at grp) into d.  Byte rows are 32 bytes, nibble rows 16; rows
// >= `rows` are zero.  Plain loads (ordered after the stage's mbarrier wait,
// which clobbers memory) and non-volatile MMAs leave the compiler free to
// overlap one group's loads with the previous group's MMAs.
__device__ __forceinline__ void group_mma(float (&d)[4], const uint8_t* grp, bool nib, int rows, int g, int t,
                                          const uint32_t (&b)[4]) {
    if (nib) {
        const uint32_t v0 = g < rows ? *reinterpret_cast<const uint32_t*>(grp + g * 16 + 4 * t) : 0u;
        const uint32_t v1 = g + 8 < rows ? *reinterpret_cast<const uint32_t*>(grp + (g + 8) * 16 + 4 * t) : 0u;
        mma_dig(d, nib_pair(v0, 0), nib_pair(v1, 0), nib_pair(v0, 1), nib_pair(v1, 1), b[0], b[1]);
        mma_dig(d, nib_pair(v0, 2), nib_pair(v1, 2), nib_pair(v0, 3), nib_pair(v1, 3), b[2], b[3]);
    } else {
        const uint2 w0 = g < rows ? *reinterpret_cast<const uint2*>(grp + g * 32 + 8 * t) : make_uint2(0u, 0u);
        const uint2 w1 =
            g + 8 < rows ? *reinterpret_cast<const uint2*>(grp + (g + 8) * 32 + 8 * t) : make_uint2(0u, 0u);
        mma_dig(d, dig_lo(w0.x), dig_lo(w1.x), dig_hi(w0.x), dig_hi(w1.x), b[0], b[1]);
        mma_dig(d, dig_lo(w0.y), dig_lo(w1.y), dig_hi(w0.y), dig_hi(w1.y), b[2], b[3]);
    }
}

// The top plane of a column task: stored digits s = d + 2^(t-1) become the
// signed digit d as a normal f16 (1024 + s, minus hb = 1024 + 2^(t-1) in both
// halves), so no offset correction is needed on the column side.
__device__ __forceinline__ uint32_t top_lo(uint32_t w, uint32_t hb) { return hsub2(prmt(w, 0x64646464u, 0x4140u), hb); }
__device__ __forceinline__ uint32_t top_hi(uint32_t w, uint32_t hb) { return hsub2(prmt(w, 0x64646464u, 0x4342u), hb); }
__device__ __forceinline__ uint32_t top_nib(uint32_t v, int k, uint32_t hb) {
    return hsub2(nib_pair(v, k) | 0x64006400u, hb);
}
__device__ __forceinline__ void group_mma_top(float (&d)[4], const uint8_t* grp, bool nib, int rows, int g, int t,
                                              const uint32_t (&b)[4], uint32_t hb) {
    // rows past `rows` contribute zero: their operands are forced to +0.0
    const bool in0 = g < rows, in1 = g + 8 < rows;
    if (nib) {
        const uint32_t v0 = in0 ? *reinterpret_cast<const uint32_t*>(grp + g * 16 + 4 * t) : 0u;
        const uint32_t v1 = in1 ? *reinterpret_cast<const uint32_t*>(grp + (g + 8) * 16 + 4 * t) : 0u;
        uint32_t a[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            a[k] = in0 ? top_nib(v0, k, hb) : 0u;
            a[4 + k] = in1 ? top_nib(v1, k, hb) : 0u;
        }
        mma_dig(d, a[0], a[4], a[1], a[5], b[0], b[1]);
        mma_dig(d, a[2], a[6], a[3], a[7], b[2], b[3]);
    } else {
        const uint2 w0 = in0 ? *reinterpret_cast<const uint2*>(grp + g * 32 + 8 * t) : make_uint2(0u, 0u);
        const uint2 w1 = in1 ? *reinterpret_cast<const uint2*>(grp + (g + 8) * 32 + 8 * t) : make_uint2(0u, 0u);
        const uint32_t a0 = in0 ? top_lo(w0.x, hb) : 0u, a2 = in0 ? top_hi(w0.x, hb) : 0u;
        const uint32_t a4 = in0 ? top_lo(w0.y, hb) : 0u, a6 = in0 ? top_hi(w0.y, hb) : 0u;
        const uint32_t a1 = in1 ? top_lo(w1.x, hb) : 0u, a3 = in1 ? top_hi(w1.x, hb) : 0u;
        const uint32_t a5 = in1 ? top_lo(w1.y, hb) : 0u, a7 = in1 ? top_hi(w1.y, hb) : 0u;
        mma_dig(d, a0, a1, a2, a3, b[0], b[1]);
        mma_dig(d, a4, a5, a6, a7, b[2], b[3]);
    }
}

// The top plane of a row k-pair: stored digits s = d + 2^(t-1) become the
// signed digit d on the lower planes' scale, d 2^-24 (a subnormal f16 for
// |d| < 1024): the f16 with exponent field 1 and mantissa s is (1024 + s)
// 2^-24, minus hb = (1024 + 2^(t-1)) 2^-24 in both halves, exactly.
__device__ __forceinline__ uint32_t rtop_lo(uint32_t w, uint32_t hb) { return hsub2(prmt(w, 0x04040404u, 0x4140u), hb); }
__device__ __forceinline__ uint32_t rtop_hi(uint32_t w, uint32_t hb) { return hsub2(prmt(w, 0x04040404u, 0x4342u), hb); }
__device__ __forceinline__ uint32_t rtop_nib(uint32_t v, int k, uint32_t hb) {
    return hsub2(nib_pair(v, k) | 0x04000400u, hb);
}
__device__ __forceinline__ void group_mma_rtop(float (&d)[4], const uint8_t* grp, bool nib, int g, int t,
                                               const uint32_t (&b)[4], uint32_t hb) {
    if (nib) {
        const uint32_t v0 = *reinterpret_cast<const uint32_t*>(grp + g * 16 + 4 * t);
        const uint32_t v1 = *reinterpret_cast<const uint32_t*>(grp + (g + 8) * 16 + 4 * t);
        mma_dig(d, rtop_nib(v0, 0, hb), rtop_nib(v1, 0, hb), rtop_nib(v0, 1, hb), rtop_nib(v1, 1, hb), b[0], b[1]);
        mma_dig(d, rtop_nib(v0, 2, hb), rtop_nib(v1, 2, hb), rtop_nib(v0, 3, hb), rtop_nib(v1, 3, hb), b[2], b[3]);
    } else {
        const uint2 w0 = *reinterpret_cast<const uint2*>(grp + g * 32 + 8 * t);
        const uint2 w1 = *reinterpret_cast<const uint2*>(grp + (g + 8) * 32 + 8 * t);
        mma_dig(d, rtop_lo(w0.x, hb), rtop_lo(w1.x, hb), rtop_hi(w0.x, hb), rtop_hi(w1.x, hb), b[0], b[1]);
        mma_dig(d, rtop_lo(w0.y, hb), rtop_lo(w1.y, hb), rtop_hi(w0.y, hb), rtop_hi(w1.y, hb), b[2], b[3]);
    }
}

// Digits of rows g, g+8 of a group as integers, in the order the MMA sees
// them (for validation): out[half][kb*4 + s], s = entries 2t, 2t+1, 2t+8, 2t+9.
__device__ __forceinline__ void group_digits(const uint8_t* grp, bool nib, int rows, int g, int t,
                                             uint32_t (&out)[2][8]) {
    uint32_t r[2][4];  // [half][kb0 lo, kb0 hi, kb1 lo, kb1 hi]
    if (nib) {
        const uint32_t v0 = g < rows ? *reinterpret_cast<const uint32_t*>(grp + g * 16 + 4 * t) : 0u;
        const uint32_t v1 = g + 8 < rows ? *reinterpret_cast<const uint32_t*>(grp + (g + 8) * 16 + 4 * t) : 0u;
        for (int k = 0; k < 4; ++k) {
            r[0][k] = nib_pair(v0, k);
            r[1][k] = nib_pair(v1, k);
        }
    } else {
        const uint2 w0 = g < rows ? *reinterpret_cast<const uint2*>(grp + g * 32 + 8 * t) : make_uint2(0u, 0u);
        const uint2 w1 =
            g + 8 < rows ? *reinterpret_cast<const uint2*>(grp + (g + 8) * 32 + 8 * t) : make_uint2(0u, 0u);
        r[0][0] = dig_lo(w0.x), r[0][1] = dig_hi(w0.x), r[0][2] = dig_lo(w0.y), r[0][3] = dig_hi(w0.y);
        r[1][0] = dig_lo(w1.x), r[1][1] = dig_hi(w1.x), r[1][2] = dig_lo(w1.y), r[1][3] = dig_hi(w1.y);
    }
    for (int hh = 0; hh < 2; ++hh)
        for (int k = 0; k < 4; ++k) {
            // pair k: k-block k >> 1, slots (2(k&1), 2(k&1) + 1)
            out[hh][(k >> 1) * 4 + 2 * (k & 1)] = r[hh][k] & 0xFFFFu;
            out[hh][(k >> 1) * 4 + 2 * (k & 1) + 1] = r[hh][k] >> 16;
        }
}
// Entry (within a 32-entry k-pair) of slot s of k-block kb for thread t.
__device__ __forceinline__ int slot_entry(int kb, int s, int t) { return 16 * kb + 2 * t + (s & 1) + 8 * (s >> 1); }

// Exact integers sum(D * 2^24) of a plane's accumulators, folded into 64-bit
// sums at weight 2^(8m).
__device__ __forceinline__ long long fold(float d, int m) {
    return (long long)__float2int_rn(d * 16777216.0f) << (8 * m);
}

__device__ __forceinline__ void st_i128(uint4* p, __int128 v) {
    *p = make_uint4(uint32_t(v), uint32_t(v >> 32), uint32_t(v >> 64), uint32_t(v >> 96));
}
__device__ __forceinline__ __int128 ld_i128(const uint4* p) {
    const uint4 v = __ldcg(p);
    return (__int128)(((unsigned __int128)v.w << 96) | ((unsigned __int128)v.z << 64) |
                      ((unsigned __int128)v.y << 32) | v.x);
}

// A row k-pair's info byte: planes | nibble top plane << 3 | (top bits - 1) << 4.
// Bytes of its digit groups, and the top plane's conversion constant.
__device__ __forceinline__ int kp_bytes(int info) { return (info & 7) * 512 - ((info >> 3) & 1) * 256; }
__device__ __forceinline__ uint32_t kp_hb(int info) { return (0x0400u | (1u << (info >> 4))) * 0x00010001u; }

}  // namespace
}  // namespace qhg
