// The plain (exact integer) form on the 5th-generation tensor cores.
//
// Digits x limbs of matvec.cu's numerics, with tcgen05.mma: the A operand is
// 128 rows of one digit plane x 64 entries (f16, written to shared memory by
// converter warps from the resident digit bytes, which bulk copies bring in),
// the B operand the eight limbs of up to eight right-hand-side columns of
// those 64 entries (N = 8 R), the accumulators FP32 in tensor memory.  A
// digit is converted once per R columns, a B operand is shared by 128 rows,
// and no warp waits on its own loads:
//
//   tc_column_kernel  rows = components of up to four tasks that share a column
//                     range and a number of planes, one accumulator per plane;
//                     V (TaskRec) is written once per component and column.
//   tc_row_kernel     rows = 64 (or 32) rows of a tile x 2 (or 4) planes;
//                     builder warps gather V and write its limbs on the tile's
//                     exponent; 128-bit row sums per item.
//   tc_combine_kernel adds a tile's items and dense row sums: y.
//
// What bounds them: not memory (16384 unknowns x 16 columns read 88 MB of codes
// in 186 us) nor the MMAs (a quarter of the issuing lane's time at 64
// columns), but the instructions of the roles between: digits -> f16 (about
// 0.8 per digit, once per R columns), V -> limbs, and the 64-bit fold of the
// sums; per step of two A tiles a handshake of each role.  Measured against
// the column-by-column kernels (device us): 16384 unknowns x 16 columns 556 ->
// 186, 8192 (3-D) x 64 columns 2654 -> 565, 2048 x 4 43 -> 28.  Tried and
// slower: one handshake per A tile (782 at 64 columns), register prefetch of V
// instead of asynchronous copies, three stages, waiting warps that sleep or
// wait on a leader.  B operands of 16 columns in the column kernel gave 3 % at
// 16 and 64 columns and lost 6 % at 24: the drains' work goes with the columns.
//
// Sums: an accumulator takes at most 128 entries, each product below 2^15 in
// magnitude times 2^-24, so it is an integer below 2^22 times 2^-24, exact (the
// MMA drops bits 2^-24 of an accumulator near 1: measured with sums that
// start at 0.75).  Adding 0.75 afterwards keeps it in [0.5, 1), where FP32 holds
// integers times 2^-24: its bits minus those of 0.75 are the sum, with no
// conversion instruction.  Limb pairs, planes and limbs are then
// combined in 32-, 64- and 128-bit integers; the integers do not depend on the
// split, so y is the same bit for bit whatever the number of columns.
#include "tc.hpp"

#include <algorithm>

#include "tcgen05.hpp"

namespace qhg {
namespace tc {
namespace {

// Warpgroups (four warps each) of both kernels: 0 issues the copies (warp 0
// codes, warp 2 x limbs of the column kernel) and the MMAs (warp 1); 1 and 2
// convert digits, taking steps in turn; in the column kernel 3 does the dense
// diagonal (FP64) and 4 .. 7 drain tensor memory (lane quarter = warp & 3),
// sharing the columns; in the row kernel 3 and 6 build the U limbs, taking
// steps in turn, and 4 and 5 drain.  Work moves in steps of at
// most two A tiles, with one barrier round and one MMA commit per step.  The
// launch's 64 registers a thread are split between them (512 in all).
constexpr int kThreads = 32 * 32;
struct ColRegs {
    static constexpr int kIssue = 40, kConvert = 56, kDrain = 72, kSide = 72;
    static_assert(kIssue + 2 * kConvert + 4 * kDrain + kSide <= 8 * 64, "register split");
};
struct RowRegs {
    static constexpr int kIssue = 56, kConvert = 56, kDrain = 96, kSide = 64, kIdle = 24;
    static_assert(kIssue + 2 * kConvert + 2 * kDrain + 2 * kSide + kIdle <= 8 * 64, "register split");
};

// Stages of raw digits and B, and of A tiles (both even: a converter group must
// see every phase of the barriers it waits on).
constexpr int kStages = 4, kColAStages = 4, kRowAStages = 2;
constexpr int kATile = 128 * 64 * 2;
constexpr int kAStage = 2 * kATile;
constexpr int kRawStage = 4 * 4096;          // four tasks (M-tiles) of at most 4 KB a step
constexpr int kAccStride = 256;              // two accumulator sets

template <int R>
struct Cfg {
    static_assert(R == 4 || R == 8, "columns at once");
    static constexpr int N = 8 * R;                      // MMA N
    static constexpr int kBCol = 64 * 16 + 16;           // B stage: [column][entry][8 limbs], columns padded (the
    static constexpr int kB = R * kBCol;                 // builders write several column pairs at once)
    static constexpr int kSplits = 4;                    // drain warpgroups
    static constexpr int kPer = R / kSplits;             // columns of each
    static constexpr int kRowSplits = 2;                 // the same for the row kernel, which needs more builders
    static constexpr int kRowPer = R / kRowSplits;
    static constexpr int kPairs = R / 2;                 // builder threads per slot, two columns each
    static constexpr int kSlots = kPairs / 2;            // slots of each (32 apart): 128 threads, 64 slots
    // row kernel: V and the slots' records on their way to a builder group, four
    // steps of each
    static constexpr int kVRing = 4 * kSlots * 128 * 16, kRecRing = 4 * kSlots * 128 * 8;
};
template <int R, int ASTAGES, bool ROW>
struct Smem {
    static constexpr int kAStages = ASTAGES;
    static constexpr int kOffRaw = ASTAGES * kAStage;
    static constexpr int kOffB = kOffRaw + kStages * kRawStage;
    static constexpr int kOffV = (kOffB + kStages * Cfg<R>::kB + 127) & ~127;
    static constexpr int kOffRec = kOffV + (ROW ? 2 * Cfg<R>::kVRing : 0);
    static constexpr int kBytes = kOffRec + (ROW ? 2 * Cfg<R>::kRecRing : 0) + 1024;
};
template <int R>
using ColSmem = Smem<R, kColAStages, false>;
template <int R>
using RowSmem = Smem<R, kRowAStages, true>;
static_assert(ColSmem<8>::kBytes <= 226 * 1024 && RowSmem<8>::kBytes <= 226 * 1024, "shared memory");

struct Bars {
    uint64_t raw_full[kStages], raw_empty[kStages];
    uint64_t a_full[kStages], b_full[kStages];
    uint64_t done[kStages];  // a step's MMAs have read its A tiles and B stage
    uint64_t acc_full[2], acc_empty[2];
    uint64_t drain;
    // What the code producer says of each step and the MMA issuer of each
    // segment, so that the roles between them walk no descriptors.  A step
    // word lives until the step's MMAs are done: eight slots (the producer is
    // at most eight steps ahead of those).
    uint32_t step[2 * kStages];
    int task[kStages][4];    // column kernel: the tasks' info words
    uint32_t segment[2];
    uint32_t tmem;
    int abort_flag;
};
// Step words: column kernel planes | chunks << 4 | last of its item << 8;
// row kernel info bytes | kSegmentEnd | kItemEnd | 64-row tile << 24.  Segment
// words: accumulators in use | last of its item << 8.
constexpr uint32_t kNoMore = 0xFFFFFFFFu;

__device__ __forceinline__ void init_bars(Bars& S, int b_writers, int drainers) {
    for (int i = 0; i < kStages; ++i) {
        mbar_init(&S.raw_full[i], 4);
        mbar_init(&S.raw_empty[i], 4);
        mbar_init(&S.a_full[i], 4);
        mbar_init(&S.b_full[i], b_writers);
        mbar_init(&S.done[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
        mbar_init(&S.acc_full[i], 2);
        mbar_init(&S.acc_empty[i], drainers);
    }
    mbar_init(&S.drain, 1);
    S.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// This CTA's (item, column block) pairs, items costliest first: rounds of one
// pair per CTA in alternating order, a pair's index being item * groups +
// group.  Advanced by precomputed steps (no division).
struct Pairs {
    int item, group, n_items, groups;
    int q[2], r[2], odd;
    __device__ __forceinline__ Pairs(int n, int g) : n_items(n), groups(g), odd(0) {
        const int ctas = int(gridDim.x), b = int(blockIdx.x);
        const int s0 = 2 * (ctas - 1 - b) + 1, s1 = 2 * b + 1;
        item = b / g, group = b % g;
        q[0] = s0 / g, r[0] = s0 % g;
        q[1] = s1 / g, r[1] = s1 % g;
    }
    __device__ __forceinline__ bool valid() const { return item < n_items; }
    __device__ __forceinline__ int some() const { return min(item, n_items - 1); }  // an item that exists
    __device__ __forceinline__ void next() {
        item += odd ? q[1] : q[0];
        group += odd ? r[1] : r[0];
        odd ^= 1;
        if (group >= groups) group -= groups, ++item;
    }
};

// B operand in the layout of the limb rows themselves (16 bytes = the limbs of
// one column and entry): N-major, no swizzle; 8-entry groups 128 bytes apart,
// columns `col` bytes apart.
__device__ __forceinline__ uint64_t limb_desc(uint32_t addr, uint32_t col) {
    uint64_t d = 0;
    d |= uint64_t((addr & 0x3FFFFu) >> 4);
    d |= uint64_t(128 >> 4) << 16;
    d |= uint64_t(col >> 4) << 32;
    d |= uint64_t(1) << 46;
    return d;
}

__device__ __forceinline__ void mma_add(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.eq.b32 p, 0, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc)
        : "memory");
}
// The MMAs of one step: M accumulators N columns apart, KS steps of 16 entries
// (k outermost: an MMA that adds to its predecessor's accumulator waits for
// it).  Accumulator m reads A at m * STRIDE (in 16-byte units) + odd half
// offsets HALF of its parity.  Unrolled with constant offsets, an MMA issues
// at the tensor core's own rate (40 cycles for N = 16, 48 for 64: shared-memory
// reads); with offsets computed per MMA it took 150 - 300.
template <int M, int KS, int N, int STRIDE, int HALF>
__device__ __forceinline__ void mma_step(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int accumulate) {
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const uint64_t am = a + uint64_t(HALF ? (m >> 1) * STRIDE + (m & 1) * HALF : m * STRIDE) + 2 * k;
            if (k == 0) mma_f16(d + m * N, am, b, idesc, accumulate);
            else mma_add(d + m * N, am, b + 16 * k, idesc);
        }
}

template <int N>
__device__ __forceinline__ void set_regs() {
    if constexpr (N < 64) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
    if constexpr (N > 64) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

template <int C>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[C]) {
    if constexpr (C == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr)
                     : "memory");
    } else if constexpr (C == 16) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr)
            : "memory");
    } else {
        static_assert(C == 32, "columns");
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr)
            : "memory");
    }
}

// v[r][t] += weight (E + kBias), E the exact sum of limbs 2t, 2t + 1 of column r
// (limb 2t + 1 times 256).  Adding 0.75 to an accumulator S 2^-24 gives the
// bits 0x3F400000 + S; the pair's bits combine to E + 257 * 0x3F400000 mod 2^32
// = E + kBias, and as |E| < 2^30 that is an unsigned 32-bit number: one
// unsigned multiply-add into 64 bits.  The biases are taken off at the end
// (join_limbs).
constexpr unsigned kBias = 0x7F400000u;
// (128 entries of digits up to 255 times limbs up to 128: adding 0.75 stays in [0.5, 1))
static_assert(128 * 255 * 128 < 1 << 22, "sums of an accumulator");
template <int PER>
__device__ __forceinline__ void add_sums(unsigned long long (&v)[PER][4], const uint32_t (&d)[8 * PER],
                                         unsigned weight) {
#pragma unroll
    for (int r = 0; r < PER; ++r)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const unsigned e = __float_as_uint(__uint_as_float(d[8 * r + 2 * t]) + 0.75f) +
                               (__float_as_uint(__uint_as_float(d[8 * r + 2 * t + 1]) + 0.75f) << 8);
            v[r][t] += (unsigned long long)e * weight;
        }
}
// The sums without their biases (`weights`: the sum of all weights added).
__device__ __forceinline__ long long pair_sum(unsigned long long v, unsigned long long weights) {
    return (long long)(v - weights * kBias);
}
__device__ __forceinline__ __int128 join_limbs(const unsigned long long (&v)[4], unsigned long long weights) {
    const unsigned long long b = weights * kBias;
    return (__int128)(long long)(v[0] - b) + ((__int128)(long long)(v[1] - b) << 16) +
           ((__int128)(long long)(v[2] - b) << 32) + ((__int128)(long long)(v[3] - b) << 48);
}

// comp_fixed (plain.hpp) of a component's columns: what does not depend on the
// column (the biases and the rounding of the first shift, as one 128-bit
// number) is made once, and the sums stay unsigned.  About half the
// instructions of comp_fixed(join_limbs(..)) a column; the drains' instructions
// are what the column kernel waits for (8192 unknowns (3-D) x 64: 327 -> 318 us).
struct CompScale {
    unsigned __int128 add;
    unsigned long long kappa;
    int shift;  // 1 .. 63
    __device__ __forceinline__ CompScale(unsigned long long weights, int shift_, unsigned long long kappa_)
        : kappa(kappa_), shift(shift_) {
        const unsigned __int128 b = weights * kBias;
        add = (unsigned __int128)(1ull << (shift - 1)) - (b + (b << 16) + (b << 32) + (b << 48));
    }
    __device__ __forceinline__ long long operator()(const unsigned long long (&v)[4]) const {
        const unsigned __int128 r = add + v[0] + ((unsigned __int128)v[1] << 16) + ((unsigned __int128)v[2] << 32) +
                                    ((unsigned __int128)v[3] << 48);
        const uint32_t w0 = uint32_t(r), w1 = uint32_t(r >> 32), w2 = uint32_t(r >> 64), w3 = uint32_t(r >> 96);
        const bool far = shift >= 32;  // (a funnel shift takes its low five bits)
        const uint32_t lo = __funnelshift_r(far ? w1 : w0, far ? w2 : w1, uint32_t(shift));
        const uint32_t hi = __funnelshift_r(far ? w2 : w1, far ? w3 : w2, uint32_t(shift));
        const unsigned long long a = ((unsigned long long)hi << 32) | lo;
        // signed a times unsigned kappa: the high 64 bits, rounded
        const unsigned __int128 p = (unsigned __int128)a * kappa;
        const unsigned long long q = (unsigned long long)(p >> 64) - (int(hi) < 0 ? kappa : 0ull);
        return (long long)(q + ((unsigned long long)p >> 63));
    }
};

// Half a tile row: 32 digits of one plane (shared address `src`, fragment
// order: 32 bytes, or 16 for a nibble plane) as f16 operands d 2^-24 in the
// four 16-byte chunks at `dst` ^ 16 j (the swizzle's low bits are in dst).  A
// lower digit is the subnormal f16 with its own bits; a signed top digit s - h
// is f16 (1024 + s) 2^-24 (exponent field 1) minus sub = (1024 + h) 2^-24.
enum PlaneKind { kLowerPlane, kTopPlane, kTopNibbles };
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void convert_half(uint32_t dst, uint32_t src, PlaneKind kind, uint32_t sub) {
    const uint4 a = lds128(src);
    if (kind == kTopNibbles) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            sts128(dst ^ (16 * k), rtop_nib(a.x, k, sub), rtop_nib(a.y, k, sub), rtop_nib(a.z, k, sub),
                   rtop_nib(a.w, k, sub));
        return;
    }
    const uint4 b = lds128(src + 16);
    if (kind == kLowerPlane) {
        sts128(dst, dig_lo(a.x), dig_lo(a.z), dig_lo(b.x), dig_lo(b.z));
        sts128(dst ^ 16, dig_hi(a.x), dig_hi(a.z), dig_hi(b.x), dig_hi(b.z));
        sts128(dst ^ 32, dig_lo(a.y), dig_lo(a.w), dig_lo(b.y), dig_lo(b.w));
        sts128(dst ^ 48, dig_hi(a.y), dig_hi(a.w), dig_hi(b.y), dig_hi(b.w));
    } else {
        sts128(dst, rtop_lo(a.x, sub), rtop_lo(a.z, sub), rtop_lo(b.x, sub), rtop_lo(b.z, sub));
        sts128(dst ^ 16, rtop_hi(a.x, sub), rtop_hi(a.z, sub), rtop_hi(b.x, sub), rtop_hi(b.z, sub));
        sts128(dst ^ 32, rtop_lo(a.y, sub), rtop_lo(a.w, sub), rtop_lo(b.y, sub), rtop_lo(b.w, sub));
        sts128(dst ^ 48, rtop_hi(a.y, sub), rtop_hi(a.w, sub), rtop_hi(b.y, sub), rtop_hi(b.w, sub));
    }
}
// Offset of half 0 of tile row `row`, first chunk (half 1: ^ 64).
__device__ __forceinline__ uint32_t row_offset(int row) {
    return uint32_t((row >> 3) * 1024 + (row & 7) * 128 + ((row & 7) << 4));
}

__device__ __forceinline__ TcTask load_task(const TcTask* p) {
    const uint4 a = ahead128(p), b = ahead128(reinterpret_cast<const uint4*>(p) + 1);
    TcTask t;
    t.off = (long long)(((unsigned long long)a.y << 32) | a.x);
    t.stride = int(a.z), t.comp_idx = int(a.w);
    t.info = int(b.x), t.split = int(b.y), t.nparts = int(b.z), t.pad = 0;
    return t;
}
__device__ __forceinline__ TcItem load_item(const TcItem* p) {
    const uint4 a = ahead128(p);
    return TcItem{int(a.x), int(a.y), int(a.z), int(a.w)};
}

// 16 columns of a dense diagonal block part x 32 tile rows x two right-hand
// sides: FP64, columns in order.
__device__ __forceinline__ void dense_part(const Arena& A, const Work& W, const DenseUnit& u, int half, int p0, int rhs,
                                           int n, int n_dslices, int lane) {
    const int row = lane + 32 * half, rows = __ldg(&A.tiles[u.tile].rows);
    if (32 * half >= rows) return;
    const int p1 = min(p0 + 1, rhs - 1);
    const bool in = row < rows;
    const TileDense D = A.tdense[u.tdense];
    const double* col = A.dense + D.off + (long long)u.k0 * D.ld + row;
    const double* x0 = W.xc + (long long)p0 * n + D.xcol + u.k0;
    const double* x1 = W.xc + (long long)p1 * n + D.xcol + u.k0;
    double s0 = 0.0, s1 = 0.0;
    int k = 0;
    for (; k + 8 <= u.cols; k += 8) {
        double c[8], a[8], b[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            c[i] = in ? __ldg(col + (long long)(k + i) * D.ld) : 0.0;
            a[i] = __ldcg(x0 + k + i);
            b[i] = __ldcg(x1 + k + i);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) s0 = fma(c[i], a[i], s0);
        if (p1 != p0)
#pragma unroll
            for (int i = 0; i < 8; ++i) s1 = fma(c[i], b[i], s1);
    }
    for (; k < u.cols; ++k) {
        const double c = in ? __ldg(col + (long long)k * D.ld) : 0.0;
        s0 = fma(c, __ldcg(x0 + k), s0);
        if (p1 != p0) s1 = fma(c, __ldcg(x1 + k), s1);
    }
    double* out = W.pdense + (long long)u.slice * 64 + row;
    out[(long long)p0 * n_dslices * 64] = s0;
    if (p1 != p0) out[(long long)p1 * n_dslices * 64] = s1;
}

// ------------------------------------------------------------ column kernel

// Chunks (32 entries) of one step of an item with P planes: at most two tiles,
// a tile holding two (plane, chunk) halves.
__device__ __forceinline__ int step_chunks(int P) { return P <= 2 ? 2 : 1; }

template <int R>
__global__ void __launch_bounds__(kThreads, 1)
    tc_column_kernel(Arena A, Work W, int n_items, int groups, int n_dense, int rhs, int pv, int n, int n_pad,
                     int n_split, int n_dslices, int* status) {
    using C = Cfg<R>;
    using M = ColSmem<R>;
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* const sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    __shared__ Bars S;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wg = warp >> 2;
    pdl_trigger();
    if (threadIdx.x == 0) init_bars(S, 1, 4 * C::kSplits);
    if (warp == 1) tmem_alloc(&S.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem;
    volatile int* abort_flag = &S.abort_flag;

    if (wg == 0) set_regs<ColRegs::kIssue>();
    if (warp == 0) {
        // ---- codes: per step the chunks of task `lane` (descriptors one item ahead)
        if (lane < 4) {
            unsigned ri = 0;
            bool ok = true;
            Pairs w(n_items, groups);
            TcItem I{}, In{};
            TcTask T{}, Tn{};
            auto load = [&](TcItem& i, TcTask& t) {
                i = load_item(A.tc_items + w.some());
                t = load_task(A.tc_tasks + 4 * w.some() + lane);
            };
            if (w.valid()) load(In, Tn);
            while (w.valid() && ok) {
                I = In, T = Tn;
                w.next();
                load(In, Tn);
                const int P = I.info & 255, kc0 = step_chunks(P);
                for (int b = 0; b < I.nchunks; b += kc0, ++ri) {
                    const int s = ri % kStages, kc = min(kc0, I.nchunks - b);
                    if (ri >= kStages) ok = wait_bar(&S.raw_empty[s], ((ri / kStages) - 1) & 1, abort_flag, status);
                    if (!ok) break;
                    S.task[s][lane] = T.info;
                    if (lane == 0) S.step[ri % (2 * kStages)] = uint32_t(P | kc << 4 | (b + kc0 >= I.nchunks) << 8);
                    mbar_expect(&S.raw_full[s], unsigned(kc * T.stride));
                    if (T.stride)
                        bulk_g2s(sm + M::kOffRaw + s * kRawStage + lane * 4096, A.qcodes + T.off + (long long)b * T.stride,
                                 unsigned(kc * T.stride), &S.raw_full[s]);
                }
            }
            // the end, for both converter groups
            for (int i = 0; i < 2 && ok; ++i, ++ri) {
                const int s = ri % kStages;
                if (ri >= kStages) ok = wait_bar(&S.raw_empty[s], ((ri / kStages) - 1) & 1, abort_flag, status);
                if (lane == 0) S.step[ri % (2 * kStages)] = kNoMore;
                mbar_arrive(&S.raw_full[s]);
            }
            if (!ok)  // copies still in flight after an abort: wait for them (bounded)
                for (unsigned k = ri > kStages ? ri - kStages : 0; k < ri; ++k)
                    for (int i = 0; i < kWaitLimit && !mbar_try(&S.raw_full[k % kStages], (k / kStages) & 1); ++i) {}
        }
    } else if (warp == 2) {
        // ---- x limbs of each step: lane = column (one lane issuing them all was
        // the kernel's slowest role at eight columns)
        pdl_wait();
        unsigned bi = 0;
        bool ok = true;
        Pairs w(n_items, groups);
        TcItem I{}, In{};
        if (w.valid()) In = load_item(A.tc_items + w.item);
        while (w.valid() && ok) {
            I = In;
            const int kc0 = step_chunks(I.info & 255);
            // (columns past the last repeat it; their V is not read)
            const uint4* x = W.xq + (long long)min(w.group * R + lane, rhs - 1) * n_pad + I.col0 + I.chunk0 * kColChunk;
            w.next();
            In = load_item(A.tc_items + w.some());
            for (int b = 0; b < I.nchunks; b += kc0, ++bi, x += kc0 * kColChunk) {
                const int s = bi % kStages, kc = min(kc0, I.nchunks - b);
                if (bi >= kStages) ok = wait_bar(&S.done[s], ((bi / kStages) - 1) & 1, abort_flag, status);
                if (!__all_sync(0xFFFFFFFFu, ok)) {
                    ok = false;
                    break;
                }
                if (lane == 0) mbar_expect(&S.b_full[s], unsigned(R * kc * 512));
                __syncwarp();
                if (lane < R)
                    bulk_g2s(sm + M::kOffB + s * C::kB + lane * C::kBCol, x, unsigned(kc * 512), &S.b_full[s]);
            }
        }
        if (!ok && lane == 0)
            for (unsigned k = bi > kStages ? bi - kStages : 0; k < bi; ++k)
                for (int i = 0; i < kWaitLimit && !mbar_try(&S.b_full[k % kStages], (k / kStages) & 1); ++i) {}
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer (one lane): segments of at most four chunks of an item,
        // each into the next of two accumulator sets (plane m at columns m N)
        if (elect_one()) {
            constexpr uint32_t idesc = mma_idesc(C::N) | (1u << 16);  // B is N-major
            constexpr int kTile = kATile >> 4;
            const uint64_t b0 = limb_desc(smem_u32(sm + M::kOffB), C::kBCol), a0 = sw128_desc(smem_u32(sm));
            unsigned seg = 0;
            int chunks = 0;  // of the current segment
            bool ok = true;
            for (unsigned ri = 0; ok; ++ri) {
                const int s = ri % kStages, buf = seg & 1;
                const unsigned ph = (ri / kStages) & 1;
                ok = wait_bar(&S.a_full[s], ph, abort_flag, status);
                if (!ok) break;
                const uint32_t word = *reinterpret_cast<volatile uint32_t*>(&S.step[ri % (2 * kStages)]);
                if (word == kNoMore) break;
                const int P = int(word & 15u), kc = int(word >> 4) & 15;
                if (chunks == 0 && seg >= 2) ok = wait_bar(&S.acc_empty[buf], ((seg >> 1) - 1) & 1, abort_flag, status);
                ok = ok && wait_bar(&S.b_full[s], ph, abort_flag, status);
                if (!ok) break;
                tc_fence_after();
                const uint64_t b = b0 + uint64_t(s * (C::kB >> 4)), a = a0 + uint64_t(int(ri % M::kAStages) * (kAStage >> 4));
                const uint32_t d = tmem + uint32_t(buf * kAccStride);
                switch (P * 2 + kc) {
                    case 3: mma_step<1, 2, C::N, kTile, 0>(d, a, b, idesc, chunks); break;
                    case 4: mma_step<1, 4, C::N, kTile, 0>(d, a, b, idesc, chunks); break;
                    case 5: mma_step<2, 2, C::N, kTile, 0>(d, a, b, idesc, chunks); break;
                    case 6: mma_step<2, 4, C::N, kTile, 0>(d, a, b, idesc, chunks); break;
                    case 7: mma_step<3, 2, C::N, kTile, 4>(d, a, b, idesc, chunks); break;
                    default: mma_step<4, 2, C::N, kTile, 4>(d, a, b, idesc, chunks); break;
                }
                mma_commit(&S.done[s]);
                chunks += kc;
                const bool end = (word >> 8) & 1u;
                if (end || chunks >= 4) {
                    S.segment[buf] = uint32_t(P) | uint32_t(end) << 8;
                    mbar_arrive(&S.acc_full[buf]);
                    mma_commit(&S.acc_full[buf]);
                    chunks = 0;
                    ++seg;
                }
            }
            mma_commit(&S.drain);
            for (int i = 0; i < kWaitLimit && !mbar_try(&S.drain, 0); ++i) {}
        }
        __syncwarp();
    } else if (wg == 1 || wg == 2) {
        // ---- converters: warp = task, lane = its row; group takes every other step
        set_regs<ColRegs::kConvert>();
        const int sub = warp & 3;
        const int q = lane >> 4, rr = lane & 15;
        const uint32_t smem0 = smem_u32(sm), row0 = row_offset(32 * sub + lane);
        for (unsigned ri = unsigned(wg - 1);; ri += 2) {
            const int s = ri % kStages;
            const unsigned ph = (ri / kStages) & 1;
            if (!warp_wait(&S.raw_full[s], ph, abort_flag, status)) break;
            const unsigned used = ri - M::kAStages;  // the step whose A stage this one takes
            const uint32_t word = *reinterpret_cast<volatile uint32_t*>(&S.step[ri % (2 * kStages)]);
            const int info = *reinterpret_cast<volatile int*>(&S.task[s][sub]);
            if (ri >= M::kAStages && !warp_wait(&S.done[used % kStages], (used / kStages) & 1, abort_flag, status)) break;
            if (word != kNoMore) {
                // (rows past the task's components convert whatever bytes are
                // there: finite values in accumulator rows that nothing reads)
                const int P = int(word & 15u), kc = int(word >> 4) & 15, count = info & 255;
                const int tb = (info >> 8) - 8 * (P - 1);
                const bool nibtop = tb <= 4;
                const uint32_t topsub = 0x04000400u + (1u << (max(tb, 1) - 1)) * 0x00010001u;
                const int row_bytes = (P - 1) * 32 + (nibtop ? 16 : 32);
                const int plane = max(0, min(16, count - 16 * q)) * 32;  // bytes from plane to plane
                const uint32_t src0 = smem0 + uint32_t(M::kOffRaw + s * kRawStage + sub * 4096 + q * 16 * row_bytes + rr * 32);
                const uint32_t top0 = src0 + uint32_t((P - 1) * plane - (nibtop ? rr * 16 : 0));
                const uint32_t tile = smem0 + (ri % M::kAStages) * uint32_t(kAStage) + row0;
                // halves i = 0, 1, ..: (plane, chunk) of a two-chunk step, planes
                // of a one-chunk step; half i & 1 of tile i >> 1.  One compact
                // loop: unrolled, the instruction fetches cost more than the work
                const int two = P <= 2 ? 1 : 0, halves = P << two;
#pragma unroll 1
                for (int i = 0; i < halves; ++i) {
                    const int m = i >> two, c = i & two;
                    if (c >= kc) continue;
                    const bool top = m == P - 1;
                    convert_half((tile + uint32_t(i >> 1) * kATile) ^ uint32_t((i & 1) << 6),
                                 (top ? top0 : src0 + uint32_t(m * plane)) + uint32_t(c * count * row_bytes),
                                 !top ? kLowerPlane : nibtop ? kTopNibbles : kTopPlane, topsub);
                }
                fence_async_smem();
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&S.a_full[s]);
                mbar_arrive(&S.raw_empty[s]);
            }
            if (word == kNoMore) break;
        }
    } else if (wg >= 4) {
        // ---- drain: warp quarter = task, lane = component
        set_regs<ColRegs::kDrain>();
        const int sub = warp & 3, e = wg - 4;
        unsigned seg = 0;
        bool ok = true;
        Pairs w(n_items, groups), wn = w;
        // tasks two items ahead, the components' records one
        TcTask T, Tn{0, 0, 0, 0, -1, 1, 0}, Tnn = Tn;
        uint4 rec_nx = make_uint4(0u, 0x100u, 0u, 0u);
        auto load_rec = [&](const TcTask& t) {
            rec_nx = ahead128(A.task_rec + t.comp_idx + min(lane, max((t.info & 255) - 1, 0)));
        };
        auto load_ahead = [&]() {
            wn.next();
            Tnn = load_task(A.tc_tasks + 4 * wn.some() + sub);
        };
        if (w.valid()) {
            Tn = load_task(A.tc_tasks + 4 * w.item + sub);
            load_rec(Tn);
            load_ahead();
        }
        for (; w.valid(); w.next()) {
            T = Tn;
            const uint4 rec = rec_nx;
            Tn = Tnn;
            load_rec(Tn);
            load_ahead();
            const int c0 = w.group * R + e * C::kPer, count = T.info & 255;
            unsigned long long v[C::kPer][4], weights = 0;
#pragma unroll
            for (int r = 0; r < C::kPer; ++r)
#pragma unroll
                for (int t = 0; t < 4; ++t) v[r][t] = 0;
            for (bool end = false; !end; ++seg) {
                const int buf = seg & 1;
                ok = warp_wait(&S.acc_full[buf], (seg >> 1) & 1, abort_flag, status);
                if (!ok) break;
                __syncwarp();
                tc_fence_after();
                const uint32_t word = *reinterpret_cast<volatile uint32_t*>(&S.segment[buf]);
                end = (word >> 8) & 1u;
                const int P = int(word & 15u);
                // (always the set's columns: no item has more planes than a set holds.
                // Without the test ptxas keeps both sets' addresses and spills sums:
                // 8192 unknowns (3-D) x 64, column kernel 318 us instead of 293)
                const int set = P <= kAccStride / C::N ? buf * kAccStride : 0;
                const uint32_t base = tmem + (uint32_t(32 * sub) << 16) + uint32_t(set + e * 8 * C::kPer);
                if (count > 0)
#pragma unroll 1
                    for (int m = 0; m < P; ++m) {
                        uint32_t d[8 * C::kPer];
                        tmem_ld<8 * C::kPer>(base + uint32_t(m * C::N), d);
                        tmem_wait_ld();
                        add_sums<C::kPer>(v, d, 1u << (8 * m));
                        weights += 1u << (8 * m);
                    }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.acc_empty[buf]);
            }
            if (!ok) break;
            if (count == 0) continue;
            const int shift = int((rec.y >> 8) & 255u);
            const unsigned long long kappa = ((unsigned long long)rec.w << 32) | rec.z;
            long long* out = W.v + (long long)int(rec.x) * pv + c0;
            if (T.nparts == 1) {
                const CompScale fixed(weights, max(shift, 1), kappa);
                long long u[C::kPer];
#pragma unroll
                for (int r = 0; r < C::kPer; ++r) u[r] = fixed(v[r]);
                if (lane < count && c0 < pv) {
                    if constexpr (C::kPer == 1) out[0] = u[0];
                    else *reinterpret_cast<longlong2*>(out) = make_longlong2(u[0], u[1]);
                }
                continue;
            }
            // a part of a split task: its limb-pair sums, as low and high
            // 32 bits, added exactly with atomics; the warp whose part
            // finishes last completes V
            if (c0 >= rhs) continue;
            long long* const blk = W.lsplit + ((long long)T.split * 33 + lane) * 8;
            const long long blk_col = (long long)n_split * 33 * 8;
            if (lane < count)
#pragma unroll
                for (int r = 0; r < C::kPer; ++r)
                    if (c0 + r < rhs)
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            const long long p = pair_sum(v[r][t], weights);
                            auto* dst = reinterpret_cast<unsigned long long*>(blk + (c0 + r) * blk_col + 2 * t);
                            atomicAdd(dst, (unsigned long long)(p & 0xFFFFFFFFll));
                            atomicAdd(dst + 1, (unsigned long long)(p >> 32));
                        }
            __threadfence();
            __syncwarp();
            int done = 0;
            if (lane == 0) done = atomicAdd(W.split_cnt + (long long)(c0 / C::kPer) * n_split + T.split, 1);
            done = __shfl_sync(0xFFFFFFFFu, done, 0);
            if (done != T.nparts - 1) continue;
            __threadfence();
            if (lane < count)
#pragma unroll
                for (int r = 0; r < C::kPer; ++r)
                    if (c0 + r < rhs) {
                        const long long* src = blk + (c0 + r) * blk_col;
                        __int128 sum = 0;
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            sum += ((__int128)__ldcg(src + 2 * t) + ((__int128)__ldcg(src + 2 * t + 1) << 32))
                                   << (16 * t);
                        out[r] = comp_fixed(sum, shift, kappa);
                    }
        }
    } else if (wg == 3) {
        // ---- dense diagonal: units x tile halves x pairs of columns, dealt
        // out over every CTA's four dense warps
        set_regs<ColRegs::kSide>();
        pdl_wait();
        const int dw = warp & 3;
        const int pairs = (rhs + 1) / 2;
        const long long parts = (long long)n_dense * 2 * pairs;
        for (long long i = (long long)dw * gridDim.x + blockIdx.x; i < parts; i += 4ll * gridDim.x) {
            const long long uh = i / pairs;
            const int4* q = reinterpret_cast<const int4*>(A.dense_units + (uh >> 1));
            const int4 a = __ldg(q);
            DenseUnit u{a.x, a.y, a.z, a.w, __ldg(&A.dense_units[uh >> 1].cols), {0, 0, 0}};
            dense_part(A, W, u, int(uh & 1), 2 * int(i % pairs), rhs, n, n_dslices, lane);
        }
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_free(tmem, 512);
}

// --------------------------------------------------------------- row kernel

__device__ __forceinline__ TcStep load_step(const TcStep* p) {
    const uint4 a = ahead128(p), b = ahead128(reinterpret_cast<const uint4*>(p) + 1);
    return TcStep{{a.x, a.y, a.z, a.w}, int(b.x), int(b.y), b.z, 0u};
}
// The part a builder needs.
__device__ __forceinline__ TcStep load_slots(const TcStep* p) {
    const uint2 b = ahead64(reinterpret_cast<const uint2*>(p) + 2);
    return TcStep{{0u, 0u, 0u, 0u}, int(b.x), int(b.y), 0u, 0u};
}
__device__ __forceinline__ TcRowItem load_row_item(const TcRowItem* p) {
    const uint4 a = ahead128(p);
    return TcRowItem{int(a.x), int(a.y), int(a.z), int(a.w)};
}

// Walk of this CTA's row items by a whole warp: lane i holds step i of the
// current run of up to 32 steps of an item, and the next run is loaded
// meanwhile (a step's descriptor loaded when its turn comes costs an L2 round
// trip per step).
template <bool CODES>
struct StepRuns {
    Pairs w, wn;      // current pair, and the one after the next
    TcRowItem I, In, Inn;
    TcStep s, sn;     // this lane's step of the current and of the next run
    int base, lane;
    bool has_next;    // In is an item

    __device__ __forceinline__ TcStep load(const Arena& A, const TcRowItem& i, int b) const {
        const TcStep* p = A.tc_steps + i.step0 + min(b + lane, i.nsteps - 1);
        return CODES ? load_step(p) : load_slots(p);
    }
    __device__ __forceinline__ void ahead(const Arena& A) {
        const bool same = base + 32 < I.nsteps || !has_next;
        TcRowItem i = same ? I : In;
        sn = load(A, i, same ? base + 32 : 0);
    }
    __device__ __forceinline__ void fetch(const Arena& A) {
        wn.next();
        Inn = load_row_item(A.tc_row_items + wn.some());
    }
    __device__ __forceinline__ StepRuns(const Arena& A, int n_items, int groups, int lane_)
        : w(n_items, groups), wn(w), base(0), lane(lane_), has_next(false) {
        I = In = Inn = TcRowItem{0, 0, 64, 0};
        s = sn = TcStep{{0u, 0u, 0u, 0u}, 0, 0, 0u, 0u};
        if (!w.valid()) return;
        I = load_row_item(A.tc_row_items + w.item);
        fetch(A);
        has_next = wn.valid();
        In = Inn;
        s = load(A, I, 0);
        ahead(A);
        fetch(A);
    }
    __device__ __forceinline__ bool valid() const { return w.valid(); }
    __device__ __forceinline__ int count() const { return min(32, I.nsteps - base); }
    __device__ __forceinline__ void next(const Arena& A) {
        s = sn;
        base += 32;
        if (base >= I.nsteps) {
            base = 0;
            w.next();
            I = In, In = Inn;
            has_next = wn.valid();
            ahead(A);
            fetch(A);
        } else {
            ahead(A);
        }
    }
};

template <int R>
__global__ void __launch_bounds__(kThreads, 1)
    tc_row_kernel(Arena A, Work W, int n_items, int groups, int rhs, int pv, int n_parts, int* status) {
    using C = Cfg<R>;
    using M = RowSmem<R>;
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* const sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    __shared__ Bars S;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wg = warp >> 2;
    pdl_trigger();
    if (threadIdx.x == 0) init_bars(S, 4, 4 * C::kRowSplits);
    if (warp == 1) tmem_alloc(&S.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem;
    volatile int* abort_flag = &S.abort_flag;

    if (wg == 0) set_regs<RowRegs::kIssue>();
    if (warp == 0) {
        // ---- codes: per step the two k-pairs of M-tile `lane`
        unsigned ri = 0;
        bool ok = true;
        for (StepRuns<true> st(A, n_items, groups, lane); st.valid() && ok; st.next(A)) {
            const int qrows = st.I.shape >> 8, count = st.count();
            const uint32_t shape = uint32_t((st.I.shape & 255) >> 6) << 24;
            const bool has = lane < qrows;
            for (int k = 0; k < count; ++k, ++ri) {
                const int s = ri % kStages;
                const uint32_t info = __shfl_sync(0xFFFFFFFFu, st.s.info, k);
                const uint32_t q0 = __shfl_sync(0xFFFFFFFFu, st.s.code[0], k), q1 = __shfl_sync(0xFFFFFFFFu, st.s.code[1], k);
                const uint32_t q2 = __shfl_sync(0xFFFFFFFFu, st.s.code[2], k), q3 = __shfl_sync(0xFFFFFFFFu, st.s.code[3], k);
                if (ri >= kStages) ok = wait_bar(&S.raw_empty[s], ((ri / kStages) - 1) & 1, abort_flag, status);
                if (!__all_sync(0xFFFFFFFFu, ok)) {
                    ok = false;
                    break;
                }
                if (lane < 4) {
                    const unsigned bytes = has ? unsigned(kp_bytes(int(info & 255u)) + kp_bytes(int((info >> 8) & 255u))) : 0u;
                    const uint32_t code = lane == 0 ? q0 : lane == 1 ? q1 : lane == 2 ? q2 : q3;
                    if (lane == 0) S.step[ri % (2 * kStages)] = info | shape;
                    mbar_expect(&S.raw_full[s], bytes);
                    if (has)
                        bulk_g2s(sm + M::kOffRaw + s * kRawStage + lane * 4096, A.pcodes + (long long)code * 256, bytes,
                                 &S.raw_full[s]);
                }
                __syncwarp();
            }
        }
        if (lane < 4) {
            for (int i = 0; i < 2 && ok; ++i, ++ri) {  // the end, for both converter groups
                const int s = ri % kStages;
                if (ri >= kStages) ok = wait_bar(&S.raw_empty[s], ((ri / kStages) - 1) & 1, abort_flag, status);
                if (lane == 0) S.step[ri % (2 * kStages)] = kNoMore;
                mbar_arrive(&S.raw_full[s]);
            }
            if (!ok)
                for (unsigned k = ri > kStages ? ri - kStages : 0; k < ri; ++k)
                    for (int i = 0; i < kWaitLimit && !mbar_try(&S.raw_full[k % kStages], (k / kStages) & 1); ++i) {}
        }
    } else if (warp == 1) {
        // ---- MMA issuer (one lane): segments of up to two steps of one split
        if (elect_one()) {
            constexpr uint32_t idesc = mma_idesc(C::N) | (1u << 16);
            constexpr int kTile = kATile >> 4;
            const uint64_t b0 = limb_desc(smem_u32(sm + M::kOffB), C::kBCol), a0 = sw128_desc(smem_u32(sm));
            unsigned seg = 0;
            uint32_t blocks = 0;  // of the current segment (planes never grow along the k axis)
            bool ok = true;
            for (unsigned ri = 0; ok; ++ri) {
                const int s = ri % kStages, buf = seg & 1;
                const unsigned ph = (ri / kStages) & 1;
                ok = wait_bar(&S.a_full[s], ph, abort_flag, status);
                if (!ok) break;
                const uint32_t word = *reinterpret_cast<volatile uint32_t*>(&S.step[ri % (2 * kStages)]);
                if (word == kNoMore) break;
                const uint32_t nblk = (word >> 24) & 1u ? ((word & 7u) + 1) >> 1 : 1u;
                const int more = int(blocks);  // accumulators already started
                if (!blocks) {
                    blocks = nblk;
                    if (seg >= 2) ok = wait_bar(&S.acc_empty[buf], ((seg >> 1) - 1) & 1, abort_flag, status);
                }
                ok = ok && wait_bar(&S.b_full[s], ph, abort_flag, status);
                if (!ok) break;
                tc_fence_after();
                const uint64_t b = b0 + uint64_t(s * (C::kB >> 4)), a = a0 + uint64_t(int(ri % M::kAStages) * (kAStage >> 4));
                const uint32_t d = tmem + uint32_t(buf * kAccStride);
                const bool two = (word >> 8) & 255u;
                if (nblk == 2) {
                    if (two) mma_step<2, 4, C::N, kTile, 0>(d, a, b, idesc, more);
                    else mma_step<2, 2, C::N, kTile, 0>(d, a, b, idesc, more);
                } else {
                    if (two) mma_step<1, 4, C::N, kTile, 0>(d, a, b, idesc, more);
                    else mma_step<1, 2, C::N, kTile, 0>(d, a, b, idesc, more);
                }
                mma_commit(&S.done[s]);
                if (word & kSegmentEnd) {
                    S.segment[buf] = blocks | ((word & kItemEnd) ? 1u << 8 : 0u) | ((word >> 24) & 1u) << 16;
                    mbar_arrive(&S.acc_full[buf]);
                    mma_commit(&S.acc_full[buf]);
                    blocks = 0;
                    ++seg;
                }
            }
            mma_commit(&S.drain);
            for (int i = 0; i < kWaitLimit && !mbar_try(&S.drain, 0); ++i) {}
        }
        __syncwarp();
    } else if (wg == 1 || wg == 2) {
        // ---- converters: thread = tile row; a group takes every other step
        set_regs<RowRegs::kConvert>();
        const int row = 32 * (warp & 3) + lane;
        const uint32_t smem0 = smem_u32(sm), row0 = row_offset(row);
        for (unsigned ri = unsigned(wg - 1);; ri += 2) {
            const int s = ri % kStages;
            const unsigned ph = (ri / kStages) & 1;
            if (!warp_wait(&S.raw_full[s], ph, abort_flag, status)) break;
            const unsigned used = ri - M::kAStages;  // the step whose A stage this one takes
            const uint32_t word = *reinterpret_cast<volatile uint32_t*>(&S.step[ri % (2 * kStages)]);
            if (ri >= M::kAStages && !warp_wait(&S.done[used % kStages], (used / kStages) & 1, abort_flag, status)) break;
            if (word != kNoMore) {
                const int wide = int(word >> 24) & 1;  // 1: 64 tile rows x 2 planes, 0: 32 x 4
                const int m0 = row >> (5 + wide), tr = row & (31 + 32 * wide), rr = tr & 15;
                const int info0 = int(word & 255u), info1 = int((word >> 8) & 255u);
                const uint32_t raw = smem0 + uint32_t(M::kOffRaw + s * kRawStage + (tr >> 4) * 4096 + m0 * 512);
                const uint32_t tile = smem0 + (ri % M::kAStages) * uint32_t(kAStage) + row0;
                const int halves = wide ? ((info0 & 7) + 1) & ~1 : 2;
                // (rows of M-tiles that the tile does not have convert whatever
                // bytes are there: nothing reads their sums)
#pragma unroll 1
                for (int i = 0; i < halves; ++i) {
                    const int m = (i & ~1) + m0, info = i & 1 ? info1 : info0, P = info & 7;  // (m: the same for the warp)
                    if (info == 0) continue;
                    const uint32_t dst = (tile + uint32_t(i >> 1) * kATile) ^ uint32_t((i & 1) << 6);
                    if (m >= P) {  // no such plane: it must add nothing
#pragma unroll
                        for (int k = 0; k < 4; ++k) sts128(dst ^ (16 * k), 0u, 0u, 0u, 0u);
                        continue;
                    }
                    const bool top = m == P - 1, nib = top && ((info >> 3) & 1);
                    convert_half(dst, raw + uint32_t((i & 1 ? kp_bytes(info0) : 0) + (i & ~1) * 512 + rr * (nib ? 16 : 32)),
                                 !top ? kLowerPlane : nib ? kTopNibbles : kTopPlane, kp_hb(info));
                }
                fence_async_smem();
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&S.a_full[s]);
                mbar_arrive(&S.raw_empty[s]);
            }
            if (word == kNoMore) break;
        }
    } else if (wg == 4 || wg == 5) {
        // ---- drain: lane = (plane, tile row); the item's 128-bit sums
        set_regs<RowRegs::kDrain>();
        const int quarter = warp & 3, e = wg - 4;
        unsigned seg = 0;
        bool ok = true;
        unsigned long long v[C::kRowPer][4], weights;
        pdl_wait();  // (the sums' buffer is the previous apply's until then)
        Pairs w(n_items, groups);
        int part = 0, part_nx = 0;
        if (w.valid()) part_nx = int(ahead32(&A.tc_row_items[w.item].part));
        while (w.valid()) {
            part = part_nx;
            const int c0 = w.group * R + e * C::kRowPer;
            w.next();
            part_nx = int(ahead32(&A.tc_row_items[w.some()].part));
#pragma unroll
            for (int r = 0; r < C::kRowPer; ++r)
#pragma unroll
                for (int t = 0; t < 4; ++t) v[r][t] = 0;
            uint32_t word = 0;
            weights = 0;
            for (bool end = false; !end; ++seg) {
                const int buf = seg & 1;
                ok = warp_wait(&S.acc_full[buf], (seg >> 1) & 1, abort_flag, status);
                if (!ok) break;
                __syncwarp();
                tc_fence_after();
                word = *reinterpret_cast<volatile uint32_t*>(&S.segment[buf]);
                end = (word >> 8) & 1u;
                const int nblk = int(word & 15u);
                const uint32_t base =
                    tmem + (uint32_t(32 * quarter) << 16) + uint32_t(buf * kAccStride + e * 8 * C::kRowPer);
#pragma unroll 1
                for (int b = 0; b < nblk; ++b) {
                    uint32_t d[8 * C::kRowPer];
                    tmem_ld<8 * C::kRowPer>(base + uint32_t(b * C::N), d);
                    tmem_wait_ld();
                    add_sums<C::kRowPer>(v, d, b ? 1u << 16 : 1u);
                    weights += b ? 1u << 16 : 1u;
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.acc_empty[buf]);
            }
            if (!ok) break;
            const int row = 32 * quarter + lane, sh = 8 * (row >> (5 + ((word >> 16) & 1u)));
#pragma unroll
            for (int r = 0; r < C::kRowPer; ++r)
                if (c0 + r < rhs)
                    st_i128(W.part + ((long long)(c0 + r) * n_parts + part) * 128 + row, join_limbs(v[r], weights) << sh);
        }
    } else if (wg == 3 || wg == 6) {
        // ---- builders: limbs of U for the 64 slots of every other step; thread =
        // (column pair, slot): a component's columns are read as whole sectors
        set_regs<RowRegs::kSide>();
        const int bt = (warp & 3) * 32 + lane;
        const int pair = bt % C::kPairs, slot0 = bt / C::kPairs;
        // Each thread copies what it will read (steps counted by group): after step
        // i the records of step i + 7 and, with the records that have arrived, V of
        // step i + 4 (both
        // come from L2 or DRAM; asynchronous copies, because registers waiting for
        // loads stall wherever the compiler moves them).  One copy group a step.
        constexpr int kS = C::kSlots;
        const uint32_t v_ring = smem_u32(sm) + uint32_t(M::kOffV + (wg == 6) * C::kVRing + bt * 16);
        const uint32_t rec_ring = smem_u32(sm) + uint32_t(M::kOffRec + (wg == 6) * C::kRecRing + bt * 8);
        StepRuns<false> st(A, n_items, groups, lane);
        int at = 0;                    // step in the run
        auto walk = [&]() {
            if (st.valid() && ++at == st.count()) {
                st.next(A);
                at = 0;
            }
        };
        const int grp = wg == 6;
        if (grp) walk();
        int q[7];                      // steps i .. i + 6: column block | slots << 24 (-1: past the end)
        uint32_t sh[kS];               // shifts of steps i .. i + 3, a byte each
        unsigned bi = unsigned(grp);
        bool ok = true;
#pragma unroll
        for (int k = 0; k < 7; ++k) q[k] = 0;
#pragma unroll
        for (int k = 0; k < kS; ++k) sh[k] = 0;
        auto copy_rec = [&](int i) {  // records of the walk's next step, for step i
            if (!st.valid()) {
                q[6] = -1;
                return;
            }
            const int s0 = __shfl_sync(0xFFFFFFFFu, st.s.slot, at), ns = __shfl_sync(0xFFFFFFFFu, st.s.nslots, at);
#pragma unroll
            for (int k = 0; k < kS; ++k)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(rec_ring + uint32_t(((i & 3) * kS + k) * 1024)),
                                 "l"(A.slot_rec + s0 + min(slot0 + 32 * k, ns - 1))
                                 : "memory");
            q[6] = st.w.group | ns << 24;
            walk();
            walk();
        };
        auto copy_v = [&](int i) {  // V of step i (q[3])
            if (q[3] < 0) return;
#pragma unroll
            for (int k = 0; k < kS; ++k) {
                int comp, info;
                asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(comp), "=r"(info) : "r"(rec_ring + uint32_t(((i & 3) * kS + k) * 1024)) : "memory");
                // a slot past the k axis (-1) has U = 0: no bytes of V are read
                // for it, the copy writes zeros (its digits are not zero, and V
                // of a component that no block holds is never written)
                const bool none = comp < 0 || slot0 + 32 * k >= q[3] >> 24;
                const long long* p = W.v + (long long)max(comp, 0) * pv + min((q[3] & 0xFFFFFF) * R + pair * 2, pv - 2);  // (past the last: not read)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(v_ring + uint32_t(((i & 3) * kS + k) * 2048)), "l"(p),
                             "r"(none ? 0 : 16)
                             : "memory");
                sh[k] = (sh[k] & 0x00FFFFFFu) | uint32_t((info >> 8) & 63) << 24;
            }
        };
        pdl_wait();  // V of this apply
        for (int i = -7;; ++i) {
            asm volatile("cp.async.wait_group 2;" ::: "memory");
            if (i >= 0) {
                if (q[0] < 0) break;
                const int sb = bi % kStages;
                if (bi >= kStages) ok = warp_wait(&S.done[sb], ((bi / kStages) - 1) & 1, abort_flag, status);
                if (!ok) break;
                uint8_t* dst = sm + M::kOffB + sb * C::kB + pair * 2 * C::kBCol + slot0 * 16;
#pragma unroll
                for (int k = 0; k < kS; ++k) {
                    const uint4 w = lds128(v_ring + uint32_t(((i & 3) * kS + k) * 2048));
                    const long long v0 = (long long)(((unsigned long long)w.y << 32) | w.x);
                    const long long v1 = (long long)(((unsigned long long)w.w << 32) | w.z);
                    const int shift = int(sh[k] & 255u);
                    *reinterpret_cast<uint4*>(dst + 512 * k) = to_limbs(tile_fixed(v0, shift));
                    *reinterpret_cast<uint4*>(dst + C::kBCol + 512 * k) = to_limbs(tile_fixed(v1, shift));
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.b_full[sb]);
                bi += 2;
            }
            // step i is done: i + 1 next
#pragma unroll
            for (int k = 0; k < kS; ++k) sh[k] >>= 8;
#pragma unroll
            for (int k = 0; k < 6; ++k) q[k] = q[k + 1];
            if (i + 4 >= 0) copy_v(i + 4);
            copy_rec(i + 7);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else if (wg == 7) {
        set_regs<RowRegs::kIdle>();
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_free(tmem, 512);
}

// Test aid: warp 0 waits for a phase that nothing completes, `polls` tests at
// most, and tells the block; warp 1 waits for another and ends when told.  out: 1
// for each lane that gave up.
__global__ void __launch_bounds__(64) give_up_kernel(int polls, int* status, int* out) {
    __shared__ uint64_t bar[2];
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&bar[i], 1);
        abort_flag = 0;
    }
    __syncthreads();
    const bool ok = warp_wait(&bar[warp], 0, &abort_flag, status + warp, warp ? kWaitLimit : polls);
    out[threadIdx.x] = ok ? 0 : 1;
}

// ------------------------------------------------------------------ combine

// Thread per (tile row, right-hand side): the tile's dense slices in column
// order plus the sums of its row items' planes, converted once.
__global__ void __launch_bounds__(64) tc_combine_kernel(Arena A, Work W, double* __restrict__ y, int n_parts,
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
    const int rs = T.parts >> 16, parts = T.parts & 0xFFFF;
    const uint4* src = W.part + ((long long)p * n_parts + T.part0) * 128 + r;
    __int128 R = 0;
    for (int i = 0; i < parts; ++i)
        for (int k = 0; k < 128; k += rs) R += ld_i128(src + i * 128 + k);
    double d = 0.0;
    for (int i = 0; i < T.nds; ++i) d += __ldcg(W.pdense + ((long long)p * n_dslices + T.ds0 + i) * 64 + r);
    const double lr = (xe && T.c_exp != kNoExp) ? i128_ldexp(R, xe + T.c_exp - 1022 - kFixBits) : 0.0;
    y[(long long)out * ld + p] = d + lr;
}

template <int R>
cudaError_t launch_column(const TcArgs& a, cudaStream_t s) {
    const int groups = (a.rhs + R - 1) / R;
    if ((long long)a.n_items * groups > INT32_MAX) return cudaErrorInvalidValue;
    if (a.n_items == 0 && a.n_dense == 0) return cudaSuccess;
    // No more blocks than there is work for: an item and a column block each, or
    // one dense part for each of a block's four dense warps.  A block holds a
    // whole SM, which another stream's kernels could use (six matrices of 300
    // unknowns, 3 columns, a stream each: 28.2 us an apply of all on a grid of every
    // SM, 16.6 on this one, 24.6 on the column-by-column kernels).
    const long long jobs = std::max((long long)a.n_items * groups, ((long long)a.n_dense * (a.rhs + 1) + 3) / 4);
    return launch_pdl(tc_column_kernel<R>, dim3(unsigned(std::min<long long>(jobs, a.sms))), dim3(kThreads), size_t(ColSmem<R>::kBytes), s, a.A, a.W,
                      a.n_items, groups, a.n_dense, a.rhs, a.pv, a.n, a.n_pad, a.n_split, a.n_dslices, a.status);
}
template <int R>
cudaError_t launch_row(const TcArgs& a, cudaStream_t s) {
    const int groups = (a.rhs + R - 1) / R;
    const long long jobs = (long long)a.n_row_items * groups;
    if (jobs > INT32_MAX) return cudaErrorInvalidValue;
    if (jobs == 0) return cudaSuccess;
    return launch_pdl(tc_row_kernel<R>, dim3(unsigned(jobs < a.sms ? jobs : a.sms)), dim3(kThreads),
                      size_t(RowSmem<R>::kBytes), s, a.A, a.W, a.n_row_items, groups, a.rhs, a.pv, a.n_parts, a.status);
}

template <class K>
cudaError_t allow_smem(K* kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace
}  // namespace tc

cudaError_t tc_setup() {
    using namespace tc;
    cudaError_t e = allow_smem(tc_column_kernel<4>, ColSmem<4>::kBytes);
    if (e == cudaSuccess) e = allow_smem(tc_column_kernel<8>, ColSmem<8>::kBytes);
    if (e == cudaSuccess) e = allow_smem(tc_row_kernel<4>, RowSmem<4>::kBytes);
    if (e == cudaSuccess) e = allow_smem(tc_row_kernel<8>, RowSmem<8>::kBytes);
    return e;
}

cudaError_t tc_debug_give_up(int polls, int* status, int* out) {
    tc::give_up_kernel<<<1, 64>>>(polls, status, out);
    return cudaGetLastError();
}

cudaError_t tc_launch(const TcArgs& a, cudaStream_t s, void (*mark)(void*, int), void* ctx) {
    using namespace tc;
    // four columns at once cost less than eight (8192 unknowns (3-D): 82 us for 3
    // or 4 columns, 92 for 5 .. 8)
    const bool few = a.rhs <= 4;
    cudaError_t e = few ? launch_column<4>(a, s) : launch_column<8>(a, s);
    if (mark) mark(ctx, 2);
    if (e == cudaSuccess) e = few ? launch_row<4>(a, s) : launch_row<8>(a, s);
    if (e == cudaSuccess)
        e = launch_pdl(tc_combine_kernel, dim3(unsigned(a.n_tiles), unsigned(a.rhs)), dim3(64), 0, s, a.A, a.W, a.y,
                       a.n_parts, a.n_dslices, a.ld);
    return e;
}

}  // namespace qhg
