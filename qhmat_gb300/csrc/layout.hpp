// Host-side ingestion of a quantized H-matrix and the resident device layout.
//
// The layout is built once per matrix on the host and uploaded as a single
// arena; every kernel reads only this arena plus the caller's x, y and
// workspace.  Nothing here depends on CUDA, so the builder is unit-testable
// on the CPU.
//
// Codes are stored as digit planes laid out for the tensor cores.  A code c of
// width w (two's complement) on P = ceil(w/8) planes with t = w - 8(P-1) top
// bits is
//     c = sum_{m<P-1} 2^(8m) d_m + 2^(8(P-1)) (d_top - 2^(t-1)),
// d_m = (c >> 8m) & 255 and d_top = (c >> 8(P-1)) + 2^(t-1) in [0, 2^t)
// (stored as a nibble when t <= 4).  The device reads the top digit as the
// signed d_top - 2^(t-1), so
//     sum_i c_i v_i = sum_m 2^(8m) sum_i digit_m,i v_i
// with no offset correction, and every inner sum is an exact small-integer
// product sum (|digits| <= 255 times 8-bit limbs of the fixed-point operand),
// which the f16 tensor-core MMA computes exactly in FP32 (no partial sum
// reaches 2^24).  Digits are
// grouped into the 16x16 A-operand fragments of mma.m16n8k16: within a
// 16-entry k-block, thread t of a fragment row needs entries 2t, 2t+1, 2t+8,
// 2t+9, and those four digits are stored together:
//   byte group row (32 bytes per 2 k-blocks): bytes 8t..8t+3 = k-block 0
//     entries (2t, 2t+1, 2t+8, 2t+9), bytes 8t+4..8t+7 = k-block 1;
//   nibble group row (16 bytes per 2 k-blocks): word t, nibble k (k = 0..3:
//     k-block k>>1, entry 2t + 8(k&1)) and nibble k+4 (the following entry).
//
//  * right factor Q (column side): components sharing a column range and a
//    width form tasks of <= 32 (two 16-row M-tiles).  Per 32-entry chunk a
//    task stores, for each M-tile q and plane m, the group of its rows_q rows;
//    entries past the range hold code 0.
//  * left factor P (row side): rows are cut into tiles of <= 64 rows inside
//    one elementary row slab.  The components of all blocks covering a tile
//    are sorted by width, widest first, and form the tile's k axis (k-pairs
//    of 32).  A k-pair's codes are all written on the planes of its widest
//    code (P and t of that width; narrower codes sign-extended).  The tile's
//    M-tile q (16 rows) and k split h own one contiguous stream (a row unit):
//    for every k-pair kp = h, h + H, ... and every plane m of the k-pair, one
//    group of 16 rows (zero past the tile or past the k axis).  Each k slot
//    has a B row, written for every apply by the column task that computes
//    its component: the eight f16 limbs of U = u in fixed point on the tile's
//    exponent; a unit's B rows are contiguous (slot = tile base + h's base +
//    32 i + lane for its i-th k-pair).
//  * dense diagonal blocks are stored column-major (value (i, k) at
//    off + k*m + i) so that lanes owning consecutive rows read consecutive
//    doubles.
#pragma once

#include <cstddef>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <vector>

namespace qhg {

using std::invalid_argument;
using std::overflow_error;
using std::runtime_error;

// Flattened host copy of a matrix, in the reference's block insertion order.
struct HostMatrix {
    uint64_t order = 0;
    std::vector<uint64_t> permutation;  // clustered position -> source index

    struct Block {
        uint64_t row0, row1, col0, col1;
        bool admissible, dense;
        uint64_t rank = 0;        // low-rank only
        uint64_t comp0 = 0;       // first component index
        uint64_t dense_off = 0;   // dense only: offset into `dense` (row-major)
        double truncation_error = 0, quantization_bound = 0;
    };
    std::vector<Block> blocks;

    // Per component (low-rank blocks, concatenated in block order).
    std::vector<uint8_t> width;
    std::vector<double> left_scale, right_scale;
    std::vector<uint64_t> left_off, right_off;  // word index into left_words/right_words
    std::vector<uint32_t> left_words, right_words;
    std::vector<double> dense;

    double reconstruction_bound() const;
};

// QHMAT001 image -> HostMatrix, with the checks and messages of
// HMatrix::load (io.cpp:173-257), the permutation check of the HMatrix
// constructor (core.cpp:205-212), check_rectangle (core.cpp:214-222) and
// finalize (core.cpp:332-358).
HostMatrix parse_qhmat(const uint8_t* bytes, size_t len);

// Validate a HostMatrix assembled from caller arrays (permutation bijection,
// rectangles, ranks, widths, finite values, partition cover).
void validate(const HostMatrix& m);

// Rows of one row tile at most.
constexpr int kTileRows = 64;
// Row units of one tile at most: its M-tiles (16 rows each) times the k
// splits, hsplit = kTileUnits / M-tiles.
constexpr int kTileUnits = 8;
// Entries of one column-side chunk (one code per lane per entry).
constexpr int kColChunk = 32;
// x entries per exponent chunk of the fixed-point right-hand side.
constexpr int kChunk = 32;

// QHMAT001 trailer: FNV-1a-64 (src/qhmat/io.cpp:18-19).
constexpr uint64_t kFnvOffsetBasis = 14695981039346656037ULL;
constexpr uint64_t kFnvPrimeValue = 1099511628211ULL;

// Device-side descriptors (32-bit indices; checked by build_layout).
struct LowRankDesc {
    int32_t row0, m, col0, n;
    int32_t rank, comp0;
};
// Column-side unit of work: chunks [chunk0, chunk0 + nchunks) of a task of
// `count` (<= 32) components of width `width` whose blocks share the column
// range [col0, col0 + n).  Chunk c of the task starts at byte off + c * stride
// and holds, for M-tile q (rows_q = min(16, count - 16q)) and plane m, rows_q
// rows of 32 bytes (16 for a nibble top plane).  A pipeline step carries
// `cps` chunks.  A task longer than kMaxPartChunks chunks is split into
// `nparts` parts whose partial sums are combined by the part that finishes
// last.  The task's components feed ndest row-side B rows, listed at
// task_dest[dest0 ..] (every part holds the same list; the finishing part
// writes them).  A unit of width 0 instead holds columns [chunk0, chunk0 + n)
// of the dense diagonal block part tdense[col0] of row tile `stride`, its row
// sums going to dense slice comp_idx.
struct ColTask {
    int32_t col0, n, count, width;
    int64_t off;
    int32_t stride, comp_idx;   // comp_idx: first of `count` entries in task_rec
    int32_t chunk0, nchunks;
    int32_t part, nparts;
    int32_t split_id;           // index of the split task (counter / partials), -1 if nparts == 1
    int32_t cps;
    int32_t dest0, ndest;
};
// A row-side B row fed by a column task: slot, and (component row in the
// task) << 16 | the right shift (0 .. 63) from the component's fixed point to
// the tile's.  A task's list is ordered by (tile, row), so that a tile's B
// rows are consecutive.
struct TaskDest {
    int32_t slot, row_cexp;
};
static_assert(sizeof(TaskDest) == 8, "TaskDest layout");
static_assert(sizeof(ColTask) == 64, "ColTask layout");
// Finalize operands of one component of a column task (one 16-byte load).
// The component's u = s t 2^(xe - 1022 - kFixBits), s = s^P s^Q, t its exact
// integer sum, is held in fixed point on the component's own exponent,
// V = round(u 2^(kFixBits - (xe - 1022 + beta))) = round(t s 2^-beta), beta a
// layout-time bound (|u| < 2^(xe - 1022 + beta), so |V| < 2^kFixBits).  With
// 2^(shift - 1) <= sum |c| < 2^shift, t 2^-shift fits 63 bits and
// s 2^(shift - beta) lies in [1/4, 1): kappa is that factor times 2^64
// (exact, the product s having 53 bits), and V = (t >> shift) kappa >> 64.
struct TaskRec {
    int32_t comp;
    uint8_t width, shift;
    uint16_t pad;
    uint64_t kappa;  // 0: u is identically zero
};
static_assert(sizeof(TaskRec) == 16, "TaskRec layout");
struct DenseDesc {
    int32_t row0, m, col0, n;
    int64_t off;  // element offset of the column-major values in the dense arena
};
// One row tile: clustered rows [row0, row0 + rows) inside one slab; qrows
// M-tiles, k axis split hsplit ways (nh of the splits have k-pairs); dense
// blocks tdense[dense0 .. dense0 + ndense), whose row sums are kept as dense
// slices ds0 .. ds0 + nds - 1 (kDenseCols columns each, in column order); u
// is put in fixed point on the exponent field xe + c_exp (xe: the largest
// exponent field of x).
struct RowTile {
    int32_t row0, rows, qrows, hsplit;
    int32_t nh, ndense, dense0, c_exp;
    int32_t ds0, nds;
    int32_t part0, parts;  // row items' partial sums; parts | rs << 16
};
static_assert(sizeof(RowTile) == 48, "RowTile layout");
// A dense diagonal block's part in a row tile: value (tile row r, column k)
// at dense[off + k * ld + r], x entries from xcol.
struct TileDense {
    int64_t off;
    int32_t ld, cols, xcol, pad;
};
static_assert(sizeof(TileDense) == 24, "TileDense layout");
// One warp's unit of row-side work: rows 16q .. 16q + 15 of a tile over the
// k-pairs kp = h, h + H, ... (nkps of them; B rows from slot0; digit groups
// from code_off; the tile's k axis has K slots), streamed in nsteps pipeline
// steps described by row_steps[step0 ..] (k-pairs | code bytes / 256 << 8 |
// the k-pairs' common info byte << 16 | 1 << 24 when the step is uniform: one
// info byte, every k-pair inside the k axis).
struct RowUnit {
    int32_t tile, q, h, H;
    int32_t nkps, K, slot0, nsteps;
    int64_t code_off, kp_off;
    int32_t step0, pad[3];
};
static_assert(sizeof(RowUnit) == 64, "RowUnit layout");

// A row-side B row slot: its component (-1: padding past the tile's k axis)
// and shift << 8 | width (shift: from the component's fixed point to the
// tile's, as in TaskDest).
struct SlotRec {
    int32_t comp, info;
};

// ---- work lists of the tensor-memory kernels (tc.cu), over the same codes.
//
// Column side: an item is up to four tasks (parts) of <= 32 components that
// share a column range, a run of chunks and a number of digit planes: task s
// gives rows 32s .. of a 128-row MMA tile.
struct TcItem {
    int32_t col0, chunk0, nchunks, info;  // info: planes | tasks << 8
};
static_assert(sizeof(TcItem) == 16, "TcItem layout");
// A task of an item: `off` is its first chunk's byte in the codes, chunks are
// `stride` bytes apart; info = components | width << 8; split: the split
// task's index (parts add their sums) or -1.
struct TcTask {
    int64_t off;
    int32_t stride, comp_idx;
    int32_t info, split, nparts, pad;
};
static_assert(sizeof(TcTask) == 32, "TcTask layout");
// Columns [k0, k0 + cols) of tdense[tdense] of a row tile, row-sum slice `slice`.
struct DenseUnit {
    int32_t tdense, tile, slice, k0, cols, pad[3];
};
static_assert(sizeof(DenseUnit) == 32, "DenseUnit layout");
// Row side: an item is a run of steps, each two k-pairs (64 slots) of one k
// split of a tile; its row sums are partial `part`.  The MMA tile's 128 rows
// are `rs` (32 or 64) tile rows for each of 128 / rs digit planes; qrows: the
// tile's 16-row M-tiles.
struct TcRowItem {
    int32_t step0, nsteps, shape, part;  // shape: rs | qrows << 8
};
static_assert(sizeof(TcRowItem) == 16, "TcRowItem layout");
// `code[q]`: the step's digit groups of M-tile q (byte offset / 256); `slot`:
// its first B row slot, `nslots` of them; info: the k-pairs' info bytes
// (second << 8, 0: none), kSegmentEnd on the last step of an accumulator
// segment (at most two steps, one split), kItemEnd on the item's last step.
struct TcStep {
    uint32_t code[4];
    int32_t slot, nslots;
    uint32_t info, pad;
};
static_assert(sizeof(TcStep) == 32, "TcStep layout");
constexpr uint32_t kSegmentEnd = 1u << 16, kItemEnd = 1u << 17;
// Steps a row item holds at least where its tile has them (shorter ones would
// be dominated by their pipeline's ends).
constexpr int kRowItemSteps = 8;

// Bytes of one column-side shared-memory stage (code groups and x rows of
// the step's chunks); one row-side stage (code groups and B rows).  Two
// stages per warp, eight warps per CTA and two CTAs per SM: 6144-byte stages
// are the largest that fit (measured: larger stages cut the per-step costs;
// 7168-byte row stages gained nothing more).
constexpr int kColSlotBytes = 6144;
constexpr int kRowSlotBytes = 6144;
// Longest run of chunks one column unit walks.
constexpr int kMaxPartChunks = 16;
// Columns of a dense block in one column-side dense unit (one slice).
constexpr int kDenseCols = 16;
// Exponent offset of a row tile without nonzero components.
constexpr int32_t kNoExp = -4000;

// Digit planes of a width-w code, and whether its top plane is a nibble.
inline int code_planes(int w) { return (w + 7) / 8; }
inline bool top_is_nibble(int w) { return w - 8 * (code_planes(w) - 1) <= 4; }

// Byte offsets of each section inside the device arena.
struct Sections {
    size_t perm, iperm, lr, dd, tasks, task_rec, task_dest, qcodes, pcodes, dense, tiles, tdense, units,
        kp_info, slot_rec, row_steps, comp_sl, comp_sr, tc_items, tc_tasks, dense_units, tc_row_items, tc_steps;
    size_t total;
};

struct Layout {
    uint64_t order = 0;
    int32_t n_lr = 0, n_dense = 0, n_comp = 0, n_tiles = 0, n_chunks = 0;
    int32_t n_tasks = 0, n_split = 0, max_parts = 1;
    int32_t n_units = 0, n_slots = 0, n_tdense = 0, n_dest = 0, n_dslices = 0;
    int32_t n_tc_items = 0, n_tc_row_items = 0, n_dense_units = 0;
    int32_t n_parts = 0;   // row-side partial sums (128 rows each)
    std::vector<uint8_t> arena;  // host image of the device arena
    Sections sec{};
    double bound = 0;
    // traffic model (reference word counts) and stored sizes
    uint64_t code_bytes = 0, left_code_bytes = 0, right_code_bytes = 0, scale_bytes = 0,
             dense_bytes = 0, flops = 0;
    uint64_t stored_q_bytes = 0, stored_p_bytes = 0;
};

Layout build_layout(const HostMatrix& m);

// SM cycles of each column task / row unit of the column-by-column kernels with
// every warp of the device resident (16 an SM).
std::vector<double> column_costs(const Layout& L);
std::vector<double> row_costs(const Layout& L);

// Longest-first assignment of units to warps: each goes to the warp with the
// least work so far.  The permutation is warp-major (each warp's units heaviest
// first), with the warps' `warps + 1` offsets.
struct Schedule {
    std::vector<int32_t> order, off;
    double total = 0, longest = 0;  // cycles: of all units, of the warp with the most
};
Schedule schedule_units(const std::vector<double>& costs, int warps);

// Which kernels an apply of `rhs` columns takes: the column-by-column ones
// (matvec.cu), which stream and convert every code once per column, or the
// tensor-memory ones (tc.cu), which do it once per four (up to four columns) or
// eight columns, in items of 128 rows and steps with a fixed handshake cost.
// Both give the same bits.  Where the line lies depends on how full the items
// are, so the times of both are predicted, in us, from the work lists; the
// coefficients are least-squares fits to whole applies of 82 matrices (1-D, 2-D
// and 3-D, 150 .. 100000 unknowns, leaves of 8 .. 128, ranks of 1 .. 33, equal and
// mixed code widths) with 3 .. 64 columns, 8 % and 6 % off.  Of those 898 applies
// four would be faster column by column by more than 1.5 % (10 % at most) and 13 on
// the other kernels (8 % at most); taking the tensor-memory kernels always made 92
// of them slower, by up to 62 %.  Column by column / tensor memory, us:
//                          3 columns   4           5           8           9           16
//   2048 (1-D, leaf 32)    32 / 25     40 / 25     48 / 28     71 / 28     81 / 35     139 / 35
//   16384 (1-D, leaf 16)   87 / 134    113 / 137   137 / 161   212 / 169   236 / 300   412 / 321
//   100000 (1-D, leaf 64)  303 / 489   394 / 495   486 / 548   765 / 582   862 / 1037  1525 / 1131
//   9001 (2-D, leaf 32)    108 / 108   140 / 110   171 / 125   266 / 132   303 / 220   520 / 232
//   16384 (2-D, leaf 64)   112 / 87    146 / 87    183 / 98    280 / 106   316 / 164   551 / 185
//   8192 (3-D, leaf 64)    133 / 82    174 / 82    212 / 91    332 / 92    372 / 158   644 / 163
// One and two columns never take them (32768 (2-D) x 1: 81 / 155, 9001 x 2: 77 / 105).
struct KernelChoice {
    double column = 0, order = 0;                           // us a column; unknowns
    double steps = 0, items = 0, row_steps = 0, dense = 0;  // per SM, of one pass over the codes
    bool tensor(size_t rhs) const;
};
KernelChoice kernel_choice(const Layout& L, const Schedule& columns, const Schedule& rows, int sms);

// Words of the bit string of `rows` codes of width w.
inline uint64_t words_for_bits(uint64_t rows, int w) { return (rows * uint64_t(w) + 31) / 32; }

}  // namespace qhg
