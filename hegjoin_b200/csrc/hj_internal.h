// hj_internal.h -- library-internal structures shared by the .cu files.
#pragma once

#include "hj_common.cuh"

// Grid parameters passed by value to kernels.
struct HjGrid {
    uint32_t k;
    uint32_t n_cells[hj::kMaxK];
    unsigned long long mult[hj::kMaxK];   // mixed-radix multipliers, dimension 0 fastest
    // Row offsets of a full stencil box (width 3 along every dimension j >= 1):
    // entry r is sum over j >= 1 of digit_j(r) * mult[j], the base-3 digits of r
    // with dimension 1 fastest; full_rows = 3^(k-1) entries.  Null (and
    // full_rows 0) for k > kRowOffMaxK.
    const unsigned long long* row_off;
    uint32_t full_rows;
    unsigned long long full_base;   // linear id of a cell minus that of its full box's first cell
};
constexpr uint32_t kRowOffMaxK = 7;   // at most 729 offsets

// Open-addressing hash of the non-empty cells, keyed by groups of four
// consecutive linear ids (g = lid >> 2).  An entry is 16 bytes: the group key
// (two words), the cell index of the group's first non-empty cell, and a 4-bit
// mask of the group's non-empty ids; the group's cells are consecutive in the
// cell table (sorted by linear id), so the cell of id g*4 + b is the first cell
// plus the number of mask bits below b.  A stencil row (up to 3 consecutive ids
// along dimension 0) spans one or two groups: one or two 16-byte loads, and
// neighbouring cells along dimension 0 hit the same entries.  Capacity is a
// power of two at least twice the number of cells (so at most half full of
// groups); free entries hold the key
// kEmptyLid (no group can have it: linear ids stay below 2^63).
// Beside it lies an occupancy bitmap: ids in segments of 32, each segment a word
// picked by a multiplicative hash (segments may share one), each cell its bit.  A
// stencil row is one load of one word -- from L2, where the table itself does not
// fit -- and three bits: the common case on sparse data, a row without cells, ends
// there.  4 bytes per table entry, 64 to 128 bits per cell: 3 to 5% of the empty
// rows find a stranger's bit and go on to the table.
struct HjCellHash {
    const uint4* entries;
    unsigned long long mask;       // capacity - 1
    const uint32_t* occ;           // occupancy bitmap
    uint32_t occ_shift;            // 64 - log2(its words)
};

// Work item of the refine kernels: queries q0..q1 (sorted positions) of cell
// `cell`, whose stencil holds `nb` candidate points.
struct HjBlock {
    uint32_t cell;
    uint32_t q0;
    uint32_t q1;
    uint32_t nb;
};

struct hj_index {
    uint32_t n = 0, d = 0, k = 0;
    int dtype = HJ_F32;
    double eps = 0;            // value in dataset type
    double thr = 0;            // largest d2 with RN(sqrt(d2)) <= eps (dataset type)
    double min_arr[hj::kMaxK] = {};
    HjGrid grid = {};
    uint64_t total_cells = 0;
    uint32_t aliasing = 0;
    uint32_t any_silent = 0;   // some cell has a coordinate of 0 and visits no cell (kernel.cu:780 wraps)
    int device = 0;
    cudaStream_t stream = nullptr;   // stream the index was built on; its memory is freed in that order

    // device arrays
    void* pts = nullptr;             // n x d, dataset type, ordered by (cell id, original id)
    uint32_t* perm = nullptr;        // sorted position -> original id (indexLookupArr)
    unsigned long long* cell_lid = nullptr;  // nC sorted linear ids
    uint32_t* cell_start = nullptr;  // nC + 1
    uint32_t nC = 0;
    uint4* hash_entries = nullptr;   // cell hash (HjCellHash)
    unsigned long long hash_mask = 0;
    uint32_t* hash_occ = nullptr;    // its occupancy bitmap
    uint8_t* cell_edge = nullptr;    // per cell: 1 if its stencil box is not full (a coordinate at the grid's edge)
    uint32_t occ_shift = 0;
    unsigned long long* row_off = nullptr;   // grid.row_off

    // workload (hj_sort_by_workload)
    bool have_workload = false;
    uint64_t total_candidates = 0;
    uint32_t* cell_nb = nullptr;     // candidates per cell (cell order)
    uint32_t* cell_order = nullptr;  // cells, heaviest first

    // tensor-core operands (built on first use)
    void* tc_a = nullptr;            // query form: K-block planes (hj_refine_tc.cu)
    void* tc_b = nullptr;            // candidate form
    uint32_t* perm_flag = nullptr;   // perm with bit 31 set for points of silent cells (null without such cells)
    uint32_t tc_kpad = 0;
    int plain_shape = 0;             // exact refine tile shape (0 or 1; autotuned per d and dtype)
    int tc_kind = -1;                // HJ_REFINE_TC_F16 / _BF16 the operands hold
    void* tc_state = nullptr;        // scale, threshold and error maxima (hj_refine_tc.cu)
};

namespace hj {

// Host: largest value x of the dataset type with RN(sqrt(x)) <= eps.
double sq_threshold(double eps, int dtype);

// Keep freed stream-ordered allocations mapped for reuse (called once per process).
void init_memory_pool();
uint64_t pool_idle_bytes();

// hj_refine_tc.cu
void tc_release(hj_index* ix);

// Largest d of the warp-per-item exact refine (hj_refine_warp.cu).
constexpr int kWarpMaxD32 = 12;
constexpr int kWarpMaxD64 = 8;

// perm with the points of silent cells marked (bit 31), for the refines' symmetric
// form; the index's own perm where no cell is silent.  Part of the index from its
// creation: joins of one index may run side by side on several threads and streams.
inline const uint32_t* flagged_perm(const hj_index* ix) { return ix->perm_flag ? ix->perm_flag : ix->perm; }

// hj_index.cu
// Work items of up to qb queries per cell, in the workload order; `align` (a
// power of two): a cell's items after its first start at multiples of it and
// fill whole groups, the first begins at the cell's first point.  Makes the workload
// order first if the index has none yet (one synchronisation for both).
hj_status build_blocks(hj_index* ix, uint32_t qb, uint32_t align, HjBlock** d_blocks, uint32_t* n_blocks,
                       cudaStream_t st);

constexpr unsigned long long kEmptyLid = ~0ull;
constexpr uint32_t kNoCell = 0xFFFFFFFFu;

inline HjCellHash cell_hash(const hj_index* ix) {
    return HjCellHash{ix->hash_entries, ix->hash_mask, ix->hash_occ, ix->occ_shift};
}

// Bitmap word of the segment of 32 ids that holds `lid`.
__host__ __device__ __forceinline__ unsigned long long occ_word(unsigned long long lid, uint32_t occ_shift) {
    return ((lid >> 5) * 0x9E3779B97F4A7C15ull) >> occ_shift;
}

// Coordinate of the cell with linear id L along dimension lane_id() for the
// lanes below k: the warp pays one 64-bit division per lane, and the other
// dimensions are fetched with shuffles, instead of k divisions per thread.
__device__ __forceinline__ uint32_t lane_cell_coord(const HjGrid& g, unsigned long long L) {
    const uint32_t j = lane_id();
    if (j >= g.k) return 0u;
    const unsigned long long q = L / g.mult[j];
    return (j + 1 < g.k) ? (uint32_t)(q % g.n_cells[j]) : (uint32_t)q;
}

// Quotient of r by a stencil width w in {1, 2, 3} (widths are 3 except where
// the stencil is clamped at the grid's edge): no integer division instruction.
__device__ __forceinline__ uint32_t div_w(uint32_t r, uint32_t w) {
    return w == 3u ? (uint32_t)(((unsigned long long)r * 0xAAAAAAABull) >> 33) : (w == 2u ? r >> 1 : r);
}

// Stencil rows of a cell's box (per dimension j the cells lo[j] .. lo[j] + w[j] - 1;
// `rows` is the product of w[1..k-1]).  Row r covers, along dimension j >= 1,
// coordinate lo[j] + the j-th mixed-radix digit of r (radices w[1], w[2], ...,
// dimension 1 fastest) and, along dimension 0, the w[0] cells from lo[0].
// A full box (every w[j] == 3 for j >= 1: the cell is not at the grid's upper
// edge) reads its rows' offsets from the grid's table; an edge box divides.
struct StencilRows {
    bool full;                  // offsets from grid.row_off
    unsigned long long first;   // linear id of row 0's first cell
};
__device__ __forceinline__ StencilRows stencil_rows(const HjGrid& g, const uint32_t* lo, uint32_t rows) {
    StencilRows s;
    s.full = g.row_off != nullptr && rows == g.full_rows;
    s.first = lo[0];
    for (uint32_t j = 1; j < g.k; ++j) s.first += (unsigned long long)lo[j] * g.mult[j];
    return s;
}
// Linear id of the first cell of row r (equal, modulo 2^64 like all linear-id
// arithmetic here, in both forms).
__device__ __forceinline__ unsigned long long stencil_row_id(const HjGrid& g, const StencilRows& s,
                                                             const uint32_t* lo, const uint32_t* w, uint32_t r) {
    if (s.full) return s.first + __ldg(g.row_off + r);
    uint32_t rem = r;
    unsigned long long id = lo[0];
    for (uint32_t j = 1; j < g.k; ++j) {
        const uint32_t qw = div_w(rem, w[j]);
        id += (unsigned long long)(lo[j] + (rem - qw * w[j])) * g.mult[j];
        rem = qw;
    }
    return id;
}

// The stencil box of a cell (kernel.cu:778-783), whole warp.  Rows are in ascending
// order of their linear ids, so the cells after the cell itself lie in its own row,
// past it, and in the rows after that one.  A full box (the cell is off the grid's
// edges; cell_edge says so) needs no coordinate: its rows are at fixed offsets from
// the cell's id.  The others take one 64-bit division per lane for the coordinates.
struct CellBox {
    unsigned long long L;
    uint32_t rows, r_own, w0;   // rows, the row that holds the cell, cells per row
    bool full, silent;          // silent: a coordinate is 0
    uint32_t lo[hj::kMaxK], w[hj::kMaxK];
};
__device__ __forceinline__ void cell_box(const HjGrid& g, unsigned long long L, bool edge, CellBox& b) {
    b.L = L;
    b.full = !edge && g.row_off != nullptr;
    b.silent = false;
    if (b.full) {
        b.rows = g.full_rows;
        b.r_own = g.full_rows >> 1;
        b.w0 = 3;
        return;
    }
    b.rows = 1;
    b.r_own = 0;
    const uint32_t cl = lane_cell_coord(g, L);
    for (uint32_t j = 0; j < g.k; ++j) {
        const uint32_t c = __shfl_sync(0xffffffffu, cl, j);
        b.silent |= c == 0u;
        b.lo[j] = c == 0u ? 0u : c - 1u;
        b.w[j] = min(g.n_cells[j] - 1u, c + 1u) - b.lo[j] + 1u;
        if (j > 0) {
            b.r_own += (c - b.lo[j]) * b.rows;
            b.rows *= b.w[j];
        }
    }
    b.w0 = b.w[0];
}
// Linear id of the first cell of row r.
__device__ __forceinline__ unsigned long long cell_box_row(const HjGrid& g, const CellBox& b, uint32_t r) {
    if (b.full) return b.L - g.full_base + __ldg(g.row_off + r);
    return stencil_row_id(g, StencilRows{false, 0ull}, b.lo, b.w, r);
}

// The entry of group g: (first cell, id mask), or a zero mask when the group has
// no cell.  Probes stop at a free entry; the table is at most half full, so the
// loop ends after a few probes (and after capacity probes at the very most).
__device__ __forceinline__ uint2 group_find(const HjCellHash& h, unsigned long long g) {
    unsigned long long i = mix64(g) & h.mask;
    for (unsigned long long probe = 0; probe <= h.mask; ++probe) {
        const uint4 e = h.entries[i];
        const unsigned long long key = ((unsigned long long)e.y << 32) | e.x;
        if (key == g) return make_uint2(e.z, e.w);
        if (key == kEmptyLid) break;
        i = (i + 1) & h.mask;
    }
    return make_uint2(kNoCell, 0u);
}

// Bit i set: the bitmap knows a cell lo + i, i < w <= 4 (or one that shares its bit).
// In the bitmap itself a cell's bit is clear.
__device__ __forceinline__ uint32_t occ_row(const HjCellHash& h, unsigned long long lo, uint32_t w) {
    const uint32_t b = (uint32_t)lo & 31u;
    uint32_t m = __ldg(h.occ + occ_word(lo, h.occ_shift)) >> b;
    if (b + w > 32u) m |= __ldg(h.occ + occ_word(lo + w - 1, h.occ_shift)) << (32u - b);
    return ~m & ((1u << w) - 1u);
}

// The existing cells among those named by `m` (occ_row's answer) from id lo on:
// consecutive in the cell table, [x, y] (x == kNoCell: none).
__device__ __forceinline__ uint2 cell_range(const HjCellHash& h, unsigned long long lo, uint32_t m) {
    uint32_t first = kNoCell, last = kNoCell;
    while (m) {
        const unsigned long long id = lo + (__ffs(m) - 1);
        const unsigned long long g = id >> 2;
        const uint2 e = group_find(h, g);
        // this group's ids among m: bit b of the group is id g * 4 + b
        const long long sh = (long long)(g * 4ull - lo);
        const uint32_t want = (sh >= 0 ? m >> sh : m << -sh) & 15u;
        m &= ~(sh >= 0 ? 15u << sh : 15u >> -sh);
        const uint32_t have = e.y & want;
        if (have == 0u) continue;
        const uint32_t f = e.x + __popc(e.y & ((1u << (__ffs(have) - 1)) - 1u));
        const uint32_t l = e.x + __popc(e.y & ((2u << (31 - __clz(have))) - 1u)) - 1u;
        if (first == kNoCell) first = f;
        last = l;
    }
    return make_uint2(first, last);
}

// Rows row0 .. row0 + 127 of a box that the bitmap does not rule out, compacted into
// `list` (row | cells << 28), and their number.  The lanes' bitmap words are loaded
// together; what is left of sparse data -- a few rows -- then goes through the
// table side by side instead of one slot of 32 rows after the other.  after: only
// the cell itself and the cells after it.  Whole warp.
constexpr uint32_t kBoxRows = 128;
__device__ __forceinline__ uint32_t box_rows_present(const HjGrid& g, const HjCellHash& h, const CellBox& b,
                                                     uint32_t row0, bool after, uint32_t* list) {
    uint32_t m[kBoxRows / 32];
#pragma unroll
    for (uint32_t i = 0; i < kBoxRows / 32; ++i) {
        const uint32_t r = row0 + i * 32 + lane_id();
        m[i] = 0;
        if (r >= b.rows) continue;
        const unsigned long long id = cell_box_row(g, b, r);
        m[i] = occ_row(h, id, b.w0);
        if (after && r == b.r_own) m[i] &= ~((1u << (uint32_t)(b.L - id)) - 1u);
    }
    uint32_t n = 0;
#pragma unroll
    for (uint32_t i = 0; i < kBoxRows / 32; ++i) {
        const uint32_t some = __ballot_sync(0xffffffffu, m[i] != 0u);
        if (m[i]) list[n + __popc(some & lanemask_lt())] = (row0 + i * 32 + lane_id()) | m[i] << 28;
        n += __popc(some);
    }
    __syncwarp();
    return n;
}

// Points of the existing cells with linear ids lo .. lo + w - 1 (consecutive
// along dimension 0, w <= 4): one contiguous span [x, y) of the cell-ordered
// points, because the non-empty cells are sorted by linear id.
__device__ __forceinline__ uint2 cell_points(const HjCellHash& h, const uint32_t* cell_start, unsigned long long lo,
                                             uint32_t m) {
    const uint2 c = cell_range(h, lo, m);
    if (c.x == kNoCell) return make_uint2(0u, 0u);
    return make_uint2(cell_start[c.x], cell_start[c.y + 1]);
}
__device__ __forceinline__ uint2 cell_span(const HjCellHash& h, const uint32_t* cell_start, unsigned long long lo,
                                           uint32_t w) {
    const uint32_t m = occ_row(h, lo, w);
    return m ? cell_points(h, cell_start, lo, m) : make_uint2(0u, 0u);
}

}  // namespace hj
