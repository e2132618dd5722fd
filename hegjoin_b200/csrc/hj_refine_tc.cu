// hj_refine_tc.cu -- tensor-core squared-distance filter with exact recheck.
//
// Reference counterpart: the refine kernelNDGridIndexGlobal (kernel.cu:727-802,
// evalPoint kernel.cu:333-370).  For high dimensions the reference's candidate
// loop is a dense distance evaluation; here each (candidate tile x query block)
// is a GEMM on the 5th-generation tensor cores:
//
//   A (M = 128 candidates, in bulk copies)  = [-2 c~, 1, 1, N_c hi, N_c lo, 0...]
//   B (N = 128 queries, resident)           = [  q~, N_q hi, N_q lo, 1, 1, 0...]
//   D' = A B^T = N_q + N_c - 2 q~.c~        (FP32 accumulate in TMEM)
//
// where x~ is the FP16 (or BF16) rounding of (x - origin) * 2^s and the norm
// terms carry the threshold: N_c = |c~|^2 - P(c), N_q = |q~|^2 - T - Q(q), with T
// the exact squared threshold and P + Q the pair's guard band (quantisation,
// tensor-core accumulation and the reference's own FP32 rounding; derivation at
// tc_band_p below).  So D' = |q~ - c~|^2 - (T + P + Q), and the sign of the MMA
// output is the filter's decision.  The origin is the per-dimension minimum and s
// is a power-of-two scale chosen per dataset so that the largest
// |x - origin|^2 * 4^s lies in [2^12, 2^14]: every stored half (coordinates up
// to 128, -2x up to 256, norm terms in [-60000, 2^14]) is finite whatever the
// data's units, and small-valued data stays clear of the FP16 subnormals.
// Scaling by 2^s is exact, so the threshold becomes T * 4^s exactly.  A pair is
//   rejected  if D' > 0 (the sign bit is clear),
//   accepted  if D' <= lo, below the band's lower edge for every pair,
//   rechecked otherwise, in FP32 in the reference's order (fma chain).
// The result set is therefore identical to the exact path.
//
// Kernel shape (one CTA per SM, persistent, 22 or 24 warps):
//   warp 0      loads: the work item's up to 512 query columns once, candidate
//               tiles through a ring of shared-memory stages, by bulk copies;
//   warps 1..4  MMA issuers, one per TMEM accumulator (4 x 128 columns, all of
//               TMEM): M = 128 x N = 128 MMAs;
//   warps 5..20 epilogue, a set of 4 per accumulator: tcgen05.ld, signs ORed or
//               gathered into masks, accumulator released;
//   the rest    emit the hits, which reach them as records in shared memory.
//
// What bounds it: the hand-over chain of an accumulator (waking the issuer and
// issuing ~330 cycles, MMAs, waking the epilogue ~100, TMEM reads with their ORs,
// vote and release ~110), the accumulators overlapping.  Per 256 columns and tile the
// floor is 273 cycles on the tensor pipe at d = 18 (two K steps) and 256 on the ALU
// (one OR per value at 128 per cycle); with the ORs left out a tile took ~350, with
// them and no hits ~750, with the hits of the data below ~820.
// Refine of 18-D points, 400,000 / 100,003 (half of the 32 x 32 chunks hold a hit),
// 90-D, 150,000 and 32-D BF16, 150,001, in ms:
//   before the sign test, symmetric form and whole-warp waits   15.9  4.7   6.7
//   the epilogue emitting                                         6.5  1.25  2.5
//   one ring of hits for all, two accumulators of 256 columns     5.83 1.06  2.06  2.21
//   sign masks in four chains of shifts, a ring per epilogue
//   warp, the accumulator released once its last read is done     5.56 0.93  1.86  1.82
//   four accumulators of 128 columns, waits without a sleep hint  5.11 0.89  1.73  1.72
// (a microbenchmark had issued N = 128 MMAs at 42% of the tensor pipe's rate, N = 256
// ones at 98%; the shorter chain is worth more).  Tried and not kept: one set of 16
// warps on every use (8.6 ms with emission, 6.3 ms without), 24 epilogue warps (5.84 ms
// against 5.83), 64-column reads (spills: 9.8 ms), named barriers instead of mbarriers
// for the release (6.5 ms), two chunks in flight (6.2 ms), three accumulators of 160
// columns, masks of the groups of four columns that hold a hit only (6.2 ms against 5.6).
// Every wait is bounded; a timeout raises an error flag that ends every later wait
// at once, and the roles walk their loops to the end (on garbage that the host
// discards, within the item's ranges), leave time for copies in flight and return.

#include <cuda_fp16.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "hj_internal.h"
#include "hj_tc.cuh"

namespace hj {
namespace {

constexpr int kTileRows = 128;               // candidate rows per tile (M of every MMA)
constexpr int kAcc = 4;                      // TMEM accumulators (a power of two)
constexpr int kAccCols = 128;                // N of one MMA: columns of one accumulator
constexpr int kQBMax = kAcc * kAccCols;      // query columns per work item at most
constexpr int kProbeThreads = 192;   // tile probe: load warp, MMA warp, 4 epilogue warps
constexpr int kProbeQB = 512;                // the tile probe evaluates 512 query rows
constexpr int kMaxStages = 8;
constexpr uint32_t kRowBytes = 64;           // one row of one K block: 32 halves
constexpr uint32_t kKBlockBytes = kTileRows * kRowBytes;   // one K block of a candidate tile
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kMaxRanges = 256;
constexpr int kEpiWarps = 16;                // 4 per accumulator: one per TMEM lane quarter
// warps that emit the hits which the epilogue finds: one keeps up with rare hits and
// leaves the most issue slots, dense hits take three (one, two and three at 18-D, 100,003
// points: 1.41, 1.03 and 0.93 ms; at 18-D, 400,000: 5.56, 5.63 and 5.77 ms)
constexpr int hit_warps(bool dense) { return dense ? 3 : 1; }
constexpr int tc_threads(bool dense) { return 32 * (1 + kAcc + kEpiWarps + hit_warps(dense)); }
// hit records between an epilogue warp and the hit warps (at least the 32 of one chunk; 32 and
// 64: 5.21 and 5.12 ms at 18-D, 400,000 points)
constexpr uint32_t kRing = 64;
constexpr long long kWaitCycles = 4000000000ll;     // ~2 s at 1.9 GHz

// Operand forms in memory: K-block planes [kb][row][64 bytes], a row's four
// 16-byte chunks permuted the way the 64-byte swizzle of shared memory wants
// them (chunk ^ (row / 2) % 4, a pattern of 8 rows).  128 rows of a plane from a
// multiple of 8 are then the shared-memory image of one K block, fetched by one
// contiguous bulk copy of 8 KB.  (A tensor-map load with a box of 64-byte rows
// delivered ~8 bytes per cycle and SM whatever d, and the refine ran at its pace.)
// Planes are padded by kRowPad zero rows: a tile may start at the last points.
constexpr uint32_t kRowPad = 512 + 8;
__host__ __device__ __forceinline__ uint64_t plane_rows(uint32_t n) { return ((uint64_t)n + 7u) / 8u * 8u + kRowPad; }

struct TcArgs {
    const HjBlock* blocks;
    uint32_t nblocks;
    uint32_t parts;             // work items per block: each takes 1/parts of the block's candidate tiles
    unsigned int* head;
    const uint32_t* perm;       // sorted position -> original id, bit 31 set for points of silent cells
    const unsigned long long* cell_lid;
    const uint32_t* cell_start;
    HjCellHash hash;
    HjGrid grid;
    const uint8_t* qform;       // operand planes
    const uint8_t* cform;
    unsigned long long plane;   // bytes of one plane
    uint32_t nkb;               // K blocks of 32 elements
    uint32_t qcols;             // query columns per work item: 512, or 256 where shared memory is short
    uint32_t stages;
    float lo;                   // accepted outright: D' <= lo (negative)
    uint32_t sym;               // every unordered pair once: see the symmetric form below
    PairSink sink;              // accepted pairs: (query id, candidate id)
    PairSink band;              // band pairs: (query sorted position, candidate sorted position)
    uint32_t count_only;
    unsigned long long* block_counts;
    unsigned long long* stats;  // [0] accepted, [1] band
    uint32_t* qcount;           // pairs per query id, added up (not in count-only mode)
    uint32_t* err;
    uint32_t fmt;               // operand format of the instruction descriptor (0 FP16, 1 BF16)
    long long wait_cycles;      // bound of every mbarrier wait (SM cycles)
};

struct __align__(16) TcShared {
    uint64_t full_a[kMaxStages];
    uint64_t empty_a[kMaxStages];
    uint64_t full_acc[kAcc];
    uint64_t empty_acc[kAcc];
    uint64_t bfull;
    uint32_t tmem_base;
    uint32_t item;
    uint32_t abort;
    uint32_t ntiles, nr;
    // a ring of hit records per epilogue warp, written by it and read by one hit warp:
    // record k lies in slot k % kRing
    uint32_t done;                         // epilogue warps through with the item
    uint32_t produced[kEpiWarps];          // records written so far
    uint32_t consumed[kEpiWarps];          // and taken
    uint4 ring[kEpiWarps][kRing];          // tile, row | chunk of 32 query columns << 7, hits, accepts
    uint32_t qid[kQBMax];                  // original ids of the query columns
    uint32_t rs[kMaxRanges];               // range start (sorted position)
    uint32_t rl[kMaxRanges];               // range length
    uint32_t tp[kMaxRanges + 1];           // tile prefix
};

// Tiles start at multiples of 8 rows (the swizzle pattern), so a range's first
// tile may begin with up to 7 rows of other points, which the epilogue masks.
__device__ __forceinline__ uint32_t range_tiles(uint32_t start, uint32_t len) {
    return len ? ((start & 7u) + len + kTileRows - 1) / kTileRows : 0u;
}

// Tiles are visited in order, so the range of tile t is found by walking r
// forward from the previous tile's range (the last r with tp[r] <= t; ranges
// without tiles are stepped over) instead of a binary search per tile.  The
// current range's first tile, end tile, start row and length stay in registers,
// so a tile inside the same range costs no shared-memory reads.
struct TileWalk {
    uint32_t start = 0, first = 0, end = 0;    // the tile's rows start + [0, 128); [first, end) are the range's
    uint32_t r = 0, t0 = 0, t1 = 0, rs = 0, rl = 0;   // range r: tiles [t0, t1), rows [rs, rs + rl)
    __device__ __forceinline__ void locate(const TcShared& S, uint32_t t) {
        if (t >= t1) {
            while (r + 1 < S.nr && S.tp[r + 1] <= t) ++r;
            t0 = S.tp[r];
            t1 = r + 1 < S.nr ? S.tp[r + 1] : 0xFFFFFFFFu;
            rs = S.rs[r];
            rl = S.rl[r];
        }
        const uint32_t off = (t - t0) * kTileRows, skip = rs & 7u;
        start = (rs & ~7u) + off;
        first = off ? 0u : skip;
        end = min((uint32_t)kTileRows, skip + rl - off);
    }
};

// The guard band of a pair (q, c): the tensor-core value D of |q~ - c~|^2 differs
// from the reference's FP32 d2 (near the threshold T) by at most
//   acc + e (2 sT + 3 e) + ref_rel (sT + e)^2
//   e   = e_c + e_q           (|x~ - x| norms; |(|q~-c~|) - |q-c|| <= e)
//   acc = gamma (2.01 (|c~|^2 + |q~|^2) + 1.01 T)  (tensor-core accumulation; 2|a.b| <= |a|^2 + |b|^2;
//                              T for the shift in the norm terms, below)
//   the last term bounds the reference's own FP32 rounding of d2 (d + 2 roundings).
// With (e_c + m)^2 <= 2 e_c^2 + 2 m^2 (m = e_q) it splits into a candidate part and a
// query part, delta <= P(c) + Q(q):
//   P(c) = gamma 2.01 |c~|^2 + e_c (2 sT + 6 e_c) + ref_rel (2 sT e_c + 2 e_c^2)
//   Q(q) = gamma (2.01 |q~|^2 + 1.01 T) + m (2 sT + 6 m) + ref_rel (sT^2 + 2 sT m + 2 m^2)
// each with a 2% margin (gamma (P + Q) of the shift itself, and rounding).
//
// The band's upper edge T + P(c) + Q(q) rides in the norm terms of the operands,
//   N_c = |c~|^2 - P(c),   N_q = |q~|^2 - T - Q(q),
// each stored as two halves that are never above it, so the MMA gives
//   D' = |q~ - c~|^2 - (T + P + Q) - (split residuals >= 0):
// a pair is rejected iff D' > 0 -- its sign bit is clear -- and accepted outright
// if D' <= -(2 P + 2 Q + residuals).  The sign test is what the epilogue is made
// of: no threshold per row or column, and three-input ORs cover two values per
// instruction where a minimum covers one.
__host__ __device__ __forceinline__ double tc_band_p(double gamma, double s_t, double ref_rel, double e, double n2) {
    return (gamma * 2.01 * n2 + e * (2.0 * s_t + 6.0 * e) + ref_rel * (2.0 * s_t * e + 2.0 * e * e)) * 1.02;
}
__host__ __device__ __forceinline__ double tc_band_q(double gamma, double s_t, double ref_rel, double e, double n2) {
    return (gamma * (2.01 * n2 + 1.01 * s_t * s_t) + e * (2.0 * s_t + 6.0 * e) +
            ref_rel * (s_t * s_t + 2.0 * s_t * e + 2.0 * e * e)) * 1.02 + 1e-30;
}

// OR of 32 words in eight independent chains (two-input ORs run at twice the rate
// of three-input ones, so the value rate is the same).
__device__ __forceinline__ uint32_t or_all(const uint32_t (&v)[32]) {
    uint32_t m[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) m[i] = (v[i] | v[i + 8]) | (v[i + 16] | v[i + 24]);
    return ((m[0] | m[1]) | (m[2] | m[3])) | ((m[4] | m[5]) | (m[6] | m[7]));
}
// Bit i = sign of at(i), in four independent chains of funnel shifts: a single chain
// of 32 took as long as the rest of an accumulator's epilogue.
template <typename At>
__device__ __forceinline__ uint32_t sign_bits(At&& at) {
    uint32_t m[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int i = 7; i >= 0; --i)
#pragma unroll
        for (int g = 0; g < 4; ++g) m[g] = __funnelshift_l(at(8 * g + i), m[g], 1);
    return (m[0] | m[1] << 8) | (m[2] << 16 | m[3] << 24);
}
__device__ __forceinline__ uint32_t sign_mask(const uint32_t (&v)[32]) {
    return sign_bits([&](int i) { return v[i]; });
}
// Bit i = (v[i] < lo), lo negative.
__device__ __forceinline__ uint32_t below_mask(const uint32_t (&v)[32], float lo) {
    return sign_bits([&](int i) { return __float_as_uint(__uint_as_float(v[i]) - lo); });
}
__device__ __forceinline__ uint32_t low_bits(uint32_t n) { return n >= 32u ? 0xFFFFFFFFu : (1u << n) - 1u; }

// Wait until a ring's counter has reached `want` (bounded like mbar_wait).
__device__ __forceinline__ uint32_t ring_wait(const uint32_t& counter, uint32_t want, volatile uint32_t* abort,
                                              uint32_t* err, long long limit_cycles) {
    const volatile uint32_t* p = &counter;
    uint32_t v = *p;
    if ((int)(v - want) < 0) {
        const long long t0 = clock64();
        while ((int)((v = *p) - want) < 0 && !*abort) {
            if (clock64() - t0 > limit_cycles) {
                *abort = 1u;
                atomicExch(err, 1u);
            }
        }
    }
    __threadfence_block();
    return v;
}

// DENSE: a chunk with a hit has its signs gathered into masks while it is in
// registers (a vote per chunk); otherwise chunks are only ORed (one vote per
// accumulator) and those with a hit are read again before the accumulator is
// released.  18-D, 400,000 points: 5.34 and 5.11 ms; 18-D, 100,003 (half of the chunks
// hold a hit, three hit warps): 0.89 and 0.93 ms; 32-D: 1.72 and 1.78 ms.
//
// Symmetric form (a.sym): d2 is the same number for (q, c) and (c, q), so a join
// that runs all its work items in one batch evaluates each unordered pair once
// and emits both orders.  An item then takes only the cells after its own in
// linear-id order (the stencil is symmetric) and, of its own cell, the points from
// its first query on; candidates before the query are masked.  Cells with a
// coordinate of 0 visit no cell in the reference's stencil (kernel.cu:780 wraps)
// although their neighbours visit them: an item of such a "silent" cell emits
// only (candidate, query) orders, and a silent candidate (bit 31 of perm) only
// (query, candidate).
//
// The epilogue does not emit: a warp that did (ids, a scan, stores: some 2,000 cycles)
// held back its whole set.  Lanes with a hit pass a record on through their warp's ring in
// shared memory, and the hit warps take up to 32 records at a time, one per lane.
//
// Work of one item.  Its query columns make one, two or four groups of up to 128; each
// tile is multiplied with all of them, group g into an accumulator h with h % groups == g,
// and an item of fewer than four groups deals its tiles to the accumulators in turn.
template <bool DENSE>
__global__ void __launch_bounds__(tc_threads(DENSE), 1) k_refine_tc(const __grid_constant__ TcArgs a) {
    extern __shared__ uint8_t smem_raw[];
    // operand tiles need 1024-byte alignment for the swizzle pattern
    uint32_t base = tc::smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (base & 1023u)) & 1023u);
    const uint32_t tile_bytes = a.nkb * kKBlockBytes;
    const uint32_t bkb_bytes = a.qcols * kRowBytes;            // one K block of the query columns
    uint8_t* b_tiles = smem;                                   // queries: [K block][qcols rows]
    uint8_t* a_tiles = smem + a.nkb * bkb_bytes;               // a.stages tiles: [K block][128 rows]
    TcShared& S = *reinterpret_cast<TcShared*>(a_tiles + a.stages * tile_bytes);

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    if (tid == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            tc::mbar_init(&S.full_a[s], 1);
            tc::mbar_init(&S.empty_a[s], kAcc);   // one arrival for each issuer
        }
        for (int j = 0; j < kAcc; ++j) {
            tc::mbar_init(&S.full_acc[j], 1);
            tc::mbar_init(&S.empty_acc[j], kEpiWarps / kAcc);   // the warps draining it
        }
        tc::mbar_init(&S.bfull, 1);
        S.abort = 0;
        tc::fence_mbar_init();
    }
    if (warp == 1) {
        tc::tmem_alloc(&S.tmem_base, kTmemCols);
        tc::tmem_relinquish();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = S.tmem_base;
    volatile uint32_t* abort = &S.abort;

    // role state carried across work items (barrier phases)
    uint32_t stage = 0, use_a = 0;   // the next tile's stage and how often it has been filled before
    uint32_t uses = 0;          // uses of its accumulator issued / drained
    uint32_t items_loaded = 0;
    WarpChunk wc_acc, wc_band;
    warp_chunk_init(wc_acc);
    warp_chunk_init(wc_band);

    for (;;) {
        __syncthreads();
        if (tid == 0) S.item = *abort ? 0xFFFFFFFFu : atomicAdd(a.head, 1u);
        __syncthreads();
        const uint32_t item = S.item;
        const uint32_t bi = item / a.parts;
        if (item == 0xFFFFFFFFu || bi >= a.nblocks) break;
        const HjBlock blk = a.blocks[bi];
        // query columns: positions qbase + [0, ncols), of which the first q0 - qbase are not the item's
        const uint32_t q0 = blk.q0, qbase = q0 & ~7u, ncols = blk.q1 - qbase;
        // column groups: accumulator h takes group h % groups of every (kAcc / groups)-th tile
        uint32_t groups = 1;
        while (groups * kAccCols < ncols) groups *= 2;
        const uint32_t round = kAcc / groups;
        bool q_silent = false;
        {
            // stencil rows of the block's cell -> candidate ranges, a row per thread
            const unsigned long long L = a.cell_lid[blk.cell];
            const uint32_t k = a.grid.k;
            uint32_t lo[kMaxK], w[kMaxK];
            uint32_t rows = 1;
            const uint32_t cl = lane_cell_coord(a.grid, L);
            for (uint32_t j = 0; j < k; ++j) {
                const uint32_t c = __shfl_sync(0xffffffffu, cl, j);
                const uint32_t h = min(a.grid.n_cells[j] - 1u, c + 1u);   // kernel.cu:781
                q_silent |= c == 0u;                                      // kernel.cu:780 wraps at 0
                lo[j] = c == 0u ? 0u : c - 1u;
                w[j] = h - lo[j] + 1u;
                if (j > 0) rows *= w[j];
            }
            if (q_silent && !a.sym) rows = 0;
            const StencilRows sr = stencil_rows(a.grid, lo, rows);
            for (uint32_t r = tid; r < rows; r += blockDim.x) {
                unsigned long long id = stencil_row_id(a.grid, sr, lo, w, r);
                uint32_t wid = w[0];
                bool own = false;
                if (a.sym) {
                    // rows before the cell's own are skipped; its own row starts at the cell itself
                    own = id <= L && L < id + wid;
                    if (own) {
                        wid -= (uint32_t)(L - id);
                        id = L;
                    } else if (id < L) {
                        wid = 0;
                    }
                }
                uint2 sp = make_uint2(0u, 0u);
                if (wid) sp = cell_span(a.hash, a.cell_start, id, wid);
                if (own) sp.x = q0;
                S.rs[r] = sp.x;
                S.rl[r] = sp.y - sp.x;
            }
            if (tid < (uint32_t)kEpiWarps) S.produced[tid] = S.consumed[tid] = 0u;
            if (tid == 0) S.done = 0u;
            for (uint32_t i = tid; i < ncols; i += blockDim.x) S.qid[i] = a.perm[qbase + i] & 0x7FFFFFFFu;
            __syncthreads();
            if (warp == 0) {
                // tiles of 128 rows: their prefix over the ranges
                const uint32_t nr = rows;
                uint32_t tiles_mine[kMaxRanges / 32];
                uint32_t my_tiles = 0;
#pragma unroll
                for (uint32_t s = 0; s < kMaxRanges / 32; ++s) {
                    const uint32_t r = lane * (kMaxRanges / 32) + s;
                    tiles_mine[s] = r < nr ? range_tiles(S.rs[r], S.rl[r]) : 0u;
                    my_tiles += tiles_mine[s];
                }
                uint32_t incl = my_tiles;
                for (int o = 1; o < 32; o <<= 1) {
                    uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= (uint32_t)o) incl += t;
                }
                uint32_t run = incl - my_tiles;
#pragma unroll
                for (uint32_t s = 0; s < kMaxRanges / 32; ++s) {
                    const uint32_t r = lane * (kMaxRanges / 32) + s;
                    if (r < nr) S.tp[r] = run;
                    run += tiles_mine[s];
                }
                if (lane == 31) {
                    S.tp[nr] = incl;
                    S.ntiles = incl;
                    S.nr = nr;
                }
            }
        }
        __syncthreads();
        // this item's tiles [t_lo, t_hi) of the block's
        const uint32_t part = item - bi * a.parts;
        const uint32_t t_lo = (uint32_t)((unsigned long long)S.ntiles * part / a.parts);
        const uint32_t t_hi = (uint32_t)((unsigned long long)S.ntiles * (part + 1) / a.parts);
        if (t_lo == t_hi) continue;

        // Every role's warp walks its loop as a whole and one elected lane issues: a wait
        // inside a one-lane branch took 600 to 1,250 cycles per hand-over against 250 converged.
        if (warp == 0) {
            // ---------------- loads: the query columns once, then the candidate tiles
            const uint32_t qbytes = ((ncols + 31u) & ~31u) * kRowBytes;
            if (tc::elect_one()) {
                tc::mbar_arrive_expect_tx(&S.bfull, a.nkb * qbytes);
                for (uint32_t kb = 0; kb < a.nkb; ++kb)
                    tc::bulk_load(b_tiles + kb * bkb_bytes, a.qform + kb * a.plane + (size_t)qbase * kRowBytes, qbytes,
                                  &S.bfull);
            }
            __syncwarp();
            TileWalk tw;
            for (uint32_t t = t_lo; t < t_hi; ++t) {
                if (use_a > 0) tc::mbar_wait<false>(&S.empty_a[stage], (use_a - 1) & 1u, abort, a.err, a.wait_cycles);
                tw.locate(S, t);
                if (tc::elect_one()) {
                    tc::mbar_arrive_expect_tx(&S.full_a[stage], tile_bytes);
                    for (uint32_t kb = 0; kb < a.nkb; ++kb)
                        tc::bulk_load(a_tiles + stage * tile_bytes + kb * kKBlockBytes,
                                      a.cform + kb * a.plane + (size_t)tw.start * kRowBytes, kKBlockBytes,
                                      &S.full_a[stage]);
                }
                __syncwarp();
                if (++stage == a.stages) { stage = 0; ++use_a; }
            }
        } else if (warp <= kAcc) {
            // ---------------- MMA issuer h (warp 1 + h), into accumulator h
            const uint32_t h = warp - 1;
            tc::mbar_wait(&S.bfull, items_loaded & 1u, abort, a.err, a.wait_cycles);
            const uint32_t first_col = h % groups * kAccCols, turn = h / groups;
            const uint64_t a_desc = tc::desc_kmajor_sw64(tc::smem_u32(a_tiles));
            const uint64_t b_desc =
                tc::desc_kmajor_sw64(tc::smem_u32(b_tiles) + first_col * kRowBytes);
            // N = this group's query columns in whole groups of 32
            const uint32_t cols = ncols > first_col ? min((uint32_t)kAccCols, ncols - first_col) : 32u;
            const uint32_t idesc = tc::idesc_f16(a.fmt, kTileRows, (cols + 31u) & ~31u);
            // A wait names a barrier's phase by one bit, so an issuer may be at most one fill of a
            // stage ahead of the last one that it saw.  Where the stages are a multiple of the round
            // (4 or 8 of them: d <= 124), a stage's tiles within an item are all the same issuer's.
            // Otherwise (2 or 3 stages) every issuer waits for every tile, and those that a tile is
            // not for arrive at the stage's release themselves: no fill is missed, none is overrun.
            const bool in_step = a.stages % round != 0u;
            const uint32_t commits = in_step ? 1u : round;
            for (uint32_t t = t_lo; t < t_hi; ++t) {
                const bool mine = ((t - t_lo) & (round - 1u)) == turn;
                if (mine || in_step) tc::mbar_wait<false>(&S.full_a[stage], use_a & 1u, abort, a.err, a.wait_cycles);
                if (mine) {
                    if (uses > 0) tc::mbar_wait<false>(&S.empty_acc[h], (uses - 1) & 1u, abort, a.err, a.wait_cycles);
                    ++uses;
                    if (tc::elect_one()) {
                        tc::fence_after();
                        uint64_t ad = a_desc + ((stage * tile_bytes) >> 4), bd = b_desc;
                        tc::mma_f16(tmem + h * kAccCols, ad, bd, idesc, 0u);
                        tc::mma_f16(tmem + h * kAccCols, ad + 2u, bd + 2u, idesc, 1u);
                        for (uint32_t kb = 1; kb < a.nkb; ++kb) {
                            ad += kKBlockBytes >> 4;
                            bd += bkb_bytes >> 4;
                            tc::mma_f16(tmem + h * kAccCols, ad, bd, idesc, 1u);
                            tc::mma_f16(tmem + h * kAccCols, ad + 2u, bd + 2u, idesc, 1u);
                        }
                        tc::mma_commit(&S.full_acc[h]);
                        for (uint32_t i = 0; i < commits; ++i) tc::mma_commit(&S.empty_a[stage]);
                    }
                    __syncwarp();
                } else if (in_step) {
                    if (lane == 0) tc::mbar_arrive(&S.empty_a[stage]);
                    __syncwarp();
                }
                if (++stage == a.stages) { stage = 0; ++use_a; }
            }
            ++items_loaded;
        } else if (warp <= kAcc + kEpiWarps) {
            // ---------------- epilogue: warps 5 .. 20, a set of 4 per accumulator, so that a slow
            // warp holds back only its own accumulator.  TMEM lane quarter = warp % 4.
            const uint32_t ew = warp - 1 - kAcc;
            constexpr uint32_t SET = kEpiWarps / kAcc;
            const uint32_t j = ew / SET;   // the accumulator this warp drains
            const uint32_t quarter = warp & 3u;
            const uint32_t row = quarter * 32u + lane;
            // this warp's columns of the accumulator, read in chunks of 32
            constexpr uint32_t COLS = kAccCols / (SET / 4), NCH = COLS / 32;
            const uint32_t acc_col = ew % SET / 4u * COLS;
            const uint32_t acc = tmem + ((quarter * 32u) << 16) + j * kAccCols + acc_col;
            const uint32_t col_base = acc_col + j % groups * kAccCols;   // in query columns
            // chunks that hold queries of this item (the rest of the accumulator is stale)
            const uint32_t nch = ncols > col_base ? min(NCH, (ncols - col_base + 31u) / 32u) : 0u;
            uint32_t prod = 0, room = kRing;   // records written, and how many may be before a look at the reader
            auto publish = [&] {
                __threadfence_block();
                __syncwarp();
                if (lane == 0) *(volatile uint32_t*)&S.produced[ew] = prod;
                __syncwarp();
            };
            for (uint32_t t = t_lo + j / groups; t < t_hi; t += round) {
                tc::mbar_wait<false>(&S.full_acc[j], uses & 1u, abort, a.err, a.wait_cycles);
                ++uses;
                tc::fence_after();
                // per chunk: signs (candidate hits) and outright accepts of this lane's row
                uint32_t hm[NCH], am[NCH];
#pragma unroll
                for (uint32_t c = 0; c < NCH; ++c) hm[c] = am[c] = 0u;
                auto release = [&] {
                    tc::fence_before();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&S.empty_acc[j]);
                };
                uint32_t seen = 0;
                if constexpr (DENSE) {
                    // the accumulator goes back as soon as the last chunk is in registers
                    if (nch == 0u) release();
#pragma unroll
                    for (uint32_t c = 0; c < NCH; ++c) {
                        if (c >= nch) break;
                        uint32_t v[32];
                        tc::tmem_ld_32(acc + c * 32u, v);
                        tc::tmem_wait_32(v);
                        if (c + 1 == nch) release();
                        if (!__any_sync(0xffffffffu, (int)or_all(v) < 0)) continue;
                        seen = 1u;
                        hm[c] = sign_mask(v);
                        am[c] = hm[c] & below_mask(v, a.lo);
                    }
                } else {
                    uint32_t v[32];
#pragma unroll
                    for (uint32_t c = 0; c < NCH; ++c) {
                        if (c >= nch) break;
                        tc::tmem_ld_32(acc + c * 32u, v);
                        tc::tmem_wait_32(v);
                        seen |= (or_all(v) >> 31) << c;
                    }
                    seen = __reduce_or_sync(0xffffffffu, seen);
                    if (!seen) {
                        release();
                        continue;
                    }
#pragma unroll
                    for (uint32_t c = 0; c < NCH; ++c) {
                        if (!((seen >> c) & 1u)) continue;
                        tc::tmem_ld_32(acc + c * 32u, v);
                        tc::tmem_wait_32(v);
                        if (seen >> c == 1u) release();   // the last one to be read again
                        hm[c] = sign_mask(v);
                        am[c] = hm[c] & below_mask(v, a.lo);
                    }
                }
                if (!seen) continue;
                // lanes with a hit pass it on
#pragma unroll
                for (uint32_t c = 0; c < NCH; ++c) {
                    const uint32_t who = __ballot_sync(0xffffffffu, hm[c] != 0u);
                    if (who == 0u) continue;
                    const uint32_t n = __popc(who);
                    if (prod + n > room) {
                        publish();
                        room = ring_wait(S.consumed[ew], prod + n - kRing, abort, a.err, a.wait_cycles) + kRing;
                        __syncwarp();
                        room = __shfl_sync(0xffffffffu, room, 0);
                    }
                    if (hm[c])
                        S.ring[ew][(prod + __popc(who & lanemask_lt())) % kRing] =
                            make_uint4(t, row | ((col_base >> 5) + c) << 7, hm[c], am[c]);
                    prod += n;
                }
                publish();
            }
            __threadfence_block();
            __syncwarp();
            if (lane == 0) atomicAdd(&S.done, 1u);
        } else {
            // ---------------- hits: batches of up to 32 records, one per lane, from this warp's rings:
            // lane l keeps the account of ring hw + l * HW
            constexpr uint32_t HW = hit_warps(DENSE), RINGS = ((uint32_t)kEpiWarps + HW - 1) / HW;
            const uint32_t hw = warp - 1 - kAcc - kEpiWarps, ring = hw + lane * HW;
            const bool mine = ring < (uint32_t)kEpiWarps;
            uint32_t taken = 0;
            uint32_t n_acc = 0, n_band = 0;
            for (;;) {
                uint32_t avail, incl, total;
                const long long t0 = clock64();
                for (uint32_t polls = 0;; ++polls) {
                    // a whole batch, a ring that is half full, what is left once every epilogue warp
                    // is through, or what has waited (its writer may need the room)
                    const uint32_t d = __shfl_sync(0xffffffffu, *(volatile uint32_t*)&S.done, 0);
                    __threadfence_block();
                    avail = mine ? *(volatile uint32_t*)&S.produced[ring] - taken : 0u;
                    const uint32_t stop = *abort;
                    incl = avail;
#pragma unroll
                    for (uint32_t o = 1; o < RINGS; o <<= 1) {
                        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += x;
                    }
                    total = __shfl_sync(0xffffffffu, incl, RINGS - 1);
                    if (__any_sync(0xffffffffu, total >= 32u || avail >= kRing / 2 || d == (uint32_t)kEpiWarps || stop ||
                                                  (total && polls >= 8u)))
                        break;
                    if (clock64() - t0 > a.wait_cycles) {
                        *abort = 1u;
                        atomicExch(a.err, 1u);
                    }
                    __nanosleep(500);
                }
                __threadfence_block();
                const uint32_t n = min(32u, total);
                if (n == 0u) break;
                const uint32_t excl = incl - avail;
                uint32_t src = 0;   // the lane whose ring holds record `lane` of the batch
#pragma unroll
                for (uint32_t l = 0; l + 1 < RINGS; ++l) src += __shfl_sync(0xffffffffu, incl, l) <= lane;
                const uint32_t at = lane - __shfl_sync(0xffffffffu, excl, src) + __shfl_sync(0xffffffffu, taken, src);
                uint4 rec = make_uint4(0u, 0u, 0u, 0u);
                if (lane < n) rec = S.ring[min(hw + src * HW, (uint32_t)kEpiWarps - 1u)][at % kRing];
                __threadfence_block();
                __syncwarp();
                if (mine && excl < n && avail) {
                    taken += min(avail, n - excl);
                    *(volatile uint32_t*)&S.consumed[ring] = taken;
                }
                // the tile's range: the last r with tp[r] <= tile
                uint32_t r = 0;
#pragma unroll
                for (uint32_t step = kMaxRanges / 2; step > 0; step >>= 1)
                    if (r + step < S.nr && S.tp[r + step] <= rec.x) r += step;
                const uint32_t rs = S.rs[r], off = (rec.x - S.tp[r]) * kTileRows, skip = rs & 7u;
                const uint32_t row = rec.y & 127u, in_range = off + row;   // from the range's aligned start
                const uint32_t cpos = (rs & ~7u) + in_range;
                const uint32_t pos0 = qbase + (rec.y >> 7) * 32u;          // query position of bit 0
                // rows past the range's end and columns past the queries are other points'; in the
                // symmetric form a candidate pairs with the queries up to its own position
                const bool in = rec.z != 0u && in_range >= skip && in_range < skip + S.rl[r];
                const uint32_t lim = in ? (a.sym ? min(blk.q1, cpos + 1u) : blk.q1) : 0u;
                uint32_t hits = lim > pos0 ? rec.z & low_bits(lim - pos0) : 0u;
                if (pos0 < q0) hits &= ~low_bits(q0 - pos0);
                // a silent candidate of a silent query: the pair is neither's
                const uint32_t cw = hits && !a.count_only ? a.perm[cpos] : 0u, cid = cw & 0x7FFFFFFFu;
                const bool fwd = !q_silent, rev = a.sym && !(cw >> 31);
                if (a.sym && !fwd && !rev) hits = 0u;
                uint32_t acc = hits & rec.w;
                uint32_t bnd = hits & ~rec.w;
                const uint32_t na = __popc(acc), nb = __popc(bnd);
                if (a.count_only) {
                    n_band += na + nb;
                } else {
                    const uint32_t self = a.sym && in ? cpos - pos0 : 0xFFFFFFFFu;   // bit of the candidate itself
                    // accepted pairs go out in both orders (symmetric form), that of a point with itself once
                    const uint32_t self_bit = self < 32u ? 1u << self : 0u;
                    // orders that the named pairs stand for, and those of them with the candidate first
                    auto reversed = [&](uint32_t m) { return rev ? (uint32_t)__popc(m & ~self_bit) : 0u; };
                    auto orders = [&](uint32_t m) { return (fwd ? (uint32_t)__popc(m) : 0u) + reversed(m); };
                    if (__any_sync(0xffffffffu, na)) {
                        const uint32_t cnt = orders(acc), cnt_rev = reversed(acc);
                        n_acc += cnt;
                        if (cnt_rev) atomicAdd(&a.qcount[cid], cnt_rev);
                        warp_emit_serial(a.sink, wc_acc, cnt, [&](auto&& put) {
                            while (acc) {
                                const uint32_t b = __ffs(acc) - 1u;
                                acc &= acc - 1u;
                                const uint32_t qid = S.qid[pos0 - qbase + b];
                                if (fwd) {
                                    put(qid, cid);
                                    atomicAdd(&a.qcount[qid], 1u);
                                }
                                if (rev && b != self) put(cid, qid);
                            }
                        });
                    }
                    if (__any_sync(0xffffffffu, nb)) {
                        n_band += orders(bnd);
                        warp_emit_serial(a.band, wc_band, nb, [&](auto&& put) {
                            while (bnd) {
                                const uint32_t b = __ffs(bnd) - 1u;
                                bnd &= bnd - 1u;
                                put(pos0 + b, cpos);
                            }
                        });
                    }
                }
            }
            unsigned long long w_acc = n_acc, w_band = n_band;
            for (int o = 16; o > 0; o >>= 1) {
                w_acc += __shfl_down_sync(0xffffffffu, w_acc, o);
                w_band += __shfl_down_sync(0xffffffffu, w_band, o);
            }
            if (lane == 0) {
                if (a.count_only) {
                    if (w_acc + w_band) atomicAdd(&a.block_counts[bi], w_acc + w_band);
                } else if (a.stats) {
                    if (w_acc) atomicAdd(&a.stats[0], w_acc);
                    if (w_band) atomicAdd(&a.stats[1], w_band);
                }
            }
        }
    }
    if (warp > kAcc + kEpiWarps && !a.count_only) {
        warp_chunk_close(a.sink, wc_acc);
        warp_chunk_close(a.band, wc_band);
    }
    if (*abort) {
        // after a timeout copies may still be in flight (a microsecond or two): let them land
        const long long t0 = clock64();
        while (clock64() - t0 < 200000ll) {}
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, kTmemCols);
    }
}

// Band pairs: exact FP32 refine in the reference's order (kernel.cu:350-355).
// sym: a pair stands for both orders (see the symmetric form above).
__global__ void k_band_recheck(const float* __restrict__ pts, const uint32_t* __restrict__ perm, uint32_t d,
                               float thr, const uint32_t* __restrict__ bq, const uint32_t* __restrict__ bc,
                               const unsigned long long* __restrict__ band_used, unsigned long long band_cap,
                               uint32_t sym, PairSink sink, uint32_t* __restrict__ qcount) {
    // after an overflow the band holds slots that were reserved and never written (the batch is
    // run again in any case)
    if (*(volatile const uint32_t*)sink.overflow) return;
    const unsigned long long n = min(*band_used, band_cap);
    WarpChunk wc;
    warp_chunk_init(wc);
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x; base < n; base += stride) {
        unsigned long long i = base + threadIdx.x;
        uint32_t qid = 0, cid = 0;
        bool fwd = false, rev = false;
        if (i < n) {
            const uint32_t qp = bq[i];
            if (qp != kSentinelKey) {
                const uint32_t cp = bc[i];
                const float* q = pts + (size_t)qp * d;
                const float* c = pts + (size_t)cp * d;
                float acc = 0.f;
                for (uint32_t l = 0; l < d; ++l) {
                    float diff = __fsub_rn(c[l], q[l]);
                    acc = __fmaf_rn(diff, diff, acc);
                }
                if (acc <= thr) {
                    const uint32_t qw = perm[qp], cw = perm[cp];
                    qid = qw & 0x7FFFFFFFu;
                    cid = cw & 0x7FFFFFFFu;
                    fwd = !(qw >> 31);
                    rev = sym && !(cw >> 31) && qp != cp;
                    if (fwd) atomicAdd(&qcount[qid], 1u);
                    if (rev) atomicAdd(&qcount[cid], 1u);
                }
            }
        }
        warp_emit(sink, wc, (fwd ? 1u : 0u) + (rev ? 1u : 0u), [&](uint32_t j) {
            return fwd && j == 0 ? make_uint2(qid, cid) : make_uint2(cid, qid);
        });
    }
    warp_chunk_close(sink, wc);
}

// Operand preparation: one thread per sorted point.
template <typename H>
__device__ __forceinline__ H to_h(double x);
template <>
__device__ __forceinline__ __half to_h<__half>(double x) { return __double2half(x); }
template <>
__device__ __forceinline__ __nv_bfloat16 to_h<__nv_bfloat16>(double x) { return __double2bfloat16(x); }
__device__ __forceinline__ double from_h(__half h) { return (double)__half2float(h); }
__device__ __forceinline__ double from_h(__nv_bfloat16 h) { return (double)__bfloat162float(h); }

// Block-wide maximum of non-negative values, folded into *out with one atomic
// per block (non-negative IEEE values order like their bit patterns).
__device__ __forceinline__ void block_max_into(double v, unsigned long long* out) {
    __shared__ double part[32];
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane_id() == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (threadIdx.x == 0 && v > 0) atomicMax(out, (unsigned long long)__double_as_longlong(v));
    }
}

// Largest |x - origin|^2 over the points, in FP64 (the scale of the operand
// forms is chosen from it), and whether any coordinate is not finite.
__global__ void k_tc_range(const float* __restrict__ pts, uint32_t n, uint32_t d, const float* __restrict__ origin,
                           unsigned long long* __restrict__ max_n2, uint32_t* __restrict__ nonfinite) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double n2 = 0;
    bool bad = false;
    if (i < n) {
        for (uint32_t l = 0; l < d; ++l) {
            const float v = pts[i * d + l];
            bad |= !isfinite(v);
            const double x = (double)v - (double)origin[l];
            n2 += x * x;
        }
    }
    if (__any_sync(0xffffffffu, bad) && lane_id() == 0) atomicOr(nonfinite, 1u);
    block_max_into(bad ? 0.0 : n2, max_n2);
}

// The two halves of a norm term N: their sum is never above it (the filter may
// only err towards the recheck).  N is at least -60000, finite in FP16: a term
// cut off there belongs to a pair whose D' is negative anyway (the other terms
// are at most 2^14).
template <typename H>
__device__ __forceinline__ H to_h_down(double x);
template <>
__device__ __forceinline__ __half to_h_down<__half>(double x) { return __float2half_rd(__double2float_rd(x)); }
template <>
__device__ __forceinline__ __nv_bfloat16 to_h_down<__nv_bfloat16>(double x) {
    return __float2bfloat16_rd(__double2float_rd(x));
}
template <typename H>
__device__ __forceinline__ double split_norm(double n, H& hi, H& lo) {
    n = fmax(n, -60000.0);
    hi = to_h<H>(n);
    lo = to_h_down<H>(n - from_h(hi));
    return n - from_h(hi) - from_h(lo);   // the residual, >= 0
}

// Constants of the guard band (scaled units).
struct TcBand {
    double thr, gamma, s_t, ref_rel;
};

// Operand forms of sorted points [row0, row0 + rows), one thread each, written to
// plane rows 0..; rows past n and up to plane_n are zero.  Units are scaled by
// `scale` (a power of two): x~ = half((x - origin) * scale).  shift: the norm
// terms carry the threshold and the guard band (the filter); otherwise they are
// |x~|^2 (the tile probe).  Folds the maxima of the bound terms into
// maxima[0..4] (float bits): e, |x~|^2, residual, 2 P + residual, 2 Q + residual.
// A block stages its 64 points in shared memory with coalesced loads (rows padded
// to an odd stride); a thread writes its rows in 16-byte chunks, neighbouring
// threads neighbouring rows.  Either form may be null.
constexpr int kTcMaxima = 5;
constexpr int kPrepRows = 64;
template <typename H>
__global__ void __launch_bounds__(kPrepRows)
    k_tc_prep(const float* __restrict__ pts, uint32_t n, uint32_t d, uint32_t nkb, const float* __restrict__ origin,
              double scale, TcBand band, uint32_t shift, uint32_t row0, unsigned long long plane_n,
              H* __restrict__ qform, H* __restrict__ cform, unsigned int* __restrict__ maxima) {
    extern __shared__ float prep_s[];
    const uint32_t stride = d | 1u;
    const unsigned long long first = (unsigned long long)blockIdx.x * kPrepRows;   // plane row
    const uint32_t src0 = row0 + (uint32_t)first;
    const uint32_t have = src0 < n ? min((uint32_t)kPrepRows, n - src0) : 0u;
    for (uint32_t f = threadIdx.x; f < have * d; f += kPrepRows) {
        const uint32_t i = f / d, l = f - i * d;
        prep_s[i * stride + l] = pts[(size_t)src0 * d + f];
    }
    __syncthreads();
    const unsigned long long row = first + threadIdx.x;
    float m[kTcMaxima] = {0.f, 0.f, 0.f, 0.f, 0.f};
    if (row < plane_n) {
        const bool real = threadIdx.x < have;
        const float* x_s = prep_s + threadIdx.x * stride;
        const H zero = to_h<H>(0.0), one = to_h<H>(1.0);
        double n2 = 0, e2 = 0;
        auto put = [&](uint32_t chunk, const H (&q)[8], const H (&c)[8]) {
            const unsigned long long at = ((unsigned long long)(chunk >> 2) * plane_n + row) * 4u +
                                          ((chunk & 3u) ^ ((uint32_t)(row >> 1) & 3u));
            if (qform) reinterpret_cast<uint4*>(qform)[at] = *reinterpret_cast<const uint4*>(q);
            if (cform) reinterpret_cast<uint4*>(cform)[at] = *reinterpret_cast<const uint4*>(c);
        };
        const uint32_t whole = d / 8u;   // chunks of coordinates only
        for (uint32_t ch = 0; ch < whole; ++ch) {
            __align__(16) H q[8], c[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t l = ch * 8u + i;
                const double x = real ? ((double)x_s[l] - (double)origin[l]) * scale : 0.0;   // exact: scale is 2^s
                const double xt = from_h(q[i] = to_h<H>(x));
                c[i] = to_h<H>(-2.0 * xt);
                e2 += (xt - x) * (xt - x);
                n2 += xt * xt;
            }
            if (!real)
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) q[i] = c[i] = zero;
            put(ch, q, c);
        }
        // the last coordinates, then the norm terms and zeros
        for (uint32_t l = whole * 8u; l < d; ++l) {
            const double x = real ? ((double)x_s[l] - (double)origin[l]) * scale : 0.0;
            const double xt = from_h(to_h<H>(x));
            e2 += (xt - x) * (xt - x);
            n2 += xt * xt;
        }
        const double e = sqrt(e2);
        const double P = tc_band_p(band.gamma, band.s_t, band.ref_rel, e, n2);
        const double Q = tc_band_q(band.gamma, band.s_t, band.ref_rel, e, n2);
        H qh, ql, cnh, cnl;
        const double rq = split_norm<H>(shift ? n2 - band.thr - Q : n2, qh, ql);
        const double rc = split_norm<H>(shift ? n2 - P : n2, cnh, cnl);
        for (uint32_t ch = whole; ch < nkb * 4u; ++ch) {
            __align__(16) H q[8], c[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t l = ch * 8u + i;
                q[i] = c[i] = zero;
                if (!real) continue;
                if (l < d) {
                    const double x = ((double)x_s[l] - (double)origin[l]) * scale;
                    q[i] = to_h<H>(x);
                    c[i] = to_h<H>(-2.0 * from_h(q[i]));
                } else if (l < d + 4u) {
                    const uint32_t w = l - d;
                    q[i] = w == 0 ? qh : w == 1 ? ql : one;
                    c[i] = w == 2 ? cnh : w == 3 ? cnl : one;
                }
            }
            put(ch, q, c);
        }
        if (real) {
            // round the bounds up: float conversion is to nearest, so scale by 1 + 2^-20
            const float up = 1.0f + 9.6e-7f;
            m[0] = (float)e * up;
            m[1] = (float)n2 * up;
            m[2] = (float)fmax(rq, rc) * up + 1e-30f;
            m[3] = (float)(2.0 * P + rc) * up + 1e-30f;
            m[4] = (float)(2.0 * Q + rq) * up + 1e-30f;
        }
    }
#pragma unroll
    for (int j = 0; j < kTcMaxima; ++j) {
        float v = m[j];
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane_id() == 0 && v > 0.f) atomicMax(&maxima[j], __float_as_uint(v));
    }
}

// Per-dimension minimum of the points: lanes walk a row's dimensions (coalesced
// reads), warps stride over rows, one atomic per (block, dimension).
__global__ void k_col_min(const float* __restrict__ pts, uint32_t n, uint32_t d, float* __restrict__ out) {
    extern __shared__ float part[];   // [warps][d]
    const uint32_t warps = blockDim.x >> 5, w = threadIdx.x >> 5;
    for (uint32_t l = lane_id(); l < d; l += 32) part[w * d + l] = INFINITY;
    for (uint32_t i = blockIdx.x * warps + w; i < n; i += gridDim.x * warps)
        for (uint32_t l = lane_id(); l < d; l += 32) part[w * d + l] = fminf(part[w * d + l], pts[(size_t)i * d + l]);
    __syncthreads();
    for (uint32_t l = threadIdx.x; l < d; l += blockDim.x) {
        float m = INFINITY;
        for (uint32_t k = 0; k < warps; ++k) m = fminf(m, part[k * d + l]);
        // non-negative floats order like their bit patterns as ints; negative ones
        // order in reverse as unsigned ints
        if (m >= 0.f) atomicMin(reinterpret_cast<int*>(out) + l, __float_as_int(m));
        else atomicMax(reinterpret_cast<unsigned int*>(out) + l, __float_as_uint(m));
    }
}

__global__ void k_fill_f32(float* p, uint32_t n, float v) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

// Debug/test kernel: one candidate tile (plane rows 0..127 of cform) against 512
// query rows (plane rows 0..511 of qform) through the same copies, descriptors and
// MMA sequence as k_refine_tc; writes every accumulator value to out[128][512].
__global__ void __launch_bounds__(kProbeThreads, 1)
    k_tc_tile_probe(const uint8_t* __restrict__ cform, const uint8_t* __restrict__ qform, unsigned long long plane,
                    uint32_t nkb, uint32_t idesc, float* __restrict__ out, uint32_t* err, uint32_t skip_mma,
                    long long wait_cycles) {
    extern __shared__ uint8_t smem_raw[];
    uint32_t base = tc::smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (base & 1023u)) & 1023u);
    const uint32_t tile_bytes = nkb * kKBlockBytes;
    constexpr uint32_t bkb_bytes = kProbeQB * kRowBytes;
    uint8_t* b_tiles = smem;
    uint8_t* a_tile = smem + nkb * bkb_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(a_tile + tile_bytes);   // [0] loads, [1] mma
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2);
    uint32_t* abortp = tslot + 1;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    if (tid == 0) {
        tc::mbar_init(&bars[0], 1);
        tc::mbar_init(&bars[1], 1);
        *abortp = 0;
        tc::fence_mbar_init();
    }
    if (warp == 1) {
        tc::tmem_alloc(tslot, kTmemCols);
        tc::tmem_relinquish();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;
    if (tid == 0) {
        tc::mbar_arrive_expect_tx(&bars[0], nkb * (bkb_bytes + kKBlockBytes));
        for (uint32_t kb = 0; kb < nkb; ++kb) {
            tc::bulk_load(a_tile + kb * kKBlockBytes, cform + kb * plane, kKBlockBytes, &bars[0]);
            tc::bulk_load(b_tiles + kb * bkb_bytes, qform + kb * plane, bkb_bytes, &bars[0]);
        }
    }
    if (tid == 32) {
        // the loads always complete before this thread goes on, so with skip_mma no
        // TMA transfer is in flight while the epilogue's wait runs out
        bool ok = tc::mbar_wait(&bars[0], 0, abortp, err, wait_cycles);
        tc::fence_after();
        if (ok && !skip_mma) {
            for (uint32_t j = 0; j < kAcc; ++j)
                for (uint32_t ks = 0; ks < nkb * 2; ++ks) {
                    const uint32_t kin = (ks & 1u) * 32u;
                    tc::mma_f16(tmem + j * kAccCols,
                                tc::desc_kmajor_sw64(tc::smem_u32(a_tile) + (ks >> 1) * kKBlockBytes + kin),
                                tc::desc_kmajor_sw64(tc::smem_u32(b_tiles) + (ks >> 1) * bkb_bytes +
                                                     j * (kAccCols * 64u) + kin),
                                idesc, ks > 0 ? 1u : 0u);
                }
        }
        // skip_mma: no MMA and no commit, so the wait below runs out (the timeout test)
        if (!skip_mma) tc::mma_commit(&bars[1]);
    }
    if (warp >= 2) {
        const uint32_t quarter = warp & 3u;
        bool ok = tc::mbar_wait(&bars[1], 0, abortp, err, wait_cycles);
        tc::fence_after();
        if (ok) {
            for (uint32_t col = 0; col < (uint32_t)kProbeQB; col += 32) {
                uint32_t v[32];
                tc::tmem_ld_32(tmem + ((quarter * 32u) << 16) + col, v);
                tc::tmem_wait_32(v);
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    out[(size_t)(quarter * 32 + lane) * kProbeQB + col + i] = __uint_as_float(v[i]);
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, kTmemCols);
    }
}

// ---- host side -------------------------------------------------------------------------
uint32_t kpad_for(uint32_t d) { return ((d + 4 + 31) / 32) * 32; }

// The float constants of the guard band, shared by the per-point terms and the kernel.
float band_s_t(double thr_s) { return (float)(std::sqrt(thr_s * (1 + 1e-4)) * (1 + 1e-6)); }   // sqrt(T (1 + 1e-4))
float band_ref_rel(uint32_t d) { return (float)((d + 2) * std::ldexp(1.0, -24) * 1.01); }
// Accumulation model: each K=16 MMA step adds 16 exact products to the FP32
// accumulator with at most 2 ulps of the largest magnitude per term lost
// (alignment and truncation); bound = (steps + 1) * 32 * 2^-23 * sum|terms|.
float band_gamma(uint32_t kpad) { return (float)((kpad / 16 + 1) * 32 * std::ldexp(1.0, -23)); }

size_t tc_smem_bytes(uint32_t nkb, uint32_t qcols, uint32_t stages) {
    return 1024 + (size_t)nkb * ((size_t)qcols * kRowBytes + (size_t)stages * kKBlockBytes) + sizeof(TcShared);
}
constexpr size_t kSmemBudget = 225 * 1024;

// Query columns per work item: 512 (each candidate tile fetched once for all four
// accumulators) where three stages fit beside them, else 256.
uint32_t tc_qcols(uint32_t nkb) { return tc_smem_bytes(nkb, kQBMax, 3) <= kSmemBudget ? kQBMax : kQBMax / 2; }

uint32_t tc_stages(uint32_t nkb) {
    uint32_t s = kMaxStages;
    while (s > 2 && tc_smem_bytes(nkb, tc_qcols(nkb), s) > kSmemBudget) --s;
    return s;
}

}  // namespace

struct TcState {
    float gamma_acc = 0;
    int scale_exp = 0;        // operand forms hold (x - origin) * 2^scale_exp
    double thr_s = 0;         // the squared threshold in those units: thr * 4^scale_exp, exact
    float max_e = 0, max_n = 0, max_r = 0;   // maxima of the per-point bound terms (scaled units)
    float lo = 0;             // accepted outright: D' <= lo
};

static TcState* tc_state(const hj_index* ix) { return reinterpret_cast<TcState*>(ix->tc_state); }

bool tc_supported(const hj_index* ix, int kind) {
    if (ix->dtype != HJ_F32 || ix->d < 8) return false;
    if (kind != HJ_REFINE_TC_F16 && kind != HJ_REFINE_TC_BF16) return false;
    uint32_t nkb = kpad_for(ix->d) / 32;
    if (tc_smem_bytes(nkb, kQBMax / 2, 2) > kSmemBudget) return false;
    uint32_t rows = 1;
    for (uint32_t j = 1; j < ix->k; ++j) rows *= 3;
    return rows <= kMaxRanges && ix->n < 0x7FFFFF00u;
}

uint32_t tc_query_block(const hj_index* ix) { return tc_qcols(kpad_for(ix->d) / 32); }

// Work items per block of queries: a list too short to fill the SMs evenly (16
// items each) has its blocks' candidate tiles cut into up to 32 parts.
static uint32_t tc_parts(uint32_t nblocks) {
    const uint32_t want = 16u * (uint32_t)num_sms(), nb = std::max<uint32_t>(nblocks, 1);
    return std::min<uint32_t>(32u, (want + nb - 1) / nb);
}

// Band recheck grid for a refine over nblocks work items: as many blocks as there
// are SMs x 8, but no more than 8 per refine CTA (small joins have small bands).
static unsigned recheck_grid(uint32_t nblocks) {
    return (unsigned)std::min<uint64_t>((uint64_t)num_sms() * 8, 8ull * std::max<uint32_t>(1, std::min<uint32_t>(nblocks, num_sms())));
}

// Upper bound on the warps that reserve chunks of one sink during one batch: the
// refine's hit warps (one CTA per SM) and the band recheck's warps (8 per block),
// each holding at most one partly filled chunk.
uint64_t tc_emit_warps(uint32_t nblocks) {
    return std::min<uint64_t>((uint64_t)num_sms(), (uint64_t)std::max<uint32_t>(nblocks, 1) * tc_parts(nblocks)) * (uint64_t)hit_warps(true) +
           (uint64_t)recheck_grid(nblocks) * 8ull;
}

// Half-width of the guard band for the worst pair of the dataset, in scaled units.
static double tc_delta_scaled(const hj_index* ix, const TcState* s) {
    const double sT = band_s_t(s->thr_s), ref = band_ref_rel(ix->d), g = s->gamma_acc;
    return tc_band_p(g, sT, ref, s->max_e, s->max_n) + tc_band_q(g, sT, ref, s->max_e, s->max_n) + 2.0 * s->max_r;
}

// The same in the dataset's units (the figure the join reports).
double tc_delta(const hj_index* ix) {
    TcState* s = tc_state(ix);
    if (!s) return 0;
    return std::ldexp(tc_delta_scaled(ix, s), -2 * s->scale_exp);
}

// Band half-width over the threshold: where it is large the filter decides
// little and nearly every neighbour goes through the exact recheck.
double tc_band_ratio(const hj_index* ix) {
    TcState* s = tc_state(ix);
    if (!s) return 1e300;
    return s->thr_s > 0 ? tc_delta_scaled(ix, s) / s->thr_s : 1e300;
}

int tc_scale_exp(const hj_index* ix) {
    TcState* s = tc_state(ix);
    return s ? s->scale_exp : 0;
}

void tc_release(hj_index* ix) {
    delete tc_state(ix);
    ix->tc_state = nullptr;
}

// Power-of-two exponent s for the operand forms: the largest |x - origin|^2
// times 4^s lands in (2^12, 2^14], and the threshold times 4^s stays a normal
// float (so scaling it is exact).  Returns false when both cannot hold.
static bool choose_scale(double max_n2, double thr, int* out) {
    int s = 0;
    if (max_n2 > 0) {
        int e2 = 0;
        std::frexp(max_n2, &e2);                 // max_n2 in [2^(e2-1), 2^e2)
        s = (14 - e2) >> 1;                      // floor((14 - e2) / 2)
        while (s > -600 && std::ldexp(max_n2, 2 * s) > 16384.0) --s;
        while (s < 600 && std::ldexp(max_n2, 2 * s + 2) <= 16384.0) ++s;
    }
    if (thr > 0) {
        // keep T * 4^s within [2^-100, 2^100]: exact in float and far from overflow
        while (std::ldexp(thr, 2 * s) > std::ldexp(1.0, 100)) --s;
        if (std::ldexp(thr, 2 * s) < std::ldexp(1.0, -100)) return false;
    }
    if (max_n2 > 0 && std::ldexp(max_n2, 2 * s) > 16384.0 * 1.0001) return false;
    *out = s;
    return true;
}

// Per-dimension minima of the points (the operand forms' origin).
static hj_status launch_col_min(const hj_index* ix, float* origin, cudaStream_t st) {
    const uint32_t n = ix->n, d = ix->d;
    k_fill_f32<<<(d + 255) / 256, 256, 0, st>>>(origin, d, INFINITY);
    HJ_LAUNCHED();
    const unsigned blocks = (unsigned)std::min<uint32_t>(num_sms() * 2, std::max<uint32_t>(1, n / 64));
    k_col_min<<<blocks, 256, (size_t)8 * d * sizeof(float), st>>>((const float*)ix->pts, n, d, origin);
    HJ_LAUNCHED();
    return HJ_OK;
}

// Operand forms of `rows` plane rows from sorted point row0 (all planes, padding rows zero).
static hj_status launch_prep(const hj_index* ix, int kind, const float* origin, int sexp, const TcBand& band,
                             uint32_t shift, uint32_t row0, uint64_t rows, void* qf, void* cf, unsigned int* mx,
                             cudaStream_t st) {
    const uint32_t n = ix->n, d = ix->d, nkb = kpad_for(d) / 32;
    const unsigned blocks = (unsigned)((rows + kPrepRows - 1) / kPrepRows);
    const size_t smem = (size_t)kPrepRows * (d | 1u) * sizeof(float);
    const double scale = std::ldexp(1.0, sexp);
    if (kind == HJ_REFINE_TC_BF16) {
        HJ_TRY(ensure_smem(k_tc_prep<__nv_bfloat16>, smem));
        k_tc_prep<__nv_bfloat16><<<blocks, kPrepRows, smem, st>>>((const float*)ix->pts, n, d, nkb, origin, scale, band,
                                                                  shift, row0, rows, (__nv_bfloat16*)qf,
                                                                  (__nv_bfloat16*)cf, mx);
    } else {
        HJ_TRY(ensure_smem(k_tc_prep<__half>, smem));
        k_tc_prep<__half><<<blocks, kPrepRows, smem, st>>>((const float*)ix->pts, n, d, nkb, origin, scale, band, shift,
                                                           row0, rows, (__half*)qf, (__half*)cf, mx);
    }
    return launch_status(__FILE__, __LINE__);
}

hj_status tc_prepare(hj_index* ix, int kind, cudaStream_t st) {
    if (ix->tc_kind == kind && ix->tc_state) return HJ_OK;
    // Drop the previous operand forms before anything else: if a step below
    // fails, nothing may be left pointing at freed buffers.
    tc_release(ix);
    ix->tc_kind = -1;
    dfree(ix->tc_a, st);
    dfree(ix->tc_b, st);
    const uint32_t kpad = kpad_for(ix->d), n = ix->n, d = ix->d;
    uint16_t *qf = nullptr, *cf = nullptr;
    float* origin = nullptr;
    unsigned long long* rng = nullptr;   // [0] max |x - origin|^2 (FP64 bits), [1] non-finite flag
    unsigned int* mx = nullptr;          // maxima of the bound terms (float bits)
    auto fail = [&](hj_status e) {
        cudaGetLastError();
        dfree(qf, st); dfree(cf, st); dfree(origin, st); dfree(rng, st); dfree(mx, st);
        return e;
    };
#define TC_TRY(x) do { hj_status e_ = (x); if (e_ != HJ_OK) return fail(e_); } while (0)
    const uint64_t rows = plane_rows(n);
    TC_TRY(dalloc(&qf, (size_t)rows * kpad, st));
    TC_TRY(dalloc(&cf, (size_t)rows * kpad, st));
    TC_TRY(dalloc(&origin, d, st));
    TC_TRY(dalloc(&rng, 2, st));
    TC_TRY(dalloc(&mx, kTcMaxima, st));
    TC_TRY(cuda_status(cudaMemsetAsync(rng, 0, 2 * sizeof(unsigned long long), st), "clear range scratch"));
    TC_TRY(cuda_status(cudaMemsetAsync(mx, 0, kTcMaxima * sizeof(unsigned int), st), "clear maxima"));
    TC_TRY(launch_col_min(ix, origin, st));
    const unsigned pblocks = std::max<uint32_t>(1, (n + 255) / 256);
    k_tc_range<<<pblocks, 256, 0, st>>>((const float*)ix->pts, n, d, origin, rng,
                                        reinterpret_cast<uint32_t*>(rng + 1));
    TC_TRY(launch_status(__FILE__, __LINE__));
    unsigned long long hr[2] = {0, 0};
    TC_TRY(cuda_status(cudaMemcpyAsync(hr, rng, sizeof(hr), cudaMemcpyDeviceToHost, st), "range to host"));
    TC_TRY(cuda_status(cudaStreamSynchronize(st), "range sync"));
    if (hr[1]) {
        set_error("the tensor-core filter needs finite coordinates (the dataset holds inf or NaN)");
        return fail(HJ_ERR_UNSUPPORTED);
    }
    double max_n2 = 0;
    std::memcpy(&max_n2, &hr[0], sizeof(double));
    int sexp = 0;
    if (!choose_scale(max_n2, ix->thr, &sexp)) {
        set_error("the tensor-core filter cannot scale this dataset: eps^2 / max |x - min|^2 = %g is below 2^-114",
                  ix->thr / max_n2);
        return fail(HJ_ERR_UNSUPPORTED);
    }
    const double thr_s = std::ldexp(ix->thr, 2 * sexp);
    const TcBand band{thr_s, band_gamma(kpad), band_s_t(thr_s), band_ref_rel(d)};
    TC_TRY(launch_prep(ix, kind, origin, sexp, band, 1u, 0, rows, qf, cf, mx, st));
    float hm[kTcMaxima];
    TC_TRY(cuda_status(cudaMemcpyAsync(hm, mx, sizeof(hm), cudaMemcpyDeviceToHost, st), "maxima to host"));
    TC_TRY(cuda_status(cudaStreamSynchronize(st), "maxima sync"));
#undef TC_TRY
    dfree(origin, st);
    dfree(rng, st);
    dfree(mx, st);
    TcState* s = new TcState();
    s->gamma_acc = (float)band.gamma;
    s->scale_exp = sexp;
    s->thr_s = thr_s;
    s->max_e = hm[0];
    s->max_n = hm[1];
    s->max_r = hm[2];
    s->lo = -std::nextafter(hm[3] + hm[4], INFINITY);
    ix->tc_a = qf;
    ix->tc_b = cf;
    ix->tc_kpad = kpad;
    ix->tc_state = s;
    ix->tc_kind = kind;
    return HJ_OK;
}

// sym: blocks[0..nblocks) is the join's whole list, each unordered pair once.  dense:
// the epilogue's form (k_refine_tc), a choice of this launch's caller alone.
hj_status launch_refine_tc(const hj_index* ix, const HjBlock* blocks, uint32_t nblocks, unsigned int* head,
                           const PairSink& sink, const PairSink& band, uint32_t count_only, bool sym, bool dense,
                           unsigned long long* block_counts, unsigned long long* stats, uint32_t* qcount,
                           uint32_t* err, cudaStream_t st) {
    if (nblocks == 0) return HJ_OK;
    const TcState* s = tc_state(ix);
    if (!s) { set_error("tensor-core operands not prepared"); return HJ_ERR_INVALID; }
    const uint32_t nkb = ix->tc_kpad / 32, qcols = tc_qcols(nkb), stages = tc_stages(nkb);
    size_t smem = tc_smem_bytes(nkb, qcols, stages);
    // one CTA per SM: ask for more than half of the SM's shared memory
    smem = std::max<size_t>(smem, 116 * 1024);
    auto kern = dense ? k_refine_tc<true> : k_refine_tc<false>;
    HJ_TRY(ensure_smem(kern, smem));
    TcArgs a{};
    a.blocks = blocks; a.nblocks = nblocks; a.parts = tc_parts(nblocks); a.head = head;
    a.perm = sym ? flagged_perm(ix) : ix->perm;
    a.cell_lid = ix->cell_lid; a.cell_start = ix->cell_start; a.grid = ix->grid;
    a.hash = cell_hash(ix);
    a.qform = (const uint8_t*)ix->tc_a; a.cform = (const uint8_t*)ix->tc_b;
    a.plane = plane_rows(ix->n) * kRowBytes;
    a.nkb = nkb; a.qcols = qcols; a.stages = stages;
    a.lo = s->lo;
    a.sym = sym ? 1u : 0u;
    a.sink = sink; a.band = band;
    a.count_only = count_only; a.block_counts = block_counts; a.stats = stats;
    a.qcount = qcount; a.err = err;
    a.fmt = ix->tc_kind == HJ_REFINE_TC_BF16 ? 1u : 0u;
    a.wait_cycles = kWaitCycles;
    unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)num_sms(), (uint64_t)nblocks * a.parts);
    kern<<<grid, tc_threads(dense), smem, st>>>(a);
    HJ_LAUNCHED();
    return HJ_OK;
}

hj_status launch_band_recheck(const hj_index* ix, const uint32_t* bq, const uint32_t* bc,
                              const unsigned long long* band_used, unsigned long long band_cap, const PairSink& sink,
                              uint32_t nblocks, bool sym, uint32_t* qcount, cudaStream_t st) {
    const unsigned grid = recheck_grid(nblocks);
    const uint32_t* perm = sym ? flagged_perm(ix) : ix->perm;
    k_band_recheck<<<grid, 256, 0, st>>>((const float*)ix->pts, perm, ix->d, (float)ix->thr, bq, bc, band_used,
                                         band_cap, sym ? 1u : 0u, sink, qcount);
    HJ_LAUNCHED();
    return HJ_OK;
}

}  // namespace hj

namespace hj {
// One launch of the tile probe.  skip_mma = 1 issues the loads but no MMA and no
// commit, so the epilogue's bounded wait runs out after wait_cycles.
static hj_status run_tile_probe(hj_index* ix, int kind, uint32_t a0, uint32_t b0, float* d_out, uint32_t skip_mma,
                                long long wait_cycles, void* h_query_rows, void* h_cand_rows, cudaStream_t st) {
    if (!ix || !d_out || !tc_supported(ix, kind)) { set_error("tensor-core tile probe: unsupported"); return HJ_ERR_INVALID; }
    HJ_TRY(tc_prepare(ix, kind, st));
    TcState* s = tc_state(ix);
    const uint32_t nkb = ix->tc_kpad / 32;
    size_t smem = 1024 + (size_t)nkb * (kProbeQB + kTileRows) * kRowBytes + 64;
    smem = std::max<size_t>(smem, 116 * 1024);
    HJ_TRY(ensure_smem(k_tc_tile_probe, smem));
    Scratch tmp(st);
    uint32_t* err = nullptr;
    HJ_TRY(tmp.alloc(&err, 1));
    HJ_CUDA(cudaMemsetAsync(err, 0, 4, st));
    // the probe's operand forms: its rows only, with plain norms, so its accumulators are
    // squared distances
    uint16_t *qf = nullptr, *cf = nullptr;
    float* origin = nullptr;
    unsigned int* mx = nullptr;
    const size_t words = (size_t)kProbeQB * ix->tc_kpad;   // halves per form (512 plane rows)
    HJ_TRY(tmp.alloc(&qf, words));
    HJ_TRY(tmp.alloc(&cf, words));
    HJ_TRY(tmp.alloc(&origin, ix->d));
    HJ_TRY(tmp.alloc(&mx, kTcMaxima));
    HJ_TRY(launch_col_min(ix, origin, st));
    HJ_TRY(launch_prep(ix, kind, origin, s->scale_exp, TcBand{}, 0u, b0, kProbeQB, qf, nullptr, mx, st));
    HJ_TRY(launch_prep(ix, kind, origin, s->scale_exp, TcBand{}, 0u, a0, kProbeQB, nullptr, cf, mx, st));
    k_tc_tile_probe<<<1, kProbeThreads, smem, st>>>((const uint8_t*)cf, (const uint8_t*)qf,
                                               (unsigned long long)kProbeQB * kRowBytes, nkb,
                                               tc::idesc_f16(kind == HJ_REFINE_TC_BF16 ? 1u : 0u, kTileRows, kAccCols),
                                               d_out, err, skip_mma, wait_cycles);
    HJ_LAUNCHED();
    uint32_t herr = 0;
    HJ_CUDA(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, st));
    // rows back in row order: out[row][kb * 32 + e] from the swizzled planes
    auto fetch = [&](const uint16_t* form, uint32_t rows, void* out) -> hj_status {
        std::vector<uint16_t> h(words);
        HJ_CUDA(cudaMemcpyAsync(h.data(), form, words * 2, cudaMemcpyDeviceToHost, st));
        HJ_CUDA(cudaStreamSynchronize(st));
        uint16_t* o = static_cast<uint16_t*>(out);
        for (uint32_t r = 0; r < rows; ++r)
            for (uint32_t ch = 0; ch < nkb * 4; ++ch)
                std::memcpy(o + (size_t)r * ix->tc_kpad + ch * 8,
                            h.data() + (((size_t)(ch >> 2) * kProbeQB + r) * 4 + ((ch & 3u) ^ ((r >> 1) & 3u))) * 8, 16);
        return HJ_OK;
    };
    if (h_query_rows) HJ_TRY(fetch(qf, std::min<uint32_t>(kProbeQB, ix->n - b0), h_query_rows));
    if (h_cand_rows) HJ_TRY(fetch(cf, std::min<uint32_t>(kTileRows, ix->n - a0), h_cand_rows));
    HJ_CUDA(cudaStreamSynchronize(st));
    if (herr) { set_error("tensor-core tile probe: a bounded wait expired"); return HJ_ERR_TIMEOUT; }
    return HJ_OK;
}
}  // namespace hj

extern "C" hj_status hj_probe_tc_tile(hj_index* ix, int kind, uint32_t a0, uint32_t b0, float* d_out,
                                      void* h_query_rows, void* h_cand_rows, void* stream) {
    using namespace hj;
    if (ix && (a0 >= ix->n || b0 >= ix->n)) { set_error("hj_probe_tc_tile: row out of range"); return HJ_ERR_INVALID; }
    return run_tile_probe(ix, kind, a0, b0, d_out, 0u, kWaitCycles, h_query_rows, h_cand_rows, as_stream(stream));
}

extern "C" hj_status hj_probe_tc_wait_timeout(hj_index* ix, int kind, uint64_t wait_cycles, void* stream) {
    using namespace hj;
    if (!ix || wait_cycles == 0 || wait_cycles > (uint64_t)kWaitCycles) {
        set_error("hj_probe_tc_wait_timeout: wait_cycles must be in [1, %lld]", kWaitCycles);
        return HJ_ERR_INVALID;
    }
    cudaStream_t st = as_stream(stream);
    Scratch tmp(st);
    float* out = nullptr;
    HJ_TRY(tmp.alloc(&out, (size_t)kTileRows * kProbeQB));
    return run_tile_probe(ix, kind, 0, 0, out, 1u, (long long)wait_cycles, nullptr, nullptr, st);
}

extern "C" hj_status hj_tc_operand_scale(const hj_index* ix, int* log2_scale) {
    using namespace hj;
    if (!ix || !log2_scale) { set_error("hj_tc_operand_scale: null argument"); return HJ_ERR_INVALID; }
    if (!ix->tc_state) { set_error("hj_tc_operand_scale: no tensor-core operands prepared"); return HJ_ERR_INVALID; }
    *log2_scale = tc_scale_exp(ix);
    return HJ_OK;
}
