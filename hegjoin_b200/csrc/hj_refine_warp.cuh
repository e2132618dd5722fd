// hj_refine_warp.cuh -- exact refine on the CUDA cores, a work item per warp.
//
// The exact path for low dimensions (float up to kWarpMaxD32, double up to
// kWarpMaxD64); the block-tiled kernel of hj_refine_plain.cu takes the rest.
// Reference counterpart and semantics as there (kernel.cu:727-802, 333-412): a
// pair (q, c) is a result iff c lies in a non-empty cell of q's 3^k stencil and
//     acc = 0; for l in 0..d-1: diff = c_l - q_l; acc = fma(diff, diff, acc)
// is at most thr.
//
// B200 design.  A warp takes an item of up to 32 queries of one cell on its own:
// no block barrier and no staging, so one-point cells cost as little as they can
// and items with few queries keep every lane busy (the block-tiled kernel gives
// its 16 query rows to the queries: 8 queries used an eighth of its threads).
//   * Lanes resolve the stencil rows through the cell hash, 128 rows per round,
//     into point ranges; the non-empty ones are compacted and laid end to end.
//   * A lane holds kWarpC candidates in registers (loaded straight from the
//     cell-ordered points: neighbouring lanes, neighbouring rows); the item's
//     queries are broadcast from shared memory, float ones as packed pairs.
//   * One ballot per query and candidate step names the hits, which leave as one
//     coalesced run with the query's id as key.
// A list of few items is cut into `parts` items per block of queries, each
// taking its slice of every round's candidates.
// Bound by instruction issue: hash probes on sparse data, ballots and stores on
// dense.  Against the block-tiled kernel: skewed 6-D, 4,000,000 points 44 -> 21 ms,
// 7-D, 300,007 points (which had no specialised kernel) 6.7 -> 3.0 ms, 5-D FP64,
// 120,000 points 1.5 -> 1.1 ms.
//
// Symmetric form (a.sym): d2 is the same number for (q, c) and (c, q), so a join
// that runs in one batch may evaluate each unordered pair once and emit both orders
// (symmetric_pays in hj_join.cu says when that is the faster form): an item takes the cells after its own in linear-id order and, of its own cell,
// the points from its first query on.  Cells with a coordinate of 0 visit no cell
// in the reference's stencil (kernel.cu:780 wraps) although their neighbours visit
// them: an item of such a cell emits only (candidate, query), a candidate of one
// (bit 31 of perm) only (query, candidate).
#pragma once

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "hj_internal.h"

namespace hj {

constexpr int kWarpC = 2;             // candidates per lane and step
constexpr uint32_t kWarpsPerBlock = 4;
constexpr uint32_t kWarpQ = 32;       // queries per work item
constexpr uint32_t kWarpRows = kBoxRows;   // stencil rows per round
constexpr uint32_t kWarpMaxBlocks = 8;   // resident blocks per SM at most

template <typename T>
struct WarpArgs {
    const T* pts;
    const uint32_t* perm;             // sorted position -> original id (sym: bit 31 set in silent cells)
    const unsigned long long* cell_lid;
    const uint32_t* cell_start;
    const uint8_t* cell_edge;
    HjCellHash hash;
    HjGrid grid;
    T thr;
    const HjBlock* blocks;
    uint32_t nblocks;
    uint32_t parts;
    uint32_t sym;
    unsigned int* head;
    PairSink sink;
    uint32_t count_only;
    unsigned long long* block_counts; // count-only mode: pairs per work item
    uint32_t* qcount;                 // pairs per query id, added up (not in count-only mode)
    // digest kernel
    uint32_t* d_count;
    unsigned long long* d_sum;
    unsigned long long* d_xor;
    unsigned long long* total;
};

// Queries in shared memory: float coordinates duplicated into packed pairs; a
// query's coordinates are padded to an even number (16-byte loads).
template <typename T, int D>
struct WarpSmem {
    static constexpr int DP = (D + 1) & ~1;
    using Q = typename std::conditional<std::is_same<T, float>::value, unsigned long long, double>::type;
    __align__(16) Q q[kWarpQ][DP];
    uint32_t qid[kWarpQ];
    uint32_t rst[kWarpRows];          // non-empty ranges of the round: start (sorted position)
    uint32_t pre[kWarpRows + 1];      // and exclusive prefix of the lengths
};

__device__ __forceinline__ unsigned long long wpack2(float lo, float hi) {
    return ((unsigned long long)__float_as_uint(hi) << 32) | __float_as_uint(lo);
}
// Packed FP32 pairs (sm_100): each half is the IEEE-rounded scalar operation.
__device__ __forceinline__ unsigned long long wsub2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long wfma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// One round of stencil rows: their non-empty point ranges, compacted into S, and
// the round's candidates (0: nothing).  Whole warp.
template <typename S_>
__device__ __forceinline__ uint32_t warp_round(const HjGrid& g, const HjCellHash& hash, const uint32_t* cell_start,
                                               const CellBox& b, uint32_t row0, bool sym, uint32_t q0, S_& S,
                                               uint32_t* n_ranges) {
    uint32_t run = 0, nr = 0;
    const uint32_t n = box_rows_present(g, hash, b, row0, sym, S.pre);
    for (uint32_t i0 = 0; i0 < n; i0 += 32) {
        uint2 sp = make_uint2(0u, 0u);
        const uint32_t x = i0 + lane_id() < n ? S.pre[i0 + lane_id()] : 0u;
        if (x) {
            const uint32_t r = x & 0x0FFFFFFFu;
            sp = cell_points(hash, cell_start, cell_box_row(g, b, r), x >> 28);
            if (sym && r == b.r_own) sp.x = q0;
        }
        // ranges replace the row list from its start: at most as many as rows read so far
        __syncwarp();
        const uint32_t len = sp.y - sp.x;
        const uint32_t some = __ballot_sync(0xffffffffu, len != 0u);
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane_id() >= (uint32_t)o) incl += t;
        }
        if (len) {
            const uint32_t at = nr + __popc(some & lanemask_lt());
            S.rst[at] = sp.x;
            S.pre[at] = run + incl - len;
        }
        run += __shfl_sync(0xffffffffu, incl, 31);
        nr += __popc(some);
        __syncwarp();
    }
    if (lane_id() == 0) S.pre[nr] = run;
    *n_ranges = nr;
    __syncwarp();
    return run;
}

// The next item of the queue (a.nblocks * a.parts and above: none left).
template <typename T>
__device__ __forceinline__ uint32_t warp_next(const WarpArgs<T>& a) {
    uint32_t it = 0;
    if (lane_id() == 0) it = atomicAdd(a.head, 1u);
    return __shfl_sync(0xffffffffu, it, 0);
}

// Reserve `n` sink slots: rank r goes to r < room ? p0 + r : p1 + (r - room).
// False on overflow (the batch is re-run).
struct WarpSlots {
    unsigned long long p0, p1;
    uint32_t room;
};
__device__ __forceinline__ bool warp_slots(const PairSink& s, WarpChunk& c, uint32_t n, WarpSlots& o) {
    o.p0 = c.base + c.used;
    o.room = c.cap - c.used;
    o.p1 = 0;
    if (n <= o.room) {
        c.used += n;
        return true;
    }
    const uint32_t need = (n - o.room + kSinkChunk - 1) / kSinkChunk * kSinkChunk;
    if (lane_id() == 0) o.p1 = atomicAdd(s.cursor, (unsigned long long)need);
    o.p1 = __shfl_sync(0xffffffffu, o.p1, 0);
    if (o.p1 + need > s.capacity) {
        if (lane_id() == 0) atomicExch(s.overflow, 1u);
        c.cap = c.used = 0;
        return false;
    }
    c.base = o.p1;
    c.used = n - o.room;
    c.cap = need;
    return true;
}

template <typename T, int D>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, D <= 8 ? 6 : 5) k_refine_warp(const __grid_constant__ WarpArgs<T> a) {
    using Smem = WarpSmem<T, D>;
    constexpr bool F32 = std::is_same<T, float>::value;
    __shared__ Smem smem[kWarpsPerBlock];
    Smem& S = smem[threadIdx.x >> 5];
    const uint32_t lane = lane_id();
    WarpChunk wc;
    warp_chunk_init(wc);
    const uint32_t n_items = a.nblocks * a.parts;
    for (uint32_t it = warp_next(a); it < n_items; it = warp_next(a)) {
        const uint32_t bi = it / a.parts, part = it - bi * a.parts;
        const HjBlock blk = a.blocks[bi];
        const uint32_t q0 = blk.q0, nq = blk.q1 - blk.q0;
        CellBox box;
        cell_box(a.grid, a.cell_lid[blk.cell], a.cell_edge[blk.cell] != 0, box);
        if (box.silent && !a.sym) continue;
        __syncwarp();
        for (uint32_t f = lane; f < nq * D; f += 32) {
            const T x = a.pts[(size_t)q0 * D + f];
            if constexpr (F32) S.q[f / D][f % D] = wpack2(x, x);
            else S.q[f / D][f % D] = x;
        }
        if (lane < nq) S.qid[lane] = a.perm[q0 + lane] & 0x7FFFFFFFu;
        const bool fwd = !box.silent;
        uint32_t my_count = 0;               // lane b: pairs of query b (or, counting only, any pairs)
        for (uint32_t row0 = a.sym ? box.r_own : 0u; row0 < box.rows; row0 += kWarpRows) {
            uint32_t nr;
            const uint32_t run = warp_round(a.grid, a.hash, a.cell_start, box, row0, a.sym != 0u, q0, S, &nr);
            const uint32_t c_lo = (uint32_t)((unsigned long long)run * part / a.parts);
            const uint32_t c_hi = (uint32_t)((unsigned long long)run * (part + 1) / a.parts);
            uint32_t j = 0;                  // this lane's current range
            for (uint32_t base = c_lo; base < c_hi; base += 32 * kWarpC) {
                uint32_t cpos[kWarpC], cw[kWarpC];
                T cv[kWarpC][D];
#pragma unroll
                for (int c = 0; c < kWarpC; ++c) {
                    const uint32_t idx = base + c * 32 + lane;
                    const bool valid = idx < c_hi;
                    if (valid)
                        while (S.pre[j + 1] <= idx) ++j;
                    const uint32_t p = valid ? S.rst[j] + (idx - S.pre[j]) : 0u;
                    cpos[c] = valid ? p : 0u;
                    cw[c] = valid && !a.count_only ? a.perm[p] : 0u;
                    // NaN coordinates: no distance of an absent candidate is at most thr
#pragma unroll
                    for (int l = 0; l < D; ++l)
                        cv[c][l] = valid ? a.pts[(size_t)p * D + l] : (T)__int_as_float(0x7FC00000);
                }
                // symmetric form: a candidate of the item's own block pairs with the queries up to itself
                uint32_t lim[kWarpC];
                bool own = false;
#pragma unroll
                for (int c = 0; c < kWarpC; ++c) {
                    lim[c] = a.sym ? cpos[c] - q0 : kWarpQ;   // query b: b <= lim (b == lim: itself)
                    own |= lim[c] < nq;
                }
                own = __any_sync(0xffffffffu, own);
                auto pairs_of = [&](uint32_t b, bool (&hit)[kWarpC]) {
                    if constexpr (F32) {
                        unsigned long long acc = 0ull;
#pragma unroll
                        for (int l = 0; l < D; ++l) {
                            const unsigned long long diff = wsub2(wpack2(cv[0][l], cv[1][l]), S.q[b][l]);
                            acc = wfma2(diff, diff, acc);
                        }
                        hit[0] = __uint_as_float((uint32_t)acc) <= a.thr;
                        hit[1] = __uint_as_float((uint32_t)(acc >> 32)) <= a.thr;
                    } else {
#pragma unroll
                        for (int c = 0; c < kWarpC; ++c) {
                            T acc = T(0);
#pragma unroll
                            for (int l = 0; l < D; ++l) {
                                const T diff = __dsub_rn(cv[c][l], S.q[b][l]);
                                acc = __fma_rn(diff, diff, acc);
                            }
                            hit[c] = acc <= a.thr;
                        }
                    }
                };
                static_assert(kWarpC == 2, "packed pairs hold two candidates");
                for (uint32_t b = 0; b < nq; ++b) {
                    bool hit[kWarpC];
                    pairs_of(b, hit);
                    if (own) {
#pragma unroll
                        for (int c = 0; c < kWarpC; ++c) hit[c] = hit[c] && b <= lim[c];
                    }
                    const uint32_t h0 = __ballot_sync(0xffffffffu, hit[0]), h1 = __ballot_sync(0xffffffffu, hit[1]);
                    if ((h0 | h1) == 0u) continue;
                    const uint32_t n0 = __popc(h0), n = n0 + __popc(h1);
                    if (lane == b) my_count += n;
                    if (a.count_only) continue;
                    const uint32_t qid = S.qid[b];
                    const uint32_t lt = lanemask_lt();
                    if (!a.sym) {
                        WarpSlots s;
                        if (!warp_slots(a.sink, wc, n, s)) continue;
#pragma unroll
                        for (int c = 0; c < kWarpC; ++c) {
                            if (!hit[c]) continue;
                            const uint32_t r = c ? n0 + __popc(h1 & lt) : __popc(h0 & lt);
                            const unsigned long long pos = r < s.room ? s.p0 + r : s.p1 + (r - s.room);
                            a.sink.keys[pos] = qid;
                            a.sink.vals[pos] = cw[c];
                        }
                    } else {
                        // both orders: forward unless the item is silent; reverse unless the candidate
                        // is, and not for the query itself
                        bool rev[kWarpC];
#pragma unroll
                        for (int c = 0; c < kWarpC; ++c) rev[c] = hit[c] && !(cw[c] >> 31) && lim[c] != b;
                        const uint32_t r0 = __ballot_sync(0xffffffffu, rev[0]), r1 = __ballot_sync(0xffffffffu, rev[1]);
                        const uint32_t nf = fwd ? n : 0u, m0 = __popc(r0);
                        WarpSlots s;
                        if (!warp_slots(a.sink, wc, nf + m0 + __popc(r1), s)) continue;
#pragma unroll
                        for (int c = 0; c < kWarpC; ++c) {
                            const uint32_t cid = cw[c] & 0x7FFFFFFFu;
                            if (hit[c] && fwd) {
                                const uint32_t r = c ? n0 + __popc(h1 & lt) : __popc(h0 & lt);
                                const unsigned long long pos = r < s.room ? s.p0 + r : s.p1 + (r - s.room);
                                a.sink.keys[pos] = qid;
                                a.sink.vals[pos] = cid;
                            }
                            if (rev[c]) {
                                const uint32_t r = nf + (c ? m0 + __popc(r1 & lt) : __popc(r0 & lt));
                                const unsigned long long pos = r < s.room ? s.p0 + r : s.p1 + (r - s.room);
                                a.sink.keys[pos] = cid;
                                a.sink.vals[pos] = qid;
                                atomicAdd(&a.qcount[cid], 1u);
                            }
                        }
                    }
                }
            }
            __syncwarp();   // the next round rewrites the ranges
        }
        if (a.count_only) {
            const uint32_t t = __reduce_add_sync(0xffffffffu, my_count);
            if (lane == 0 && t) atomicAdd(&a.block_counts[bi], (unsigned long long)t);
        } else if (fwd) {
            if (lane < nq && my_count) atomicAdd(&a.qcount[S.qid[lane]], my_count);
        }
    }
    if (!a.count_only) warp_chunk_close(a.sink, wc);
}

// Digests without pairs: for a streamed join whose batches nobody reads, each
// query's (count, sum of mix64(id), xor of mix64(id ^ salt)) straight from the
// refine.  Lanes are queries here, so a query's totals stay in its lane's
// registers; candidates are staged 32 at a time with their hashes and broadcast.
// Bound by the arithmetic of the pairs (FP64 for double data): at 2-D, 1,000,000
// points and 4.7e9 pairs the pairs alone are 75 GB of traffic when they are
// written, grouped and folded: 91 ms, against 8.2 ms for this whole join.
template <typename T, int D>
struct DigestSmem {
    static constexpr int DP = (D + 1) & ~1;
    __align__(16) T c[32][DP < 4 && sizeof(T) == 4 ? 4 : DP];
    ulonglong2 h[32];
    uint32_t rst[kWarpRows];
    uint32_t pre[kWarpRows + 1];
};
template <typename T, int D>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_refine_digest(const __grid_constant__ WarpArgs<T> a) {
    using Smem = DigestSmem<T, D>;
    __shared__ Smem smem[kWarpsPerBlock];
    Smem& S = smem[threadIdx.x >> 5];
    const uint32_t lane = lane_id();
    const uint32_t n_items = a.nblocks * a.parts;
    unsigned long long total = 0;
    for (uint32_t it = warp_next(a); it < n_items; it = warp_next(a)) {
        const uint32_t bi = it / a.parts, part = it - bi * a.parts;
        const HjBlock blk = a.blocks[bi];
        const uint32_t q0 = blk.q0, nq = blk.q1 - blk.q0;
        CellBox box;
        cell_box(a.grid, a.cell_lid[blk.cell], a.cell_edge[blk.cell] != 0, box);
        if (box.silent) continue;
        T qv[D];
#pragma unroll
        for (int l = 0; l < D; ++l) qv[l] = lane < nq ? a.pts[(size_t)(q0 + lane) * D + l] : (T)__int_as_float(0x7FC00000);
        uint32_t cnt = 0;
        unsigned long long sum = 0, xr = 0;
        for (uint32_t row0 = 0; row0 < box.rows; row0 += kWarpRows) {
            uint32_t nr;
            const uint32_t run = warp_round(a.grid, a.hash, a.cell_start, box, row0, false, q0, S, &nr);
            const uint32_t c_lo = (uint32_t)((unsigned long long)run * part / a.parts);
            const uint32_t c_hi = (uint32_t)((unsigned long long)run * (part + 1) / a.parts);
            uint32_t j = 0;
            for (uint32_t base = c_lo; base < c_hi; base += 32) {
                const uint32_t idx = base + lane;
                __syncwarp();
                if (idx < c_hi) {
                    while (S.pre[j + 1] <= idx) ++j;
                    const uint32_t p = S.rst[j] + (idx - S.pre[j]);
#pragma unroll
                    for (int l = 0; l < D; ++l) S.c[lane][l] = a.pts[(size_t)p * D + l];
                    const uint64_t id = a.perm[p];
                    S.h[lane] = make_ulonglong2(mix64(id), mix64(id ^ 0x5bd1e9955bd1e995ull));
                }
                __syncwarp();
                const uint32_t m = min(32u, c_hi - base);
                auto one = [&](uint32_t i) {
                    T acc = T(0);
#pragma unroll
                    for (int l = 0; l < D; ++l) {
                        if constexpr (std::is_same<T, float>::value) {
                            const T diff = __fsub_rn(S.c[i][l], qv[l]);
                            acc = __fmaf_rn(diff, diff, acc);
                        } else {
                            const T diff = __dsub_rn(S.c[i][l], qv[l]);
                            acc = __fma_rn(diff, diff, acc);
                        }
                    }
                    const ulonglong2 h = S.h[i];
                    if (acc <= a.thr) {
                        ++cnt;
                        sum += h.x;
                        xr ^= h.y;
                    }
                };
                if (m == 32u) {
#pragma unroll 8
                    for (uint32_t i = 0; i < 32; ++i) one(i);
                } else {
                    for (uint32_t i = 0; i < m; ++i) one(i);
                }
            }
            __syncwarp();
        }
        if (lane < nq && cnt) {
            const uint32_t id = a.perm[q0 + lane];
            atomicAdd(&a.d_count[id], cnt);
            atomicAdd(&a.d_sum[id], sum);
            atomicXor(&a.d_xor[id], xr);
        }
        total += cnt;
    }
    for (int o = 16; o > 0; o >>= 1) total += __shfl_down_sync(0xffffffffu, total, o);
    if (lane == 0 && total) atomicAdd(a.total, total);
}

// One persistent launch: as many blocks as fit on the GPU (at most kWarpMaxBlocks
// per SM), and no more warps than items.
template <typename T, int D, bool DIGEST>
hj_status launch_warp(const WarpArgs<T>& a, cudaStream_t st) {
    auto kern = DIGEST ? k_refine_digest<T, D> : k_refine_warp<T, D>;
    static std::atomic<int> s_per_sm{0};   // asked once per kernel (a driver call)
    int per_sm = s_per_sm.load(std::memory_order_relaxed);
    if (per_sm == 0) {
        HJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kWarpsPerBlock, 0));
        per_sm = std::max(1, std::min(per_sm, (int)kWarpMaxBlocks));
        s_per_sm.store(per_sm, std::memory_order_relaxed);
    }
    const uint64_t items = (uint64_t)a.nblocks * a.parts;
    const unsigned grid =
        (unsigned)std::min<uint64_t>((uint64_t)per_sm * num_sms(), (items + kWarpsPerBlock - 1) / kWarpsPerBlock);
    kern<<<grid, 32 * kWarpsPerBlock, 0, st>>>(a);
    HJ_LAUNCHED();
    return HJ_OK;
}

template <typename T, int D, int MaxD, bool DIGEST>
hj_status dispatch_warp(const WarpArgs<T>& a, uint32_t d, cudaStream_t st) {
    if (d == (uint32_t)D) return launch_warp<T, D, DIGEST>(a, st);
    if constexpr (D < MaxD) return dispatch_warp<T, D + 1, MaxD, DIGEST>(a, d, st);
    set_error("exact refine: no warp kernel for d = %u", d);
    return HJ_ERR_UNSUPPORTED;
}

}  // namespace hj
