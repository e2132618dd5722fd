// hj_refine_warp.cu -- host side of the warp-per-item exact refine.
#include "hj_refine_warp.cuh"

namespace hj {

hj_status refine_warp_f32(const WarpArgs<float>& a, uint32_t d, bool digest, cudaStream_t st);
hj_status refine_warp_f64(const WarpArgs<double>& a, uint32_t d, bool digest, cudaStream_t st);

// A candidate's coordinates lie in registers (two candidates per lane): the
// dimensions up to which that leaves room for enough warps.
bool warp_refine_supported(const hj_index* ix) {
    return ix->d <= (uint32_t)(ix->dtype == HJ_F32 ? kWarpMaxD32 : kWarpMaxD64);
}

// Queries per work item: 32 (a candidate is loaded once for all of them) where that
// leaves four items per resident warp, fewer for fewer points -- down to 4: an item
// runs alone in its warp, and the heaviest one is the join's critical path (6-D,
// 20,011 points, whole join with CSR: 1.56 ms with 32 and the estimator taking whole
// items, 1.08 ms with 4).
uint32_t warp_query_block(uint32_t n) {
    const uint32_t items = 4u * kWarpMaxBlocks * kWarpsPerBlock * (uint32_t)num_sms();
    uint32_t q = kWarpQ;
    while (q > 4 && n / q < items) q >>= 1;
    return q;
}

// Items per block of queries: a list that would leave warps idle (fewer than two
// items per resident warp) is cut so that an item still has about 8,192 pairs to
// evaluate; `avg` = mean pairs (queries x candidates) per block of the join.  The
// estimator's sample is cut whatever the mean: its first items are the heaviest of
// the join, and one of them alone took as long as the join (6-D, 20,011 points: 142
// us of 270).
static uint32_t warp_parts(uint32_t nblocks, double avg, bool sample) {
    const uint64_t want = 2ull * kWarpMaxBlocks * kWarpsPerBlock * (uint64_t)num_sms();
    const uint64_t nb = std::max<uint32_t>(nblocks, 1);
    const uint64_t by_work = sample ? 64u : (uint64_t)(avg / 8192.0);
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>({64, (want + nb - 1) / nb, by_work}));
}

// Slots that partly filled chunks can leave unused in one launch.
uint64_t warp_chunk_slack(uint32_t nblocks, double avg) {
    const uint64_t items = (uint64_t)std::max<uint32_t>(nblocks, 1) * warp_parts(nblocks, avg, false) + kWarpsPerBlock - 1;
    return std::min<uint64_t>((uint64_t)kWarpMaxBlocks * kWarpsPerBlock * num_sms(), items) * kSinkChunk;
}

template <typename T>
static WarpArgs<T> make_args(const hj_index* ix, const HjBlock* blocks, uint32_t nblocks, double avg, bool sample,
                             bool sym, unsigned int* head) {
    WarpArgs<T> a{};
    a.pts = (const T*)ix->pts;
    a.perm = sym ? flagged_perm(ix) : ix->perm;
    a.cell_lid = ix->cell_lid;
    a.cell_start = ix->cell_start;
    a.cell_edge = ix->cell_edge;
    a.hash = cell_hash(ix);
    a.grid = ix->grid;
    a.thr = (T)ix->thr;
    a.blocks = blocks;
    a.nblocks = nblocks;
    a.parts = warp_parts(nblocks, avg, sample);
    a.sym = sym ? 1u : 0u;
    a.head = head;
    return a;
}

// Runs the refine over work items blocks[0..nblocks).  `head` must be zero on
// entry.  count_only: per-item pair counts go to block_counts.  sym: the items are
// the join's whole list, each unordered pair once.  Each query's pairs are added to
// qcount, by original id (not with count_only).
hj_status launch_refine_warp(const hj_index* ix, const HjBlock* blocks, uint32_t nblocks, double avg, unsigned int* head,
                             const PairSink& sink, uint32_t count_only, bool sym, unsigned long long* block_counts,
                             uint32_t* qcount, cudaStream_t st) {
    if (nblocks == 0) return HJ_OK;
    auto run = [&](auto zero, auto refine) -> hj_status {
        using T = decltype(zero);
        WarpArgs<T> a = make_args<T>(ix, blocks, nblocks, avg, count_only != 0u, sym, head);
        a.sink = sink;
        a.count_only = count_only;
        a.block_counts = block_counts;
        a.qcount = qcount;
        return refine(a, ix->d, false, st);
    };
    return ix->dtype == HJ_F32 ? run(0.f, refine_warp_f32) : run(0.0, refine_warp_f64);
}

// The digests of hj_result_digest for every query of the items, and the number of
// pairs, without writing a pair.  The arrays and *total are added to.
hj_status launch_refine_digest(const hj_index* ix, const HjBlock* blocks, uint32_t nblocks, double avg, unsigned int* head,
                               uint32_t* d_count, unsigned long long* d_sum, unsigned long long* d_xor,
                               unsigned long long* total, cudaStream_t st) {
    if (nblocks == 0) return HJ_OK;
    auto run = [&](auto zero, auto refine) -> hj_status {
        using T = decltype(zero);
        WarpArgs<T> a = make_args<T>(ix, blocks, nblocks, avg, false, false, head);
        a.d_count = d_count;
        a.d_sum = d_sum;
        a.d_xor = d_xor;
        a.total = total;
        return refine(a, ix->d, true, st);
    };
    return ix->dtype == HJ_F32 ? run(0.f, refine_warp_f32) : run(0.0, refine_warp_f64);
}

}  // namespace hj
