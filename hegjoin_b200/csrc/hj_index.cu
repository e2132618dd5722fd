// hj_index.cu -- grid geometry, grid-index build and workload order.
//
// Reference counterparts:
//   generateNDGridDimensions   main.cu:449-520
//   gridIndexingGPU            GPU.cu:74-398 (kernelIndexComputeNonemptyCells kernel.cu:34-66)
//   sortByWorkLoad             SortByWorkload.cu:19-247 (sortByWorkLoadGlobal kernel.cu:74-144)
//
// B200 design: everything stays on the device.  Cell ids are computed once,
// (cell id, point id) pairs are radix-sorted on only the bits totalCells
// needs, the non-empty-cell table comes from a run-boundary scan instead of the
// reference's device->host copy and host loop (GPU.cu:293-324), and the
// points are gathered into cell order so the refine kernels stream each
// cell's points as one contiguous range.  The workload pass resolves each
// cell's 3^k stencil once per cell as 3^(k-1) contiguous point ranges (the
// cells along dimension 0 are consecutive linear ids), one warp per cell.

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <limits>
#include <map>
#include <mutex>

#include <cuda.h>

#include "hj_internal.h"

namespace hj {

// ---- error state ----------------------------------------------------------------
static thread_local char g_err[1024] = "";
void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
static std::atomic<uint64_t> g_launches{0};
static thread_local uint64_t t_launches = 0;
void count_launch() {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    ++t_launches;
}
uint64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }
uint64_t thread_launch_count() { return t_launches; }

static thread_local Workspace* t_workspace = nullptr;
Workspace* current_workspace() { return t_workspace; }
void set_current_workspace(Workspace* ws) { t_workspace = ws; }

static std::atomic<int64_t> g_fail_alloc_in{0};
bool injected_alloc_failure_armed() { return g_fail_alloc_in.load(std::memory_order_relaxed) > 0; }
bool injected_alloc_failure() {
    if (g_fail_alloc_in.load(std::memory_order_relaxed) <= 0) return false;
    return g_fail_alloc_in.fetch_sub(1, std::memory_order_relaxed) == 1;
}

// Through the runtime's driver entry-point query (the library does not link libcuda).
uint64_t context_id() {
    using Current = CUresult (*)(CUcontext*);
    using Id = CUresult (*)(CUcontext, unsigned long long*);
    auto entry = [](const char* name) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess
                   ? p
                   : nullptr;
    };
    static const Current current = reinterpret_cast<Current>(entry("cuCtxGetCurrent"));
    static const Id id_of = reinterpret_cast<Id>(entry("cuCtxGetId"));
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (current && id_of && current(&c) == CUDA_SUCCESS && c) id_of(c, &id);
    return id;
}

namespace {
// A readback buffer lives as long as the context that it was allocated in.
struct Pinned {
    void* p;
    int dev;
    uint64_t ctx;
};
// Buffers of ended threads wait for the next thread (a server's workers come and go
// with it, and allocating pinned memory stops the device for a moment); at most
// kReadbackKept of them.  Those of a context that is gone are forgotten.
constexpr size_t kReadbackKept = 32;
std::mutex g_readback_mu;
std::vector<Pinned> g_readback_free;
struct Readback {
    std::vector<Pinned> bufs;   // one per context that the thread has used
    ~Readback() {
        for (const Pinned& b : bufs) {
            if (cudaSetDevice(b.dev) != cudaSuccess || context_id() != b.ctx) continue;
            {
                std::lock_guard<std::mutex> lk(g_readback_mu);
                if (g_readback_free.size() < kReadbackKept) {
                    g_readback_free.push_back(b);
                    continue;
                }
            }
            cudaFreeHost(b.p);
        }
    }
};
thread_local Readback t_readback;
}  // namespace
hj_status readback_buffer(void** p) {
    Pinned b{nullptr, 0, context_id()};
    if (b.ctx == 0) {
        HJ_CUDA(cudaFree(nullptr));   // makes the device's context current
        b.ctx = context_id();
    }
    for (const Pinned& have : t_readback.bufs)
        if (have.ctx == b.ctx) {
            *p = have.p;
            return HJ_OK;
        }
    HJ_CUDA(cudaGetDevice(&b.dev));
    auto gone = [&](const Pinned& x) { return x.dev == b.dev && x.ctx != b.ctx; };
    auto& bufs = t_readback.bufs;
    bufs.erase(std::remove_if(bufs.begin(), bufs.end(), gone), bufs.end());
    {
        std::lock_guard<std::mutex> lk(g_readback_mu);
        auto& free = g_readback_free;
        free.erase(std::remove_if(free.begin(), free.end(), gone), free.end());
        auto it = std::find_if(free.begin(), free.end(), [&](const Pinned& x) { return x.ctx == b.ctx; });
        if (it != free.end()) {
            b.p = it->p;
            free.erase(it);
        }
    }
    if (!b.p) HJ_CUDA(cudaHostAlloc(&b.p, kReadbackBytes, cudaHostAllocDefault));
    bufs.push_back(b);
    *p = b.p;
    return HJ_OK;
}

constexpr size_t kDefaultSmem = 48 * 1024;
constexpr size_t kStaticSmemMax = 16 * 1024;   // no kernel here that takes dynamic shared memory has more
hj_status ensure_smem_ptr(const void* kern, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<uint64_t, const void*>, size_t> done;   // by context: each has its own limits
    // the 48 KB that need no raised limit hold the kernel's static shared memory too
    if (bytes <= kDefaultSmem - kStaticSmemMax) return HJ_OK;
    std::lock_guard<std::mutex> lk(mu);
    size_t& have = done[{context_id(), kern}];
    if (bytes <= have) return HJ_OK;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) {
        set_error("cudaFuncSetAttribute(%zu bytes): %s", bytes, cudaGetErrorString(e));
        return HJ_ERR_CUDA;
    }
    have = bytes;
    return HJ_OK;
}

void init_memory_pool() {
    static std::atomic<bool> done{false};
    if (done.exchange(true)) return;
    int dev = 0;
    cudaMemPool_t pool;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
        uint64_t keep = ~0ull;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        // Concurrent joins (the serving loop's workers) allocate and free on their own
        // streams.  By default the pool may hand one stream memory another stream freed
        // by making the allocation wait for that stream, which couples the requests;
        // reuse only memory whose free has completed, or that was freed on the same stream.
        int no = 0;
        cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &no);
    }
    cudaGetLastError();
}

// Bytes that the memory pool holds and nobody uses (0 when it cannot say).
uint64_t pool_idle_bytes() {
    int dev = 0;
    cudaMemPool_t pool;
    uint64_t reserved = 0, used = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetDefaultMemPool(&pool, dev) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return reserved > used ? reserved - used : 0;
}

template <typename T>
static T sq_threshold_t(T eps) {
    // sqrt is correctly rounded and monotone, so {x : RN(sqrt(x)) <= eps} is
    // {x <= T}; walk from RN(eps^2) to its largest member.
    T x = eps * eps;
    while (x > T(0) && std::sqrt(x) > eps) x = std::nextafter(x, T(0));
    while (true) {
        T nx = std::nextafter(x, std::numeric_limits<T>::infinity());
        if (std::sqrt(nx) <= eps) x = nx; else break;
    }
    return x;
}
double sq_threshold(double eps, int dtype) {
    if (dtype == HJ_F32) return (double)sq_threshold_t<float>((float)eps);
    return sq_threshold_t<double>(eps);
}

namespace {

template <typename T>
struct GeoT {
    T min_arr[kMaxK];
    T eps;
};

// kernel.cu:56 / kernel.cu:779: (unsigned)((x - minArr) / eps), IEEE ops in T.
__device__ __forceinline__ uint32_t cell_coord(float x, float mn, float eps) {
    return __float2uint_rz(__fdiv_rn(__fsub_rn(x, mn), eps));
}
__device__ __forceinline__ uint32_t cell_coord(double x, double mn, double eps) {
    return __double2uint_rz(__ddiv_rn(__dsub_rn(x, mn), eps));
}

// ---- geometry: per-dimension min / max ----------------------------------------------
// Per block the minimum and maximum of each of the k indexed dimensions (partials
// [dim][block]), KN >= k of them in registers, so that the points are read once.
// Comparisons keep the reference's order: a NaN never replaces a value (but a first
// NaN stays).
template <typename T, int KN>
__global__ void __launch_bounds__(512) k_minmax(const T* __restrict__ db, uint32_t n, uint32_t d, uint32_t k, T* out_min,
                                                T* out_max) {
    __shared__ T smin[16], smax[16];
    T mn[KN], mx[KN];
#pragma unroll
    for (int j = 0; j < KN; ++j) mn[j] = mx[j] = (uint32_t)j < k ? db[j] : T(0);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int j = 0; j < KN; ++j) {
            if ((uint32_t)j >= k) break;
            const T v = db[i * d + j];
            mn[j] = v < mn[j] ? v : mn[j];
            mx[j] = v > mx[j] ? v : mx[j];
        }
    }
#pragma unroll
    for (int j = 0; j < KN; ++j) {
        if ((uint32_t)j >= k) break;
        T lo = mn[j], hi = mx[j];
        for (int o = 16; o > 0; o >>= 1) {
            T a = __shfl_down_sync(0xffffffffu, lo, o), b = __shfl_down_sync(0xffffffffu, hi, o);
            lo = a < lo ? a : lo;
            hi = b > hi ? b : hi;
        }
        if (lane_id() == 0) { smin[threadIdx.x >> 5] = lo; smax[threadIdx.x >> 5] = hi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
                lo = smin[w] < lo ? smin[w] : lo;
                hi = smax[w] > hi ? smax[w] : hi;
            }
            out_min[(size_t)j * gridDim.x + blockIdx.x] = lo;
            out_max[(size_t)j * gridDim.x + blockIdx.x] = hi;
        }
        __syncthreads();
    }
}

template <typename T>
hj_status geometry_t(const T* db, uint32_t n, uint32_t d, uint32_t k, T eps, double* h_min, double* h_max,
                     uint32_t* h_ncells, uint64_t* h_total, cudaStream_t st) {
    constexpr int kGeoBlocks = 148;
    const int blocks = std::min<int>(kGeoBlocks, std::max<uint32_t>(1, (n + 511) / 512));
    Scratch tmp(st);
    T* part = nullptr;
    HJ_TRY(tmp.alloc(&part, (size_t)2 * blocks * k));
    if (k <= 2) k_minmax<T, 2><<<blocks, 512, 0, st>>>(db, n, d, k, part, part + (size_t)k * blocks);
    else if (k <= 6) k_minmax<T, 6><<<blocks, 512, 0, st>>>(db, n, d, k, part, part + (size_t)k * blocks);
    else k_minmax<T, kMaxK><<<blocks, 512, 0, st>>>(db, n, d, k, part, part + (size_t)k * blocks);
    HJ_LAUNCHED();
    static_assert(2 * kGeoBlocks * kMaxK * sizeof(double) <= kReadbackBytes, "the blocks' partials are read back");
    T* hp = nullptr;
    HJ_TRY(readback_buffer(reinterpret_cast<void**>(&hp)));
    HJ_CUDA(cudaMemcpyAsync(hp, part, (size_t)2 * blocks * k * sizeof(T), cudaMemcpyDeviceToHost, st));
    HJ_CUDA(cudaStreamSynchronize(st));
    uint64_t total = 1;
    for (uint32_t j = 0; j < k; ++j) {
        T mn = hp[(size_t)j * blocks], mx = hp[(size_t)(k + j) * blocks];
        for (int b = 1; b < blocks; ++b) {
            mn = std::min(mn, hp[(size_t)j * blocks + b]);
            mx = std::max(mx, hp[(size_t)(k + j) * blocks + b]);
        }
        // main.cu:489-509, in T
        T mnA = mn - eps;
        T mxA = mx + eps;
        T r = (mxA - mnA) / eps;
        uint32_t nc = (uint32_t)std::ceil(r);
        if (h_min) h_min[j] = (double)mnA;
        if (h_max) h_max[j] = (double)mxA;
        if (h_ncells) h_ncells[j] = nc;
        total *= nc;
    }
    if (h_total) *h_total = total;
    return HJ_OK;
}

// ---- index build -----------------------------------------------------------------------
template <typename T>
__global__ void k_cell_ids(const T* __restrict__ db, uint32_t n, uint32_t d, GeoT<T> geo, HjGrid grid,
                           unsigned long long* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t* alias, uint32_t* silent) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned long long lid = 0;
    bool al = false, zero = false;
    for (uint32_t j = 0; j < grid.k; ++j) {
        uint32_t c = cell_coord(db[(uint64_t)i * d + j], geo.min_arr[j], geo.eps);
        al |= c >= grid.n_cells[j];
        zero |= c == 0u;
        lid += (unsigned long long)c * grid.mult[j];
    }
    keys[i] = lid;
    vals[i] = zero ? i | 0x80000000u : i;   // the sort carries the mark to the point's place
    if (al) atomicExch(alias, 1u);
    if (zero) atomicExch(silent, 1u);
}

// 1 where a run of equal keys begins.
__global__ void k_run_flags(const unsigned long long* __restrict__ keys, uint32_t n, uint32_t* __restrict__ flags) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    flags[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

// pos: exclusive scan of the run flags.
__global__ void k_cells(const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ pos, uint32_t n,
                        unsigned long long* __restrict__ cell_lid, uint32_t* __restrict__ cell_start,
                        uint32_t* n_cells_out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool first = i == 0 || keys[i] != keys[i - 1];
    if (first) {
        cell_lid[pos[i]] = keys[i];
        cell_start[pos[i]] = i;
    }
    if (i == n - 1) {
        uint32_t nc = pos[i] + (first ? 1u : 0u);
        cell_start[nc] = n;
        *n_cells_out = nc;
    }
}

// Points in cell order.  A warp takes 32 rows at a time: their ids once, then the
// rows' values in flat order (coalesced stores; loads coalesce within a row).
template <typename T>
__global__ void __launch_bounds__(256) k_gather_rows(const T* __restrict__ db, const uint32_t* __restrict__ perm,
                                                      uint32_t n, uint32_t d, T* __restrict__ out) {
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32u; r0 < n; r0 += warps * 32u) {
        const uint32_t rows = min(32u, n - r0);
        const uint32_t id = lane_id() < rows ? perm[r0 + lane_id()] & 0x7FFFFFFFu : 0u;
        T* dst = out + (size_t)r0 * d;
        for (uint32_t f0 = 0; f0 < rows * d; f0 += 32) {
            const uint32_t f = f0 + lane_id();
            const uint32_t i = f / d, l = f - i * d;
            const uint32_t src = __shfl_sync(0xffffffffu, id, i & 31u);
            if (f < rows * d) dst[f] = db[(size_t)src * d + l];
        }
    }
}

// The sorted lookup array with the marks of silent cells' points (bit 31) into `marked`,
// and without them in place.
__global__ void k_split_marks(uint32_t* __restrict__ perm, uint32_t* __restrict__ marked, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t x = perm[i];
    marked[i] = x;
    perm[i] = x & 0x7FFFFFFFu;
}

// ---- workload ------------------------------------------------------------------------
}  // namespace

// Per non-empty cell: number of candidates in its stencil (kernel.cu:74-144).
// One warp per cell; the rows of the stencil (tuples over dimensions 1..k-1) are
// split over the lanes, each row being one contiguous range of linear ids.  The
// stencil is symmetric, so a cell looks only at the cells after it -- half of the
// rows -- and adds each neighbour's points to its own count and its own points to
// the neighbour's.  Silent cells (a coordinate of 0: they visit no cell) are
// cleared by k_cell_keys.
// Bound by the bitmap probes (L2 latency and ALU): 6.8M cells of the skewed 6-D
// data, 122 rows each.
__global__ void __launch_bounds__(256) k_cell_workload(const unsigned long long* __restrict__ cell_lid,
                                                        const uint32_t* __restrict__ cell_start,
                                                        const uint8_t* __restrict__ cell_edge, uint32_t nC, HjGrid grid,
                                                        HjCellHash hash, uint32_t* __restrict__ cell_nb) {
    __shared__ uint32_t lists[8][kBoxRows];
    const uint32_t cell = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (cell >= nC) return;
    CellBox box;
    cell_box(grid, cell_lid[cell], cell_edge[cell] != 0, box);
    const uint32_t pop = cell_start[cell + 1] - cell_start[cell];
    uint32_t cnt = 0;
    uint32_t* list = lists[threadIdx.x >> 5];
    for (uint32_t r0 = box.r_own; r0 < box.rows; r0 += kBoxRows) {
        const uint32_t n = box_rows_present(grid, hash, box, r0, true, list);
        for (uint32_t i = lane_id(); i < n; i += 32) {
            const uint32_t x = list[i];
            const uint2 c = cell_range(hash, cell_box_row(grid, box, x & 0x0FFFFFFFu), x >> 28);
            if (c.x == kNoCell) continue;
            uint32_t s = cell_start[c.x];
            for (uint32_t j = c.x; j <= c.y; ++j) {
                const uint32_t e = cell_start[j + 1];
                cnt += e - s;
                if (j != cell) atomicAdd(&cell_nb[j], pop);
                s = e;
            }
        }
        __syncwarp();
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane_id() == 0) atomicAdd(&cell_nb[cell], cnt);
}

namespace {

// After k_cell_workload: clears the silent cells' counts, writes the sort keys of
// the workload order (top - candidates: ascending keys, descending candidates) and
// adds totalCandidates up in *out.
__global__ void __launch_bounds__(256) k_cell_keys(const unsigned long long* __restrict__ cell_lid,
                                                    const uint32_t* __restrict__ cell_start, uint32_t nC, HjGrid g,
                                                    uint32_t any_silent, uint32_t top, uint32_t* __restrict__ cell_nb,
                                                    uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                    unsigned long long* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long work = 0;
    if (i < nC) {
        uint32_t nb = cell_nb[i];
        if (any_silent) {
            unsigned long long L = cell_lid[i];
            bool silent = false;
            for (uint32_t j = 0; j < g.k; ++j) {
                const unsigned long long q = L / g.n_cells[j];
                silent |= L == q * g.n_cells[j];
                L = q;
            }
            if (silent) cell_nb[i] = nb = 0;
        }
        keys[i] = top - nb;
        vals[i] = i;
        work = (unsigned long long)nb * (cell_start[i + 1] - cell_start[i]);
    }
    for (int o = 16; o > 0; o >>= 1) work += __shfl_down_sync(0xffffffffu, work, o);
    __shared__ unsigned long long ws[8];
    if (lane_id() == 0) ws[threadIdx.x >> 5] = work;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 1; j < 8; ++j) work += ws[j];
        if (work) atomicAdd(out, work);
    }
}

__global__ void k_block_counts(const uint32_t* __restrict__ order, const uint32_t* __restrict__ cell_start, uint32_t nC,
                               uint32_t qb, uint32_t align, uint32_t* __restrict__ cnt) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == nC) cnt[nC] = 0;   // the scan's total goes there
    if (i >= nC) return;
    uint32_t c = order[i];
    uint32_t s = cell_start[c] & ~(align - 1u);
    cnt[i] = (cell_start[c + 1] - s + qb - 1) / qb;
}

__global__ void k_make_blocks(const uint32_t* __restrict__ order, const uint32_t* __restrict__ cell_start,
                              const uint32_t* __restrict__ cell_nb, const uint32_t* __restrict__ off, uint32_t nC,
                              uint32_t qb, uint32_t align, HjBlock* __restrict__ blocks) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nC) return;
    uint32_t c = order[i];
    uint32_t s = cell_start[c], e = cell_start[c + 1];
    uint32_t o = off[i];
    for (uint32_t q = s & ~(align - 1u); q < e; q += qb, ++o)
        blocks[o] = HjBlock{c, max(q, s), min(e, q + qb), cell_nb[c]};
}

// Points in the workload order: a thread per cell writes a few points itself; cells
// of more are written by the warp together, one after the other.  (A warp per cell
// took 1.09 ms for 6.8M cells of 1.5 points on average.)
__global__ void __launch_bounds__(256) k_origin_index(const uint32_t* __restrict__ order,
                                                       const uint32_t* __restrict__ cell_start,
                                                       const uint32_t* __restrict__ perm, const uint32_t* __restrict__ off,
                                                       uint32_t nC, uint32_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t s = 0, e = 0, o = 0;
    if (i < nC) {
        const uint32_t c = order[i];
        s = cell_start[c];
        e = cell_start[c + 1];
        o = off[i];
    }
    const bool many = e - s > 8u;
    if (!many)
        for (uint32_t q = s; q < e; ++q) out[o + (q - s)] = perm[q];
    uint32_t todo = __ballot_sync(0xffffffffu, many);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1u;
        const uint32_t ws = __shfl_sync(0xffffffffu, s, src), we = __shfl_sync(0xffffffffu, e, src),
                       wo = __shfl_sync(0xffffffffu, o, src);
        for (uint32_t q = ws + lane_id(); q < we; q += 32) out[wo + (q - ws)] = perm[q];
    }
}

__global__ void k_pop_in_order(const uint32_t* __restrict__ order, const uint32_t* __restrict__ cell_start, uint32_t nC,
                               uint32_t* __restrict__ pop) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nC) return;
    uint32_t c = order[i];
    pop[i] = cell_start[c + 1] - cell_start[c];
}

__global__ void k_export_index(const unsigned long long* __restrict__ cell_lid, const uint32_t* __restrict__ cell_start,
                               uint32_t nC, hj_grid_cell_lookup* lookup, hj_grid* grid) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nC) return;
    if (lookup) lookup[i] = hj_grid_cell_lookup{i, 0u, cell_lid[i]};
    if (grid) grid[i] = hj_grid{(int32_t)cell_start[i], (int32_t)cell_start[i + 1] - 1};
}

__global__ void k_export_sched(const uint32_t* __restrict__ order, const uint32_t* __restrict__ nb, uint32_t nC,
                               hj_scheduling_cell* out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nC) return;
    uint32_t c = order[i];
    out[i] = hj_scheduling_cell{(int32_t)nb[c], (int32_t)c};
}

template <typename T>
hj_status index_create_t(const T* d_db, uint32_t n, uint32_t d, uint32_t k, T eps, const double* h_min,
                         const uint32_t* h_ncells, cudaStream_t st, hj_index* ix) {
    ix->n = n; ix->d = d; ix->k = k;
    ix->eps = (double)eps;
    ix->thr = sq_threshold((double)eps, ix->dtype);
    GeoT<T> geo{};
    geo.eps = eps;
    ix->grid.k = k;
    unsigned long long mul = 1;
    ix->total_cells = 1;
    for (uint32_t j = 0; j < k; ++j) {
        geo.min_arr[j] = (T)h_min[j];
        ix->min_arr[j] = (double)geo.min_arr[j];
        ix->grid.n_cells[j] = h_ncells[j];
        ix->grid.mult[j] = mul;
        mul *= h_ncells[j];
        ix->total_cells *= h_ncells[j];
    }
    // temporaries: freed on every return path; the index's own arrays are freed by free_index on failure
    Scratch tmp(st);
    unsigned long long *keys = nullptr, *keys_tmp = nullptr;
    uint32_t *vals_tmp = nullptr, *pos = nullptr, *scalars = nullptr;
    HJ_TRY(tmp.alloc(&keys, n));
    HJ_TRY(tmp.alloc(&keys_tmp, n));
    HJ_TRY(dalloc(&ix->perm, n, st));
    HJ_TRY(tmp.alloc(&vals_tmp, n));
    HJ_TRY(tmp.alloc(&scalars, 4));
    HJ_CUDA(cudaMemsetAsync(scalars, 0, 4 * sizeof(uint32_t), st));
    unsigned grid1 = (n + 255) / 256;
    k_cell_ids<T><<<grid1, 256, 0, st>>>(d_db, n, d, geo, ix->grid, keys, ix->perm, scalars,
                                          scalars + 2);
    HJ_LAUNCHED();
    uint32_t nbits = bits_for(ix->total_cells > 0 ? ix->total_cells - 1 : 0);
    HJ_TRY(radix_sort_u64_u32(reinterpret_cast<uint64_t*>(keys), ix->perm, reinterpret_cast<uint64_t*>(keys_tmp),
                              vals_tmp, n, nbits, st));
    tmp.release(keys_tmp);
    tmp.release(vals_tmp);
    HJ_TRY(tmp.alloc(&pos, n));
    k_run_flags<<<grid1, 256, 0, st>>>(keys, n, pos);
    HJ_LAUNCHED();
    HJ_TRY(scan_u32_inplace(pos, n, st));
    HJ_TRY(dalloc(&ix->cell_lid, (size_t)n, st));
    HJ_TRY(dalloc(&ix->cell_start, (size_t)n + 1, st));
    k_cells<<<grid1, 256, 0, st>>>(keys, pos, n, ix->cell_lid, ix->cell_start, scalars + 1);
    HJ_LAUNCHED();
    T* pts = nullptr;
    HJ_TRY(dalloc(&pts, (size_t)n * d, st));
    ix->pts = pts;
    unsigned grid2 = (unsigned)std::min<uint64_t>(((uint64_t)n + 255) / 256, (uint64_t)num_sms() * 8);
    k_gather_rows<T><<<grid2, 256, 0, st>>>(d_db, ix->perm, n, d, pts);
    HJ_LAUNCHED();
    uint32_t* hs = nullptr;
    HJ_TRY(readback_buffer(reinterpret_cast<void**>(&hs)));
    HJ_CUDA(cudaMemcpyAsync(hs, scalars, 3 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    HJ_CUDA(cudaStreamSynchronize(st));
    ix->aliasing = hs[0];
    ix->nC = hs[1];
    ix->any_silent = hs[2];
    if (ix->aliasing) {
        set_error("grid aliasing: a point's cell coordinate reaches nCells in some indexed dimension "
                  "(epsilon below the coordinates' rounding granularity); unsupported");
        return HJ_ERR_UNSUPPORTED;
    }
    if (ix->any_silent) {
        HJ_TRY(dalloc(&ix->perm_flag, n, st));
        k_split_marks<<<grid1, 256, 0, st>>>(ix->perm, ix->perm_flag, n);
        HJ_LAUNCHED();
    }
    return HJ_OK;
}

// The first cell of each group inserts the group's entry: key, first cell, mask
// of the group's ids (its cells are the next ones in the table, at most four).
// The key word pair is claimed with a 64-bit compare-and-swap on the entry's
// first 8 bytes; first cell and mask are written after it.  The first cell of
// each segment of 32 ids clears the segment's bits in the bitmap (a clear bit is a
// cell: the bitmap and the table start as one array of set bits).  Every cell notes
// whether a coordinate lies at the grid's edge.  The first threads also write the
// grid's row offsets (HjGrid::row_off): entry r is the sum over j >= 1 of r's base-3
// digits times the multipliers.
__global__ void k_hash_insert(const unsigned long long* __restrict__ lid, uint32_t nC, HjGrid grid, uint4* entries,
                              unsigned long long mask, uint32_t* occ, uint32_t occ_shift, uint8_t* __restrict__ edge,
                              unsigned long long* __restrict__ row_off) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < grid.full_rows) {
        uint32_t rem = i;
        unsigned long long o = 0;
        for (uint32_t j = 1; j < grid.k; ++j) {
            o += (unsigned long long)(rem % 3u) * grid.mult[j];
            rem /= 3u;
        }
        row_off[i] = o;
    }
    if (i >= nC) return;
    const unsigned long long me = lid[i], before = i > 0 ? lid[i - 1] : ~me;
    {
        unsigned long long rest = me;
        bool e = false;
        for (uint32_t j = 0; j < grid.k; ++j) {
            const unsigned long long q = rest / grid.n_cells[j];
            const uint32_t c = (uint32_t)(rest - q * grid.n_cells[j]);
            e |= c == 0u || c + 1u >= grid.n_cells[j];
            rest = q;
        }
        edge[i] = e ? 1 : 0;
    }
    if (i == 0 || (before >> 5) != (me >> 5)) {
        uint32_t bits = 0;
        for (uint32_t j = i; j < nC && (lid[j] >> 5) == (me >> 5); ++j) bits |= 1u << (uint32_t)(lid[j] & 31u);
        atomicAnd(occ + occ_word(me, occ_shift), ~bits);
    }
    const unsigned long long g = me >> 2;
    if (i > 0 && (before >> 2) == g) return;
    uint32_t m = 0;
    for (uint32_t j = i; j < nC && j < i + 4 && (lid[j] >> 2) == g; ++j) m |= 1u << (uint32_t)(lid[j] & 3u);
    unsigned long long s = mix64(g) & mask;
    for (unsigned long long probe = 0; probe <= mask; ++probe) {   // the table is at most half full
        unsigned long long* kw = reinterpret_cast<unsigned long long*>(&entries[s]);
        const unsigned long long prev = atomicCAS(kw, kEmptyLid, g);
        if (prev == kEmptyLid) {
            entries[s].z = i;
            entries[s].w = m;
            return;
        }
        s = (s + 1) & mask;
    }
}

// The cell hash of an index whose cell table is built: the table (capacity: the
// power of two at least twice the number of cells, an upper bound on the groups
// that needs no count from the device, at least 64), its bitmap (a word per entry)
// and, for k <= kRowOffMaxK, the grid's row offsets.
hj_status build_cell_hash(hj_index* ix, cudaStream_t st) {
    unsigned long long cap = 64;
    while (cap < 2ull * ix->nC) cap <<= 1;
    HJ_TRY(dalloc(&ix->hash_entries, (size_t)(cap + cap / 4), st));
    HJ_CUDA(cudaMemsetAsync(ix->hash_entries, 0xFF, (size_t)(cap + cap / 4) * sizeof(uint4), st));
    ix->hash_mask = cap - 1;
    ix->hash_occ = reinterpret_cast<uint32_t*>(ix->hash_entries + cap);
    ix->occ_shift = 65 - bits_for(cap);   // cap = 2^(bits - 1)
    HJ_TRY(dalloc(&ix->cell_edge, ix->nC, st));
    if (ix->grid.k <= kRowOffMaxK) {
        uint32_t rows = 1;
        ix->grid.full_base = 1;
        for (uint32_t j = 1; j < ix->grid.k; ++j) {
            rows *= 3;
            ix->grid.full_base += ix->grid.mult[j];
        }
        HJ_TRY(dalloc(&ix->row_off, rows, st));
        ix->grid.full_rows = rows;
        ix->grid.row_off = ix->row_off;
    }
    k_hash_insert<<<(std::max(ix->nC, ix->grid.full_rows) + 255) / 256, 256, 0, st>>>(
        ix->cell_lid, ix->nC, ix->grid, ix->hash_entries, ix->hash_mask, ix->hash_occ, ix->occ_shift, ix->cell_edge,
        ix->row_off);
    HJ_LAUNCHED();
    return HJ_OK;
}

void free_index(hj_index* ix, cudaStream_t st) {
    tc_release(ix);
    dfree(ix->hash_entries, st);
    ix->hash_occ = nullptr;   // part of the table's allocation
    dfree(ix->cell_edge, st);
    dfree(ix->row_off, st);
    ix->grid.row_off = nullptr;
    ix->grid.full_rows = 0;
    dfree(ix->pts, st);
    dfree(ix->perm, st);
    dfree(ix->cell_lid, st);
    dfree(ix->cell_start, st);
    dfree(ix->cell_nb, st);
    dfree(ix->cell_order, st);
    dfree(ix->tc_a, st);
    dfree(ix->tc_b, st);
    dfree(ix->perm_flag, st);
}

}  // namespace

// Launches of the workload order; **total (in tmp) then holds totalCandidates, for workload_done.
static hj_status workload_launch(hj_index* ix, Scratch& tmp, unsigned long long** total_out, cudaStream_t st) {
    const uint32_t nC = ix->nC;
    // a previous attempt that failed part-way may have left these allocated
    dfree(ix->cell_nb, st);
    dfree(ix->cell_order, st);
    unsigned long long* total = nullptr;
    uint32_t *keys = nullptr, *keys_tmp = nullptr, *vals_tmp = nullptr;
    HJ_TRY(dalloc(&ix->cell_nb, nC, st));
    HJ_TRY(dalloc(&ix->cell_order, nC, st));
    HJ_TRY(tmp.alloc(&total, 1));
    HJ_TRY(tmp.alloc(&keys, nC));
    HJ_TRY(tmp.alloc(&keys_tmp, nC));
    HJ_TRY(tmp.alloc(&vals_tmp, nC));
    HJ_CUDA(cudaMemsetAsync(ix->cell_nb, 0, (size_t)nC * 4, st));
    HJ_CUDA(cudaMemsetAsync(total, 0, sizeof(unsigned long long), st));
    unsigned g = (unsigned)(((uint64_t)nC * 32 + 255) / 256);
    k_cell_workload<<<g, 256, 0, st>>>(ix->cell_lid, ix->cell_start, ix->cell_edge, nC, ix->grid, cell_hash(ix),
                                       ix->cell_nb);
    HJ_LAUNCHED();
    // no count exceeds n: the sort needs only that many bits
    const uint32_t nbits = bits_for(ix->n);
    k_cell_keys<<<(nC + 255) / 256, 256, 0, st>>>(ix->cell_lid, ix->cell_start, nC, ix->grid, ix->any_silent,
                                                  (uint32_t)((1ull << nbits) - 1), ix->cell_nb, keys, ix->cell_order,
                                                  total);
    HJ_LAUNCHED();
    HJ_TRY(radix_sort_u32_u32(keys, ix->cell_order, keys_tmp, vals_tmp, nC, nbits, st));
    *total_out = total;
    return HJ_OK;
}
static void workload_done(hj_index* ix, unsigned long long total) {
    ix->total_candidates = total;
    ix->have_workload = true;
}

hj_status build_blocks(hj_index* ix, uint32_t qb, uint32_t align, HjBlock** d_blocks, uint32_t* n_blocks,
                       cudaStream_t st) {
    const uint32_t nC = ix->nC;
    Scratch tmp(st);
    unsigned long long *total = nullptr, *back = nullptr;
    HJ_TRY(readback_buffer(reinterpret_cast<void**>(&back)));
    if (!ix->have_workload) HJ_TRY(workload_launch(ix, tmp, &total, st));
    uint32_t* cnt = nullptr;
    HJ_TRY(tmp.alloc(&cnt, (size_t)nC + 1));
    k_block_counts<<<nC / 256 + 1, 256, 0, st>>>(ix->cell_order, ix->cell_start, nC, qb, align, cnt);
    HJ_LAUNCHED();
    HJ_TRY(scan_u32_inplace(cnt, (uint64_t)nC + 1, st));
    // nothing that can fail for want of memory stands between a copy and the wait for it
    if (total) HJ_CUDA(cudaMemcpyAsync(back + 1, total, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    HJ_CUDA(cudaMemcpyAsync(back, cnt + nC, 4, cudaMemcpyDeviceToHost, st));
    HJ_CUDA(cudaStreamSynchronize(st));
    if (total) workload_done(ix, back[1]);
    const uint32_t nb = *reinterpret_cast<const uint32_t*>(back);
    HjBlock* blocks = nullptr;
    HJ_TRY(tmp.alloc_pool(&blocks, (size_t)std::max<uint32_t>(nb, 1)));   // handed to the caller
    k_make_blocks<<<(nC + 255) / 256, 256, 0, st>>>(ix->cell_order, ix->cell_start, ix->cell_nb, cnt, nC, qb, align,
                                                    blocks);
    HJ_LAUNCHED();
    *d_blocks = tmp.keep(blocks);
    *n_blocks = nb;
    return HJ_OK;
}

}  // namespace hj

using namespace hj;

extern "C" {

const char* hj_last_error(void) { return hj::g_err; }

void hj_debug_fail_alloc(uint64_t nth) { hj::g_fail_alloc_in.store((int64_t)nth, std::memory_order_relaxed); }

hj_status hj_debug_pool_used(uint64_t* bytes) {
    if (!bytes) { set_error("hj_debug_pool_used: null argument"); return HJ_ERR_INVALID; }
    int dev = 0;
    cudaMemPool_t pool;
    HJ_CUDA(cudaGetDevice(&dev));
    HJ_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
    unsigned long long used = 0;   // cudaMemPoolAttrUsedMemCurrent is a 64-bit count
    HJ_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
    *bytes = (uint64_t)used;
    return HJ_OK;
}
hj_status hj_debug_pool_peak(uint64_t* bytes, int reset) {
    if (!bytes) { set_error("hj_debug_pool_peak: null argument"); return HJ_ERR_INVALID; }
    int dev = 0;
    cudaMemPool_t pool;
    HJ_CUDA(cudaGetDevice(&dev));
    HJ_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
    unsigned long long high = 0;
    HJ_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &high));
    *bytes = (uint64_t)high;
    if (reset) {
        unsigned long long zero = 0;   // resets the high-water mark to the current use
        HJ_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &zero));
    }
    return HJ_OK;
}
const char* hj_version(void) { return "hegjoin_b200 0.1 (sm_100a)"; }
uint64_t hj_kernel_launch_count(void) { return hj::launch_count(); }

hj_status hj_grid_geometry(const void* d_db, uint32_t n, uint32_t d, uint32_t k, int dtype, double eps,
                           double* h_min_arr, double* h_max_arr, uint32_t* h_n_cells, uint64_t* h_total_cells,
                           void* stream) {
    if (!d_db || n == 0 || d == 0 || k == 0 || k > (uint32_t)kMaxK || k > d || !(eps > 0)) {
        set_error("hj_grid_geometry: invalid arguments (n=%u d=%u k=%u eps=%g)", n, d, k, eps);
        return HJ_ERR_INVALID;
    }
    cudaStream_t st = as_stream(stream);
    if (dtype == HJ_F32)
        return geometry_t<float>((const float*)d_db, n, d, k, (float)eps, h_min_arr, h_max_arr, h_n_cells,
                                 h_total_cells, st);
    if (dtype == HJ_F64)
        return geometry_t<double>((const double*)d_db, n, d, k, eps, h_min_arr, h_max_arr, h_n_cells, h_total_cells,
                                  st);
    set_error("hj_grid_geometry: unknown dtype %d", dtype);
    return HJ_ERR_INVALID;
}

hj_status hj_index_create(const void* d_db, uint32_t n, uint32_t d, uint32_t k, int dtype, double eps,
                          const double* h_min_arr, const uint32_t* h_n_cells, void* stream, hj_index** out) {
    if (!out) { set_error("hj_index_create: null out"); return HJ_ERR_INVALID; }
    *out = nullptr;
    if (!d_db || n == 0 || d == 0 || d > (uint32_t)kMaxD || k == 0 || k > (uint32_t)kMaxK || k > d || !(eps > 0) ||
        (dtype != HJ_F32 && dtype != HJ_F64) || n >= 0x7FFFFFFFu) {
        set_error("hj_index_create: invalid arguments (n=%u d=%u k=%u dtype=%d eps=%g)", n, d, k, dtype, eps);
        return HJ_ERR_INVALID;
    }
    cudaStream_t st = as_stream(stream);
    double mn[kMaxK], mx[kMaxK];
    uint32_t nc[kMaxK];
    if (!h_min_arr || !h_n_cells) {
        HJ_TRY(hj_grid_geometry(d_db, n, d, k, dtype, eps, mn, mx, nc, nullptr, stream));
        h_min_arr = mn;
        h_n_cells = nc;
    }
    uint64_t tot = 1;
    for (uint32_t j = 0; j < k; ++j) {
        if (h_n_cells[j] == 0) { set_error("hj_index_create: nCells[%u] == 0", j); return HJ_ERR_INVALID; }
        if (tot > ~0ull / h_n_cells[j]) { set_error("hj_index_create: totalCells overflows 64 bits"); return HJ_ERR_UNSUPPORTED; }
        tot *= h_n_cells[j];
    }
    init_memory_pool();
    hj_index* ix = new hj_index();
    ix->dtype = dtype;
    ix->stream = st;
    cudaGetDevice(&ix->device);
    hj_status s = (dtype == HJ_F32)
                      ? index_create_t<float>((const float*)d_db, n, d, k, (float)eps, h_min_arr, h_n_cells, st, ix)
                      : index_create_t<double>((const double*)d_db, n, d, k, eps, h_min_arr, h_n_cells, st, ix);
    // linear ids are below totalCells <= 2^64 - 1, so none equals the hash's free-slot mark
    if (s == HJ_OK) s = build_cell_hash(ix, st);
    if (s != HJ_OK) {
        free_index(ix, st);
        cudaStreamSynchronize(st);
        delete ix;
        return s;
    }
    *out = ix;
    return HJ_OK;
}

hj_status hj_index_destroy(hj_index* ix) {
    if (!ix) return HJ_OK;
    // stream-ordered frees on the index's own stream: no device-wide synchronisation,
    // so concurrent joins on other streams keep running
    free_index(ix, ix->stream);
    delete ix;
    return HJ_OK;
}

hj_status hj_index_get_info(const hj_index* ix, hj_index_info* o) {
    if (!ix || !o) { set_error("hj_index_get_info: null argument"); return HJ_ERR_INVALID; }
    *o = hj_index_info{};
    o->n = ix->n; o->d = ix->d; o->k = ix->k; o->dtype = (uint32_t)ix->dtype;
    o->n_nonempty_cells = ix->nC;
    o->grid_aliasing = ix->aliasing;
    o->total_cells = ix->total_cells;
    o->total_candidates = ix->total_candidates;
    o->eps = ix->eps;
    o->sq_threshold = ix->thr;
    for (uint32_t j = 0; j < ix->k; ++j) {
        o->min_arr[j] = ix->min_arr[j];
        o->n_cells[j] = ix->grid.n_cells[j];
    }
    return HJ_OK;
}

hj_status hj_index_export(const hj_index* ix, hj_grid_cell_lookup* d_lookup, hj_grid* d_grid, uint32_t* d_index_lookup,
                          void* stream) {
    if (!ix) { set_error("hj_index_export: null index"); return HJ_ERR_INVALID; }
    cudaStream_t st = as_stream(stream);
    if (d_lookup || d_grid) {
        k_export_index<<<(ix->nC + 255) / 256, 256, 0, st>>>(ix->cell_lid, ix->cell_start, ix->nC, d_lookup, d_grid);
        HJ_LAUNCHED();
    }
    if (d_index_lookup)
        HJ_CUDA(cudaMemcpyAsync(d_index_lookup, ix->perm, (size_t)ix->n * 4, cudaMemcpyDeviceToDevice, st));
    return HJ_OK;
}

hj_status hj_index_views(const hj_index* ix, const void** pts, const uint32_t** perm, const uint64_t** cell_lid,
                         const uint32_t** cell_start) {
    if (!ix) { set_error("hj_index_views: null index"); return HJ_ERR_INVALID; }
    if (pts) *pts = ix->pts;
    if (perm) *perm = ix->perm;
    if (cell_lid) *cell_lid = reinterpret_cast<const uint64_t*>(ix->cell_lid);
    if (cell_start) *cell_start = ix->cell_start;
    return HJ_OK;
}

hj_status hj_sort_by_workload(hj_index* ix, void* stream, uint64_t* total_candidates) {
    if (!ix) { set_error("hj_sort_by_workload: null index"); return HJ_ERR_INVALID; }
    cudaStream_t st = as_stream(stream);
    if (!ix->have_workload) {
        Scratch tmp(st);
        unsigned long long *total = nullptr, *back = nullptr;
        HJ_TRY(readback_buffer(reinterpret_cast<void**>(&back)));
        HJ_TRY(hj::workload_launch(ix, tmp, &total, st));
        HJ_CUDA(cudaMemcpyAsync(back, total, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
        HJ_CUDA(cudaStreamSynchronize(st));
        hj::workload_done(ix, *back);
    }
    if (total_candidates) *total_candidates = ix->total_candidates;
    return HJ_OK;
}

hj_status hj_workload_export(const hj_index* ix, hj_scheduling_cell* d_sched, uint32_t* d_origin, void* stream) {
    if (!ix || !ix->have_workload) { set_error("hj_workload_export: run hj_sort_by_workload first"); return HJ_ERR_INVALID; }
    cudaStream_t st = as_stream(stream);
    uint32_t nC = ix->nC;
    if (d_sched) {
        k_export_sched<<<(nC + 255) / 256, 256, 0, st>>>(ix->cell_order, ix->cell_nb, nC, d_sched);
        HJ_LAUNCHED();
    }
    if (d_origin) {
        Scratch tmp(st);
        uint32_t* off = nullptr;
        HJ_TRY(tmp.alloc(&off, nC));
        k_pop_in_order<<<(nC + 255) / 256, 256, 0, st>>>(ix->cell_order, ix->cell_start, nC, off);
        HJ_LAUNCHED();
        HJ_TRY(scan_u32_inplace(off, nC, st));
        k_origin_index<<<(nC + 255) / 256, 256, 0, st>>>(ix->cell_order, ix->cell_start, ix->perm, off, nC, d_origin);
        HJ_LAUNCHED();
    }
    return HJ_OK;
}

}  // extern "C"
