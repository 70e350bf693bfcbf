// tcr_search.cu -- compact-hashing fixed-radius neighbour search for sm_100a, with a C ABI.
//
// One engine serves a single search and a batch of independent clouds (the scenes or timesteps
// of a simulation sweep, of uneven sizes, each with its own domain, periodicity, supports and
// hashMapLength); a single search is a batch of one cloud.  Every phase is one set of launches
// over all clouds, on one CUDA stream, with no host synchronisation inside a phase:
//   build:  per-cloud support max-reductions -> per-cloud grid parameters (compute_h) -> wrap and
//           pack reference points into float4 (x, y, z, h) with (cloud, linear cell) sort keys ->
//           one cooperative launch: stable radix sort, placement, run-length cell table (begin,
//           coords, bucket, cloud) and one lin -> cell map region per cloud.
//   count:  query packing (a self search reuses the reference order) -> query groups (cells) ->
//           work units of <= 32 queries of one group -> warp-per-unit candidate walk that tests
//           every (query, candidate) pair once as tensor-core products, counts, and stages
//           per-unit hit records -> exact decisions of the pairs near the threshold -> scan.
//   emit:   expansion of the staged records into CSR/COO slots; units that were not staged are
//           walked again.
// The candidate set of every query is the reference's (cppSrc/neighborhood.h:73-132): the
// stencil cells of its own cell, found by linear index inside the bucket of the stencil cell's
// hash; the pair test is the reference's float test (tcr_common.cuh).  Clouds never see each
// other: keys, cells, map regions and work units all carry the cloud.
#include <cstdio>
#include <cstring>
#include <cstdarg>
#include <cstddef>
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

#include <cuda_fp16.h>

#include "tcr_common.cuh"
#include "tcr_scan.cuh"
#include "tcr_sort.cuh"
#include "../../include/tcr_b200.h"

namespace tcr {

// ------------------------------------------------------------------------------------------
// error reporting (set_error / g_err: tcr_common.cuh)
#define TCR_CUDA(call)                                                                         \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            return set_error(TCR_ERR_CUDA, "%s:%d %s", __FILE__, __LINE__, cudaGetErrorString(e_)); \
    } while (0)

// ------------------------------------------------------------------------------------------
// workspace layout
static inline int64_t align256(int64_t x) { return (x + 255) & ~int64_t(255); }
static inline int64_t next_pow2(int64_t x) {
    int64_t p = 1;
    while (p < x) p <<= 1;
    return p;
}
// Map slots of a cloud with n reference points: a power of two >= 2n (load factor <= 1/2).
static inline int64_t hash_capacity(int64_t n_ref, int64_t min_cap) {
    return std::max<int64_t>(min_cap, next_pow2(2 * std::max<int64_t>(n_ref, 1)));
}
constexpr int64_t kSingleMapMin = 1024;  // one search
constexpr int64_t kBatchMapMin = 64;     // per cloud of a batch
// Work counters: [0] count walk, [1] emit walk, [2 + cls] / [8 + cls] the count / emit walk of
// one cloud class (cls = dim * 2 + periodic, 2..7) in a batch that mixes classes, [30] the expansion.
constexpr int kWorkCounters = 32;
constexpr int kExpandCounter = 30;  // the record expansion

// Default tuning of a search (tcr_search_desc / tcr_batch_desc unit_queries and walk_blocks_per_sm):
// queries per work unit and blocks per SM of the walk's grid (the count walk has six or seven of them
// resident; the others take over as those end).  Neither changes a result: a query's
// candidates and their order do not depend on how queries are grouped into units.
constexpr int kDefaultUnitQueries = 32;
constexpr int kDefaultWalkBlocksPerSM = 12;

struct Carve {
    char* base;
    int64_t off;
    template <typename T>
    T* take(int64_t count) {
        T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
        off += align256(count * (int64_t)sizeof(T));
        return p;
    }
};

// Persistent structure (reference side); kept alive for reuse.
struct Structure {
    GridParams* grid;         // [C] per cloud
    int32_t* num_cells;       // [3] cells; set when the build's sort gave up waiting; blocks of the statistics that finished
    int32_t* bad_grids;       // [1] clouds with points on both sides and no valid grid
    float4* rsorted;          // [nr] wrapped reference points in (cloud, cell) order, .w = support
    int32_t* rsidx;           // [nr] global index of each sorted point
    int32_t* cell_start;      // [nr+1]
    int32_t* cell_lin;        // [nr]
    int32_t* cell_coords;     // [3*nr]
    int32_t* cell_bucket;     // [nr] reference hash of the cell's coordinates mod hashMapLength
    int32_t* cell_cloud;      // [nr]
    unsigned long long* map;  // [map_total] per-cloud regions of (lin << 32 | cell), empty = ~0
    int64_t map_total;
};

static Structure carve_structure(void* buf, int64_t nr, int64_t C, int64_t map_total, int64_t* bytes) {
    Carve c{(char*)buf, 0};
    Structure s;
    s.grid = c.take<GridParams>(C);
    s.num_cells = c.take<int32_t>(3);
    s.bad_grids = c.take<int32_t>(1);
    s.rsorted = c.take<float4>(nr);
    s.rsidx = c.take<int32_t>(nr);
    s.cell_start = c.take<int32_t>(nr + 1);
    s.cell_lin = c.take<int32_t>(nr);
    s.cell_coords = c.take<int32_t>(3 * nr);
    s.cell_bucket = c.take<int32_t>(nr);
    s.cell_cloud = c.take<int32_t>(nr);
    s.map_total = map_total;
    s.map = c.take<unsigned long long>(map_total);
    if (bytes) *bytes = c.off;
    return s;
}

// Per-search scratch.
struct Scratch {
    CloudParams* table;     // [C] this search's cloud table
    int32_t* query_prefix;  // [C+1] global index of each cloud's first query (last: total)
    int32_t* ref_prefix;    // [C+1] the same for reference points
    QueryParams* qparams;   // [C]
    void* sort_state;       // SortState32 or SortState64
    int32_t* num_qgroups;   // [2] query groups; set when this search's query sort gave up waiting
    int32_t* num_units;     // [1]
    int32_t* num_stray;     // [1]
    int32_t* work;          // [kWorkCounters] work distribution counters
    int64_t* total;         // [1]
    int64_t* info;          // [8] see tcr_count
    int32_t* num_flagged;   // [1]
    int32_t* exact_clouds;  // [1] clouds whose every pair takes the exact test
    int32_t* num_exact;     // [3] pairs inside the count walk's band: listed one by one, decided with their window;
                            // windows listed
    int32_t* unit_cap;      // [1] queries per work unit of this search (set by the count phase)
    unsigned long long* cursor;  // [2] staging fill, staging capacity
    float4* pack;           // [max(nq,nr)] packed input points before sorting
    void* keys[2];          // [max(nq,nr)] 64-bit slots (32-bit keys use the first half)
    int32_t* vals[2];
    int32_t* hist;
    int32_t* tile_sums;
    int64_t* scan_tiles64;  // [scan_tiles(max)]
    int32_t* scan_tiles32;  // [scan_tiles(max)]
    float4* qsorted;        // [nq]
    int32_t* qsidx;         // [nq] global query index of each sorted query
    int32_t* qgroup_start;  // [nq+1]
    int32_t* qgroup_coords; // [3*nq]
    int32_t* qgroup_cloud;  // [nq]
    int32_t* unit_group;    // [nq]
    int32_t* unit_t0;       // [nq]
    int32_t* counts;        // [nq] global query order
    int32_t* stray;         // [nq]
    int32_t* rec;           // [nq] per unit: offset of its record in the staging list (-1: not staged)
    int32_t* flagged;       // [nq] units re-walked by the emit pass
    // incremental re-sort (builds given the previous cell of every reference point), else null
    int32_t* stay;          // [nr] 1: the point is still in its previous cell
    void* stay_keys;        // [nr] keys of the unmoved points, input order (sorted when the hint holds)
    int32_t* stay_idx;      // [nr]
    void* moved_keys[2];    // [nr] keys of the moved points (sorted in place)
    int32_t* moved_vals[2]; // [nr]
    void* moved_state;      // SortState of the moved points' sort
    int32_t* inc_count;     // [2] unmoved points, hint broken (1: fall back to the full sort)
};

static Scratch carve_scratch(void* buf, int64_t nq, int64_t nr, int64_t C, bool incremental, int64_t* bytes) {
    Carve c{(char*)buf, 0};
    Scratch s;
    const int64_t nmax = std::max<int64_t>(std::max<int64_t>(nq, nr), 1);
    s.table = c.take<CloudParams>(C);
    s.query_prefix = c.take<int32_t>(C + 1);
    s.ref_prefix = c.take<int32_t>(C + 1);
    s.qparams = c.take<QueryParams>(C);
    s.sort_state = c.take<SortState64>(1);
    s.num_qgroups = c.take<int32_t>(2);
    s.num_units = c.take<int32_t>(1);
    s.num_stray = c.take<int32_t>(1);
    s.work = c.take<int32_t>(kWorkCounters);
    s.total = c.take<int64_t>(1);
    s.info = c.take<int64_t>(8);
    s.num_flagged = c.take<int32_t>(1);
    s.exact_clouds = c.take<int32_t>(1);
    s.num_exact = c.take<int32_t>(3);
    s.unit_cap = c.take<int32_t>(1);
    s.cursor = c.take<unsigned long long>(2);
    s.pack = c.take<float4>(nmax);
    s.keys[0] = c.take<unsigned long long>(nmax);
    s.keys[1] = c.take<unsigned long long>(nmax);
    s.vals[0] = c.take<int32_t>(nmax);
    s.vals[1] = c.take<int32_t>(nmax);
    s.hist = c.take<int32_t>(sort_hist_elems(nmax));
    s.tile_sums = c.take<int32_t>(kBins);  // the sort's digit totals
    s.scan_tiles64 = c.take<int64_t>(scan_tiles(nmax + 1));
    s.scan_tiles32 = c.take<int32_t>(scan_tiles(nmax + 1));
    const int64_t q = std::max<int64_t>(nq, 1);
    s.qsorted = c.take<float4>(q);
    s.qsidx = c.take<int32_t>(q);
    s.qgroup_start = c.take<int32_t>(q + 1);
    s.qgroup_coords = c.take<int32_t>(3 * q);
    s.qgroup_cloud = c.take<int32_t>(q);
    s.unit_group = c.take<int32_t>(q);
    s.unit_t0 = c.take<int32_t>(q);
    s.counts = c.take<int32_t>(q);
    s.stray = c.take<int32_t>(q);
    s.rec = c.take<int32_t>(q);
    s.flagged = c.take<int32_t>(q);
    const int64_t ni = incremental ? std::max<int64_t>(nr, 1) : 0;
    s.stay = incremental ? c.take<int32_t>(ni) : nullptr;
    s.stay_keys = incremental ? c.take<unsigned long long>(ni) : nullptr;
    s.stay_idx = incremental ? c.take<int32_t>(ni) : nullptr;
    for (int k = 0; k < 2; ++k) {
        s.moved_keys[k] = incremental ? c.take<unsigned long long>(ni) : nullptr;
        s.moved_vals[k] = incremental ? c.take<int32_t>(ni) : nullptr;
    }
    s.moved_state = incremental ? c.take<SortState64>(1) : nullptr;
    s.inc_count = incremental ? c.take<int32_t>(2) : nullptr;
    if (bytes) *bytes = c.off;
    return s;
}

template <typename K>
static SortWorkspaceT<K> sort_workspace(const Scratch& W) {
    SortWorkspaceT<K> s;
    s.keys[0] = reinterpret_cast<K*>(W.keys[0]);
    s.keys[1] = reinterpret_cast<K*>(W.keys[1]);
    s.vals[0] = W.vals[0];
    s.vals[1] = W.vals[1];
    s.hist = W.hist;
    s.tile_sums = W.tile_sums;
    s.state = reinterpret_cast<SortStateT<K>*>(W.sort_state);
    return s;
}

// ------------------------------------------------------------------------------------------
// the cloud table

// Host -> device copy of the table as kernel parameters (no pageable copy, so it also records
// into a CUDA graph): up to kUploadChunk clouds travel with the phase's init kernel; of more, all but the last
// with launches of up to kWideChunk clouds (kernel parameters hold 32 KB; 24 clouds a launch cost a batch of 256
// 22 launches, 162 us).
constexpr int kUploadChunk = 24;
constexpr int kWideChunk = 220;
template <int N>
struct CloudChunk {
    int32_t first, count, n_clouds, query_total, ref_total, pad;
    CloudParams p[N];
};
static_assert(sizeof(CloudChunk<kUploadChunk>) <= 4000 && sizeof(CloudChunk<kWideChunk>) <= 32000,
              "kernel parameter block too large");

template <int N>
__device__ __forceinline__ void upload_chunk(const CloudChunk<N>& ch, CloudParams* table, int32_t* query_prefix,
                                             int32_t* ref_prefix) {
    for (int i = threadIdx.x; i < ch.count; i += blockDim.x) {
        const int c = ch.first + i;
        table[c] = ch.p[i];
        query_prefix[c] = ch.p[i].query_base;
        ref_prefix[c] = ch.p[i].ref_base;
    }
    if (threadIdx.x == 0 && ch.first + ch.count == ch.n_clouds) {
        query_prefix[ch.n_clouds] = ch.query_total;
        ref_prefix[ch.n_clouds] = ch.ref_total;
    }
}
// Lanes reading different kernel parameters are served one by one, so the chunk is spread over blocks.
constexpr int kUploadPerBlock = 8;
__global__ void upload_clouds_kernel(const __grid_constant__ CloudChunk<kWideChunk> ch, CloudParams* table,
                                     int32_t* query_prefix, int32_t* ref_prefix) {
    const int i = blockIdx.x * kUploadPerBlock + threadIdx.x;
    if (threadIdx.x >= kUploadPerBlock || i >= ch.count) return;
    table[ch.first + i] = ch.p[i];
    query_prefix[ch.first + i] = ch.p[i].query_base;
    ref_prefix[ch.first + i] = ch.p[i].ref_base;
}

// Cloud of global point index i: the last c with prefix[c] <= i (empty clouds are skipped).
__device__ __forceinline__ int cloud_of(const int32_t* __restrict__ prefix, int C, int64_t i) {
    if (C == 1) return 0;
    int lo = 0, hi = C;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= i) lo = mid; else hi = mid;
    }
    return lo;
}

// ------------------------------------------------------------------------------------------
// build kernels

// Block reduction of max / or; one atomic per block and field.
__device__ __forceinline__ void block_reduce_stats(uint32_t kmax, int bad, SupportStats* out) {
    __shared__ uint32_t s_max[32];
    __shared__ int s_bad[32];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) { s_max[w] = kmax; s_bad[w] = bad; }
    __syncthreads();
    if (w == 0) {
        kmax = lane < nw ? s_max[lane] : 0u;
        bad = lane < nw ? s_bad[lane] : 0;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
            bad |= __shfl_xor_sync(0xffffffffu, bad, o);
        }
        if (lane == 0) {
            atomicMax(&out->max_key, kmax);
            if (bad) atomicOr(&out->bad, 1);
        }
    }
}

__device__ __forceinline__ SupportStats* stats_at(char* base, int64_t stride, int c) {
    return reinterpret_cast<SupportStats*>(base + stride * c);
}
__device__ __forceinline__ void stats_atomic(SupportStats* s, uint32_t kmax, int bad) {
    if (kmax) atomicMax(&s->max_key, kmax);
    if (bad) atomicOr(&s->bad, 1);
}

__device__ __forceinline__ void support_stat(float v, uint32_t& kmax, int& bad) {
    kmax = max(kmax, float_key(v));
    bad |= !(v >= 1e-18f && v <= 1e18f);
}
// The threads' statistics of the cloud each ended in (-1: it had no point): one atomic per block and field
// where the block stayed in one cloud.
__device__ __forceinline__ void block_stats(int cur, uint32_t kmax, int bad, char* out, int64_t stride) {
    __shared__ int s_cloud;
    if (threadIdx.x == 0) s_cloud = cur;  // thread 0 holds the block's first point, if it has any
    __syncthreads();
    if (__syncthreads_and(cur < 0 || cur == s_cloud)) {
        if (s_cloud >= 0) block_reduce_stats(kmax, bad, stats_at(out, stride, s_cloud));
    } else if (cur >= 0) {
        stats_atomic(stats_at(out, stride, cur), kmax, bad);
    }
}
// Whether this block is the last of its launch to get here; the others' writes before are visible then.
__device__ __forceinline__ bool last_block(int32_t* done) {
    __shared__ int s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();  // (cumulative: the block's atomics before its arrival)
        s_last = atomicAdd(done, 1) == (int)gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    return s_last != 0;
}

// Per cloud: util.py:28-79 compute_h and cellTable.py:27-29, float32 throughout.
// same_sup: the query supports are the reference support array (statistics reduced once).
__device__ __forceinline__ void grid_params(const CloudParams* __restrict__ table, GridParams* grid, int C,
                                            int32_t* bad_grids, int same_sup, int first, int stride) {
    const float grow = 1.00010001659393310546875f;  // fl32(1e-4 + 1)
    for (int cl = first; cl < C; cl += stride) {
        const CloudParams& sp = table[cl];
        GridParams* g = &grid[cl];
        if (same_sup) g->build_query_stats = g->ref_stats;
        // computeGridSupport: scatter reads the reference supports, gather the query supports,
        // (super)symmetric both (torch.max propagates NaN, as the key maximum does).
        uint32_t key = 0;
        if (sp.mode != kGather) key = max(key, g->ref_stats.max_key);
        if (sp.mode != kScatter) key = max(key, g->build_query_stats.max_key);
        const float hmax = key_float(key);
        float ext[3], nc[3], h[3];
        bool any = false;
        for (int d = 0; d < sp.dim; ++d) {
            ext[d] = __fsub_rn(sp.dmax[d], sp.dmin[d]);
            nc[d] = floorf(__fdiv_rn(ext[d], hmax));
            h[d] = __fdiv_rn(ext[d], nc[d]);
        }
        for (int d = 0; d < sp.dim; ++d) any |= __fsub_rn(__fdiv_rn(ext[d], h[d]), nc[d]) > 0.0f;
        if (any)
            for (int d = 0; d < sp.dim; ++d) {
                nc[d] = __fsub_rn(nc[d], 1.0f);
                h[d] = __fdiv_rn(ext[d], nc[d]);
            }
        any = false;
        for (int d = 0; d < sp.dim; ++d) {
            const float r = __fdiv_rn(ext[d], h[d]);
            any |= ceilf(r) > r;
        }
        if (any)
            for (int d = 0; d < sp.dim; ++d) h[d] = __fmul_rn(h[d], grow);
        float hc = h[0];
        for (int d = 1; d < sp.dim; ++d) {
            const float v = h[d];
            if (hc != hc) break;
            if (v != v || v > hc) hc = v;  // torch.max propagates NaN
        }
        g->hmax = hmax;
        g->hcell = hc;
        if (sp.hcell_override[0] > 0.0f) {  // caller-chosen grid (multi-level search)
            hc = sp.hcell_override[0];
            for (int d = 0; d < 3; ++d) {
                g->hcell_d[d] = d < sp.dim ? sp.hcell_override[d] : 1.0f;
                hc = fminf(hc, g->hcell_d[d]);
            }
            for (int d = 0; d < 3; ++d) {
                if (d >= sp.dim) { g->count[d] = 1; continue; }
                const float r = __fdiv_rn(ext[d], g->hcell_d[d]);
                // periodic dims of a clamped grid hold a whole number of cells (ext / n each);
                // rounding must not add a sliver cell at the seam
                g->count[d] = (sp.dedupe && ((sp.periodic_mask >> d) & 1)) ? max(1, (int32_t)rintf(r))
                                                                             : (int32_t)ceilf(r);
            }
        } else {
            for (int d = 0; d < 3; ++d) {
                g->hcell_d[d] = hc;
                g->count[d] = d < sp.dim ? (int32_t)ceilf(__fdiv_rn(ext[d], hc)) : 1;
            }
        }
        g->always_exact = ((sp.mode != kGather && g->ref_stats.bad) || (sp.mode != kScatter && g->build_query_stats.bad))
                              ? 1 : 0;
        int err = 0;
        if (!(hc > 0.0f) || !isfinite(hc)) err = 1;  // no valid grid (support larger than the domain, NaN, ...)
        if (sp.dedupe) {  // clamped grid: linear indices must not wrap
            double cells = 1.0;
            for (int d = 0; d < sp.dim; ++d) cells *= (double)max(g->count[d], 1);
            if (cells >= 2147483647.0) err = 1;
        }
        for (int d = 0; d < sp.dim; ++d)
            if (((sp.periodic_mask >> d) & 1) && g->count[d] <= 0) err = 1;
        g->error = err;
        if (err && sp.n_query > 0 && sp.n_ref > 0) atomicAdd(bad_grids, 1);
    }
}
__global__ void grid_params_kernel(const CloudParams* __restrict__ table, GridParams* grid, int C, int32_t* bad_grids,
                                   int same_sup) {
    grid_params(table, grid, C, bad_grids, same_sup, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// Per-cloud maximum support (computeGridSupport, cellTable.py:40-81, needs it) and whether every
// support lies in [1e-18, 1e18] (else the exact test decides every pair).  Each block reduces a
// contiguous range, so a thread changes cloud only at cloud boundaries; a block that stayed in one
// cloud issues one atomic per field.  The record of cloud c is at out + c * stride.  With `done` (a
// build's last statistics) the last block to finish writes the clouds' grid parameters.
__global__ void support_stats_kernel(const CloudParams* __restrict__ table, const int32_t* __restrict__ prefix, int C,
                                     int64_t n, int query_side, char* out, int64_t stride, GridParams* grid = nullptr,
                                     int32_t* bad_grids = nullptr, int same_sup = 0, int32_t* done = nullptr) {
    const int64_t per = (n + gridDim.x - 1) / gridDim.x;
    const int64_t lo = (int64_t)blockIdx.x * per;
    const int64_t hi = min(n, lo + per);
    int cur = -1;
    int64_t cbase = 0, cend = 0;
    const float* h = nullptr;
    uint32_t kmax = 0;
    int bad = 0;
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        if (cur < 0 || i >= cend) {
            if (cur >= 0) stats_atomic(stats_at(out, stride, cur), kmax, bad);
            cur = cloud_of(prefix, C, i);
            cbase = prefix[cur];
            cend = prefix[cur + 1];
            h = query_side ? table[cur].query_sup : table[cur].ref_sup;
            kmax = 0;
            bad = 0;
        }
        if (h) support_stat(h[i - cbase], kmax, bad);
    }
    block_stats(cur, kmax, bad, out, stride);
    if (done && last_block(done)) grid_params(table, grid, C, bad_grids, same_sup, threadIdx.x, blockDim.x);
}

// Start of a build: the (last clouds of the) table, per-cloud statistics and flags, counters, the sort
// state, an empty map.
template <typename K>
__global__ void grid_init_kernel(const __grid_constant__ CloudChunk<kUploadChunk> ch, GridParams* g, int C, Structure S,
                                 Scratch W) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
        g[c].ref_stats.max_key = 0;
        g[c].ref_stats.bad = 0;
        g[c].build_query_stats.max_key = 0;
        g[c].build_query_stats.bad = 0;
        g[c].error = 0;
        g[c].out_of_grid = 0;
    }
    ulonglong2* map = reinterpret_cast<ulonglong2*>(S.map);  // capacities are powers of two >= 64
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < S.map_total / 2;
         i += (int64_t)gridDim.x * blockDim.x)
        map[i] = make_ulonglong2(~0ull, ~0ull);
    if (blockIdx.x != 0) return;
    upload_chunk(ch, W.table, W.query_prefix, W.ref_prefix);
    if (threadIdx.x == 0) {
        *S.bad_grids = 0;
        S.num_cells[0] = S.num_cells[1] = S.num_cells[2] = 0;
        sort_state_reset(reinterpret_cast<SortStateT<K>*>(W.sort_state));
    }
}

template <typename K>
__global__ void sort_state_init_kernel(SortStateT<K>* st) { sort_state_reset(st); }

// End of the last cell (or query group): cell_start[C] = n.
__global__ void finish_cells_kernel(int32_t* cell_start, const int32_t* num_cells, int64_t n) {
    cell_start[*num_cells] = (int32_t)n;
}

// A cloud's largest query support, as the lean test's band takes it, and whether every pair takes the exact
// test; derived from the statistics by whoever reads them.
__device__ __forceinline__ bool query_limits(const CloudParams& cp, const GridParams& g, const QueryParams& q,
                                             float& qmax) {
    // (every field is read first: as short-circuits the reads waited for each other)
    const int mode = cp.mode, qbad = q.stats.bad, rbad = g.ref_stats.bad;
    const uint32_t key = q.stats.max_key;
    const bool has_q = (cp.query_sup != nullptr) & (mode != kScatter);
    qmax = has_q ? key_float(key) : 0.0f;
    return (has_q & (qbad != 0)) | ((mode != kGather) & (rbad != 0)) | !(fabsf(qmax) <= 1e18f);
}

// Start of a count: the (last clouds of the) table; zeroes the per-search counters, the per-cloud query
// statistics and the per-query counts.  same_sorted: the queries are the structure's sorted points, whose
// statistics are there.
__global__ void count_init_kernel(const __grid_constant__ CloudChunk<kUploadChunk> ch, const GridParams* grid, Scratch W,
                                  int C, int unit_cap, int64_t nq, int64_t stage_cap, int same_sorted) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += (int64_t)gridDim.x * blockDim.x)
        W.counts[i] = 0;
    if (blockIdx.x != 0) return;
    upload_chunk(ch, W.table, W.query_prefix, W.ref_prefix);
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        const SupportStats none = {0u, 0};
        W.qparams[c].stats = same_sorted ? grid[c].ref_stats : none;
        W.qparams[c].coord_key = 0;
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < kWorkCounters; ++k) W.work[k] = 0;
        W.num_qgroups[0] = W.num_qgroups[1] = 0;
        *W.num_stray = 0;
        *W.num_units = 0;
        *W.num_flagged = 0;
        *W.exact_clouds = 0;
        W.num_exact[0] = W.num_exact[1] = W.num_exact[2] = 0;
        *W.unit_cap = unit_cap;
        W.cursor[0] = 0ull;
        W.cursor[1] = (unsigned long long)stage_cap;
    }
}

__device__ __forceinline__ float4 load_point(const float* x, const float* h, int64_t i, int dim) {
    float4 v = make_float4(0.f, 0.f, 0.f, h ? h[i] : 0.0f);
    const float* p = x + i * dim;
    v.x = p[0];
    if (dim > 1) v.y = p[1];
    if (dim > 2) v.z = p[2];
    return v;
}

__device__ __forceinline__ float4 wrap_point(int dim, int mask, const float* dmin, const float* ext, float4 v,
                                             int times) {
    for (int d = 0; d < dim; ++d)
        if ((mask >> d) & 1) {
            float c = comp(v, d);
            for (int t = 0; t < times; ++t) c = wrap_coord(c, dmin[d], ext[d]);
            if (d == 0) v.x = c; else if (d == 1) v.y = c; else v.z = c;
        }
    return v;
}

// Integer cell of a point; a clamped grid (dedupe) puts every point in a cell of [0, count):
// no aliasing, no short seam cell.
__device__ __forceinline__ void cell_of(int dim, int dedupe, const float* dmin, const float* hcell,
                                        const int32_t* count, const float4& v, int32_t* c) {
    c[0] = cell_coord(v.x, dmin[0], hcell[0]);
    c[1] = dim > 1 ? cell_coord(v.y, dmin[1], hcell[1]) : 0;
    c[2] = dim > 2 ? cell_coord(v.z, dmin[2], hcell[2]) : 0;
    if (dedupe)
        for (int d = 0; d < dim; ++d) c[d] = min(max(c[d], 0), count[d] - 1);
}

// (cloud, signed-order linear index) sort keys; one cloud needs no cloud bits.
__device__ __forceinline__ void make_key(uint32_t& k, int, uint32_t lin_key) { k = lin_key; }
__device__ __forceinline__ void make_key(unsigned long long& k, int cloud, uint32_t lin_key) {
    k = ((unsigned long long)(uint32_t)cloud << 32) | lin_key;
}
__device__ __forceinline__ int key_cloud(uint32_t) { return 0; }
__device__ __forceinline__ int key_cloud(unsigned long long k) { return (int)(k >> 32); }
__device__ __forceinline__ uint32_t key_low(uint32_t k) { return k; }
__device__ __forceinline__ uint32_t key_low(unsigned long long k) { return (uint32_t)k; }
template <typename K>
__device__ __forceinline__ K kmin2(K a, K b) { return a < b ? a : b; }
template <typename K>
__device__ __forceinline__ K kmax2(K a, K b) { return a < b ? b : a; }

// What a point-parallel kernel needs of the point's cloud, reloaded when a thread crosses into
// another cloud.
struct PointCtx {
    int32_t cloud, dim, periodic_mask, dedupe, error;
    int64_t base, end;
    float dmin[3], ext[3], hcell[3];
    int32_t count[3];
    const float* pos;
    const float* sup;
};
__device__ __forceinline__ void load_point_ctx(PointCtx& p, const CloudParams* __restrict__ table,
                                               const GridParams* grid, const int32_t* __restrict__ prefix, int c,
                                               bool query_side) {
    const CloudParams& cp = table[c];
    const GridParams& g = grid[c];
    p.cloud = c;
    p.dim = cp.dim;
    p.periodic_mask = cp.periodic_mask;
    p.dedupe = cp.dedupe;
    p.error = g.error;
    p.base = prefix[c];
    p.end = prefix[c + 1];
    for (int d = 0; d < 3; ++d) {
        p.dmin[d] = cp.dmin[d];
        p.ext[d] = cp.ext[d];
        p.hcell[d] = g.hcell_d[d];
        p.count[d] = g.count[d];
    }
    p.pos = query_side ? cp.query_pos : cp.ref_pos;
    p.sup = query_side ? cp.query_sup : cp.ref_sup;
}

// Wrap (twice for the reference cloud, cppSearch.py:221 after neighborhood.py:203; once for a
// query cloud), pack to float4 and emit the (cloud, linear cell) key.  A cloud without a valid
// grid gets one constant key (its points form one cell that no walk visits).
// hint (incremental build): the point's previous linear cell; stay[i] = it is still there.
template <typename K>
__global__ void pack_points_kernel(const CloudParams* __restrict__ table, GridParams* grid,
                                   const int32_t* __restrict__ prefix, int C, int64_t n, int query_side, int wraps,
                                   int track_grid, float4* __restrict__ pack, K* __restrict__ keys,
                                   int32_t* __restrict__ vals, SortStateT<K>* st,
                                   const int32_t* __restrict__ hint = nullptr, int32_t* __restrict__ stay = nullptr) {
    K kmin = ~(K)0, kmax = 0;
    const int64_t per = (n + gridDim.x - 1) / gridDim.x;
    const int64_t lo = (int64_t)blockIdx.x * per;
    const int64_t hi = min(n, lo + per);
    PointCtx p;
    p.cloud = -1;
    p.end = 0;
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        if (p.cloud < 0 || i >= p.end) load_point_ctx(p, table, grid, prefix, cloud_of(prefix, C, i), query_side != 0);
        float4 v = load_point(p.pos, p.sup, i - p.base, p.dim);
        uint32_t lin = 0;
        if (!p.error) {
            v = wrap_point(p.dim, p.periodic_mask, p.dmin, p.ext, v, wraps);
            int32_t c[3];
            cell_of(p.dim, p.dedupe, p.dmin, p.hcell, p.count, v, c);
            if (track_grid) {
                bool out = false;
                for (int d = 0; d < p.dim; ++d) out |= c[d] < 0 || c[d] >= p.count[d];
                if (out && !*(volatile int32_t*)&grid[p.cloud].out_of_grid) atomicOr(&grid[p.cloud].out_of_grid, 1);
            }
            lin = (uint32_t)linear_index(p.dim, c, p.count);
        }
        K key;
        make_key(key, p.cloud, lin ^ 0x80000000u);
        if (stay) stay[i] = (!p.error && hint[i] == (int32_t)lin) ? 1 : 0;
        pack[i] = v;
        keys[i] = key;
        vals[i] = (int32_t)i;
        kmin = kmin2(kmin, key);
        kmax = kmax2(kmax, key);
    }
    __shared__ K s_min[32], s_max[32];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        kmin = kmin2(kmin, (K)__shfl_xor_sync(0xffffffffu, kmin, o));
        kmax = kmax2(kmax, (K)__shfl_xor_sync(0xffffffffu, kmax, o));
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) { s_min[w] = kmin; s_max[w] = kmax; }
    __syncthreads();
    if (w == 0) {
        kmin = lane < nw ? s_min[lane] : ~(K)0;
        kmax = lane < nw ? s_max[lane] : (K)0;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            kmin = kmin2(kmin, (K)__shfl_xor_sync(0xffffffffu, kmin, o));
            kmax = kmax2(kmax, (K)__shfl_xor_sync(0xffffffffu, kmax, o));
        }
        if (lane == 0) {
            atomicMin(&st->key_min, kmin);
            atomicMax(&st->key_max, kmax);
        }
    }
}

__device__ __forceinline__ uint32_t mix32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x85ebca6bu;
    x ^= x >> 13;
    x *= 0xc2b2ae35u;
    x ^= x >> 16;
    return x;
}

// A cloud whose points all lie in a grid of no more cells than its map region has slots keeps them in place:
// slot = linear index (returned: the cells; 0: the region is an open-addressing table).  A unit's 27
// look-ups then read neighbouring slots, one read each, instead of 27 scattered probe chains.
__device__ __forceinline__ uint32_t direct_cells(int dim, const int32_t* count, int out_of_grid, int64_t cap) {
    double cells = 1.0;
    for (int d = 0; d < dim; ++d) cells *= (double)max(count[d], 1);
    return (!out_of_grid && cells <= (double)cap && cells < 2147483648.0) ? (uint32_t)cells : 0u;
}

__device__ __forceinline__ void map_insert(unsigned long long* map, int64_t cap, int32_t lin, int32_t cell) {
    const unsigned long long entry = ((unsigned long long)(uint32_t)lin << 32) | (uint32_t)cell;
    uint64_t slot = mix32((uint32_t)lin) & (cap - 1);
    for (int64_t probe = 0; probe < cap; ++probe) {
        unsigned long long prev = atomicCAS(&map[slot], ~0ull, entry);
        if (prev == ~0ull || (uint32_t)(prev >> 32) == (uint32_t)lin) return;
        slot = (slot + 1) & (cap - 1);
    }
}

__device__ __forceinline__ int32_t map_find(const unsigned long long* __restrict__ map, int64_t cap, uint32_t direct,
                                            int32_t lin) {
    if (direct) {  // (an empty slot holds -1; a linear index outside the grid names no cell)
        if ((uint32_t)lin >= direct) return -1;
        return (int32_t)__ldg(reinterpret_cast<const uint2*>(map) + (uint32_t)lin).x;
    }
    const uint32_t mask = (uint32_t)(cap - 1);  // capacities are at most 2^32
    uint32_t slot = mix32((uint32_t)lin) & mask;
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const uint2 e = __ldg(reinterpret_cast<const uint2*>(map) + slot);  // (cell, lin)
        if (e.y == (uint32_t)lin && (int32_t)e.x >= 0) return (int32_t)e.x;
        if (e.x == 0xffffffffu && e.y == 0xffffffffu) return -1;
        if (probe == 0xffffffffu) return -1;
        slot = (slot + 1) & mask;
    }
    return -1;
}

// What the build does with its sorted points: places each one (the point, its input index and, for the
// serving loop, its linear cell and input index), and writes one cell record per run of equal keys
// (unique_consecutive, hashTable.py:193): begin, lin, cloud, coords of the run's first point, bucket, and
// the cell's entry in its cloud's map region.
template <typename K>
struct BuildTail {
    static constexpr bool kPlace = true, kRuns = true;
    int32_t* starts;   // cell_start
    int32_t* num_runs;
    const float4* __restrict__ pack;
    float4* sorted;
    int32_t* sidx;
    int32_t* lin_out;
    int32_t* order_out;
    const CloudParams* table;
    const GridParams* grid;
    int32_t* cell_lin;
    int32_t* cell_coords;
    int32_t* cell_bucket;
    int32_t* cell_cloud;
    unsigned long long* map;
    int64_t n;
    __device__ __forceinline__ void place(int64_t i, K key, int32_t p) const {
        if (!TCR_GUARD(p, n)) return;
        sorted[i] = pack[p];
        sidx[i] = p;
        if (lin_out) lin_out[i] = (int32_t)(key_low(key) ^ 0x80000000u);
        if (order_out) order_out[i] = p;
    }
    __device__ __forceinline__ void run(const K* keys, int64_t i, int32_t cell) const {
        const K key = keys[i];
        const int cloud = key_cloud(key);
        const int32_t lin = (int32_t)(key_low(key) ^ 0x80000000u);
        const CloudParams& cp = table[cloud];
        const GridParams& g = grid[cloud];
        int32_t c[3] = {0, 0, 0};
        uint32_t bucket = 0;
        if (!g.error) {
            cell_of(cp.dim, cp.dedupe, cp.dmin, g.hcell_d, g.count, sorted[i], c);
            bucket = ref_hash(cp.dim, c, cp.hash_len);
            const uint32_t direct = direct_cells(cp.dim, g.count, g.out_of_grid, cp.map_cap);
            if (!direct)
                map_insert(map + cp.map_base, cp.map_cap, lin, cell);
            else if ((uint32_t)lin < direct)
                map[cp.map_base + lin] = ((unsigned long long)(uint32_t)lin << 32) | (uint32_t)cell;
        }
        cell_lin[cell] = lin;
        cell_cloud[cell] = cloud;
        cell_coords[3 * cell + 0] = c[0];
        cell_coords[3 * cell + 1] = c[1];
        cell_coords[3 * cell + 2] = c[2];
        cell_bucket[cell] = (int32_t)bucket;
    }
};

// The order and cells a caller of the incremental build receives when the sort gave up: the order it came
// in, and its hint.
__global__ void abandoned_order_kernel(const int32_t* __restrict__ failed, int64_t n, const int32_t* __restrict__ hint,
                                       int32_t* lin_out, int32_t* order_out) {
    if (!*failed) return;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (lin_out) lin_out[i] = hint ? hint[i] : 0;
        if (order_out) order_out[i] = (int32_t)i;
    }
}

// What BuildTail does, for queries sorted by their own cells: one query group per run.
template <typename K>
struct QueryTail {
    static constexpr bool kPlace = true, kRuns = true;
    int32_t* starts;   // qgroup_start
    int32_t* num_runs;
    const float4* __restrict__ pack;
    float4* sorted;
    int32_t* sidx;
    const CloudParams* table;
    const GridParams* grid;
    int32_t* group_coords;
    int32_t* group_cloud;
    int64_t n;
    __device__ __forceinline__ void place(int64_t i, K, int32_t p) const {
        if (!TCR_GUARD(p, n)) return;
        sorted[i] = pack[p];
        sidx[i] = p;
    }
    __device__ __forceinline__ void run(const K* keys, int64_t i, int32_t group) const {
        const int cloud = key_cloud(keys[i]);
        const CloudParams& cp = table[cloud];
        const GridParams& g = grid[cloud];
        int32_t c[3] = {0, 0, 0};
        if (!g.error) cell_of(cp.dim, cp.dedupe, cp.dmin, g.hcell_d, g.count, sorted[i], c);
        group_cloud[group] = cloud;
        group_coords[3 * group + 0] = c[0];
        group_coords[3 * group + 1] = c[1];
        group_coords[3 * group + 2] = c[2];
    }
};

// ------------------------------------------------------------------------------------------
// incremental re-sort
//
// A build may be given the reference points in the cell order of a previous build, with each
// point's previous linear cell (the hint).  The points still in their cell ("unmoved") then form
// a subsequence already sorted by (key, input index); only the moved points are radix-sorted, and
// the two sorted lists are merged by (key, input index) -- exactly the stable sort of the input.
// The unmoved subsequence is verified on the device; if it is not sorted (a wrong hint), or too
// many points moved, the full radix sort runs instead.  Every kernel reads the decision from the
// device, so the build enqueues without a host round trip.

struct StayIn {
    const int32_t* stay;
    __device__ int32_t operator()(int64_t i) const { return stay[i]; }
};
template <typename K>
struct StayOut {
    const K* keys;        // the pack output, input order
    K* stay_keys;
    int32_t* stay_idx;
    K* moved_keys;
    int32_t* moved_vals;
    __device__ void operator()(int64_t i, int32_t ex, int32_t flag) const {
        if (flag) {
            stay_keys[ex] = keys[i];
            stay_idx[ex] = (int32_t)i;
        } else {
            moved_keys[i - ex] = keys[i];
            moved_vals[i - ex] = (int32_t)i;
        }
    }
};

template <typename K>
__global__ void inc_check_kernel(const K* __restrict__ stay_keys, const int32_t* n_stay, int32_t* bad) {
    const int64_t n = *n_stay;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    bool ok = true;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k + 1 < n; k += stride)
        ok &= stay_keys[k] <= stay_keys[k + 1];
    if (!__all_sync(0xffffffffu, ok) && (threadIdx.x & 31) == 0) atomicOr(bad, 1);
}

// Chooses the path: the moved points' sort and the merge, or the full sort (one thread).
template <typename K>
__global__ void inc_decide_kernel(SortStateT<K>* full, SortStateT<K>* moved, const int32_t* counts, int64_t n) {
    const int64_t n_stay = counts[0];
    const bool fallback = counts[1] != 0 || 2 * n_stay < n;  // wrong hint, or most points moved
    sort_state_reset(moved);
    if (fallback) {
        moved->key_min = moved->key_max = 0;  // no moved sort
        return;
    }
    moved->key_min = full->key_min;  // a superset of the moved keys' range
    moved->key_max = full->key_max;
    moved->n_dev = n - n_stay;
    full->key_min = full->key_max = 0;  // no full sort: the merge writes the sorted keys in place
}

// Number of list entries ordered before (key, idx); the list is sorted by (key, idx).
template <typename K>
__device__ __forceinline__ int64_t count_before(const K* keys, const int32_t* idx, int64_t n, K key, int32_t i) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        const K km = keys[mid];
        if (km < key || (km == key && idx[mid] < i)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Merges the unmoved and the sorted moved points into keys/vals (input buffer 0 of the full sort,
// whose passes are all skipped on this path).
template <typename K>
__global__ void inc_merge_kernel(const K* __restrict__ stay_keys, const int32_t* __restrict__ stay_idx,
                                 const K* moved_k0, const K* moved_k1, const int32_t* moved_v0,
                                 const int32_t* moved_v1, const SortStateT<K>* moved, const int32_t* counts,
                                 int64_t n, K* __restrict__ keys, int32_t* __restrict__ vals) {
    if (counts[1] != 0 || 2 * (int64_t)counts[0] < n) return;  // the full sort runs instead
    const int64_t n_stay = counts[0], n_moved = n - n_stay;
    const int s = moved->sel[key_passes<K>()];
    const K* mk = s ? moved_k1 : moved_k0;
    const int32_t* mv = s ? moved_v1 : moved_v0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += stride) {
        K key;
        int32_t i;
        int64_t pos;
        if (t < n_stay) {
            key = stay_keys[t];
            i = stay_idx[t];
            pos = t + count_before(mk, mv, n_moved, key, i);
        } else {
            key = mk[t - n_stay];
            i = mv[t - n_stay];
            pos = (t - n_stay) + count_before(stay_keys, stay_idx, n_stay, key, i);
        }
        keys[pos] = key;
        vals[pos] = i;
    }
}

// ------------------------------------------------------------------------------------------
// query side

// Self search: query i is reference i, so the reference order and cells group the queries.
// Positions are the once-wrapped query coordinates (only periodic dims differ from rsorted), supports the
// caller's of this call: a kept structure may be searched with others than it was built from.  Their
// statistics are reduced on the way, as support_stats_kernel does.
__global__ void pack_self_queries_kernel(const CloudParams* __restrict__ table, const GridParams* grid,
                                         const int32_t* __restrict__ prefix, int C, const int32_t* __restrict__ rsidx,
                                         int64_t n, float4* __restrict__ qsorted, int32_t* __restrict__ qsidx,
                                         QueryParams* qp) {
    const int64_t per = (n + gridDim.x - 1) / gridDim.x;
    const int64_t lo = (int64_t)blockIdx.x * per;
    const int64_t hi = min(n, lo + per);
    char* const out = reinterpret_cast<char*>(&qp->stats);
    constexpr int64_t stride = (int64_t)sizeof(QueryParams);
    PointCtx p;
    p.cloud = -1;
    p.base = p.end = 0;
    uint32_t kmax = 0;
    int bad = 0;
    for (int64_t t = lo + threadIdx.x; t < hi; t += blockDim.x) {
        const int32_t i = rsidx[t];
        if (!TCR_GUARD(i, n)) continue;  // (the build's sort gave up)
        if (p.cloud < 0 || i < p.base || i >= p.end) {
            if (p.cloud >= 0) stats_atomic(stats_at(out, stride, p.cloud), kmax, bad);
            load_point_ctx(p, table, grid, prefix, cloud_of(prefix, C, i), true);
            kmax = 0;
            bad = 0;
        }
        const float4 v = load_point(p.pos, p.sup, i - p.base, p.dim);
        if (p.sup) support_stat(v.w, kmax, bad);
        qsorted[t] = wrap_point(p.dim, p.periodic_mask, p.dmin, p.ext, v, 1);
        qsidx[t] = i;
    }
    // A warp that stayed in one cloud reduces first.  No barriers, and an atomic only where it raises the maximum:
    // reduced by blocks, 1M periodic points took 29 us instead of 25.
    const int c0 = __shfl_sync(0xffffffffu, p.cloud, 0);
    const bool one = __all_sync(0xffffffffu, p.cloud < 0 || p.cloud == c0);
    if (one) {
        kmax = __reduce_max_sync(0xffffffffu, kmax);
        bad = __reduce_or_sync(0xffffffffu, bad);
    }
    if (p.cloud >= 0 && (!one || (threadIdx.x & 31) == 0)) {
        SupportStats* st = stats_at(out, stride, p.cloud);
        if (kmax > *(volatile uint32_t*)&st->max_key) atomicMax(&st->max_key, kmax);
        if (bad && *(volatile int32_t*)&st->bad == 0) atomicOr(&st->bad, 1);
    }
}

// Group count comes from a device scalar; the scan kernels are launched over the upper bound
// and read the true count through the functor.  A unit holds at most `cap` (<= 32) queries.
// After a sort that gave up there are no groups and so no units: nothing is walked, counted or emitted.
struct BoundedUnitCountIn {
    const int32_t* group_start;
    const int32_t* num_groups;
    int32_t cap;
    const int32_t* build_failed;
    const int32_t* sort_failed;
    __device__ int32_t operator()(int64_t g) const {
        // (read-only loads, so that a thread's elements share them and none waits for another)
        const int32_t groups = __ldg(num_groups), failed = __ldg(build_failed) | __ldg(sort_failed);
        if (failed != 0 || g >= groups) return 0;
        const int32_t n = __ldg(&group_start[g + 1]) - __ldg(&group_start[g]);
        return (n + cap - 1) / cap;
    }
};
struct BoundedUnitOut {
    const int32_t* group_start;
    int32_t* unit_group;
    int32_t* unit_t0;
    int32_t cap;
    int64_t bound;  // entries of unit_group / unit_t0
    __device__ void operator()(int64_t g, int32_t ex, int32_t nunits) const {
        if (nunits <= 0) return;
        const int32_t s = group_start[g];
        for (int32_t u = 0; u < nunits; ++u) {
            if (!TCR_GUARD(ex + u, bound)) break;
            unit_group[ex + u] = (int32_t)g;
            unit_t0[ex + u] = s + u * cap;
        }
    }
};

// ------------------------------------------------------------------------------------------
// the candidate walk
//
// Work unit: <= 32 queries of one query group (cell).  One warp takes a unit, looks up its
// cloud (one copy of the cloud's parameters in shared memory, refreshed when the warp moves to
// another cloud), finds the unit's 3^d stencil cells and walks their candidates in chunks of 32.
// The count walk tests every (query, candidate) pair once and writes the unit's record -- its
// candidate runs and the 32-bit hit mask of every (query, chunk) -- to a staging list; the emit
// pass expands the records into CSR/COO slots.  A unit that finds the staging list full is only
// counted and is walked again by the emit walk, which writes its pairs directly.

// Float64 inputs (tcr_count_f64 / tcr_emit_f64): the walks find and test candidates on the float32
// copies and decide every pair inside the widened rounding band on these double arrays with the
// reference's double expression.  qpos == null: a float32 search.
struct F64Walk {
    const double* qpos;      // [nq * dim] queries, wrapped as the reference wraps them
    const double* qsup;      // [nq] or null
    const double4* rsorted;  // [nr] the references in the structure's cell order, .w = support
    double ext[3];           // max - min of the domain, in double
};

// common.h:106-129 and neighborhoodDynamic.h:59-70 at scalar_t = double: per dimension
// diff = moduloOp(x_i, x_j, max - min) = ((x_i - x_j + h/2) - floor((x_i - x_j + h/2) / h) * h) - h/2
// on periodic dimensions, x_i - x_j otherwise; sum += diff * diff; sqrt(sum) < the mode's
// threshold.  Explicit intrinsics keep every operation rounded on its own (no FMA).
__device__ __noinline__ bool f64_pair_test(int dim, int mask, int mode, const double* ext, const double* xi,
                                           double hi, const double* xj, double hj) {
    double sum = 0.0;
    for (int d = 0; d < dim; ++d) {
        double diff;
        if ((mask >> d) & 1) {
            const double h = ext[d];
            const double half = __ddiv_rn(h, 2.0);
            const double t = __dadd_rn(__dsub_rn(xi[d], xj[d]), half);
            diff = __dsub_rn(__dsub_rn(t, __dmul_rn(floor(__ddiv_rn(t, h)), h)), half);
        } else {
            diff = __dsub_rn(xi[d], xj[d]);
        }
        sum = __dadd_rn(sum, __dmul_rn(diff, diff));
    }
    const double dist = __dsqrt_rn(sum);
    double thr;
    switch (mode) {
        case kGather: thr = hi; break;
        case kScatter: thr = hj; break;
        case kSymmetric: thr = __ddiv_rn(__dadd_rn(hi, hj), 2.0); break;
        default: thr = hi < hj ? hj : hi; break;  // std::max
    }
    return dist < thr;
}

// Pair (cloud-local query qi, sorted reference j) of a float64 search decided on the double arrays.
__device__ __noinline__ bool f64_pair_decide(F64Walk f, int dim, int mask, int mode, int64_t qi, int32_t j) {
    double xi[3] = {0.0, 0.0, 0.0};
    for (int d = 0; d < dim; ++d) xi[d] = f.qpos[qi * dim + d];
    const double4 c = f.rsorted[j];
    const double xj[3] = {c.x, c.y, c.z};
    return f64_pair_test(dim, mask, mode, f.ext, xi, f.qsup ? f.qsup[qi] : 0.0, xj, c.w);
}

// The tensor-core test's constants (see split_pair): the band relative to the largest product, the
// largest scaled support it takes, the scaled distance beyond which a candidate sends its unit to
// fix_unit, the scaled place of the lanes past a unit's candidates (farther than any support), and the
// norm of a query row that must never hit.
constexpr float kMmaBand = 4e-6f;
constexpr float kMmaSupport = 4.0f;
constexpr float kMmaReach = 16.0f;
constexpr float kMmaPad = 15.0f;
constexpr float kMmaFar = 60000.0f;
// Lanes with a pair inside the band, over the chunks of a window, from which on the window is listed as a whole, if
// they are also one a pair of chunks; fewer list their pairs.  A random cloud's window has one at most nearly always,
// and 0.3 on average where 32 queries meet 16 pairs of chunks (20k points in 4^3 periodic cells: 654 us when four
// lanes there listed the window, which takes one warp 30 us); a lattice's has four even in 1D (1M points: 1.18 ms,
// 1.45 when eight were asked for).
constexpr int kBandLanes = 4;

// The unit's cloud, as the walk kernels read it (shared memory, warp-uniform).
struct UnitCtx {
    int32_t cloud, dim, periodic_mask, dedupe;
    uint32_t hash_len;
    int32_t error, exact_all;
    int32_t count[3];
    int32_t qshift, rshift;  // subtracted from global query / reference indices (cloud-local numbering)
    float dmin[3], hcell[3], ext[3];
    float rmax, qmax;        // largest reference / query support (band of the fast test)
    float f64_err;           // float64 inputs: bound on the error of a float32 coordinate difference
    int32_t shift_ok;        // the periodic dims hold enough cells: candidates across a seam are shifted
    float shift_delta;       // bound on the error a shift adds to a difference
    // the tensor-core test: power-of-two scale that puts the largest cell edge (scale_cell) in [1, 2), the
    // half width of the band its result must leave (in scaled units; mma_seam more for shifted
    // candidates), and whether every support is in its range
    float scale, scale_cell, mma_band, mma_seam;
    int32_t mma_ok;
    int32_t plain_cells;  // every point lies in the grid and linear indices do not wrap: an in-range cell's linear
                          // index names that cell only, so its bucket needs no check
    int64_t map_base, map_cap;
    uint32_t map_direct;     // direct_cells of the cloud
};

struct WalkArgs {
    const CloudParams* __restrict__ table;
    const GridParams* grid;
    const QueryParams* __restrict__ qparams;
    const int32_t* __restrict__ query_prefix;
    int32_t num_clouds;
    int32_t local_index;          // 1: rows and columns numbered within each cloud
    int32_t mode;
    int32_t no_stray_check;       // self search, no periodic dims, same positions: a query's cell is its
                                  // group's where linear indices name one cell each (UnitCtx.plain_cells)
    int32_t class_filter;         // >= 0: walk only units of clouds of this class (dim * 2 + periodic)
    int32_t self;                 // self search: sorted query t is sorted reference t, wrapped once less
    const float4* __restrict__ rsorted;
    const int32_t* __restrict__ rsidx;
    const int32_t* __restrict__ cell_start;
    const int32_t* __restrict__ cell_bucket;
    const unsigned long long* __restrict__ map;
    const float4* __restrict__ qsorted;
    const int32_t* __restrict__ qsidx;
    const int32_t* __restrict__ group_start;
    const int32_t* __restrict__ group_coords;
    const int32_t* __restrict__ group_cloud;
    const int32_t* __restrict__ unit_group;
    const int32_t* __restrict__ unit_t0;
    const int32_t* __restrict__ num_units;
    const int32_t* __restrict__ unit_cap;   // queries per unit
    const int32_t* __restrict__ unit_list;  // emit re-walk: the units to walk
    const int32_t* __restrict__ num_list;
    int32_t* work;
    int32_t* stray;
    int32_t* num_stray;
    int32_t* counts;              // [nq] count output, global query order
    int32_t* rec;                 // [units] offset of each unit's record in the staging list, negative if not staged
    int32_t* flagged;             // [units] units to re-walk in the emit pass
    int32_t* num_flagged;
    int32_t* num_exact;           // [3] pairs inside the product's band, listed; decided with their window; windows listed
    int32_t* exact_clouds;
    int4* band_pairs;             // [nq] (sorted query, sorted reference, mask word of the staging list, bit)
    unsigned long long* band_windows;  // [band_cap] unit << 32 | window << 16 | its marked pairs of chunks
    int64_t band_cap;
    unsigned long long* cursor;   // staging list fill
    int32_t* stage;               // staging list
    int64_t stage_cap;
    const int32_t* __restrict__ query_ids;  // optional: row written for global query q is query_ids[q]
    const int32_t* __restrict__ ref_ids;    // optional: column written for global reference j is ref_ids[j]
    const int64_t* offsets;       // emit input [nq+1]
    int64_t* row_out;             // emit: COO rows or null
    int64_t* col_out;             // emit: columns
    int64_t out_cap;              // emit: entries of row_out/col_out; writes beyond are dropped
    F64Walk f64;                  // float64 inputs, or qpos == null
    int64_t nq_total, nr_total;   // point counts (bounds of the checked build)
};

__device__ __forceinline__ void load_unit_ctx(UnitCtx& u, const WalkArgs& a, int cloud) {
    const CloudParams& cp = a.table[cloud];
    const GridParams& g = a.grid[cloud];
    const QueryParams& q = a.qparams[cloud];
    u.cloud = cloud;
    u.dim = cp.dim;
    u.periodic_mask = cp.periodic_mask;
    u.dedupe = cp.dedupe;
    u.hash_len = cp.hash_len;
    u.error = g.error;
    u.exact_all = query_limits(cp, g, q, u.qmax);
    for (int d = 0; d < 3; ++d) {
        u.count[d] = g.count[d];
        u.dmin[d] = cp.dmin[d];
        u.hcell[d] = g.hcell_d[d];
        u.ext[d] = cp.ext[d];
    }
    u.qshift = a.local_index ? cp.query_base : 0;
    u.rshift = a.local_index ? cp.ref_base : 0;
    u.rmax = key_float(g.ref_stats.max_key);
    // a float32 copy of a double coordinate x is off by <= |x| 2^-24, the float difference adds one
    // rounding: 2^-21 of the largest |coordinate| bounds a difference's error with room to spare
    u.f64_err = a.f64.qpos ? key_float(q.coord_key) * 4.76837158203125e-7f : 0.0f;
    // Candidates of a stencil cell across the periodic seam can be moved by +-ext, so that the fast test
    // needs no wrap, where the reference's moduloOp wraps exactly the moved cells.  Two points of a
    // stencil are less than 2 cells apart.  With five cells or more on a dimension that is at most half the
    // extent (the last cell may be a sliver: ext > 4 cells), so only moved candidates wrap.  With four
    // cells (3 cells < ext <= 4 cells) a difference D between ext / 2 and 2 cells wraps too, to
    // ext - D >= ext - 2 cells: beyond every threshold, and so is D, when thresholds end at ext - 2 cells
    // (less what rounding a coordinate to its cell can add).  A moved candidate is at most 2 cells away
    // with five cells, ext - 2 cells with four: ext / 2 at most.  A shift
    // changes a difference by at most one rounding of the shifted coordinate plus the reference's
    // own rounding of q - c before its exact wrap: shift_delta bounds both.
    bool ok = cp.periodic_mask != 0;
    float delta = 0.0f;
    const float tmax = fmaxf(a.mode == kScatter ? 0.0f : u.qmax, a.mode == kGather ? 0.0f : u.rmax);
    for (int d = 0; d < cp.dim; ++d)
        if ((cp.periodic_mask >> d) & 1) {
            // two roundings of magnitude <= half an ulp of (|coordinate| + ext) each: <= 2^-23 of it
            const float one = (fmaxf(fabsf(cp.dmin[d]), fabsf(cp.dmax[d])) + cp.ext[d]) * 1.1920928955078125e-7f;
            const float room = fmaf(-2.0f, g.hcell_d[d], cp.ext[d]) - fmaf(4.0f, one, 2.0f * u.f64_err);
            ok = ok && (g.count[d] >= 5 || (g.count[d] == 4 && tmax <= room));
            delta = fmaxf(delta, one);
        }
    u.shift_ok = ok && isfinite(delta);
    u.shift_delta = delta;
    u.map_base = cp.map_base;
    u.map_cap = cp.map_cap;
    u.plain_cells = direct_cells(cp.dim, g.count, g.out_of_grid, int64_t(1) << 31) != 0;
    u.map_direct = direct_cells(cp.dim, g.count, g.out_of_grid, cp.map_cap);
    float cell = 0.0f;
    for (int d = 0; d < cp.dim; ++d) cell = fmaxf(cell, g.hcell_d[d]);
    const uint32_t ex = min(max((__float_as_uint(cell) >> 23) & 0xffu, 1u), 253u);
    u.scale = __uint_as_float((254u - ex) << 23);
    u.scale_cell = cell * u.scale;
    // |Q| is at most sqrt(3) * 0.55 cells, a candidate near the threshold at most that plus thr away
    const float hq = a.mode == kScatter ? 0.0f : u.qmax * u.scale, hc = a.mode == kGather ? 0.0f : u.rmax * u.scale;
    const float t = a.mode == kSymmetric ? 0.5f * (hq + hc) : fmaxf(hq, hc);
    const float e = fmaf(0.96f, u.scale_cell, t), fe = u.f64_err * u.scale, dl = u.shift_delta * u.scale;
    u.mma_band = kMmaBand * e * e + kBandEps * t * t + fmaf(2.0f * 1.7320508f * t, fe, 3.0f * fe * fe);
    u.mma_seam = fmaf(2.0f * t, dl, dl * dl);
    u.mma_ok = !u.exact_all && hq <= kMmaSupport && hc <= kMmaSupport && u.scale_cell >= 1.0f && u.scale_cell <= 2.0f;
}

__device__ __forceinline__ ExactCtx unit_exact_ctx(const UnitCtx& u, int mode) {
    ExactCtx c;
    c.dim = u.dim;
    c.mode = mode;
    c.periodic_mask = u.periodic_mask;
    c.ext[0] = u.ext[0];
    c.ext[1] = u.ext[1];
    c.ext[2] = u.ext[2];
    return c;
}

// Looks up stencil cell `o` (getOffsets order, last coordinate fastest) around cell gc with the
// reference's semantics; returns the sorted range or an empty one, inside the sorted points.
template <int DIM>
__device__ __forceinline__ void stencil_lookup(const WalkArgs& a, const UnitCtx& u, const int32_t* gc, int o,
                                               int32_t& beg, int32_t& cnt) {
    int32_t c[3] = {0, 0, 0};
    int rem = o;
    bool dup = false, inside = true;
#pragma unroll
    for (int d = DIM - 1; d >= 0; --d) {
        const int32_t off = rem % 3 - 1;
        rem /= 3;
        int32_t v = gc[d] + off;
        const int32_t n = u.count[d];
        if ((u.periodic_mask >> d) & 1) {
            // a neighbour of a cell inside the grid wraps by one extent at most
            const int32_t v1 = v < 0 ? v + n : (v >= n ? v - n : v);
            v = (uint32_t)v1 < (uint32_t)n ? v1 : pymod(v, n);
            // with fewer than 3 cells the wrapped offsets repeat a cell; the clamped grid visits it once
            if (u.dedupe && ((n == 1 && off != 0) || (n == 2 && off == 1))) dup = true;
        } else if (u.dedupe && (v < 0 || v >= n)) {
            dup = true;  // clamped grid: nothing lies outside it
        }
        inside &= (uint32_t)v < (uint32_t)n;
        c[d] = v;
    }
    beg = 0;
    cnt = 0;
    if (dup) return;
    const int32_t lin = linear_index(DIM, c, u.count);
    const int32_t cell = map_find(a.map + u.map_base, u.map_cap, u.map_direct, lin);
    if (cell < 0 || !TCR_GUARD(cell, a.nr_total)) return;
    const int32_t b = __ldg(&a.cell_start[cell]), e = __ldg(&a.cell_start[cell + 1]);
    // queryHashMap matches the linear index inside bucket hash(c) only.
    if (!(inside && u.plain_cells) && (uint32_t)__ldg(&a.cell_bucket[cell]) != ref_hash(DIM, c, u.hash_len)) return;
    if (b < 0 || e < b || e > a.nr_total) return;
    beg = b;
    cnt = e - b;
}
__device__ __forceinline__ void stencil_lookup_any(const WalkArgs& a, const UnitCtx& u, const int32_t* gc, int o,
                                                   int32_t& beg, int32_t& cnt) {
    if (u.dim == 1) stencil_lookup<1>(a, u, gc, o, beg, cnt);
    else if (u.dim == 2) stencil_lookup<2>(a, u, gc, o, beg, cnt);
    else stencil_lookup<3>(a, u, gc, o, beg, cnt);
}

template <int DIM>
__device__ __forceinline__ bool same_cell(const int32_t* a, const int32_t* b) {
    bool s = a[0] == b[0];
    if (DIM > 1) s &= a[1] == b[1];
    if (DIM > 2) s &= a[2] == b[2];
    return s;
}

// Per-candidate pieces of the lean test: the candidate's share of the threshold and the half
// width of the band (conservative over every query: qmax is the largest query support).
template <int MODE>
__device__ __forceinline__ float cand_share(float hc) {
    return MODE == kSymmetric ? 0.5f * hc : hc;
}
template <int MODE>
__device__ __forceinline__ float cand_band(float cw, float qmax) {
    float t;
    if (MODE == kGather) t = qmax;
    else if (MODE == kScatter) t = cw;
    else if (MODE == kSymmetric) t = fmaf(qmax, 0.5f, cw);
    else t = fmaxf(qmax, cw);
    return kBandEps * t * t;
}
// thr for (query support hq, candidate share cw), float-exact as the reference evaluates it.
template <int MODE>
__device__ __forceinline__ float pair_thr(float hq, float cw) {
    if (MODE == kGather) return hq;
    if (MODE == kScatter) return cw;
    if (MODE == kSymmetric) return fmaf(hq, 0.5f, cw);  // fl(hq/2 + hc/2) == fl(hq + hc) / 2
    return fmaxf(hq, cw);
}

// Per-dimension constants of the fast periodic difference: the extent h, the half extent at which
// a difference wraps (+inf on a non-periodic dimension, which never wraps) and the band around it
// inside which the wrap decision is left to the exact test.
struct WrapCtx {
    float h[3], half[3], epsh[3];
};
__device__ __forceinline__ WrapCtx wrap_ctx(int periodic_mask, const float* ext) {
    WrapCtx w;
    for (int d = 0; d < 3; ++d) {
        const bool p = (periodic_mask >> d) & 1;
        w.h[d] = ext[d];
        w.half[d] = p ? 0.5f * ext[d] : __int_as_float(0x7f800000);
        w.epsh[d] = p ? kBandEps * ext[d] : 0.0f;
    }
    return w;
}

// Float difference q - c along dimension d, wrapped once into [-h/2, h/2] on a periodic dimension
// (the reference's moduloOp decides exactly; a difference within the band of +-h/2 sets wrap_unc).
template <bool PERIODIC>
__device__ __forceinline__ float fast_diff(const WrapCtx& wc, int d, float q, float c, bool& wrap_unc) {
    float diff = q - c;
    if (PERIODIC) {
        const float ad = fabsf(diff);
        wrap_unc |= fabsf(ad - wc.half[d]) <= wc.epsh[d];
        if (ad >= wc.half[d]) diff -= copysignf(wc.h[d], diff);
    }
    return diff;
}

// One (query, candidate) test.  in: decided; unc: needs the exact reference test.
template <int DIM, bool PERIODIC, int MODE>
__device__ __forceinline__ void lean_test(const WrapCtx& wc, const float4& q, const float4& c, float cw, float band,
                                          bool& in, bool& unc) {
    bool wrap_unc = false;
    float dd[3];
#pragma unroll
    for (int d = 0; d < DIM; ++d) dd[d] = fast_diff<PERIODIC>(wc, d, comp(q, d), comp(c, d), wrap_unc);
    float d2 = dd[0] * dd[0];
    if (DIM > 1) d2 = fmaf(dd[1], dd[1], d2);
    if (DIM > 2) d2 = fmaf(dd[2], dd[2], d2);
    const float thr = pair_thr<MODE>(q.w, cw);
    const float r = fmaf(-thr, thr, d2);  // d2 - thr^2, one rounding; sign exact
    in = r < 0.0f;
    unc = (fabsf(r) <= band) || wrap_unc;
}

constexpr int kWalkWarps = 4;
// Resident blocks per SM the count walk is compiled for (registers <= 65536 / (128 * blocks)): seven
// (72 registers) on non-periodic clouds, six (80) on periodic ones.  8/7/6 blocks measured
// 239/216/219 us on the 1M workload, 168/162/163 us for 131k queries against it, 42/39/37 us on 65k periodic
// points and 1274/1168/1098 us on the periodic 3D clouds of a batch of 256.
#ifndef TCR_WALK_MIN_BLOCKS
#define TCR_WALK_MIN_BLOCKS 7
#endif
#ifndef TCR_WALK_MIN_BLOCKS_PERIODIC
#define TCR_WALK_MIN_BLOCKS_PERIODIC 6
#endif
constexpr int kWalkMinBlocks = TCR_WALK_MIN_BLOCKS;
constexpr int kWalkMinBlocksPeriodic = TCR_WALK_MIN_BLOCKS_PERIODIC;

// Record of a staged unit in the staging list (int32 words):
//   [0] chunks of 32 candidates   [1] R, candidate runs   [2] nb, queries   [3] 0 (unused)
//   [4, 4 + R)          first sorted index of each run
//   [4 + R, 5 + 2R)     candidate prefix of each run; entry R is the unit's candidate count M
//   [5 + 2R, ...)       hit masks, chunk-major: word c * nb + q, bit j set when query q meets
//                       candidate 32 c + j
// A run is a stretch of consecutive sorted points: one non-empty stencil cell, so R is at most 27.
constexpr int kRecHeader = 4;
__host__ __device__ __forceinline__ int64_t record_words(int32_t runs, int32_t nchunks, int32_t nb) {
    return kRecHeader + 2 * (int64_t)runs + 1 + (int64_t)nchunks * nb;
}

constexpr int kWalkWin = 1024;  // candidates whose runs are laid out at a time
struct WalkSmem {
    alignas(128) uint4 cand[kWalkWarps][2][2][32];  // two chunks' candidates as A fragments: first and second 8 factors (cand_slot)
    uint4 query[kWalkWarps][32][2];     // the queries as B fragments
    float csq[kWalkWarps][2][32];       // superSymmetric: the candidates' squared supports (scaled)
    float qsq[kWalkWarps][32];          // and the queries'
    // per chunk of the window (and the pair after it): bit k, a run starts at its candidate k; runs before it, minus one
    uint2 starts[kWalkWarps][kWalkWin / 32 + 2];
    int32_t delta[kWalkWarps][32];      // per run: its first sorted index minus its first candidate
    float shift[kWalkWarps][3][32];     // per run: +-ext on the dimensions its cell lies across a seam
    UnitCtx u[kWalkWarps];
};

// Candidate k of the unit (prefix pre[0..S]): returns its sorted index.
__device__ __forceinline__ int32_t cand_index(const int32_t* pre, const int32_t* beg, int S, int32_t k) {
    int lo = 0, hi = S;  // pre[lo] <= k < pre[hi]
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (pre[mid] <= k) lo = mid; else hi = mid;
    }
    return beg[lo] + (k - pre[lo]);
}

// The query's share of the test, kept in the .w of its shared-memory copy: gather hq^2 (the test is
// d2 - hq^2), symmetric hq / 2 (thr = hq / 2 + hc / 2 == fl(hq + hc) / 2), superSymmetric hq.
template <int MODE>
__device__ __forceinline__ float query_share(float hq) {
    return MODE == kSymmetric ? 0.5f * hq : (MODE == kGather ? hq * hq : hq);
}

// The largest threshold candidate c (share cw) can meet over every query (qmax: the largest query
// support); the band of the fast test is kBandEps times its square.
template <int MODE>
__device__ __forceinline__ float cand_tmax(float cw, float qmax) {
    if (MODE == kGather) return qmax;
    if (MODE == kScatter) return cw;
    if (MODE == kSymmetric) return fmaf(qmax, 0.5f, cw);
    return fmaxf(qmax, cw);
}

// Float test of query q (share in q.w) against candidate c (share cw): r < 0 means inside.
template <int DIM, bool PERIODIC, int MODE>
__device__ __forceinline__ float pair_residual(const WrapCtx& wc, const float4& q, const float4& c, float cw,
                                               bool& wrap_unc) {
    float dd[3];
#pragma unroll
    for (int d = 0; d < DIM; ++d) dd[d] = fast_diff<PERIODIC>(wc, d, comp(q, d), comp(c, d), wrap_unc);
    float d2 = dd[0] * dd[0];
    if (DIM > 1) d2 = fmaf(dd[1], dd[1], d2);
    if (DIM > 2) d2 = fmaf(dd[2], dd[2], d2);
    if (MODE == kGather) return d2 - q.w;  // same sign as d2 - hq * hq up to the band
    if (MODE == kScatter) return fmaf(-c.w, c.w, d2);
    const float thr = MODE == kSymmetric ? q.w + cw : fmaxf(q.w, c.w);
    return fmaf(-thr, thr, d2);
}

// Warp-wide 32 x 32 bit transpose: lane j holds row j (bit k = entry (j, k)); lane k receives
// column k (bit j = entry (j, k)).  Five butterfly stages swap ever smaller off-diagonal blocks
// with the partner lane (lane ^ s): the 16- and 8-bit stages are one byte permutation of the own
// and the partner's row each; in the 4-, 2- and 1-bit stages a lane keeps its own bits under a
// lane-dependent mask and takes the partner's row rotated into place (right by s in the upper
// lane of a pair, left by s in the lower one) under the complement.  The per-lane selectors,
// masks and rotations depend on the lane only, so a loop over chunks computes them once.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x, int lane) {
    const uint32_t sel16 = (lane & 16) ? 0x3276u : 0x5410u;
    const uint32_t sel8 = (lane & 8) ? 0x3715u : 0x6240u;
    const uint32_t keep4 = (lane & 4) ? 0xf0f0f0f0u : 0x0f0f0f0fu, rot4 = (lane & 4) ? 4u : 28u;
    const uint32_t keep2 = (lane & 2) ? 0xccccccccu : 0x33333333u, rot2 = (lane & 2) ? 2u : 30u;
    const uint32_t keep1 = (lane & 1) ? 0xaaaaaaaau : 0x55555555u, rot1 = (lane & 1) ? 1u : 31u;
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), sel16);
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), sel8);
    uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4);
    x = (x & keep4) | (__funnelshift_r(y, y, rot4) & ~keep4);
    y = __shfl_xor_sync(0xffffffffu, x, 2);
    x = (x & keep2) | (__funnelshift_r(y, y, rot2) & ~keep2);
    y = __shfl_xor_sync(0xffffffffu, x, 1);
    x = (x & keep1) | (__funnelshift_r(y, y, rot1) & ~keep1);
    return x;
}

// The lane's candidate against queries K4-1 .. 0 of the unit (K4 a multiple of 4; rows past the
// unit's queries are NaN and never hit): bit k of the result is query k's hit, taken from the sign
// of the residual (an arithmetic NaN is positive).  `unc` collects pairs inside the band.
template <int DIM, bool P, int MODE>
__device__ __forceinline__ uint32_t chunk_hits(const WrapCtx& wc, const float4* __restrict__ qsm, int K4,
                                               const float4& cv, float cw, float band, bool& unc) {
    uint32_t hit = 0;
    for (int k = K4 - 4; k >= 0; k -= 4) {
#pragma unroll
        for (int i = 3; i >= 0; --i) {
            const float4 q = qsm[k + i];
            bool wu = false;
            const float r = pair_residual<DIM, P, MODE>(wc, q, cv, cw, wu);
            hit = __funnelshift_l(__float_as_uint(r), hit, 1);
            unc |= (fabsf(r) <= band) || wu;
        }
    }
    return hit;
}

// ---- the tensor-core test
//
// d^2 - thr^2 of every (query, candidate) pair of a unit is one small matrix product: with positions
// relative to the unit's cell centre (scaled by a power of two so that a cell's edge lies in [1, 2)),
//   |Q - C|^2 - thr^2 = N_q + N_c - 2 Q.C [- hq hc / 2],
// N_q = |Q|^2 - (gather hq^2, symmetric hq^2 / 4), N_c = |C|^2 - (scatter hc^2, symmetric hc^2 / 4), and
// the last term in symmetric mode (thr = (hq + hc) / 2).  Every factor is split into two float16
// (hi + lo: 22 bits); hi*hi, hi*lo and lo*hi of the three coordinates and the supports and both
// halves of both norms are 16 products: one mma.m16n8k16 tests 16 candidates against 8 queries, with
// float32 accumulation.  What bounds the walk is issue slots: the float32x2 form took ~9 instructions a
// lane and test, the product leaves 1.5 (collect the sign, keep the smallest magnitude), and its
// accumulator layout hands each lane 4 candidates of two queries, so the hit masks need three
// shuffles per 16 queries and 64 candidates instead of a 32 x 32 bit transpose per chunk.  mma.sync and
// not tcgen05: a unit has ~16 queries and a chunk 32 candidates, so a 128-row tile would span several
// warps and wait on its commit for a product that takes 8 of a chunk's ~100 issue slots.
//
// The product only decides pairs outside a band.  Its error for a pair near the threshold: 16
// products, each at most E = (|Q| + thr + ..)^2, aligned and summed in about 24 bits (<= 16 * 2^-24 E;
// measured 2^-21.4 of the largest product), dropped lo*lo terms and the halves' rounding (<= 8e-7 E).
// kMmaBand = 4e-6 covers the sum twice (measured over random cells: 1.7e-7 E).  The pairs inside the band
// (three in a thousand queries have one) are listed, alone or as a window, and decided exactly after the walk.
__device__ __forceinline__ uint32_t h2bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
// (a, b) as float16 pairs: hi = fl16(a, b), lo = fl16((a, b) - hi).
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    hi = h2bits(h);
    lo = h2bits(__floats2half2_rn(a - f.x, b - f.y));
}
// One number as the float16 pair (hi, lo).
__device__ __forceinline__ uint32_t split_one(float n) {
    return h2bits(__floats2half2_rn(n, n - __half2float(__float2half_rn(n))));
}
constexpr uint32_t kHalfOnes = 0x3c003c00u;

// The 16 factors of a candidate, as 8 pairs of float16 (two 16-byte rows): (xy hi, z hc hi, xy lo,
// z hc lo) and (xy hi, z hc hi, N_c, ones).  A query's, which meet them: -2 xy and (-2 z, -hq / 2) hi twice,
// and (their lo parts, ones, N_q).
template <int MODE>
__device__ __forceinline__ void store_query_frag(uint4* f, float x, float y, float z, float h, bool live) {
    uint32_t xyh = 0, xyl = 0, zhh = 0, zhl = 0;
    float n = kMmaFar;
    if (live) {
        n = fmaf(x, x, fmaf(y, y, z * z));
        if (MODE == kGather) n = fmaf(-h, h, n);
        if (MODE == kSymmetric) n = fmaf(-0.25f * h, h, n);
        split_pair(-2.0f * x, -2.0f * y, xyh, xyl);
        split_pair(-2.0f * z, MODE == kSymmetric ? -0.5f * h : 0.0f, zhh, zhl);
    }
    f[0] = make_uint4(xyh, zhh, xyh, zhh);
    f[1] = make_uint4(xyl, zhl, kHalfOnes, split_one(n));
}
// Returns false when the candidate is too far off for float16 (or NaN): its products decide nothing.
// (The last pair of the second row, the ones, stays from one chunk to the next.)
template <int MODE>
__device__ __forceinline__ bool store_cand_frag(uint4* first, uint4* second, float x, float y, float z, float h) {
    uint4 f;
    const float d = fmaf(x, x, fmaf(y, y, z * z));
    float n = d;
    if (MODE == kScatter) n = fmaf(-h, h, n);
    if (MODE == kSymmetric) n = fmaf(-0.25f * h, h, n);
    split_pair(x, y, f.x, f.z);
    split_pair(z, MODE == kSymmetric ? h : 0.0f, f.y, f.w);
    *first = f;
    *reinterpret_cast<uint2*>(second) = make_uint2(f.x, f.y);
    reinterpret_cast<uint32_t*>(second)[2] = split_one(n);
    return d <= kMmaReach * kMmaReach;
}
// Candidates are the product's 16 rows, queries its 8 columns (units hold any number of queries, so the
// finer step wastes less).  Row r + 8 i of tile t is candidate 4r + 2t + i of the chunk, so that lane
// (g = lane >> 2, t = lane & 3) holds candidates 4g .. 4g + 3 of queries 2t and 2t + 1 in the two tiles'
// accumulators.  Candidate k's place in shared memory is k with its low bits mixed so that neither the
// stores nor ldmatrix's eight rows (4 apart) meet in a bank.
__device__ __forceinline__ int cand_slot(int k) { return k ^ ((k >> 3) & 3); }
static_assert(kWalkWin == 32 * kWarp, "one chunk's starts per lane");
static_assert(kMmaPad > 3.0f * kMmaSupport, "the lanes past the candidates must not hit");

// Four 8 x 8 matrices of float16: one register each, lane (g, t) holding pair t of row g.
__device__ __forceinline__ void load_matrix(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void mma_16x8(float (&d)[4], const uint32_t (&c)[4], uint32_t q0, uint32_t q1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%10, %10, %10, %10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(q0), "r"(q1), "f"(0.0f));
}

// The 32 candidates of tiles c0, c1 against the 8 queries (q0, q1): shifts 8 hits into `hit`, bits 0..3 query
// 2t's among candidates 4g .. 4g + 3, bits 4..7 query 2t + 1's.  umin collects the smallest magnitude.
// superSymmetric: the product is d^2, compared with max(hq, hc)^2 (cs, qs: the squared supports).
template <int MODE>
__device__ __forceinline__ uint32_t mma_hits(uint32_t hit, const uint32_t (&c0)[4], const uint32_t (&c1)[4],
                                             const float4& cs, uint32_t q0, uint32_t q1, const float2& qs,
                                             float& umin) {
    float d0[4], d1[4];
    mma_16x8(d0, c0, q0, q1);
    mma_16x8(d1, c1, q0, q1);
    if (MODE == kSuperSymmetric) {
        d0[0] -= fmaxf(qs.x, cs.x), d0[1] -= fmaxf(qs.y, cs.x), d0[2] -= fmaxf(qs.x, cs.y), d0[3] -= fmaxf(qs.y, cs.y);
        d1[0] -= fmaxf(qs.x, cs.z), d1[1] -= fmaxf(qs.y, cs.z), d1[2] -= fmaxf(qs.x, cs.w), d1[3] -= fmaxf(qs.y, cs.w);
    }
    hit = __funnelshift_l(__float_as_uint(d1[3]), hit, 1);
    hit = __funnelshift_l(__float_as_uint(d1[1]), hit, 1);
    hit = __funnelshift_l(__float_as_uint(d0[3]), hit, 1);
    hit = __funnelshift_l(__float_as_uint(d0[1]), hit, 1);
    hit = __funnelshift_l(__float_as_uint(d1[2]), hit, 1);
    hit = __funnelshift_l(__float_as_uint(d1[0]), hit, 1);
    hit = __funnelshift_l(__float_as_uint(d0[2]), hit, 1);
    hit = __funnelshift_l(__float_as_uint(d0[0]), hit, 1);
#pragma unroll
    for (int i = 0; i < 4; ++i) umin = fminf(umin, fminf(fabsf(d0[i]), fabsf(d1[i])));
    return hit;
}

// 8 x 8 transpose of nibbles across the lanes of equal t: nibble i of lane g goes to nibble g of lane i.
__device__ __forceinline__ uint32_t nibble_transpose(uint32_t x, int lane) {
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), (lane & 16) ? 0x3276u : 0x5410u);
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), (lane & 8) ? 0x3715u : 0x6240u);
    const uint32_t keep = (lane & 4) ? 0xf0f0f0f0u : 0x0f0f0f0fu, rot = (lane & 4) ? 4u : 28u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4);
    return (x & keep) | (__funnelshift_r(y, y, rot) & ~keep);
}

// The same with every pair inside the band decided by the reference's exact test, on the original
// (unshifted) candidate of sorted index j -- in double on the double arrays for float64 inputs;
// rare units only, so out of line.
template <int DIM, int MODE>
__device__ __noinline__ uint32_t chunk_hits_exact(ExactCtx xc, const float4* qsm, const float* qh, const int32_t* qid,
                                                  int K4, float4 cv, int32_t j, float band, F64Walk f64) {
    const WrapCtx wc = wrap_ctx(xc.periodic_mask, xc.ext);
    const float cw = cand_share<MODE>(cv.w);
    uint32_t hit = 0;
    for (int k = K4 - 1; k >= 0; --k) {
        const float4 q = qsm[k];
        bool wu = false;
        const float r = pair_residual<DIM, true, MODE>(wc, q, cv, cw, wu);
        bool in = r < 0.0f;
        if ((fabsf(r) <= band) || wu)
            in = f64.qpos ? f64_pair_decide(f64, DIM, xc.periodic_mask, MODE, qid[k], j)
                          : exact_pair_test(xc, q, qh[k], cv, cv.w);
        hit = (hit << 1) | (in ? 1u : 0u);
    }
    return hit;
}

// A unit as both walks start it: its queries (one per lane), its stencil cells (one per lane) and where
// the cells' candidates lie in the unit's sequence.
struct Unit {
    int32_t nb, M;        // queries, candidates
    int32_t gc[3];
    float4 q;             // the lane's query (NaN past the unit's queries and for strays)
    int32_t qorig;
    bool active;          // the lane holds a query of this unit's cell
    int32_t beg, cnt, pre;  // the lane's stencil cell: first sorted point, points, first candidate
    float sh[3];          // its seam shift
    bool shift_mode, seam;
};

// STRAYS: append the queries whose own cell is not the unit's to the stray list.
template <int DIM, bool PERIODIC, bool STRAYS>
__device__ __forceinline__ Unit open_unit(const WalkArgs& a, const UnitCtx& u, int32_t unit, int32_t grp, int lane) {
    constexpr int S = DIM == 1 ? 3 : (DIM == 2 ? 9 : 27);
    Unit n;
    const int32_t t0 = a.unit_t0[unit];
    n.nb = min(*a.unit_cap, a.group_start[grp + 1] - t0);
    for (int d = 0; d < 3; ++d) n.gc[d] = a.group_coords[3 * grp + d];
    // the unit's queries, loaded before the stencil look-ups so that both latencies overlap
    const float4 nan4 = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
    const bool qlane = lane < n.nb && TCR_IN(t0 + lane, a.nq_total);
    n.q = nan4;
    n.qorig = 0;
    if (qlane) {
        n.q = a.qsorted[t0 + lane];
        n.qorig = a.qsidx[t0 + lane];
    }
    n.beg = n.cnt = 0;
    if (lane < S) stencil_lookup<DIM>(a, u, n.gc, lane, n.beg, n.cnt);
    n.shift_mode = PERIODIC && u.shift_ok;
    n.sh[0] = n.sh[1] = n.sh[2] = 0.f;
    if (n.shift_mode) {  // in stencil_lookup's offset order
        int rem = lane;
#pragma unroll
        for (int d = DIM - 1; d >= 0; --d) {
            const int32_t v = n.gc[d] + rem % 3 - 1;
            rem /= 3;
            if (lane < S && ((u.periodic_mask >> d) & 1))
                n.sh[d] = v < 0 ? -u.ext[d] : (v >= u.count[d] ? u.ext[d] : 0.f);
        }
    }
    n.seam = n.shift_mode && __any_sync(0xffffffffu, n.sh[0] != 0.f || n.sh[1] != 0.f || n.sh[2] != 0.f);
    const int32_t inc = warp_inclusive_scan(n.cnt);
    n.M = __shfl_sync(0xffffffffu, inc, 31);
    n.pre = inc - n.cnt;
    // a query whose own cell differs from the group's leaves for the serial path
    n.active = false;
    if (qlane) {
        n.active = TCR_IN(n.qorig, a.nq_total);
        // (equal positions, and equal cells of the sorted point and its group, are not enough where linear
        // indices wrap: two cells of the grid can then share one key, one run and one group)
        bool check = !a.no_stray_check || !u.plain_cells;
        if (check && a.self && u.plain_cells) {
            // the group's cell is the reference's; where the second wrap changed nothing it is the query's
            // too (three compares instead of three divisions)
            const float4 r = __ldg(&a.rsorted[t0 + lane]);
            check = !(r.x == n.q.x && (DIM < 2 || r.y == n.q.y) && (DIM < 3 || r.z == n.q.z));
        }
        if (n.active && check) {
            int32_t qc[3];
            cell_of(DIM, u.dedupe, u.dmin, u.hcell, u.count, n.q, qc);
            n.active = same_cell<DIM>(qc, n.gc);
        }
        if (!n.active) {  // own cell differs from the group's (aliasing or wrap rounding)
            if (STRAYS) {
                const int32_t k = atomicAdd(a.num_stray, 1);
                if (TCR_IN(k, a.nq_total)) a.stray[k] = t0 + lane;
            }
            n.q = nan4;
        }
    }
    return n;
}

// What fix_unit keeps in shared memory, in place of the candidates' fragments.
struct FixSmem {
    float4 q[32];        // the unit's queries: x, y, z and the query's share of the test
    float qh[32];        // the queries' supports (for the exact test)
    int32_t qid[32];     // the queries' cloud-local indices (float64 inputs)
    int32_t pre[33];     // candidate prefix of the stencil cells
    int32_t beg[32];
    float shift[3][32];
};
static_assert(sizeof(FixSmem) <= sizeof(uint4) * 2 * 2 * 32, "fits the fragments of one warp");

// A unit the product did not take: a periodic cloud with so few cells that differences wrap, supports
// outside the fast test's range, points far outside their cell, more windows at the threshold than can be listed.  One candidate per lane against every
// query in float32; a chunk with a pair inside the float32 band once more with those pairs decided by
// the reference's exact test; the hit bits transposed into the masks.  Out of line, at the unit's end, so
// that its registers do not cost the main loop spills.
template <int DIM, bool PERIODIC, int MODE>
__device__ __noinline__ void fix_unit(const WalkArgs& a, WalkSmem& wsm, int32_t unit, int32_t grp, int lane, int w) {
    const UnitCtx& u = wsm.u[w];
    FixSmem& sm = *reinterpret_cast<FixSmem*>(&wsm.cand[w][0][0][0]);
    const float4 nan4 = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
    const Unit n = open_unit<DIM, PERIODIC, false>(a, u, unit, grp, lane);
    constexpr int S = DIM == 1 ? 3 : (DIM == 2 ? 9 : 27);
    sm.pre[lane] = n.pre;
    if (lane == 0) sm.pre[S] = n.M;
    sm.beg[lane] = n.beg;
    for (int d = 0; d < 3; ++d) sm.shift[d][lane] = n.sh[d];
    sm.q[lane] = make_float4(n.q.x, n.q.y, n.q.z, query_share<MODE>(n.q.w));  // rows >= nb: NaN, never hit
    sm.qh[lane] = n.q.w;
    sm.qid[lane] = n.qorig - u.qshift;
    __syncwarp();
    const int32_t base = a.rec[unit];
    uint32_t* msk = nullptr;
    if (base >= 0 && TCR_GUARD(base + kRecHeader, a.stage_cap)) {
        const int32_t* rec = a.stage + base;
        msk = reinterpret_cast<uint32_t*>(a.stage + base + kRecHeader + 2 * rec[1] + 1);
    }
    const WrapCtx wc = wrap_ctx(u.periodic_mask, u.ext);
    const int K4 = (n.nb + 3) & ~3;
    const int32_t nchunks = (n.M + 31) >> 5;
    const bool has = msk != nullptr && lane < n.nb;
    int32_t count = 0;
    for (int32_t c = 0; c < nchunks; ++c) {
        const int32_t k = (c << 5) + lane;
        float4 cv = nan4, cs = nan4;
        int32_t j = 0;
        if (k < n.M) {
            int lo = 0, hi = S;  // pre[lo] <= k < pre[hi]
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (sm.pre[mid] <= k) lo = mid; else hi = mid;
            }
            j = sm.beg[lo] + (k - sm.pre[lo]);
            if (TCR_GUARD(j, a.nr_total)) cv = __ldg(&a.rsorted[j]);
            cs = cv;
            if (PERIODIC && n.seam) {
                cs.x += sm.shift[0][lo];
                if (DIM > 1) cs.y += sm.shift[1][lo];
                if (DIM > 2) cs.z += sm.shift[2][lo];
            }
        }
        const float cw = cand_share<MODE>(cv.w);
        const float t = cand_tmax<MODE>(cw, u.qmax);
        float band = u.exact_all ? __int_as_float(0x7f800000) : kBandEps * t * t;
        // float64 inputs: the band also covers the rounding of the coordinates to float32
        if (u.f64_err > 0.0f) band += fmaf(2.0f * 1.7320508f * t, u.f64_err, 3.0f * u.f64_err * u.f64_err);
        // shifted candidates: the band also covers the shift's rounding (|d2 error| <= 2 T delta + delta^2)
        const float bs = n.seam ? band + fmaf(2.0f * t, u.shift_delta, u.shift_delta * u.shift_delta) : band;
        bool unc = false;
        uint32_t hit;
        if (!PERIODIC || n.shift_mode)
            hit = chunk_hits<DIM, false, MODE>(wc, sm.q, K4, cs, cw, bs, unc);
        else
            hit = chunk_hits<DIM, PERIODIC, MODE>(wc, sm.q, K4, cv, cw, bs, unc);
        if (__any_sync(0xffffffffu, unc)) {
            hit = chunk_hits_exact<DIM, MODE>(unit_exact_ctx(u, MODE), sm.q, sm.qh, sm.qid, K4, cv, j, band,
                                              a.f64);
        }
        const uint32_t m = warp_transpose32(hit, lane);
        if (lane < n.nb) {
            count += __popc(m);
            if (has) msk[c * n.nb + lane] = m;
        }
    }
    if (n.active) a.counts[n.qorig] = count;
    __syncwarp();
    wsm.cand[w][0][1][lane].w = wsm.cand[w][1][1][lane].w = kHalfOnes;
}

// The pairs inside the band among a window's marked chunks, listed: their products again, tile by tile, each lane
// keeping its own.  Many of them, or no place for them: the window itself.  Returns true when there is no
// place for that either.  Out of line, so that the walk's registers hold none of it (in line, the walk took 2 to 5%
// longer in half of the modes).
template <int DIM, bool PERIODIC, int MODE>
__device__ __noinline__ bool list_band(const WalkArgs& a, WalkSmem& sm, int32_t unit, int32_t grp, int32_t w0, int32_t M,
                                       uint32_t marked, bool seam, int lane, int w) {
    const UnitCtx& u = sm.u[w];
    const int32_t wn = min(M - w0, kWalkWin), nb = min(*a.unit_cap, a.group_start[grp + 1] - a.unit_t0[unit]);
    const float s = u.scale;
    float os[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
        os[d] = d < DIM ? -s * fmaf((float)a.group_coords[3 * grp + d] + 0.5f, u.hcell[d], u.dmin[d]) : 0.f;
    float band = u.mma_band;
    if (PERIODIC && seam) band += u.mma_seam;
    const int g = lane >> 2, tq = lane & 3, slot = cand_slot(lane);
    const uint32_t crow = (uint32_t)__cvta_generic_to_shared(
        &sm.cand[w][0][lane >> 4][cand_slot(4 * (lane & 7) + ((lane >> 3) & 1))]);
    const int32_t base = a.rec[unit];
    const int32_t masks = base >= 0 ? base + kRecHeader + 2 * a.stage[base + 1] + 1 : 0;
    auto run_of = [&](int32_t k) -> int32_t {
        const uint2 st = sm.starts[w][k >> 5];
        return (int32_t)st.y + __popc(st.x & ((2u << (k & 31)) - 1u));
    };
    bool full = base < 0 || (int32_t)(marked >> 16) >= max(kBandLanes, (wn + 63) >> 6);
    const bool list = !full;  // the pairs one by one
    marked &= 0xffffu;
#pragma unroll 1
    for (int32_t c = 0; list && 32 * c < wn && (marked >> (c >> 1)); ++c) {
        if (!((marked >> (c >> 1)) & 1u)) continue;
        const int32_t kl = min(32 * c + lane, wn - 1), run = run_of(kl);
        const float4 v = __ldg(&a.rsorted[sm.delta[w][run] + w0 + kl]);
        float x = v.x, y = v.y, z = v.z;
        if (PERIODIC && seam) {
            x += sm.shift[w][0][run];
            if (DIM > 1) y += sm.shift[w][1][run];
            if (DIM > 2) z += sm.shift[w][2][run];
        }
        store_cand_frag<MODE>(&sm.cand[w][0][0][slot], &sm.cand[w][0][1][slot], fmaf(x, s, os[0]),
                              DIM > 1 ? fmaf(y, s, os[1]) : 0.f, DIM > 2 ? fmaf(z, s, os[2]) : 0.f, v.w * s);
        if (MODE == kSuperSymmetric) sm.csq[w][0][lane] = (v.w * s) * (v.w * s);
        __syncwarp();
#pragma unroll 1
        for (int i = 0; 8 * (i >> 1) < nb; ++i) {  // tile i & 1 of the candidates, i >> 1 of the queries
            uint32_t cf[4];
            load_matrix(cf, crow ^ (32u * (i & 1)));
            const uint32_t* qf = reinterpret_cast<const uint32_t*>(&sm.query[w][8 * (i >> 1) + g][0]);
            float d[4];
            mma_16x8(d, cf, qf[tq], qf[4 + tq]);
            const int q0 = 8 * (i >> 1) + 2 * tq, k0 = 32 * c + 4 * g + 2 * (i & 1);  // of d[0]; d[j]: q0 + (j & 1), k0 + (j >> 1)
            uint32_t close = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float r = d[j];
                if (MODE == kSuperSymmetric) r -= fmaxf(sm.qsq[w][q0 + (j & 1)], sm.csq[w][0][(k0 + (j >> 1)) & 31]);
                close |= (fabsf(r) <= band && q0 + (j & 1) < nb && k0 + (j >> 1) < wn ? 1u : 0u) << j;
            }
            for (; close; close &= close - 1) {
                const int j = __ffs(close) - 1, q = q0 + (j & 1), k = k0 + (j >> 1);
                const int32_t f = atomicAdd(a.num_exact, 1);
                if (f < a.nq_total)
                    a.band_pairs[f] = make_int4(a.unit_t0[unit] + q, sm.delta[w][run_of(k)] + w0 + k,
                                                masks + ((w0 + k) >> 5) * nb + q, k & 31);
                else
                    full = true;  // the list is
            }
            __syncwarp();
        }
    }
    bool lost = false;
    if (__any_sync(0xffffffffu, full) && lane == 0) {
        // (every place that is claimed is written)
        const bool named = w0 < (kWalkWin << 16);
        const int32_t f = named ? atomicAdd(&a.num_exact[2], 1) : 0;
        lost = !named || f >= a.band_cap;
        if (!lost)
            a.band_windows[f] = ((unsigned long long)(uint32_t)unit << 32) | (uint32_t)(w0 / kWalkWin) << 16 | marked;
    }
    __syncwarp();
    return lost;
}

// Count walk of one unit: test every (query, candidate) once, count, and stage the unit's record.
//
// The unit's candidates stream two chunks of 32 at a time, one per lane and chunk (a lane finds its
// candidate's run by its rank among the runs' starts), loaded a pair ahead of their use; they are written to
// shared memory as A fragments and meet the unit's queries (B fragments, in registers) in
// tensor-core products.
template <int DIM, bool PERIODIC, int MODE>
__device__ __forceinline__ void count_unit(const WalkArgs& a, WalkSmem& sm, int32_t unit, int32_t grp, int lane,
                                           int w) {
    const UnitCtx& u = sm.u[w];
    const Unit n = open_unit<DIM, PERIODIC, true>(a, u, unit, grp, lane);
    const int32_t nb = n.nb, M = n.M;
    // runs: the non-empty stencil cells
    const bool starts = n.cnt > 0;
    const uint32_t smask = __ballot_sync(0xffffffffu, starts);
    const int32_t R = __popc(smask);
    const int rid = __popc(smask & ((1u << lane) - 1u));
    if (starts) {
        sm.delta[w][rid] = n.beg - n.pre;
        if (PERIODIC) {
            sm.shift[w][0][rid] = n.sh[0];
            sm.shift[w][1][rid] = n.sh[1];
            sm.shift[w][2][rid] = n.sh[2];
        }
    }
    // scaled positions relative to the cell's centre: fma(x, s, -centre * s) is exact up to one rounding
    const float s = u.scale;
    float os[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) os[d] = d < DIM ? -s * fmaf((float)n.gc[d] + 0.5f, u.hcell[d], u.dmin[d]) : 0.f;
    const float X = fmaf(n.q.x, s, os[0]), Y = DIM > 1 ? fmaf(n.q.y, s, os[1]) : 0.f,
                Z = DIM > 2 ? fmaf(n.q.z, s, os[2]) : 0.f, H = n.q.w * s;
    store_query_frag<MODE>(sm.query[w][lane], X, Y, Z, H, n.active);
    if (MODE == kSuperSymmetric) sm.qsq[w][lane] = H * H;
    // the product takes the unit when its points are where their cell says (a query is at most half a
    // cell off the centre) and every support is in its range; otherwise fix_unit tests it
    const float far = u.scale_cell * 0.55f;
    const bool near = !n.active || (fabsf(X) <= far && fabsf(Y) <= far && fabsf(Z) <= far);
    const bool product = u.mma_ok && (!PERIODIC || n.shift_mode) && __all_sync(0xffffffffu, near);
    // the unit's record, reserved up front
    const int32_t nchunks = (M + 31) >> 5;
    bool stage = false;
    uint32_t* msk = nullptr;
    if (a.stage_cap > 0 && nchunks > 0) {
        const int64_t words = record_words(R, nchunks, nb);
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.cursor, (unsigned long long)words);
        base = __shfl_sync(0xffffffffu, base, 0);
        stage = base + (unsigned long long)words <= (unsigned long long)a.stage_cap;
        if (stage) {
            int32_t* rec = a.stage + base;
            if (lane == 0) {
                rec[0] = nchunks;
                rec[1] = R;
                rec[2] = nb;
                rec[3] = 0;
                rec[kRecHeader + 2 * R] = M;
                a.rec[unit] = (int32_t)base;
            }
            if (starts) {
                rec[kRecHeader + rid] = n.beg;
                rec[kRecHeader + R + rid] = n.pre;
            }
            msk = reinterpret_cast<uint32_t*>(rec + kRecHeader + 2 * R + 1);
        }
    }
    if (lane == 0 && !stage && TCR_IN(unit, a.nq_total)) {
        a.rec[unit] = -1;
        if (nchunks > 0) {  // not staged: the emit walk tests the unit again
            const int32_t f = atomicAdd(a.num_flagged, 1);
            if (TCR_IN(f, a.nq_total)) a.flagged[f] = unit;
        }
    }
    __syncwarp();
    uint32_t count = 0;
    bool redo = false;  // the unit goes to fix_unit after all
    if (product) {
        float band = u.mma_band;
        if (PERIODIC && n.seam) band += u.mma_seam;
        const int g = lane >> 2, tq = lane & 3;
        const int slot = cand_slot(lane);
        // ldmatrix row of this lane: matrix i = lane >> 3 is factors 8 (i >> 1) .. of rows 8 (i & 1) .. of a tile
        // (the second tile's candidates are two on: the place with bit 1 flipped)
        const uint32_t crow = (uint32_t)__cvta_generic_to_shared(
            &sm.cand[w][0][lane >> 4][cand_slot(4 * (lane & 7) + ((lane >> 3) & 1))]);
        // the masks this lane ends up with: query (and 16 more), chunk of the pair
        const int row0 = 8 * ((lane >> 3) & 1) + 2 * tq + (g & 1), half = lane >> 4;
        const bool keep0 = stage && row0 < nb, keep1 = stage && row0 + 16 < nb;
        uint32_t* out = msk + half * nb + row0;
        uint32_t count1 = 0;
        const uint32_t le = (2u << lane) - 1u;  // bits 0 .. lane
        for (int32_t w0 = 0; w0 < M; w0 += kWalkWin) {
            // where the window's runs start, and the rank of each chunk's first run
            const int32_t wn = min(M - w0, kWalkWin);
            sm.starts[w][lane] = make_uint2(0u, 0u);
            __syncwarp();
            const int32_t at = n.pre - w0;
            if (starts && at >= 0 && at < kWalkWin) atomicOr(&sm.starts[w][at >> 5].x, 1u << (at & 31));
            __syncwarp();
            const int32_t before = __popc(__ballot_sync(0xffffffffu, starts && at < 0));
            const int32_t here = __popc(sm.starts[w][lane].x);
            const int32_t upto = before + warp_inclusive_scan(here) - 1;
            sm.starts[w][lane].y = (uint32_t)(upto - here);
            if (lane == 31) sm.starts[w][32] = sm.starts[w][33] = make_uint2(0u, (uint32_t)upto);
            __syncwarp();
            // candidate k of the window (lanes past the last one repeat it)
            auto run_of = [&](int32_t k) -> int32_t {
                const uint2 st = sm.starts[w][k >> 5];
                return (int32_t)st.y + __popc(st.x & le);
            };
            auto fetch = [&](int32_t k, int32_t& run) -> float4 {
                run = run_of(k);
                const int32_t j = sm.delta[w][run] + (w0 + min(k, wn - 1));
                return __ldg(&a.rsorted[j]);
            };
            uint32_t marked = 0;  // bits 0 .. 15: the window's pairs of chunks with a pair inside the band; then: lanes with one
            // one copy of the loop per number of query tiles: a tile costs no branch
            auto pairs = [&](auto tiles) {
                constexpr int NT = decltype(tiles)::value;
                uint32_t qa[4], qb[4];  // (first, second row) of query tiles 0, 1 and 2, 3
                float2 qs[4];
                const uint32_t qrow = (uint32_t)__cvta_generic_to_shared(
                    &sm.query[w][8 * (lane >> 4) + (lane & 7)][(lane >> 3) & 1]);
                load_matrix(qa, qrow);
                if (NT >= 3) load_matrix(qb, qrow + 16 * 2 * 16);
                if (MODE == kSuperSymmetric)
#pragma unroll
                    for (int i = 0; i < NT; ++i) qs[i] = *reinterpret_cast<const float2*>(&sm.qsq[w][8 * i + 2 * tq]);
                int32_t run[2];
                float4 v[2];
                v[0] = fetch(lane, run[0]);
                v[1] = fetch(32 + lane, run[1]);
                for (int32_t k0 = 0; k0 < wn; k0 += 64) {
                    float umin = __int_as_float(0x7f800000);
                    bool far = false;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float x = v[e].x, y = v[e].y, z = v[e].z;
                        if (PERIODIC && n.seam) {
                            x += sm.shift[w][0][run[e]];
                            if (DIM > 1) y += sm.shift[w][1][run[e]];
                            if (DIM > 2) z += sm.shift[w][2][run[e]];
                        }
                        x = k0 + 32 * e + lane < wn ? fmaf(x, s, os[0]) : kMmaPad;
                        y = DIM > 1 ? fmaf(y, s, os[1]) : 0.f;
                        z = DIM > 2 ? fmaf(z, s, os[2]) : 0.f;
                        const float h = v[e].w * s;
                        far |= !store_cand_frag<MODE>(&sm.cand[w][e][0][slot], &sm.cand[w][e][1][slot], x, y, z, h);
                        if (MODE == kSuperSymmetric) sm.csq[w][e][lane] = h * h;
                    }
                    __syncwarp();
                    v[0] = fetch(k0 + 64 + lane, run[0]);
                    v[1] = fetch(k0 + 96 + lane, run[1]);
                    // nibbles: (query 2t, 2t + 1) x (queries 0 .. 7, 8 .. 15) x (chunk 0, 1); p1 the same for queries 16 ..
                    uint32_t p0 = 0, p1 = 0;
#pragma unroll
                    for (int e = 1; e >= 0; --e) {
                        if (e == 1 && k0 + 32 >= wn) continue;
                        uint32_t c0[4], c1[4];
                        load_matrix(c0, crow + e * (2 * 32 * 16));
                        load_matrix(c1, (crow ^ 32u) + e * (2 * 32 * 16));
                        float4 cs;
                        if (MODE == kSuperSymmetric) cs = *reinterpret_cast<const float4*>(&sm.csq[w][e][4 * g]);
                        if (NT >= 2) p0 = mma_hits<MODE>(p0, c0, c1, cs, qa[2], qa[3], qs[1], umin);
                        else p0 <<= 8;
                        p0 = mma_hits<MODE>(p0, c0, c1, cs, qa[0], qa[1], qs[0], umin);
                        if (NT >= 4) p1 = mma_hits<MODE>(p1, c0, c1, cs, qb[2], qb[3], qs[3], umin);
                        else if (NT >= 3) p1 <<= 8;
                        if (NT >= 3) p1 = mma_hits<MODE>(p1, c0, c1, cs, qb[0], qb[1], qs[2], umin);
                    }
                    redo |= far;
                    const uint32_t close = __ballot_sync(0xffffffffu, umin <= band);
                    if (close) marked += (1u << (k0 >> 6)) + ((uint32_t)__popc(close) << 16);
                    const bool in = k0 + 32 * half < wn;
                    const uint32_t m0 = nibble_transpose(p0, lane);
                    count += __popc(m0);
                    if (keep0 && in) out[0] = m0;
                    if (NT >= 3) {
                        const uint32_t m1 = nibble_transpose(p1, lane);
                        count1 += __popc(m1);
                        if (keep1 && in) out[16] = m1;
                    }
                    out += 2 * nb;
                    __syncwarp();  // the fragments are read before the next pair's are written
                }
            };
            if (nb <= 8) pairs(std::integral_constant<int, 1>());
            else if (nb <= 16) pairs(std::integral_constant<int, 2>());
            else if (nb <= 24) pairs(std::integral_constant<int, 3>());
            else pairs(std::integral_constant<int, 4>());
            // rare: the pairs inside the band are listed, to be decided after the walk
            if (marked) redo |= list_band<DIM, PERIODIC, MODE>(a, sm, unit, grp, w0, M, marked, PERIODIC && n.seam, lane, w);
        }
        redo = __any_sync(0xffffffffu, redo);
        // the two chunks of a pair were counted by different lanes; query q's count to lane q
        count += __shfl_xor_sync(0xffffffffu, count, 16);
        count1 += __shfl_xor_sync(0xffffffffu, count1, 16);
        const int from = (lane & 8) | ((lane & 1) << 2) | ((lane >> 1) & 3);
        const uint32_t ca = __shfl_sync(0xffffffffu, count, from), cb = __shfl_sync(0xffffffffu, count1, from);
        count = lane < 16 ? ca : cb;
    }
    if (n.active) a.counts[n.qorig] = (int32_t)count;
    __syncwarp();
    if (nchunks > 0 && (!product || redo)) {
        if (lane == 0 && a.rec[unit] < 0) a.rec[unit] = -2;  // not staged, and no listed window of it needs deciding
        fix_unit<DIM, PERIODIC, MODE>(a, sm, unit, grp, lane, w);
    }
}

// Class (dim * 2 + any periodic dim) of a cloud, the key of the walk kernels' template.
__device__ __forceinline__ int cloud_class(const CloudParams& cp) { return cp.dim * 2 + (cp.periodic_mask ? 1 : 0); }

// Next units of a warp.  Without a class filter one unit per atomic; with one (a batch that mixes
// classes runs one launch per class) a chunk of 32 consecutive units, of which the units of other
// classes are dropped by one ballot -- units of a cloud are consecutive, so chunks rarely mix.
__device__ __forceinline__ uint32_t next_units(const WalkArgs& a, int32_t* counter, const int32_t* list,
                                               int32_t nlist, int lane, int32_t& base) {
    const bool filter = a.class_filter >= 0;
    int32_t b = 0;
    if (lane == 0) b = atomicAdd(counter, filter ? 32 : 1);
    base = __shfl_sync(0xffffffffu, b, 0);
    if (base >= nlist) return 0u;
    if (!filter) return 1u;
    bool mine = false;
    if (base + lane < nlist) {
        const int32_t unit = list ? list[base + lane] : base + lane;
        const int32_t grp = a.unit_group[unit];
        mine = cloud_class(a.table[a.group_cloud[grp]]) == a.class_filter;
    }
    return __ballot_sync(0xffffffffu, mine);  // bit k: unit base + k belongs to this launch
}

template <int DIM, bool PERIODIC, int MODE>
__global__ void __launch_bounds__(kWalkWarps * 32, PERIODIC ? kWalkMinBlocksPeriodic : kWalkMinBlocks)
    walk_count_kernel(const __grid_constant__ WalkArgs a) {
    __shared__ WalkSmem sm;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int e = 0; e < 2; ++e) sm.cand[w][e][1][lane].w = kHalfOnes;
    const int32_t nunits = *a.num_units;
    int32_t* counter = &a.work[a.class_filter >= 0 ? 2 + a.class_filter : 0];
    int cur = -1;
    const bool filter = a.class_filter >= 0;
    // the first claim of every warp is its own number, the counter's come after them
    const int32_t step = filter ? 32 : 1, first = (int32_t)(gridDim.x * kWalkWarps) * step;
    int32_t claim = (int32_t)(blockIdx.x * kWalkWarps + w) * step;
    for (;;) {
        const int32_t base = __shfl_sync(0xffffffffu, claim, 0);
        if (base >= nunits) break;
        uint32_t todo = 1u;
        if (filter) {  // a chunk of 32 consecutive units; the units of other classes are dropped
            bool mine = false;
            if (base + lane < nunits) mine = cloud_class(a.table[a.group_cloud[a.unit_group[base + lane]]]) ==
                                             a.class_filter;
            todo = __ballot_sync(0xffffffffu, mine);
        }
        // the next claim is issued before this one's units run and read after them, so the
        // atomic's latency overlaps their work
        if (lane == 0) claim = first + atomicAdd(counter, step);
        while (todo) {
            const int32_t unit = base + (__ffs(todo) - 1);
            todo &= todo - 1;
            const int32_t grp = a.unit_group[unit];
            const int cloud = a.num_clouds == 1 ? 0 : a.group_cloud[grp];
            if (cloud != cur) {
                __syncwarp();
                if (lane == 0) load_unit_ctx(sm.u[w], a, cloud);
                cur = cloud;
                __syncwarp();
            }
            if (sm.u[w].error) {  // no grid: nothing found, nothing staged
                if (lane == 0) a.rec[unit] = -1;
                continue;
            }
            count_unit<DIM, PERIODIC, MODE>(a, sm, unit, grp, lane, w);
        }
    }
}

struct EmitSmem {
    int32_t pre[kWalkWarps][33];
    int32_t beg[kWalkWarps][32];
    float4 q[kWalkWarps][32];
    UnitCtx u[kWalkWarps];
};

// Emit walk of one unit that was not staged: walk again and write the pairs straight to their slots.
template <int DIM, bool PERIODIC, int MODE>
__device__ __forceinline__ void emit_unit(const WalkArgs& a, EmitSmem& sm, int32_t unit, int32_t grp, int lane,
                                          int w) {
    constexpr int S = DIM == 1 ? 3 : (DIM == 2 ? 9 : 27);
    const UnitCtx& u = sm.u[w];
    const WrapCtx wc = wrap_ctx(u.periodic_mask, u.ext);
    const float qmax = u.qmax;
    const bool exact_all = u.exact_all != 0;
    const unsigned lt = (1u << lane) - 1u;
    const float4 nan4 = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
    const int32_t t0 = a.unit_t0[unit];
    const int32_t nb = min(*a.unit_cap, a.group_start[grp + 1] - t0);
    const int32_t gc[3] = {a.group_coords[3 * grp], a.group_coords[3 * grp + 1], a.group_coords[3 * grp + 2]};
    int32_t beg = 0, cnt = 0;
    if (lane < S) stencil_lookup<DIM>(a, u, gc, lane, beg, cnt);
    const int32_t inc = warp_inclusive_scan(cnt);
    sm.pre[w][lane + 1] = inc;
    if (lane == 0) sm.pre[w][0] = 0;
    sm.beg[w][lane] = beg;
    const int32_t M = __shfl_sync(0xffffffffu, inc, 31);
    int32_t qorig = 0;
    float4 qv = nan4;
    int64_t obase = 0;
    if (lane < nb) {
        const int32_t t = t0 + lane;
        qv = a.qsorted[t];
        qorig = a.qsidx[t];
        int32_t qc[3];
        cell_of(DIM, u.dedupe, u.dmin, u.hcell, u.count, qv, qc);
        if (same_cell<DIM>(qc, gc)) obase = a.offsets[qorig];
        else qv = nan4;  // stray: written by the serial kernel
    }
    sm.q[w][lane] = qv;
    __syncwarp();
    for (int32_t base = 0; base < M; base += 32) {
        const int32_t k = base + lane;
        float4 cv = nan4;
        int32_t j = 0;
        if (k < M) {
            j = cand_index(sm.pre[w], sm.beg[w], S, k);
            if (TCR_GUARD(j, a.nr_total)) cv = __ldg(&a.rsorted[j]);
            else j = 0;
        }
        int32_t jl = __ldg(&a.rsidx[j]);
        jl = a.ref_ids ? __ldg(&a.ref_ids[jl]) : jl - u.rshift;
        const int64_t jorig = (int64_t)jl;
        const float cw = cand_share<MODE>(cv.w);
        float band = exact_all ? __int_as_float(0x7f800000) : cand_band<MODE>(cw, qmax);
        if (u.f64_err > 0.0f) {  // float64 inputs: the coordinates' rounding to float32 widens the band
            const float t = cand_tmax<MODE>(cw, qmax), fe = u.f64_err;
            band += fmaf(2.0f * 1.7320508f * t, fe, 3.0f * fe * fe);
        }
        for (int qi = 0; qi < nb; ++qi) {
            const float4 q = sm.q[w][qi];
            bool in, unc;
            lean_test<DIM, PERIODIC, MODE>(wc, q, cv, cw, band, in, unc);
            const uint32_t ub = __ballot_sync(0xffffffffu, unc);
            int32_t qrow = __shfl_sync(0xffffffffu, qorig, qi);
            if (ub && unc)
                in = a.f64.qpos ? f64_pair_decide(a.f64, DIM, u.periodic_mask, MODE, qrow - u.qshift, j)
                                : exact_pair_test(unit_exact_ctx(u, MODE), q, q.w, cv, cv.w);
            const uint32_t b = __ballot_sync(0xffffffffu, in);
            const int64_t qb = __shfl_sync(0xffffffffu, obase, qi);
            qrow = a.query_ids ? __ldg(&a.query_ids[qrow]) : qrow - u.qshift;
            if (in) {
                const int64_t pos = qb + __popc(b & lt);
                if (pos < a.out_cap) {
                    a.col_out[pos] = jorig;
                    if (a.row_out) a.row_out[pos] = (int64_t)qrow;
                }
            }
            if (lane == qi) obase += __popc(b);
        }
    }
    __syncwarp();
}

template <int DIM, bool PERIODIC, int MODE>
__global__ void __launch_bounds__(kWalkWarps * 32) walk_emit_kernel(WalkArgs a) {
    __shared__ EmitSmem sm;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t nlist = *a.num_list;
    if (nlist == 0) return;  // every unit was staged: no claim atomics at all
    int32_t* counter = a.class_filter >= 0 ? &a.work[8 + a.class_filter] : &a.work[1];
    int cur = -1;
    for (;;) {
        int32_t base;
        uint32_t todo = next_units(a, counter, a.unit_list, nlist, lane, base);
        if (base >= nlist) break;
        while (todo) {
            const int32_t unit = a.unit_list[base + (__ffs(todo) - 1)];
            todo &= todo - 1;
            const int32_t grp = a.unit_group[unit];
            const int cloud = a.num_clouds == 1 ? 0 : a.group_cloud[grp];
            if (cloud != cur) {
                __syncwarp();
                if (lane == 0) load_unit_ctx(sm.u[w], a, cloud);
                cur = cloud;
                __syncwarp();
            }
            if (sm.u[w].error) continue;
            emit_unit<DIM, PERIODIC, MODE>(a, sm, unit, grp, lane, w);
        }
    }
}

// Position of the highest set bit of a non-zero word (one bfind).
__device__ __forceinline__ uint32_t top_set_bit(uint32_t m) {
    uint32_t b;
    asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(m));
    return b;
}

// Emit pass for staged units: expand each unit's record into its queries' CSR/COO slots, one warp per unit,
// window by window of up to kExpandWin chunks.  The window's hit masks come into shared memory in
// (query, chunk) order, an equal share of consecutive words per lane; every lane turns the set bits of its share
// into 16-bit tags (word and bit) in the shared output table, which so is in output order.  The
// window's candidate columns are gathered (consecutive sorted indices; each lane finds its candidate's run
// by a rank in the window's run-start bitmap) and lanes over output positions write consecutive slots.
//
// The expansion is bound by issue slots (11% of the mask bits are set), then by the output's HBM
// writes.  A lane walks its share in one loop over its set bits, all lanes together as many steps as the
// fullest share has (42 of 25 on the 1M workload); a loop per word, as long as the fullest word of 32
// each time, took 99.  Units are claimed one by one: a fixed share per warp left the SMs idle for 20% of the
// 1M workload and 70% of a 65k one.
constexpr int kExpandWarps = 8;
constexpr int kExpandWin = 16;    // chunks per window: 512 candidates
constexpr int kExpandTab = 1920;  // outputs one table holds (four blocks of eight warps fit an SM)
struct ExpandSmem {
    union {
        uint32_t word[kExpandWarps][kExpandWin * 32];  // hit masks: word i of lane L's share at 32 i + L
        int32_t col[kExpandWarps][kExpandWin * 32];    // then the output column of each candidate of the window
    };
    uint16_t tab[kExpandWarps][kExpandTab];        // (word << 5) | bit of each output, word = query * chunks + chunk
    uint2 starts[kExpandWarps][kExpandWin];        // per chunk: bit k, a run starts at its candidate k; runs before it, minus one
    int32_t delta[kExpandWarps][32];               // per run: its first sorted index minus its first candidate
    long long* qcol[kExpandWarps][32];             // column output of table entry 0 of each query (this window)
    int32_t qrow[kExpandWarps][32];
};
// ceil(2^16 / k): x / k == x * kInverse[k] >> 16 for x < 2^16 / k.
__constant__ uint32_t kInverse[33] = {0,    65536, 32768, 21846, 16384, 13108, 10923, 9363, 8192, 7282, 6554,
                                      5958, 5462,  5042,  4682,  4370,  4096,  3856,  3641, 3450, 3277, 3121,
                                      2979, 2850,  2731,  2622,  2521,  2428,  2341,  2260, 2185, 2115, 2048};

// One step of a lane through its share (words 128 bytes apart, last first): takes the next word when the
// current one, m, is spent, and writes the tag of its highest set bit below pos.  Predicated by hand:
// as branches the two halves diverge in every step (217 against 199 us for the 1M workload's expansion).
__device__ __forceinline__ void expand_step(uint32_t base, uint32_t& at, uint32_t& m, uint32_t& tag, uint32_t& pos) {
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        ".reg .u32 b, t;\n"
        ".reg .u16 h;\n"
        "setp.gt.u32 p, %0, %4;\n"
        "setp.eq.and.u32 p, %1, 0, p;\n"
        "@p sub.u32 %0, %0, 128;\n"
        "@p sub.u32 %2, %2, 32;\n"
        "@p ld.shared.u32 %1, [%0];\n"
        "setp.ne.u32 q, %1, 0;\n"
        "bfind.u32 b, %1;\n"
        "add.u32 t, %2, b;\n"
        "cvt.u16.u32 h, t;\n"
        "@q sub.u32 %3, %3, 2;\n"
        "@q st.shared.u16 [%3], h;\n"
        "shl.b32 t, 1, b;\n"  // (no bit: shifted out)
        "xor.b32 %1, %1, t;\n"
        "}\n"
        : "+r"(at), "+r"(m), "+r"(tag), "+r"(pos)
        : "r"(base)
        : "memory");
}

struct ExpandArgs {
    const int32_t* __restrict__ stage;
    const int32_t* __restrict__ rec;
    const int32_t* __restrict__ num_units;
    const int32_t* __restrict__ unit_t0;
    const int32_t* __restrict__ unit_group;
    const int32_t* __restrict__ group_cloud;
    const int32_t* __restrict__ qsidx;
    const int32_t* __restrict__ col_of;  // [nr] column of each sorted reference (composed: with ref_ids applied)
    int32_t composed;
    const int64_t* __restrict__ offsets;
    const int32_t* __restrict__ query_ids;
    const CloudParams* __restrict__ table;
    int32_t num_clouds;
    int32_t local_index;
    int64_t* __restrict__ row_out;
    int64_t* __restrict__ col_out;
    int64_t out_cap;
    int32_t* work;              // the next unit to claim
    const unsigned long long* __restrict__ stage_cap;  // words of the staging list
    int64_t nq, nr;
};

__global__ void __launch_bounds__(kExpandWarps * 32, 4) expand_records_kernel(const __grid_constant__ ExpandArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ExpandSmem& sm = *reinterpret_cast<ExpandSmem*>(smem_raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t nu = *a.num_units;
    uint32_t* __restrict__ word = sm.word[w];
    int32_t* __restrict__ cols = sm.col[w];
    uint16_t* __restrict__ tab = sm.tab[w];
    const uint32_t le = (2u << lane) - 1u;  // bits 0 .. lane
    const int64_t cap = (int64_t)*a.stage_cap;
    // A unit is claimed three iterations before it runs, its record offset and first query are read two
    // before, its record's first 64 words (the header and the runs) and query rows (lane < 32 covers every
    // unit size) one before, so a unit starts with them at hand instead of dependent round trips.
    // (the first two are the warp's own number and the next round's, the counter's come after them)
    const int32_t warps = (int32_t)gridDim.x * kExpandWarps;
    auto claim = [&]() -> int32_t { return lane == 0 ? 2 * warps + atomicAdd(a.work, 1) : 0; };
    auto words_of = [&](int32_t r0, int32_t k) -> int32_t {
        return (r0 >= 0 && (int64_t)r0 + k < cap) ? a.stage[r0 + k] : 0;
    };
    auto qrows = [&](int32_t v, int32_t t0) -> int32_t {
        return (v < nu && TCR_GUARD(t0 + lane, a.nq)) ? a.qsidx[t0 + lane] : -1;
    };
    int32_t ua = (int32_t)blockIdx.x * kExpandWarps + w, ub = ua + warps;
    if (ua >= nu) return;
    int32_t next = ub < nu ? claim() : nu;
    int32_t r0a = ua < nu ? a.rec[ua] : -1, t0a = ua < nu ? a.unit_t0[ua] : 0;
    int32_t r0b = ub < nu ? a.rec[ub] : -1, t0b = ub < nu ? a.unit_t0[ub] : 0;
    int32_t ha = words_of(r0a, lane), hb = words_of(r0a, 32 + lane), qa = qrows(ua, t0a);
    while (ua < nu) {
        const int32_t u = ua, r0 = r0a, h0 = ha, h1 = hb, qrow_l = qa;
        ha = words_of(r0b, lane);
        hb = words_of(r0b, 32 + lane);
        qa = qrows(ub, t0b);
        ua = ub;
        r0a = r0b;
        ub = __shfl_sync(0xffffffffu, next, 0);
        r0b = -1;
        if (ub < nu) {
            r0b = a.rec[ub];
            t0b = a.unit_t0[ub];
        }
        next = claim();
        if (r0 < 0) continue;  // no candidates, or re-tested by the emit walk
        const int32_t nchunks = __shfl_sync(0xffffffffu, h0, 0), R = __shfl_sync(0xffffffffu, h0, 1),
                      nb = __shfl_sync(0xffffffffu, h0, 2);
        if (!TCR_GUARD(R, 28) || !TCR_GUARD(nb - 1, 32) || !TCR_GUARD(r0 + record_words(R, nchunks, nb) - 1, cap))
            continue;
        const int32_t* rec = a.stage + r0;
        const uint32_t* masks = reinterpret_cast<const uint32_t*>(rec + kRecHeader + 2 * R + 1);
        int32_t rshift = 0, qshift = 0;
        if (a.local_index) {
            const CloudParams& cp = a.table[a.num_clouds == 1 ? 0 : a.group_cloud[a.unit_group[u]]];
            rshift = a.composed ? 0 : cp.ref_base;
            qshift = cp.query_base;
        }
        auto word_at = [&](int32_t k) -> int32_t {  // word k of the record, k < 64
            const int32_t x = __shfl_sync(0xffffffffu, h0, k & 31), y = __shfl_sync(0xffffffffu, h1, k & 31);
            return k < 32 ? x : y;
        };
        const int32_t beg = word_at(kRecHeader + lane);
        const int32_t pre = word_at(min(kRecHeader + R + lane, 63));  // candidate prefix of the runs, then M
        if (lane < R) sm.delta[w][lane] = beg - pre;
        const int32_t M = __shfl_sync(0xffffffffu, pre, R);
        const bool mine = lane < nb && TCR_GUARD(qrow_l, a.nq);
        int64_t qoff = 0;  // lane q: output position of query q's next hit
        if (mine) {
            qoff = a.offsets[qrow_l];
            if (a.row_out) sm.qrow[w][lane] = a.query_ids ? a.query_ids[qrow_l] : qrow_l - qshift;
        }
        const uint32_t inb = kInverse[nb];
        int32_t nc = 0;
        for (int32_t c0 = 0; c0 < nchunks; c0 += nc) {
            nc = min(kExpandWin, nchunks - c0);
            int32_t words, share, nw, bits, steps, end, n;
            for (;;) {
                // the window's masks: read in the record's order (chunk, query), stored in output order
                words = nb * nc;
                share = (words + 31) >> 5;
                const uint32_t ishare = kInverse[share];
                const uint32_t* src = masks + (int64_t)c0 * nb;
                __syncwarp();
                auto place = [&](int32_t i0, auto count) {
                    constexpr int N = decltype(count)::value;
                    uint32_t m[N];
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        const int32_t x = ((i0 + i) << 5) + lane;
                        m[i] = x < words ? __ldcs(&src[x]) : 0u;
                    }
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        const uint32_t x = ((i0 + i) << 5) + lane;
                        const uint32_t c = (x * inb) >> 16, q = x - c * nb, v = q * nc + c;
                        const uint32_t owner = (v * ishare) >> 16;
                        if (x < (uint32_t)words) word[((v - owner * share) << 5) + owner] = m[i];
                    }
                };
                if (share > 4)
                    for (int32_t i0 = 0; i0 < share; i0 += 8) place(i0, std::integral_constant<int, 8>());
                else
                    place(0, std::integral_constant<int, 4>());
                __syncwarp();
                nw = min(max(words - lane * share, 0), share);  // words of this lane's share
                bits = 0;
                steps = 0;
                for (int32_t i = 0; i < nw; ++i) {
                    const int32_t p = __popc(word[(i << 5) + lane]);
                    bits += p;
                    steps += max(p, 1);
                }
                end = warp_inclusive_scan(bits);
                n = __shfl_sync(0xffffffffu, end, 31);
                if (n <= kExpandTab) break;
                nc = (nc + 1) >> 1;  // more outputs than the table holds (one chunk's always fit)
            }
            // lane q: the table entries before query q's first (its first word is word `off` of lane `owner`'s
            // share), and its own
            int32_t qpre, qv;
            {
                const int32_t first = min(lane, nb) * nc, owner = min((int32_t)((first * kInverse[share]) >> 16), 31),
                              off = first - owner * share;
                qpre = __shfl_sync(0xffffffffu, end - bits, owner);
                for (int32_t i = 0; i < off; ++i) qpre += first < words ? __popc(word[(i << 5) + owner]) : 0;
                if (first >= words) qpre = n;
                qv = __shfl_down_sync(0xffffffffu, qpre, 1) - qpre;
                if (lane >= nb) qv = 0;
                else if (lane == 31) qv = n - qpre;
            }
            // every lane expands its share, last word and highest bit first
            {
                const uint32_t base = (uint32_t)__cvta_generic_to_shared(word) + 4 * lane;
                uint32_t pos = (uint32_t)__cvta_generic_to_shared(tab) + 2 * end;
                uint32_t at = base + 128 * nw, m = 0, tag = (uint32_t)(lane * share + nw) << 5;
                const int32_t T = __reduce_max_sync(0xffffffffu, steps);
                for (int32_t t = 0; t < T; t += 4) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) expand_step(base, at, m, tag, pos);
                }
            }
            // the window's runs: start bits and ranks
            const int32_t wbase = c0 << 5;
            if (lane < kExpandWin) sm.starts[w][lane] = make_uint2(0u, 0u);
            __syncwarp();
            const int32_t at = pre - wbase;
            if (lane < R && at >= 0 && at < (nc << 5)) atomicOr(&sm.starts[w][at >> 5].x, 1u << (at & 31));
            const int32_t before = __popc(__ballot_sync(0xffffffffu, lane < R && at < 0));
            __syncwarp();
            const int32_t here = lane < kExpandWin ? __popc(sm.starts[w][lane].x) : 0;
            const int32_t upto = before + warp_inclusive_scan(here) - 1;
            if (lane < kExpandWin) sm.starts[w][lane].y = (uint32_t)(upto - here);
            __syncwarp();
            // the candidate columns, in place of the masks; the loads of each batch issued together so that
            // their latencies overlap (lanes past the last candidate repeat it)
            auto gather = [&](int32_t cc0, auto count) {
                constexpr int N = decltype(count)::value;
                int32_t jl[N];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const int32_t cc = min(cc0 + i, nc - 1);
                    const uint2 st = sm.starts[w][cc];
                    const int32_t run = (int32_t)st.y + __popc(st.x & le);
                    const int32_t j = sm.delta[w][run & 31] + min(wbase + (cc << 5) + lane, M - 1);
                    jl[i] = TCR_GUARD(j, a.nr) ? __ldg(&a.col_of[j]) : 0;
                }
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (cc0 + i < nc) cols[((cc0 + i) << 5) + lane] = jl[i] - rshift;
            };
            for (int32_t cc0 = 0; cc0 < nc;) {
                if (nc - cc0 > 4) {
                    gather(cc0, std::integral_constant<int, 8>());
                    cc0 += 8;
                } else {
                    gather(cc0, std::integral_constant<int, 4>());
                    cc0 += 4;
                }
            }
            // per query: the output slot of its table entry 0, and whether all of the window's outputs
            // fit the output buffer (then the loops write without checks)
            sm.qcol[w][lane] = reinterpret_cast<long long*>(a.col_out) + (qoff - qpre);
            const bool fits = __all_sync(0xffffffffu, !mine || qoff + qv <= a.out_cap);
            qoff += qv;
            __syncwarp();
            const uint32_t inc = kInverse[nc], per = (uint32_t)nc << 5;
            if (fits && !a.row_out) {
#pragma unroll 4
                for (int32_t o = lane; o < n; o += 32) {
                    const uint32_t v = tab[o], q = ((v >> 5) * inc) >> 16;
                    __stcs(sm.qcol[w][q] + o, (long long)cols[v - q * per]);
                }
            } else if (fits) {  // COO: the row of an output sits at the same slot of row_out
                const int64_t rd = ((intptr_t)a.row_out - (intptr_t)a.col_out) / 8;  // both int64-aligned
#pragma unroll 4
                for (int32_t o = lane; o < n; o += 32) {
                    const uint32_t v = tab[o], q = ((v >> 5) * inc) >> 16;
                    long long* p = sm.qcol[w][q] + o;
                    __stcs(p, (long long)cols[v - q * per]);
                    __stcs(p + rd, (long long)sm.qrow[w][q]);
                }
            } else {
                for (int32_t o = lane; o < n; o += 32) {
                    const uint32_t v = tab[o], q = ((v >> 5) * inc) >> 16;
                    const int64_t pos = (sm.qcol[w][q] - reinterpret_cast<long long*>(a.col_out)) + o;
                    if (TCR_GUARD(pos, a.out_cap)) {
                        __stcs(reinterpret_cast<long long*>(&a.col_out[pos]), (long long)cols[v - q * per]);
                        if (a.row_out) __stcs(reinterpret_cast<long long*>(&a.row_out[pos]), (long long)sm.qrow[w][q]);
                    }
                }
            }
            __syncwarp();
        }
    }
}

// The caller's id of every sorted reference, for the expansion of a search with ref_ids: composed once
// here, where composing it per unit read the ids 27 times over in random order (0.25 of 0.43 ms for 500k
// adaptive points).
__global__ void compose_ids_kernel(const int32_t* __restrict__ rsidx, const int32_t* __restrict__ ref_ids, int64_t n,
                                   int32_t* __restrict__ out) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) {
        const int32_t p = rsidx[j];
        out[j] = TCR_GUARD(p, n) ? ref_ids[p] : 0;
    }
}

// Sets hit `bit` of a mask to what the exact test found: 1 or -1 where that is a change.  (A pair may be listed by
// itself and with its window; one of the two finds the change.)
__device__ __forceinline__ int set_hit(uint32_t* mask, int bit, bool in) {
    const uint32_t b = 1u << bit;
    if (in) return (atomicOr(mask, b) & b) ? 0 : 1;
    return (atomicAnd(mask, ~b) & b) ? -1 : 0;
}

// Where a window's runs start (at: the lane's run, relative to the window), and the rank of each chunk's first run.
__device__ __forceinline__ void lay_window(WalkSmem& sm, int lane, int w, bool starts, int32_t at) {
    sm.starts[w][lane] = make_uint2(0u, 0u);
    __syncwarp();
    if (starts && at >= 0 && at < kWalkWin) atomicOr(&sm.starts[w][at >> 5].x, 1u << (at & 31));
    __syncwarp();
    const int32_t before = __popc(__ballot_sync(0xffffffffu, starts && at < 0));
    const int32_t here = __popc(sm.starts[w][lane].x);
    const int32_t upto = before + warp_inclusive_scan(here) - 1;
    sm.starts[w][lane].y = (uint32_t)(upto - here);
    if (lane == 31) sm.starts[w][32] = sm.starts[w][33] = make_uint2(0u, (uint32_t)upto);
    __syncwarp();
}

// A pair inside the product's band decided by the reference's exact test after the walk, its hit bit and its query's
// count corrected where the product's sign said otherwise.
__device__ __forceinline__ void decide_band_pair(const WalkArgs& a, const int4& p) {
    if (!TCR_GUARD(p.x, a.nq_total) || !TCR_GUARD(p.y, a.nr_total) || !TCR_GUARD(p.z, a.stage_cap)) return;
    const int32_t qorig = a.qsidx[p.x];
    const CloudParams& cp = a.table[cloud_of(a.query_prefix, a.num_clouds, qorig)];
    const bool was = ((uint32_t)a.stage[p.z] >> (p.w & 31)) & 1u;
    bool in;
    if (a.f64.qpos) {
        in = f64_pair_decide(a.f64, cp.dim, cp.periodic_mask, a.mode, qorig - (a.local_index ? cp.query_base : 0), p.y);
    } else {
        ExactCtx xc;
        xc.dim = cp.dim;
        xc.mode = a.mode;
        xc.periodic_mask = cp.periodic_mask;
        for (int d = 0; d < 3; ++d) xc.ext[d] = cp.ext[d];
        const float4 q = a.qsorted[p.x], c = a.rsorted[p.y];
        in = exact_pair_test(xc, q, q.w, c, c.w);
    }
    if (in == was) return;  // (nearly always)
    if (const int change = set_hit(reinterpret_cast<uint32_t*>(&a.stage[p.z]), p.w & 31, in)) atomicAdd(&a.counts[qorig], change);
}

// What decide_window keeps in shared memory, in place of the second chunk's fragments.
struct BandSmem {
    uint32_t pair[64];   // bit 31: the product's decision, [10, 15): query, [0, 10): candidate of the window
    int32_t change[32];  // per query: pairs found less pairs lost
};
static_assert(sizeof(BandSmem) <= sizeof(uint4) * 2 * 32 && kWalkWin <= 1024, "fits the fragments of one chunk");

// A window of a unit's candidates with many pairs inside the product's band (points on a lattice whose spacing
// divides the support: most queries have some): the products of its marked pairs of chunks again, the pairs
// inside the band queued in shared memory and decided 32 at a time by the exact test, one per lane.  (Tested again
// by fix_unit, one candidate per lane against every query, 1M lattice points took 2.75 ms, of 0.6 ms without pairs at
// the threshold; now NNN.)  Not in the walk, whose registers and code it would share.
template <int DIM, int MODE>
__device__ __noinline__ void decide_window(const WalkArgs& a, WalkSmem& sm, unsigned long long entry, int lane, int w) {
    const UnitCtx& u = sm.u[w];
    BandSmem& near = *reinterpret_cast<BandSmem*>(&sm.cand[w][1][0][0]);
    const int32_t unit = (int32_t)(entry >> 32), w0 = (int32_t)((entry >> 16) & 0xffffu) * kWalkWin;
    const uint32_t marked = (uint32_t)entry & 0xffffu;
    const int32_t t0 = a.unit_t0[unit], base = a.rec[unit];
    if (base < -1) return;  // the unit was tested again as a whole
    const Unit n = open_unit<DIM, true, false>(a, u, unit, a.unit_group[unit], lane);
    const int32_t wn = min(n.M - w0, kWalkWin);
    uint32_t* msk = nullptr;  // the window's first hit mask
    if (base >= 0 && TCR_GUARD(base + kRecHeader, a.stage_cap))
        msk = reinterpret_cast<uint32_t*>(a.stage + base + kRecHeader + 2 * a.stage[base + 1] + 1) + (int64_t)(w0 >> 5) * n.nb;
    // runs, queries and scale as count_unit has them
    const bool starts = n.cnt > 0;
    const uint32_t smask = __ballot_sync(0xffffffffu, starts), lt = (1u << lane) - 1u;
    const int rid = __popc(smask & lt);
    if (starts) {
        sm.delta[w][rid] = n.beg - n.pre;
        for (int d = 0; d < 3; ++d) sm.shift[w][d][rid] = n.sh[d];
    }
    const float s = u.scale;
    float os[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) os[d] = d < DIM ? -s * fmaf((float)n.gc[d] + 0.5f, u.hcell[d], u.dmin[d]) : 0.f;
    const float H = n.q.w * s;
    store_query_frag<MODE>(sm.query[w][lane], fmaf(n.q.x, s, os[0]), DIM > 1 ? fmaf(n.q.y, s, os[1]) : 0.f,
                           DIM > 2 ? fmaf(n.q.z, s, os[2]) : 0.f, H, n.active);
    if (MODE == kSuperSymmetric) sm.qsq[w][lane] = H * H;
    lay_window(sm, lane, w, starts, n.pre - w0);
    const float band = u.mma_band + (n.seam ? u.mma_seam : 0.f);
    const int g = lane >> 2, tq = lane & 3, slot = cand_slot(lane);
    const uint32_t crow = (uint32_t)__cvta_generic_to_shared(
        &sm.cand[w][0][lane >> 4][cand_slot(4 * (lane & 7) + ((lane >> 3) & 1))]);
    near.change[lane] = 0;
    int32_t waiting = 0, decided = 0;
    auto run_of = [&](int32_t k) -> int32_t {  // candidate k of the window
        const uint2 st = sm.starts[w][k >> 5];
        return (int32_t)st.y + __popc(st.x & ((2u << (k & 31)) - 1u));
    };
    auto decide = [&]() {  // the first 32 waiting pairs (the rest moves up)
        __syncwarp();
        const int32_t m = min(waiting, 32);
        if (lane < m) {
            const uint32_t e = near.pair[lane];
            const int q = (e >> 10) & 31, k = e & 1023;
            const int32_t j = sm.delta[w][run_of(k)] + w0 + k;
            bool in;
            if (a.f64.qpos) {
                in = f64_pair_decide(a.f64, DIM, u.periodic_mask, MODE, a.qsidx[t0 + q] - u.qshift, j);
            } else {
                const float4 x = a.qsorted[t0 + q], c = a.rsorted[j];
                in = exact_pair_test(unit_exact_ctx(u, MODE), x, x.w, c, c.w);
            }
            if (in != ((e >> 31) != 0)) {
                const int change = msk ? set_hit(&msk[(k >> 5) * n.nb + q], k & 31, in) : (in ? 1 : -1);
                if (change) atomicAdd(&near.change[q], change);
            }
        }
        waiting -= m;
        decided += m;
        __syncwarp();
        const uint32_t rest = near.pair[32 + lane];
        __syncwarp();
        if (lane < waiting) near.pair[lane] = rest;
        __syncwarp();
    };
#pragma unroll 1
    for (int32_t c = 0; 32 * c < wn; ++c) {
        if (!((marked >> (c >> 1)) & 1u)) continue;
        const int32_t k0 = min(32 * c + lane, wn - 1), run = run_of(k0);  // (lanes past the last candidate repeat it)
        const float4 v = __ldg(&a.rsorted[sm.delta[w][run] + w0 + k0]);
        float x = v.x, y = v.y, z = v.z;
        if (n.seam) {
            x += sm.shift[w][0][run];
            if (DIM > 1) y += sm.shift[w][1][run];
            if (DIM > 2) z += sm.shift[w][2][run];
        }
        __syncwarp();  // (the last chunk's fragments are read)
        store_cand_frag<MODE>(&sm.cand[w][0][0][slot], &sm.cand[w][0][1][slot], fmaf(x, s, os[0]),
                              DIM > 1 ? fmaf(y, s, os[1]) : 0.f, DIM > 2 ? fmaf(z, s, os[2]) : 0.f, v.w * s);
        if (MODE == kSuperSymmetric) sm.csq[w][0][lane] = (v.w * s) * (v.w * s);
        __syncwarp();
#pragma unroll 1
        for (int i = 0; 8 * (i >> 1) < n.nb; ++i) {  // tile i & 1 of the candidates, i >> 1 of the queries
            uint32_t cf[4];
            load_matrix(cf, crow ^ (32u * (i & 1)));
            const uint32_t* qf = reinterpret_cast<const uint32_t*>(&sm.query[w][8 * (i >> 1) + g][0]);
            float d[4];
            mma_16x8(d, cf, qf[tq], qf[4 + tq]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int q = 8 * (i >> 1) + 2 * tq + (j & 1), k = 32 * c + 4 * g + 2 * (i & 1) + (j >> 1);
                float r = d[j];
                if (MODE == kSuperSymmetric) r -= fmaxf(sm.qsq[w][q], sm.csq[w][0][k & 31]);
                const bool close = fabsf(r) <= band && q < n.nb && k < wn;
                const uint32_t m = __ballot_sync(0xffffffffu, close);
                if (m == 0) continue;
                if (close) near.pair[waiting + __popc(m & lt)] = (__float_as_uint(r) & 0x80000000u) | (uint32_t)(q << 10 | k);
                waiting += __popc(m);
                if (waiting >= 32) decide();
            }
        }
    }
    if (waiting > 0) decide();
    __syncwarp();
    if (n.active && near.change[lane] != 0) atomicAdd(&a.counts[n.qorig], near.change[lane]);
    if (lane == 0) atomicAdd(&a.num_exact[1], decided);
    __syncwarp();
}

template <int DIM>
__device__ __forceinline__ void decide_window_mode(const WalkArgs& a, WalkSmem& sm, unsigned long long entry, int lane, int w) {
    switch (a.mode) {
        case kGather: return decide_window<DIM, kGather>(a, sm, entry, lane, w);
        case kScatter: return decide_window<DIM, kScatter>(a, sm, entry, lane, w);
        case kSymmetric: return decide_window<DIM, kSymmetric>(a, sm, entry, lane, w);
        default: return decide_window<DIM, kSuperSymmetric>(a, sm, entry, lane, w);
    }
}

// The listed windows, one warp each.
__device__ __forceinline__ void decide_windows(const WalkArgs& a, int32_t n) {
    if (n == 0) return;
    __shared__ WalkSmem sm;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    sm.cand[w][0][1][lane].w = kHalfOnes;
    const int32_t units = *a.num_units;
    int cur = -1;
    for (int32_t i = blockIdx.x * kWalkWarps + w; i < n; i += gridDim.x * kWalkWarps) {
        const unsigned long long entry = a.band_windows[i];
        if (!TCR_GUARD(entry >> 32, units)) continue;
        const int32_t grp = a.unit_group[entry >> 32];
        const int cloud = a.num_clouds == 1 ? 0 : a.group_cloud[grp];
        if (cloud != cur) {
            __syncwarp();
            if (lane == 0) load_unit_ctx(sm.u[w], a, cloud);
            cur = cloud;
            __syncwarp();
        }
        if (sm.u[w].dim == 1) decide_window_mode<1>(a, sm, entry, lane, w);
        else if (sm.u[w].dim == 2) decide_window_mode<2>(a, sm, entry, lane, w);
        else decide_window_mode<3>(a, sm, entry, lane, w);
    }
}

// Resident blocks per SM of the launch after the count walk (registers <= 65536 / (128 * blocks)): a listed window is a
// chain of reads for one warp, so warps in flight decide (1M lattice points in 3D / 1D: 1.22 / 1.18 ms with five, 1.18 /
// 1.13 with seven).
constexpr int kStrayBlocks = 7;

// Serial walk for queries whose own cell differs from their group's (one thread per query).  After the count
// walk also: the pairs inside the product's band (one thread per listed pair, one warp per listed window).
template <bool EMIT>
__global__ void __launch_bounds__(kWalkWarps * 32, EMIT ? 1 : kStrayBlocks) stray_kernel(const __grid_constant__ WalkArgs a) {
    // (read together: as they are used, each would wait for the work before it)
    const int32_t ns = *a.num_stray, listed = a.num_exact[0], windows = a.num_exact[2];
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, threads = (int64_t)gridDim.x * blockDim.x;
    // the last launch of a count or an emit leaves the work counters ready for the next emit
    if (blockIdx.x == 0 && threadIdx.x < kWorkCounters) a.work[threadIdx.x] = 0;
    if constexpr (!EMIT) {
        for (int64_t c = threads - 1 - first; c < a.num_clouds; c += threads) {  // (from the end: the first have pairs)
            float qmax;
            const bool any = a.table[c].n_query > 0;
            if (query_limits(a.table[c], a.grid[c], a.qparams[c], qmax) & any) atomicAdd(a.exact_clouds, 1);
        }
        const int64_t nband = min((int64_t)listed, a.nq_total);
        for (int64_t i = first; i < nband; i += threads) decide_band_pair(a, a.band_pairs[i]);
        decide_windows(a, (int32_t)min((int64_t)windows, a.band_cap));
    }
    for (int32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
        const int32_t t = a.stray[s];
        const float4 q = a.qsorted[t];
        const int32_t qorig = a.qsidx[t];
        UnitCtx u;
        load_unit_ctx(u, a, cloud_of(a.query_prefix, a.num_clouds, qorig));
        if (u.error) continue;
        const int S = u.dim == 1 ? 3 : (u.dim == 2 ? 9 : 27);
        const ExactCtx xc = unit_exact_ctx(u, a.mode);
        int32_t qc[3];
        cell_of(u.dim, u.dedupe, u.dmin, u.hcell, u.count, q, qc);
        int64_t pos = EMIT ? a.offsets[qorig] : 0;
        int32_t n = 0;
        for (int o = 0; o < S; ++o) {
            int32_t beg, cnt;
            stencil_lookup_any(a, u, qc, o, beg, cnt);
            for (int32_t j = beg; j < beg + cnt; ++j) {
                const float4 cv = a.rsorted[j];
                const bool in = a.f64.qpos ? f64_pair_decide(a.f64, u.dim, u.periodic_mask, a.mode, qorig - u.qshift, j)
                                           : exact_pair_test(xc, q, q.w, cv, cv.w);
                if (in) {
                    if (EMIT) {
                        if (pos < a.out_cap) {
                            const int32_t jl = a.rsidx[j];
                            a.col_out[pos] = (int64_t)(a.ref_ids ? a.ref_ids[jl] : jl - u.rshift);
                            if (a.row_out) a.row_out[pos] = a.query_ids ? a.query_ids[qorig] : qorig - u.qshift;
                        }
                        ++pos;
                    } else {
                        ++n;
                    }
                }
            }
        }
        if (!EMIT) a.counts[qorig] = n;
    }
}

// ------------------------------------------------------------------------------------------
// float64 inputs (the reference dispatches its operators on float and double,
// neighborhoodDynamic_cpu.cpp:504,531).  The structure is built from float32 copies with a cell
// size no smaller than the reference's double one, so every pair within the double support lies
// in the query's 3^d stencil; the walks then test candidates on the float32 copies with a band
// widened by the copies' rounding, and every pair inside the band is decided on the caller's double
// positions and supports by the reference's double expression.
struct F64Args {
    const double* qpos;  // [nq * dim], wrapped as the reference wraps queries
    const double* qsup;  // [nq] or null
    const double* rpos;  // [nr * dim], reference j at row j, wrapped as the reference wraps references
    const double* rsup;  // [nr] or null
    double4* rsorted;    // [nr] the references in the structure's cell order, .w = support
    double ext[3];       // max - min of the domain, in double
    int64_t nq, nr;
};

static F64Walk f64_walk(const F64Args& f) {
    F64Walk w;
    w.qpos = f.qpos;
    w.qsup = f.qsup;
    w.rsorted = f.rsorted;
    for (int d = 0; d < 3; ++d) w.ext[d] = f.ext[d];
    return w;
}

// The double references in cell order (a stencil cell's candidates are one contiguous run), and the
// largest |coordinate| of the double positions (NaN ignored, rounded up) for the band of the float
// test.
__global__ void f64_prep_kernel(const int32_t* __restrict__ rsidx, F64Args f, int dim, QueryParams* qp) {
    float m = 0.0f;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < f.nr; j += stride) {
        const int64_t jl = rsidx[j];
        if (!TCR_GUARD(jl, f.nr)) continue;  // (the build's sort gave up)
        double4 v = make_double4(0.0, 0.0, 0.0, f.rsup ? f.rsup[jl] : 0.0);
        v.x = f.rpos[jl * dim];
        if (dim > 1) v.y = f.rpos[jl * dim + 1];
        if (dim > 2) v.z = f.rpos[jl * dim + 2];
        f.rsorted[j] = v;
        m = fmaxf(m, __double2float_ru(fmax(fabs(v.x), fmax(fabs(v.y), fabs(v.z)))));
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < f.nq * dim; i += stride)
        m = fmaxf(m, __double2float_ru(fabs(f.qpos[i])));
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(&qp->coord_key, float_key(m));
}

// The inputs of a float64 search in one pass: wrapped positions, float32 copies, and the maxima the cell
// size is computed from.  (As torch operations -- a remainder, a difference and a sum per column and
// wrap, stacks, casts and five reductions, each read back by itself -- this was 49 launches and five host
// waits, 390 of 740 us for 150k points.)
__device__ __forceinline__ double wrap_coord64(double x, double lo, double ext) {
    double m = fmod(__dsub_rn(x, lo), ext);
    if (m != 0.0 && ((ext < 0.0) != (m < 0.0))) m = __dadd_rn(m, ext);
    return __dadd_rn(m, lo);
}
// Ordered encoding of doubles (NaN above everything, 0 below everything: no value).
__device__ __forceinline__ unsigned long long double_key(double v) {
    if (v != v) return ~0ull;
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ void block_max_key(unsigned long long k, unsigned long long* out) {
    __shared__ unsigned long long s[32];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, k, o);
        k = other > k ? other : k;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = k;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 1; w < blockDim.x / 32; ++w) k = s[w] > k ? s[w] : k;
        if (k) atomicMax(out, k);
    }
}
__global__ void f64_prepare_kernel(const __grid_constant__ tcr_f64_prepare_desc d) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long* stats = static_cast<unsigned long long*>(d.stats);
    unsigned long long kq = 0, kr = 0, khq = 0, khr = 0;
    for (int64_t i = first; i < d.n_query * d.dim; i += stride) {
        const int c = (int)(i % d.dim);
        const bool per = (d.periodic_mask >> c) & 1;
        const double lo = d.domain_min[c], ext = __dsub_rn(d.domain_max[c], lo);
        double v = d.query_pos[i];
        if (per) v = wrap_coord64(v, lo, ext);
        d.query_wrapped[i] = v;
        d.query_pos_f[i] = __double2float_rn(v);
        kq = max(kq, double_key(fabs(v)));
        if (d.self_search) {
            if (per) v = wrap_coord64(v, lo, ext);
            d.ref_wrapped[i] = v;
            kr = max(kr, double_key(fabs(v)));
        }
    }
    if (!d.self_search && d.ref_pos)
        for (int64_t i = first; i < d.n_ref * d.dim; i += stride) {
            const int c = (int)(i % d.dim);
            const double lo = d.domain_min[c], ext = __dsub_rn(d.domain_max[c], lo);
            double v = d.ref_pos[i];
            if ((d.periodic_mask >> c) & 1) v = wrap_coord64(wrap_coord64(v, lo, ext), lo, ext);
            d.ref_wrapped[i] = v;
            d.ref_pos_f[i] = __double2float_rn(v);
            kr = max(kr, double_key(fabs(v)));
        }
    if (d.query_sup)
        for (int64_t i = first; i < d.n_query; i += stride) {
            const double h = d.query_sup[i];
            if (d.query_sup_f) d.query_sup_f[i] = __double2float_rn(h);
            khq = max(khq, double_key(h));
        }
    if (d.ref_sup)
        for (int64_t i = first; i < d.n_ref; i += stride) {
            const double h = d.ref_sup[i];
            if (d.ref_sup_f) d.ref_sup_f[i] = __double2float_rn(h);
            khr = max(khr, double_key(h));
        }
    block_max_key(kq, &stats[0]);
    block_max_key(kr, &stats[1]);
    block_max_key(khq, &stats[2]);
    block_max_key(khr, &stats[3]);
}
// The keys as doubles (one thread per number).
__global__ void f64_stats_kernel(unsigned long long* stats) {
    const unsigned long long k = stats[threadIdx.x];
    unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    if (k == 0) u = 0xfff0000000000000ull;   // no value: -infinity
    if (k == ~0ull) u = 0x7ff8000000000000ull;
    stats[threadIdx.x] = u;
}

// counts -> offsets (int64, nq+1), optional CSR indptr (int32) and rowEntries (int64).
struct CountIn {
    const int32_t* counts;
    int64_t n;
    __device__ int64_t operator()(int64_t i) const { return i < n ? (int64_t)counts[i] : 0; }
};
struct OffsetOut {
    int64_t n;
    int64_t* offsets;
    int32_t* indptr;
    int64_t* entries;
    // the search's info block, written with the total (element n)
    const int32_t* bad_grids;
    const int32_t* build_failed;
    const int32_t* sort_failed;
    const int32_t* num_stray;
    const int32_t* exact_clouds;
    const unsigned long long* cursor;
    const int32_t* num_flagged;
    const int32_t* num_exact;
    const int32_t* inc_count;
    int64_t n_ref;
    int64_t* info;
    __device__ void operator()(int64_t i, int64_t ex, int64_t v) const {
        offsets[i] = ex;
        if (indptr) indptr[i] = (int32_t)ex;
        if (i < n) {
            if (entries) entries[i] = v;
            return;
        }
        info[0] = ex;
        info[1] = *build_failed || *sort_failed ? -1 : *bad_grids;  // -1: a sort gave up waiting, nothing was searched
        info[2] = *num_stray;
        info[3] = *exact_clouds;
        info[4] = (int64_t)*cursor;
        info[5] = *num_flagged;
        info[6] = min((int64_t)num_exact[0], n) + num_exact[1];
        // incremental build: points sorted by the small sort (-1: the full sort ran); -2: no hint
        info[7] = inc_count ? ((inc_count[1] != 0 || 2 * (int64_t)inc_count[0] < n_ref) ? -1 : n_ref - inc_count[0]) : -2;
    }
};

// ------------------------------------------------------------------------------------------
// host orchestration

// One search as the kernels see it: the cloud table plus what holds for all clouds.
struct HostBatch {
    int32_t C = 0, mode = 0, self = 0, local_index = 0;
    std::vector<CloudParams> clouds;
    int64_t nq = 0, nr = 0, map_total = 0;
    const int32_t* query_ids = nullptr;
    const int32_t* ref_ids = nullptr;
    bool any_query_sup = false, any_ref_sup = false;
    bool same_sorted = false;     // self search, no periodic dims, queries are the references (same arrays)
    bool same_positions = false;  // self search, no periodic dims, same position arrays
    bool same_supports = false;   // self search, the queries' supports are the references' arrays
    int walk_class = 0;           // dim * 2 + (any periodic dim) when every cloud shares it, else 0
    uint32_t class_mask = 0;      // bit cls: some cloud with queries has class cls
    bool wide = false;            // 64-bit (cloud, cell) sort keys
    const int32_t* lin_hint = nullptr;  // incremental build: previous linear cell of every reference point
    int32_t* lin_out = nullptr;         // receives the linear cell of every sorted reference point
    int32_t* order_out = nullptr;       // receives the input index of every sorted reference point
    int unit_cap = kDefaultUnitQueries;           // queries per work unit
    int walk_bps = kDefaultWalkBlocksPerSM;       // blocks per SM of the walk's grid
};

// The descriptors' tuning fields (0: default).
static int take_tuning(HostBatch& b, int32_t unit_queries, int32_t walk_blocks_per_sm) {
    if (unit_queries != 0 && unit_queries != 8 && unit_queries != 16 && unit_queries != 32)
        return set_error(TCR_ERR_INVALID, "unit_queries must be 8, 16 or 32 (0: default 32)");
    if (walk_blocks_per_sm < 0 || walk_blocks_per_sm > 64)
        return set_error(TCR_ERR_INVALID, "walk_blocks_per_sm must be in [1, 64] (0: default 12)");
    b.unit_cap = unit_queries ? unit_queries : kDefaultUnitQueries;
    b.walk_bps = walk_blocks_per_sm ? walk_blocks_per_sm : kDefaultWalkBlocksPerSM;
    return TCR_OK;
}

// Validation shared by both descriptors.  level 0: sizes only; 1: query phases (the reference
// supports come from the structure); 2: structure build.
static int check_cloud(const char* who, int dim, int mode, int64_t L, int64_t nq, int64_t nr, const void* qpos,
                       const void* qsup, const void* rpos, const void* rsup, int self, int level) {
    if (dim < 1 || dim > 3) return set_error(TCR_ERR_INVALID, "%sdim must be 1, 2 or 3 (got %d)", who, dim);
    if (mode < 0 || mode > 3) return set_error(TCR_ERR_INVALID, "%sinvalid mode %d", who, mode);
    if (nq < 0 || nr < 0 || nq > 0x7fffffffLL || nr > 0x7ffffff0LL)
        return set_error(TCR_ERR_INVALID, "%spoint counts must be in [0, 2^31)", who);
    if (self && nq != nr) return set_error(TCR_ERR_INVALID, "%sself search needs one cloud", who);
    if (level == 0) return TCR_OK;
    if (L <= 0 || L > 0xffffffffLL) return set_error(TCR_ERR_INVALID, "%shashMapLength must be in [1, 2^32)", who);
    if ((nq && !qpos) || (nr && !rpos)) return set_error(TCR_ERR_INVALID, "%smissing positions", who);
    if ((mode == kGather || mode == kSymmetric || mode == kSuperSymmetric) && nq && !qsup)
        return set_error(TCR_ERR_INVALID, "%sthis mode needs query supports", who);
    if (level >= 2 && (mode == kScatter || mode == kSymmetric || mode == kSuperSymmetric) && nr && !rsup)
        return set_error(TCR_ERR_INVALID, "%sthis mode needs reference supports", who);
    return TCR_OK;
}

static int finish_batch(HostBatch& b, int64_t map_min) {
    int64_t qb = 0, rb = 0, mb = 0;
    bool same_pos = b.self != 0, same_sorted = b.self != 0, same_sup = b.self != 0;
    int cls = -1;
    bool mixed = false;
    b.any_query_sup = b.any_ref_sup = false;
    b.class_mask = 0;
    for (CloudParams& cp : b.clouds) {
        cp.query_base = (int32_t)qb;
        cp.ref_base = (int32_t)rb;
        qb += cp.n_query;
        rb += cp.n_ref;
        if (qb > 0x7ffffff0LL || rb > 0x7ffffff0LL)
            return set_error(TCR_ERR_INVALID, "the clouds hold more than 2^31 query or reference points");
        cp.map_cap = hash_capacity(cp.n_ref, map_min);
        cp.map_base = mb;
        mb += cp.map_cap;
        same_pos = same_pos && cp.periodic_mask == 0 && cp.query_pos == cp.ref_pos;
        same_sorted = same_sorted && cp.periodic_mask == 0 && cp.query_pos == cp.ref_pos && cp.query_sup == cp.ref_sup;
        same_sup = same_sup && cp.query_sup == cp.ref_sup;
        b.any_query_sup = b.any_query_sup || cp.query_sup != nullptr;
        b.any_ref_sup = b.any_ref_sup || cp.ref_sup != nullptr;
        const int c = cp.dim * 2 + (cp.periodic_mask != 0 ? 1 : 0);
        if (cls < 0) cls = c;
        else if (c != cls) mixed = true;
        if (cp.n_query > 0) b.class_mask |= 1u << c;
    }
    b.nq = qb;
    b.nr = rb;
    b.map_total = mb;
    b.same_positions = same_pos;
    b.same_sorted = same_sorted;
    b.same_supports = same_sup;
    b.walk_class = mixed ? 0 : cls;
    b.wide = b.C > 1;
    return TCR_OK;
}

static void fill_domain(CloudParams& cp, int dim, const float* lo, const float* hi) {
    for (int k = 0; k < 3; ++k) {
        cp.dmin[k] = k < dim ? lo[k] : 0.f;
        cp.dmax[k] = k < dim ? hi[k] : 1.f;
        cp.ext[k] = cp.dmax[k] - cp.dmin[k];
    }
}

static int batch_of_desc(const tcr_search_desc* d, int level, HostBatch& b) {
    if (!d) return set_error(TCR_ERR_INVALID, "null descriptor");
    int rc = check_cloud("", d->dim, d->mode, d->hash_map_length, d->n_query, d->n_ref, d->query_pos, d->query_sup,
                         d->ref_pos, d->ref_sup, d->self_search, level);
    if (rc) return rc;
    if (d->hcell[0] > 0.0f)
        for (int k = 0; k < d->dim; ++k)
            if (!(d->hcell[k] > 0.0f) || !(d->hcell[k] < 3.0e38f))
                return set_error(TCR_ERR_INVALID, "cell size override must be positive and finite in every dimension");
    CloudParams cp;
    memset(&cp, 0, sizeof(cp));
    cp.dim = d->dim;
    cp.mode = d->mode;
    cp.periodic_mask = d->periodic_mask;
    cp.hash_len = (uint32_t)d->hash_map_length;
    fill_domain(cp, d->dim, d->domain_min, d->domain_max);
    for (int k = 0; k < 3; ++k) cp.hcell_override[k] = d->hcell[0] > 0.0f ? (k < d->dim ? d->hcell[k] : 1.0f) : 0.0f;
    cp.dedupe = d->clamped_grid ? 1 : 0;
    cp.n_query = (int32_t)d->n_query;
    cp.n_ref = (int32_t)d->n_ref;
    cp.query_pos = d->query_pos;
    cp.query_sup = d->query_sup;
    cp.ref_pos = d->ref_pos;
    cp.ref_sup = d->ref_sup;
    b = HostBatch();
    b.C = 1;
    b.mode = d->mode;
    b.self = d->self_search ? 1 : 0;
    b.query_ids = d->query_ids;
    b.ref_ids = d->ref_ids;
    b.clouds.push_back(cp);
    if ((rc = take_tuning(b, d->unit_queries, d->walk_blocks_per_sm))) return rc;
    return finish_batch(b, kSingleMapMin);
}

static int batch_of(const tcr_batch_desc* bd, int level, HostBatch& b) {
    if (!bd) return set_error(TCR_ERR_INVALID, "null batch descriptor");
    if (bd->n_clouds < 1 || bd->n_clouds > (1 << 22))
        return set_error(TCR_ERR_INVALID, "n_clouds must be in [1, 2^22] (got %d)", bd->n_clouds);
    if (!bd->clouds) return set_error(TCR_ERR_INVALID, "missing cloud table");
    b = HostBatch();
    b.C = bd->n_clouds;
    b.mode = bd->mode;
    b.self = bd->self_search ? 1 : 0;
    b.local_index = bd->local_index ? 1 : 0;
    b.query_ids = bd->query_ids;
    b.ref_ids = bd->ref_ids;
    b.lin_hint = bd->ref_lin_hint;
    b.lin_out = bd->ref_lin_out;
    b.order_out = bd->ref_order_out;
    b.clouds.resize(bd->n_clouds);
    if (int rc = take_tuning(b, bd->unit_queries, bd->walk_blocks_per_sm)) return rc;
    char who[48];
    for (int k = 0; k < bd->n_clouds; ++k) {
        const tcr_cloud_desc& c = bd->clouds[k];
        snprintf(who, sizeof(who), "cloud %d: ", k);
        int rc = check_cloud(who, c.dim, bd->mode, c.hash_map_length, c.n_query, c.n_ref, c.query_pos, c.query_sup,
                             c.ref_pos, c.ref_sup, bd->self_search, level);
        if (rc) return rc;
        if (level >= 1 && c.hcell[0] > 0.0f)
            for (int d = 0; d < c.dim; ++d)
                if (!(c.hcell[d] > 0.0f) || !(c.hcell[d] < 3.0e38f))
                    return set_error(TCR_ERR_INVALID, "%scell size override must be positive and finite", who);
        CloudParams& cp = b.clouds[k];
        memset(&cp, 0, sizeof(cp));
        cp.dim = c.dim;
        cp.mode = bd->mode;
        cp.periodic_mask = c.periodic_mask & ((1 << c.dim) - 1);
        for (int d = 0; d < 3; ++d) cp.hcell_override[d] = c.hcell[0] > 0.0f ? (d < c.dim ? c.hcell[d] : 1.0f) : 0.0f;
        cp.dedupe = c.clamped_grid ? 1 : 0;
        cp.hash_len = (uint32_t)c.hash_map_length;
        fill_domain(cp, c.dim, c.domain_min, c.domain_max);
        cp.n_query = (int32_t)c.n_query;
        cp.n_ref = (int32_t)c.n_ref;
        cp.query_pos = c.query_pos;
        cp.query_sup = c.query_sup;
        cp.ref_pos = c.ref_pos;
        cp.ref_sup = c.ref_sup;
    }
    return finish_batch(b, kBatchMapMin);
}

static void batch_sizes(const HostBatch& b, int64_t* s, int64_t* w) {
    if (s) carve_structure(nullptr, b.nr, b.C, b.map_total, s);
    if (w) carve_scratch(nullptr, b.nq, b.nr, b.C, b.lin_hint != nullptr, w);
}

static inline unsigned grid_for(int64_t n, int threads, int max_blocks = 148 * 16) {
    int64_t b = (n + threads - 1) / threads;
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(b, max_blocks));
}

static int num_sms() {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

// Optional per-launch timing of the two heaviest kernels (count walk, record expansion): events
// recorded around the launch on its own stream; read back with tcr_profile_kernel_ms.
static std::mutex g_prof_mu;
static int g_prof_on = 0;
static int g_prof_dev = -1;
static cudaEvent_t g_prof_ev[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
static int g_prof_recorded[2] = {0, 0};

static void prof_mark(int kernel, int end, cudaStream_t st) {
    if (!g_prof_on) return;
    std::lock_guard<std::mutex> lk(g_prof_mu);
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != g_prof_dev) return;
    // External: under stream capture the record becomes an event node of the graph, so replays
    // of a recorded search time the kernel too
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) return;
    const unsigned flags = cs == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : cudaEventRecordDefault;
    if (cudaEventRecordWithFlags(g_prof_ev[kernel][end], st, flags) == cudaSuccess && end) g_prof_recorded[kernel] = 1;
}

template <int N>
static CloudChunk<N> cloud_chunk(const HostBatch& b, int first, int count) {
    CloudChunk<N> ch;
    ch.first = first;
    ch.count = count;
    ch.n_clouds = b.C;
    ch.query_total = (int32_t)b.nq;
    ch.ref_total = (int32_t)b.nr;
    ch.pad = 0;
    memcpy(ch.p, &b.clouds[first], sizeof(CloudParams) * count);
    return ch;
}
// Uploads all but the table's last chunk, which is returned for the phase's init kernel.
static int upload_table(const HostBatch& b, const Scratch& W, cudaStream_t st, CloudChunk<kUploadChunk>& last) {
    const int tail = b.C <= kUploadChunk ? b.C : 1, before = b.C - tail;
    for (int first = 0; first < before; first += kWideChunk) {
        const int count = std::min(kWideChunk, before - first);
        upload_clouds_kernel<<<(count + kUploadPerBlock - 1) / kUploadPerBlock, 32, 0, st>>>(
            cloud_chunk<kWideChunk>(b, first, count), W.table, W.query_prefix, W.ref_prefix);
        note_launches(1);
    }
    last = cloud_chunk<kUploadChunk>(b, before, tail);
    TCR_CUDA(cudaGetLastError());
    return TCR_OK;
}

static WalkArgs make_walk(const HostBatch& b, const Structure& S, const Scratch& W) {
    WalkArgs a;
    memset(&a, 0, sizeof(a));
    a.table = W.table;
    a.grid = S.grid;
    a.qparams = W.qparams;
    a.query_prefix = W.query_prefix;
    a.num_clouds = b.C;
    a.local_index = b.local_index;
    a.mode = b.mode;
    a.no_stray_check = b.same_positions ? 1 : 0;
    a.self = b.self;
    a.rsorted = S.rsorted;
    a.rsidx = S.rsidx;
    a.cell_start = S.cell_start;
    a.cell_bucket = S.cell_bucket;
    a.map = S.map;
    a.qsorted = b.same_sorted ? S.rsorted : W.qsorted;
    a.qsidx = b.same_sorted ? S.rsidx : W.qsidx;
    a.group_start = b.self ? S.cell_start : W.qgroup_start;
    a.group_coords = b.self ? S.cell_coords : W.qgroup_coords;
    a.group_cloud = b.self ? S.cell_cloud : W.qgroup_cloud;
    a.unit_group = W.unit_group;
    a.unit_t0 = W.unit_t0;
    a.num_units = W.num_units;
    a.unit_cap = W.unit_cap;
    a.unit_list = W.flagged;
    a.num_list = W.num_flagged;
    a.work = W.work;
    a.stray = W.stray;
    a.num_stray = W.num_stray;
    a.counts = W.counts;
    a.rec = W.rec;
    a.flagged = W.flagged;
    a.num_flagged = W.num_flagged;
    a.num_exact = W.num_exact;
    a.exact_clouds = W.exact_clouds;
    a.band_pairs = reinterpret_cast<int4*>(W.pack);  // the packed points are sorted away by now
    a.band_windows = reinterpret_cast<unsigned long long*>(W.keys[1]);  // and so are the keys
    a.band_cap = std::max(b.nq, b.nr);
    a.cursor = W.cursor;
    a.query_ids = b.query_ids;
    a.ref_ids = b.ref_ids;
    a.nq_total = b.nq;
    a.nr_total = b.nr;
    return a;
}

// Dispatches a walk kernel template on a cloud class (dim * 2 + any periodic dim) and the mode.
template <template <int, bool, int> class L>
static cudaError_t dispatch_walk(const WalkArgs& a, int cls, int mode, dim3 grid, dim3 block, size_t smem,
                                 cudaStream_t st) {
#define TCR_M(D, P)                                                                    \
    switch (mode) {                                                                    \
        case kGather: return L<D, P, kGather>::launch(a, grid, block, smem, st);       \
        case kScatter: return L<D, P, kScatter>::launch(a, grid, block, smem, st);     \
        case kSymmetric: return L<D, P, kSymmetric>::launch(a, grid, block, smem, st); \
        default: return L<D, P, kSuperSymmetric>::launch(a, grid, block, smem, st);    \
    }
    switch (cls) {
        case 2: TCR_M(1, false)
        case 3: TCR_M(1, true)
        case 4: TCR_M(2, false)
        case 5: TCR_M(2, true)
        case 6: TCR_M(3, false)
        default: TCR_M(3, true)
    }
#undef TCR_M
}

// Raises a kernel's dynamic shared memory limit once per device (not a stream operation, so a
// search can be recorded into a CUDA graph after its first eager run).
template <typename F>
static cudaError_t ensure_smem(F* kernel, int bytes, uint64_t* done_mask) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (__atomic_load_n(done_mask, __ATOMIC_ACQUIRE) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) __atomic_fetch_or(done_mask, bit, __ATOMIC_ACQ_REL);
    return e;
}

template <int D, bool P, int M>
struct CountLaunch {
    static cudaError_t launch(const WalkArgs& a, dim3 g, dim3 b, size_t, cudaStream_t st) {
        walk_count_kernel<D, P, M><<<g, b, 0, st>>>(a);
        return cudaGetLastError();
    }
};
template <int D, bool P, int M>
struct EmitLaunch {
    static cudaError_t launch(const WalkArgs& a, dim3 g, dim3 b, size_t, cudaStream_t st) {
        walk_emit_kernel<D, P, M><<<g, b, 0, st>>>(a);
        return cudaGetLastError();
    }
};

// One walk launch for a batch of one class; one per class present (each filtering its units)
// when the clouds mix classes.
template <template <int, bool, int> class L>
static cudaError_t launch_walks(const HostBatch& b, WalkArgs a, dim3 grid, dim3 block, size_t smem,
                                cudaStream_t st) {
    if (b.walk_class != 0) {
        a.class_filter = -1;
        note_launches(1);
        return dispatch_walk<L>(a, b.walk_class, b.mode, grid, block, smem, st);
    }
    for (int cls = 2; cls <= 7; ++cls) {
        if (!((b.class_mask >> cls) & 1)) continue;
        a.class_filter = cls;
        note_launches(1);
        cudaError_t e = dispatch_walk<L>(a, cls, b.mode, grid, block, smem, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Persistent walk grid: the blocks loop over units through an atomic counter, so the size only
// sets the parallelism -- about two units per query group's worth of full units per warp.
static unsigned walk_blocks(const HostBatch& b, int64_t nq) {
    const int64_t max_units = 2 * nq / b.unit_cap + 1;
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)num_sms() * b.walk_bps,
                                                            (max_units + kWalkWarps - 1) / kWalkWarps));
}

template <typename K>
static int build_impl(const HostBatch& b, const Structure& S, const Scratch& W, cudaStream_t st) {
    const SortWorkspaceT<K> sw = sort_workspace<K>(W);
    const int C = b.C;
    const int64_t nr = b.nr, nq = b.nq;
    CloudChunk<kUploadChunk> chunk;
    int rc = upload_table(b, W, st, chunk);
    if (rc) return rc;
    grid_init_kernel<K><<<grid_for(std::max<int64_t>(C, S.map_total / 8), 256, num_sms() * 8), 256, 0, st>>>(
        chunk, S.grid, C, S, W);
    note_launches(1);
    // computeGridSupport: which supports set hMax depends on the mode; the last statistics also write the
    // grid parameters
    const bool ref_stats = b.any_ref_sup && nr > 0, query_stats = b.any_query_sup && nq > 0 && !b.same_supports;
    const int same_sup = b.same_supports ? 1 : 0;
    if (ref_stats) {
        support_stats_kernel<<<grid_for(nr, 256, num_sms() * 4), 256, 0, st>>>(
            W.table, W.ref_prefix, C, nr, 0, reinterpret_cast<char*>(S.grid) + offsetof(GridParams, ref_stats),
            (int64_t)sizeof(GridParams), S.grid, S.bad_grids, same_sup, query_stats ? nullptr : S.num_cells + 2);
        note_launches(1);
    }
    if (query_stats) {
        support_stats_kernel<<<grid_for(nq, 256, num_sms() * 4), 256, 0, st>>>(
            W.table, W.query_prefix, C, nq, 1,
            reinterpret_cast<char*>(S.grid) + offsetof(GridParams, build_query_stats), (int64_t)sizeof(GridParams),
            S.grid, S.bad_grids, same_sup, S.num_cells + 2);
        note_launches(1);
    }
    if (!ref_stats && !query_stats) {
        grid_params_kernel<<<grid_for(C, 128), 128, 0, st>>>(W.table, S.grid, C, S.bad_grids, same_sup);
        note_launches(1);
    }
    if (nr > 0) {
        const bool inc = b.lin_hint != nullptr;
        // few blocks: each ends with one atomic on the key range, so thousands of them would queue
        pack_points_kernel<K><<<grid_for(nr, 256, num_sms() * 4), 256, 0, st>>>(
            W.table, S.grid, W.ref_prefix, C, nr, 0, 2, 1, W.pack, sw.keys[0], sw.vals[0], sw.state,
            inc ? b.lin_hint : nullptr, inc ? W.stay : nullptr);
        note_launches(1);
        if (inc) {
            SortWorkspaceT<K> mw = sw;
            mw.keys[0] = reinterpret_cast<K*>(W.moved_keys[0]);
            mw.keys[1] = reinterpret_cast<K*>(W.moved_keys[1]);
            mw.vals[0] = W.moved_vals[0];
            mw.vals[1] = W.moved_vals[1];
            mw.state = reinterpret_cast<SortStateT<K>*>(W.moved_state);
            TCR_CUDA(cudaMemsetAsync(W.inc_count, 0, 2 * sizeof(int32_t), st));
            StayOut<K> so{sw.keys[0], reinterpret_cast<K*>(W.stay_keys), W.stay_idx, mw.keys[0], mw.vals[0]};
            TCR_CUDA(device_exclusive_scan<int32_t>(StayIn{W.stay}, so, nr, W.scan_tiles32, W.inc_count, st));
            inc_check_kernel<K><<<grid_for(nr, 256), 256, 0, st>>>(reinterpret_cast<const K*>(W.stay_keys),
                                                                   W.inc_count, W.inc_count + 1);
            inc_decide_kernel<K><<<1, 1, 0, st>>>(sw.state, mw.state, W.inc_count, nr);
            note_launches(2);
            TCR_CUDA(sort_coop<K>(mw, nr, S.num_cells + 1, 0, NoTail(), st));
            inc_merge_kernel<K><<<grid_for(nr, 256), 256, 0, st>>>(
                reinterpret_cast<const K*>(W.stay_keys), W.stay_idx, mw.keys[0], mw.keys[1], mw.vals[0], mw.vals[1],
                mw.state, W.inc_count, nr, sw.keys[0], sw.vals[0]);
            note_launches(1);
        }
        TCR_CUDA(sort_coop<K>(sw, nr, S.num_cells + 1, inc ? 1 : 0,
                              BuildTail<K>{S.cell_start, S.num_cells, W.pack, S.rsorted, S.rsidx, b.lin_out, b.order_out,
                                           W.table, S.grid, S.cell_lin, S.cell_coords, S.cell_bucket, S.cell_cloud,
                                           S.map, nr},
                              st));
        if (b.lin_out || b.order_out) {
            abandoned_order_kernel<<<grid_for(nr, 256, num_sms()), 256, 0, st>>>(S.num_cells + 1, nr, b.lin_hint,
                                                                               b.lin_out, b.order_out);
            note_launches(1);
        }
    } else {
        finish_cells_kernel<<<1, 1, 0, st>>>(S.cell_start, S.num_cells, nr);
        note_launches(1);
    }
    TCR_CUDA(cudaGetLastError());
    return TCR_OK;
}

template <typename K>
static int count_impl(const HostBatch& b, const Structure& S, const Scratch& W, int32_t* stage, int64_t stage_cap,
                      int64_t* offsets, int32_t* indptr_out, int64_t* row_entries_out, int64_t* info_out,
                      cudaStream_t st, const F64Args* f64) {
    const int C = b.C;
    const int64_t nq = b.nq;
    CloudChunk<kUploadChunk> chunk;
    int rc = upload_table(b, W, st, chunk);
    if (rc) return rc;
    const int unit_cap = b.unit_cap;
    // The query supports' statistics: the structure's where the queries are its sorted points themselves, with
    // the packing of other self searches, else by a launch of their own.
    const bool packed = b.self && !b.same_sorted && nq > 0;
    count_init_kernel<<<grid_for(std::max<int64_t>(C, nq), 256), 256, 0, st>>>(chunk, S.grid, W, C, unit_cap, nq, stage_cap,
                                                                               b.same_sorted ? 1 : 0);
    note_launches(1);
    if (b.any_query_sup && nq > 0 && !b.self) {
        support_stats_kernel<<<grid_for(nq, 256, num_sms() * 4), 256, 0, st>>>(
            W.table, W.query_prefix, C, nq, 1, reinterpret_cast<char*>(W.qparams) + offsetof(QueryParams, stats),
            (int64_t)sizeof(QueryParams));
        note_launches(1);
    }
    if (f64 && (b.nr > 0 || nq > 0)) {
        f64_prep_kernel<<<grid_for(std::max<int64_t>(b.nr, nq * b.clouds[0].dim), 256), 256, 0, st>>>(
            S.rsidx, *f64, b.clouds[0].dim, W.qparams);
        note_launches(1);
    }
    if (nq > 0) {
        const int32_t* gstart;
        const int32_t* ngroups;
        if (b.self) {
            if (packed) {
                pack_self_queries_kernel<<<grid_for(nq, 256), 256, 0, st>>>(
                    W.table, S.grid, W.query_prefix, C, S.rsidx, nq, W.qsorted, W.qsidx, W.qparams);
                note_launches(1);
            }
            gstart = S.cell_start;
            ngroups = S.num_cells;
        } else {
            // sort the queries by their own (cloud, cell)
            const SortWorkspaceT<K> sw = sort_workspace<K>(W);
            sort_state_init_kernel<K><<<1, 1, 0, st>>>(sw.state);
            note_launches(1);
            pack_points_kernel<K><<<grid_for(nq, 256, num_sms() * 4), 256, 0, st>>>(
                W.table, S.grid, W.query_prefix, C, nq, 1, 1, 0, W.pack, sw.keys[0], sw.vals[0], sw.state);
            note_launches(1);
            TCR_CUDA(sort_coop<K>(sw, nq, W.num_qgroups + 1, 0,
                                  QueryTail<K>{W.qgroup_start, W.num_qgroups, W.pack, W.qsorted, W.qsidx, W.table,
                                               S.grid, W.qgroup_coords, W.qgroup_cloud, nq},
                                  st));
            gstart = W.qgroup_start;
            ngroups = W.num_qgroups;
        }
        BoundedUnitCountIn ui{gstart, ngroups, unit_cap, S.num_cells + 1, W.num_qgroups + 1};
        BoundedUnitOut uo{gstart, W.unit_group, W.unit_t0, unit_cap, nq};
        TCR_CUDA(device_exclusive_scan<int32_t>(ui, uo, nq, W.scan_tiles32, W.num_units, st));
        WalkArgs a = make_walk(b, S, W);
        if (f64) a.f64 = f64_walk(*f64);
        a.stage = stage;
        a.stage_cap = stage_cap;
        prof_mark(TCR_PROFILE_COUNT_WALK, 0, st);
        TCR_CUDA(launch_walks<CountLaunch>(b, a, dim3(walk_blocks(b, nq)), dim3(kWalkWarps * 32), 0, st));
        prof_mark(TCR_PROFILE_COUNT_WALK, 1, st);
        stray_kernel<false><<<grid_for(nq, 128, num_sms() * kStrayBlocks), kWalkWarps * 32, 0, st>>>(a);
        note_launches(1);
    }
    CountIn ci{W.counts, nq};
    OffsetOut oo{nq, offsets, indptr_out, row_entries_out, S.bad_grids, S.num_cells + 1, W.num_qgroups + 1, W.num_stray, W.exact_clouds, W.cursor,
                 W.num_flagged, W.num_exact, b.lin_hint && b.nr > 0 ? W.inc_count : nullptr, b.nr, W.info};
    TCR_CUDA(device_exclusive_scan<int64_t>(ci, oo, nq + 1, W.scan_tiles64, W.total, st));
    if (info_out) TCR_CUDA(cudaMemcpyAsync(info_out, W.info, 8 * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    return TCR_OK;
}

static int emit_impl(const HostBatch& b, const Structure& S, const Scratch& W, const int32_t* stage,
                     const int64_t* offsets, int64_t* row_out, int64_t* col_out, int64_t out_capacity,
                     cudaStream_t st, const F64Args* f64) {
    const int64_t nq = b.nq;
    if (out_capacity < 0 || (out_capacity > 0 && !col_out)) return set_error(TCR_ERR_INVALID, "bad output buffer");
    if (nq <= 0) return TCR_OK;
    WalkArgs a = make_walk(b, S, W);
    if (f64) a.f64 = f64_walk(*f64);
    a.offsets = offsets;
    a.row_out = row_out;
    a.col_out = col_out;
    a.out_cap = out_capacity;
    if (stage) {
        const int nsm = num_sms();
        // resident blocks (four an SM), no more than about two units per query group's worth of full ones
        const unsigned blocks = (unsigned)std::max<int64_t>(
            1, std::min<int64_t>((int64_t)nsm * 4, (2 * nq / b.unit_cap + kExpandWarps) / kExpandWarps));
        ExpandArgs e;
        e.stage = stage;
        e.rec = W.rec;
        e.num_units = W.num_units;
        e.unit_t0 = W.unit_t0;
        e.unit_group = W.unit_group;
        e.group_cloud = a.group_cloud;
        e.qsidx = a.qsidx;
        e.col_of = S.rsidx;
        if (b.ref_ids && b.nr > 0) {  // (the sort's values are spent by now)
            compose_ids_kernel<<<grid_for(b.nr, 256), 256, 0, st>>>(S.rsidx, b.ref_ids, b.nr, W.vals[0]);
            note_launches(1);
            e.col_of = W.vals[0];
        }
        e.offsets = offsets;
        e.query_ids = b.query_ids;
        e.composed = b.ref_ids ? 1 : 0;
        e.table = W.table;
        e.num_clouds = b.C;
        e.local_index = b.local_index;
        e.row_out = row_out;
        e.col_out = col_out;
        e.out_cap = out_capacity;
        e.work = W.work + kExpandCounter;
        e.stage_cap = W.cursor + 1;
        e.nq = nq;
        e.nr = b.nr;
        static uint64_t expand_attr_done = 0;
        TCR_CUDA(ensure_smem(expand_records_kernel, (int)sizeof(ExpandSmem), &expand_attr_done));
        prof_mark(TCR_PROFILE_EXPAND, 0, st);
        expand_records_kernel<<<blocks, kExpandWarps * 32, sizeof(ExpandSmem), st>>>(e);
        prof_mark(TCR_PROFILE_EXPAND, 1, st);
        note_launches(1);
    }
    TCR_CUDA(launch_walks<EmitLaunch>(b, a, dim3(walk_blocks(b, nq)), dim3(kWalkWarps * 32), 0, st));
    stray_kernel<true><<<grid_for(nq, 128, num_sms() * 4), kWalkWarps * 32, 0, st>>>(a);
    note_launches(1);
    return TCR_OK;
}

static int run_build(const HostBatch& b, void* structure, int64_t structure_bytes, void* scratch,
                     int64_t scratch_bytes, void* stream) {
    int64_t need_s = 0, need_w = 0;
    batch_sizes(b, &need_s, &need_w);
    if (!structure || !scratch || structure_bytes < need_s || scratch_bytes < need_w)
        return set_error(TCR_ERR_INVALID, "workspace too small (structure %lld/%lld, scratch %lld/%lld)",
                         (long long)structure_bytes, (long long)need_s, (long long)scratch_bytes, (long long)need_w);
    const Structure S = carve_structure(structure, b.nr, b.C, b.map_total, nullptr);
    const Scratch W = carve_scratch(scratch, b.nq, b.nr, b.C, b.lin_hint != nullptr, nullptr);
    cudaStream_t st = (cudaStream_t)stream;
    return b.wide ? build_impl<unsigned long long>(b, S, W, st) : build_impl<uint32_t>(b, S, W, st);
}

static int run_count(const HostBatch& b, const void* structure, void* scratch, int64_t scratch_bytes, int32_t* stage,
                     int64_t stage_capacity, int64_t* offsets, int32_t* indptr_out, int64_t* row_entries_out,
                     int64_t* info_out, void* stream, const F64Args* f64 = nullptr) {
    int64_t need_w = 0;
    batch_sizes(b, nullptr, &need_w);
    if (!structure || !scratch || scratch_bytes < need_w || !offsets)
        return set_error(TCR_ERR_INVALID, "workspace too small or offsets missing");
    if (stage_capacity < 0 || stage_capacity > 0x7fffffffLL || (stage_capacity > 0 && !stage))
        return set_error(TCR_ERR_INVALID, "stage capacity must be in [0, 2^31) with a buffer");
    const Structure S = carve_structure(const_cast<void*>(structure), b.nr, b.C, b.map_total, nullptr);
    const Scratch W = carve_scratch(scratch, b.nq, b.nr, b.C, b.lin_hint != nullptr, nullptr);
    cudaStream_t st = (cudaStream_t)stream;
    return b.wide ? count_impl<unsigned long long>(b, S, W, stage, stage_capacity, offsets, indptr_out,
                                                   row_entries_out, info_out, st, f64)
                  : count_impl<uint32_t>(b, S, W, stage, stage_capacity, offsets, indptr_out, row_entries_out,
                                         info_out, st, f64);
}

static int run_emit(const HostBatch& b, const void* structure, void* scratch, int64_t scratch_bytes,
                    const int32_t* stage, const int64_t* offsets, int64_t* row_out, int64_t* col_out,
                    int64_t out_capacity, void* stream, const F64Args* f64 = nullptr) {
    int64_t need_w = 0;
    batch_sizes(b, nullptr, &need_w);
    if (!structure || !scratch || scratch_bytes < need_w || !offsets)
        return set_error(TCR_ERR_INVALID, "workspace too small or offsets missing");
    const Structure S = carve_structure(const_cast<void*>(structure), b.nr, b.C, b.map_total, nullptr);
    const Scratch W = carve_scratch(scratch, b.nq, b.nr, b.C, b.lin_hint != nullptr, nullptr);
    return emit_impl(b, S, W, stage, offsets, row_out, col_out, out_capacity, (cudaStream_t)stream, f64);
}

}  // namespace tcr

using namespace tcr;

extern "C" {

const char* tcr_last_error(void) { return g_err; }

int tcr_version(void) { return TCR_ABI_VERSION; }

int64_t tcr_desc_bytes(void) { return (int64_t)sizeof(tcr_search_desc); }

int64_t tcr_cloud_desc_bytes(void) { return (int64_t)sizeof(tcr_cloud_desc); }

int64_t tcr_batch_desc_bytes(void) { return (int64_t)sizeof(tcr_batch_desc); }

int64_t tcr_kernel_launches(void) { return (int64_t)__atomic_load_n(&g_launches, __ATOMIC_RELAXED); }

int tcr_profile_kernels(int32_t enable) {
    std::lock_guard<std::mutex> lk(g_prof_mu);
    if (!enable) {
        g_prof_on = 0;
        return TCR_OK;
    }
    int dev = 0;
    TCR_CUDA(cudaGetDevice(&dev));
    if (dev != g_prof_dev) {
        for (auto& pair : g_prof_ev)
            for (auto& e : pair) {
                if (e) cudaEventDestroy(e);
                e = nullptr;
            }
        for (auto& pair : g_prof_ev)
            for (auto& e : pair) TCR_CUDA(cudaEventCreate(&e));
        g_prof_dev = dev;
    }
    g_prof_recorded[0] = g_prof_recorded[1] = 0;
    g_prof_on = 1;
    return TCR_OK;
}

int tcr_profile_kernel_ms(int32_t kernel, float* ms) {
    if (kernel < 0 || kernel > 1 || !ms) return set_error(TCR_ERR_INVALID, "invalid kernel id or output");
    std::lock_guard<std::mutex> lk(g_prof_mu);
    if (!g_prof_recorded[kernel]) return set_error(TCR_ERR_INVALID, "no profiled launch of kernel %d", kernel);
    TCR_CUDA(cudaEventSynchronize(g_prof_ev[kernel][1]));
    TCR_CUDA(cudaEventElapsedTime(ms, g_prof_ev[kernel][0], g_prof_ev[kernel][1]));
    return TCR_OK;
}

#ifdef TCR_CHECKED
// Checked build only: the first failed bounds check (source line, index, bound), then cleared.
int tcr_debug_checks(int64_t* out3) {
    unsigned long long h[3] = {0, 0, 0};
    TCR_CUDA(cudaMemcpyFromSymbol(h, g_check, sizeof(h)));
    const unsigned long long z[3] = {0, 0, 0};
    TCR_CUDA(cudaMemcpyToSymbol(g_check, z, sizeof(z)));
    for (int k = 0; k < 3; ++k) out3[k] = (int64_t)h[k];
    return TCR_OK;
}
#endif

int tcr_search_sizes(int64_t n_query, int64_t n_ref, int32_t dim, int64_t* structure_bytes, int64_t* scratch_bytes) {
    if (dim < 1 || dim > 3 || n_query < 0 || n_ref < 0) return set_error(TCR_ERR_INVALID, "invalid sizes");
    if (structure_bytes) carve_structure(nullptr, n_ref, 1, hash_capacity(n_ref, kSingleMapMin), structure_bytes);
    if (scratch_bytes) carve_scratch(nullptr, n_query, n_ref, 1, false, scratch_bytes);
    return TCR_OK;
}

int tcr_structure_offsets(int64_t n_ref, int64_t* offsets, int32_t n) {
    if (n_ref < 0 || !offsets || n < TCR_STRUCT_NFIELDS) return set_error(TCR_ERR_INVALID, "invalid arguments");
    char* const base = reinterpret_cast<char*>(256);  // any non-null base; offsets are relative
    const Structure s = carve_structure(base, n_ref, 1, hash_capacity(n_ref, kSingleMapMin), nullptr);
    auto off = [&](const void* p) { return (int64_t)((const char*)p - base); };
    offsets[TCR_STRUCT_GRID] = off(s.grid);
    offsets[TCR_STRUCT_NUM_CELLS] = off(s.num_cells);
    offsets[TCR_STRUCT_SORTED_POINTS] = off(s.rsorted);
    offsets[TCR_STRUCT_SORT_INDEX] = off(s.rsidx);
    offsets[TCR_STRUCT_CELL_START] = off(s.cell_start);
    offsets[TCR_STRUCT_CELL_LIN] = off(s.cell_lin);
    offsets[TCR_STRUCT_CELL_COORDS] = off(s.cell_coords);
    offsets[TCR_STRUCT_CELL_BUCKET] = off(s.cell_bucket);
    offsets[TCR_STRUCT_MAP] = off(s.map);
    offsets[TCR_STRUCT_MAP_CAPACITY] = s.map_total;
    return TCR_OK;
}

int tcr_build_structure(const tcr_search_desc* d, void* structure, int64_t structure_bytes, void* scratch,
                        int64_t scratch_bytes, void* stream) {
    NvtxRange nvtx_("tcr_build_structure");
    HostBatch b;
    int rc = batch_of_desc(d, 2, b);
    if (rc) return rc;
    return run_build(b, structure, structure_bytes, scratch, scratch_bytes, stream);
}

int tcr_count(const tcr_search_desc* d, const void* structure, void* scratch, int64_t scratch_bytes, int32_t* stage,
              int64_t stage_capacity, int64_t* offsets, int32_t* indptr_out, int64_t* row_entries_out, int64_t* info_out,
              void* stream) {
    NvtxRange nvtx_("tcr_count");
    HostBatch b;
    int rc = batch_of_desc(d, 1, b);
    if (rc) return rc;
    return run_count(b, structure, scratch, scratch_bytes, stage, stage_capacity, offsets, indptr_out, row_entries_out,
                     info_out, stream);
}

int tcr_emit(const tcr_search_desc* d, const void* structure, void* scratch, int64_t scratch_bytes,
             const int32_t* stage, const int64_t* offsets, int64_t* row_out, int64_t* col_out, int64_t out_capacity,
             void* stream) {
    NvtxRange nvtx_("tcr_emit");
    HostBatch b;
    int rc = batch_of_desc(d, 1, b);
    if (rc) return rc;
    return run_emit(b, structure, scratch, scratch_bytes, stage, offsets, row_out, col_out, out_capacity, stream);
}

static int f64_args(const tcr_search_desc* d, const tcr_f64_inputs* in, F64Args& f) {
    if (!in) return set_error(TCR_ERR_INVALID, "missing float64 inputs");
    if ((d->n_query > 0 && !in->query_pos) || (d->n_ref > 0 && (!in->ref_pos || !in->ref_sorted)))
        return set_error(TCR_ERR_INVALID, "missing float64 positions or the sorted-reference workspace");
    if (d->mode != TCR_SCATTER && d->n_query > 0 && !in->query_sup)
        return set_error(TCR_ERR_INVALID, "this mode needs float64 query supports");
    if (d->mode != TCR_GATHER && d->n_ref > 0 && !in->ref_sup)
        return set_error(TCR_ERR_INVALID, "this mode needs float64 reference supports");
    if (d->hcell[0] <= 0.0f) return set_error(TCR_ERR_INVALID, "float64 searches need the cell size in hcell");
    if (d->clamped_grid) return set_error(TCR_ERR_INVALID, "float64 searches use the reference's unclamped grid");
    f.qpos = in->query_pos;
    f.qsup = in->query_sup;
    f.rpos = in->ref_pos;
    f.rsup = in->ref_sup;
    f.rsorted = reinterpret_cast<double4*>(in->ref_sorted);
    for (int k = 0; k < 3; ++k) f.ext[k] = in->domain_max[k] - in->domain_min[k];
    f.nq = d->n_query;
    f.nr = d->n_ref;
    return TCR_OK;
}

int tcr_f64_prepare(const tcr_f64_prepare_desc* d, double* stats_host, void* stream) {
    NvtxRange nvtx_("tcr_f64_prepare");
    if (!d) return set_error(TCR_ERR_INVALID, "null descriptor");
    if (d->dim < 1 || d->dim > 3) return set_error(TCR_ERR_INVALID, "dim must be 1, 2 or 3 (got %d)", d->dim);
    if (d->n_query < 0 || d->n_ref < 0 || d->n_query > 0x7fffffffLL || d->n_ref > 0x7ffffff0LL)
        return set_error(TCR_ERR_INVALID, "point counts must be in [0, 2^31)");
    if (!d->stats || (d->n_query && (!d->query_pos || !d->query_wrapped || !d->query_pos_f)))
        return set_error(TCR_ERR_INVALID, "missing query positions, their outputs or stats");
    if (d->self_search ? (d->n_query != d->n_ref || (d->n_ref && !d->ref_wrapped))
                       : (d->ref_pos && d->n_ref && (!d->ref_wrapped || !d->ref_pos_f)))
        return set_error(TCR_ERR_INVALID, "missing reference outputs");
    cudaStream_t st = (cudaStream_t)stream;
    TCR_CUDA(cudaMemsetAsync(d->stats, 0, 4 * sizeof(unsigned long long), st));
    f64_prepare_kernel<<<grid_for(std::max<int64_t>(std::max(d->n_query, d->n_ref) * d->dim, 1), 256, num_sms() * 8), 256, 0,
                         st>>>(*d);
    f64_stats_kernel<<<1, 4, 0, st>>>(static_cast<unsigned long long*>(d->stats));
    note_launches(2);
    TCR_CUDA(cudaGetLastError());
    if (stats_host) TCR_CUDA(cudaMemcpyAsync(stats_host, d->stats, 4 * sizeof(double), cudaMemcpyDeviceToHost, st));
    return TCR_OK;
}

int tcr_count_f64(const tcr_search_desc* d, const tcr_f64_inputs* in, const void* structure, void* scratch,
                  int64_t scratch_bytes, int32_t* stage, int64_t stage_capacity, int64_t* offsets,
                  int32_t* indptr_out, int64_t* row_entries_out, int64_t* info_out, void* stream) {
    NvtxRange nvtx_("tcr_count_f64");
    HostBatch b;
    int rc = batch_of_desc(d, 1, b);
    if (rc) return rc;
    F64Args f;
    rc = f64_args(d, in, f);
    if (rc) return rc;
    return run_count(b, structure, scratch, scratch_bytes, stage, stage_capacity, offsets, indptr_out, row_entries_out,
                     info_out, stream, &f);
}

int tcr_emit_f64(const tcr_search_desc* d, const tcr_f64_inputs* in, const void* structure, void* scratch,
                 int64_t scratch_bytes, const int32_t* stage, const int64_t* offsets, int64_t* row_out,
                 int64_t* col_out, int64_t out_capacity, void* stream) {
    NvtxRange nvtx_("tcr_emit_f64");
    HostBatch b;
    int rc = batch_of_desc(d, 1, b);
    if (rc) return rc;
    F64Args f;
    rc = f64_args(d, in, f);
    if (rc) return rc;
    return run_emit(b, structure, scratch, scratch_bytes, stage, offsets, row_out, col_out, out_capacity, stream, &f);
}

int tcr_batch_sizes(const tcr_batch_desc* bd, int64_t* structure_bytes, int64_t* scratch_bytes) {
    HostBatch b;
    int rc = batch_of(bd, 0, b);
    if (rc) return rc;
    batch_sizes(b, structure_bytes, scratch_bytes);
    return TCR_OK;
}

int tcr_batch_build_structure(const tcr_batch_desc* bd, void* structure, int64_t structure_bytes, void* scratch,
                              int64_t scratch_bytes, void* stream) {
    NvtxRange nvtx_("tcr_batch_build_structure");
    HostBatch b;
    int rc = batch_of(bd, 2, b);
    if (rc) return rc;
    return run_build(b, structure, structure_bytes, scratch, scratch_bytes, stream);
}

int tcr_batch_count(const tcr_batch_desc* bd, const void* structure, void* scratch, int64_t scratch_bytes,
                    int32_t* stage, int64_t stage_capacity, int64_t* offsets, int32_t* indptr_out,
                    int64_t* row_entries_out, int64_t* info_out, void* stream) {
    NvtxRange nvtx_("tcr_batch_count");
    HostBatch b;
    int rc = batch_of(bd, 1, b);
    if (rc) return rc;
    return run_count(b, structure, scratch, scratch_bytes, stage, stage_capacity, offsets, indptr_out, row_entries_out,
                     info_out, stream);
}

int tcr_batch_emit(const tcr_batch_desc* bd, const void* structure, void* scratch, int64_t scratch_bytes,
                   const int32_t* stage, const int64_t* offsets, int64_t* row_out, int64_t* col_out,
                   int64_t out_capacity, void* stream) {
    NvtxRange nvtx_("tcr_batch_emit");
    HostBatch b;
    int rc = batch_of(bd, 1, b);
    if (rc) return rc;
    return run_emit(b, structure, scratch, scratch_bytes, stage, offsets, row_out, col_out, out_capacity, stream);
}

}  // extern "C"

// ------------------------------------------------------------------------------------------
// Search without any device allocation.
//
// Some callers cannot allocate device memory at search time: a host application that hands the
// search a fixed memory arena at start-up and forbids cudaMalloc afterwards (cudaMalloc can
// synchronise the device and stall a real-time loop), or a plugin host whose allocator the
// search cannot reach.  tcr_search_noalloc serves them: the structure and the scratch of one
// whole search live in the file-scope device array below, so the caller passes only its inputs
// and its output buffers.  The array is kTcrStaticScratchBytes (32 MiB) on every GPU that loads
// this library, held until the process exits.
namespace tcr {
constexpr int64_t kTcrStaticScratchBytes = 32ll << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kTcrStaticScratchBytes];

constexpr int kMaxDevices = 64;
static void* g_static_ptr[kMaxDevices] = {nullptr};
static int g_static_err[kMaxDevices] = {0};
static std::once_flag g_static_once[kMaxDevices];

// Device address of g_static_scratch on the current device.  In host code the symbol's name is
// only a host-side stand-in, so the address is asked from the runtime, once per device, with that
// device current.
static int static_scratch_address(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(TCR_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return set_error(TCR_ERR_INVALID, "device ordinal %d out of range", dev);
    std::call_once(g_static_once[dev], [dev]() {
        void* p = nullptr;
        cudaError_t r = cudaGetSymbolAddress(&p, g_static_scratch);
        if (r == cudaSuccess) g_static_ptr[dev] = p;
        else g_static_err[dev] = (int)r;
    });
    if (!g_static_ptr[dev])
        return set_error(TCR_ERR_CUDA, "cudaGetSymbolAddress(static scratch) failed on device %d: %s", dev,
                         cudaGetErrorString((cudaError_t)g_static_err[dev]));
    *out = g_static_ptr[dev];
    return TCR_OK;
}
}  // namespace tcr

extern "C" int tcr_search_noalloc(const tcr_search_desc* d, int64_t* offsets, int32_t* indptr_out,
                                  int64_t* row_entries_out, int64_t* row_out, int64_t* col_out,
                                  int64_t pair_capacity, int64_t* total_out, void* stream) {
    using namespace tcr;
    NvtxRange nvtx_("tcr_search_noalloc");
    HostBatch b;
    int rc = batch_of_desc(d, 2, b);
    if (rc) return rc;
    if (!offsets || (pair_capacity > 0 && !col_out) || pair_capacity < 0)
        return set_error(TCR_ERR_INVALID, "offsets and a column buffer of pair_capacity entries are required");
    int64_t s_bytes = 0, w_bytes = 0;
    batch_sizes(b, &s_bytes, &w_bytes);
    if (s_bytes + w_bytes > kTcrStaticScratchBytes)
        return set_error(TCR_ERR_INVALID,
                         "tcr_search_noalloc: %lld query and %lld reference points need %lld bytes of structure "
                         "and scratch, more than the static %lld bytes; use tcr_build_structure/tcr_count/tcr_emit "
                         "with caller-allocated buffers",
                         (long long)d->n_query, (long long)d->n_ref, (long long)(s_bytes + w_bytes),
                         (long long)kTcrStaticScratchBytes);
    void* base = nullptr;
    rc = static_scratch_address(&base);
    if (rc) return rc;
    void* structure = base;
    void* scratch = static_cast<char*>(base) + s_bytes;
    // The rest of the array is the staging list: units whose records fit are expanded by the emit
    // without being tested again.
    const int64_t stage_off = align256(s_bytes + w_bytes);
    const int64_t stage_words = std::min<int64_t>((kTcrStaticScratchBytes - stage_off) / 4, 0x7fffffff);
    int32_t* stage = stage_words > 0 ? reinterpret_cast<int32_t*>(static_cast<char*>(base) + stage_off) : nullptr;
    // Every kernel below initialises what it reads (counters, map, sort state), so the contents a
    // previous call left in the array do not matter.
    rc = tcr_build_structure(d, structure, s_bytes, scratch, w_bytes, stream);
    if (rc) return rc;
    int64_t info[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    rc = tcr_count(d, structure, scratch, w_bytes, stage, stage ? stage_words : 0, offsets, indptr_out,
                   row_entries_out, info, stream);
    if (rc) return rc;
    TCR_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    if (total_out) *total_out = info[0];
    if (info[1] < 0) return set_error(TCR_ERR_CUDA, "tcr_search_noalloc: a sort on the device gave up waiting; nothing was searched");
    if (info[1]) return set_error(TCR_ERR_INVALID, "no valid cell grid for this domain and support");
    if (info[0] > pair_capacity)
        return set_error(TCR_ERR_INVALID, "tcr_search_noalloc: %lld pairs do not fit the %lld-entry output",
                         (long long)info[0], (long long)pair_capacity);
    if (info[0] == 0) return TCR_OK;
    return tcr_emit(d, structure, scratch, w_bytes, stage, offsets, row_out, col_out, pair_capacity, stream);
}
