// tcr_sort.cuh -- stable LSD radix sort of (key, int32 value) pairs, 32- or 64-bit keys.
//
// Per 8-bit digit: a tile histogram, a per-digit scan of the tiles' counts and a stable
// scatter, as phases of one cooperative launch (sort_coop_kernel, the searches' sorts) or as
// three launches (radix_sort_pairs, the scatter operators' sort).  Inside a tile the scatter ranks keys with warp match/ballot so equal digits
// keep their input order; tiles are concatenated in order, so the whole sort is stable.  A pass
// whose digit is the same for every key is skipped on the device without a host round trip:
// digits above the highest bit in which two keys differ (from the key range the producer
// reduced) are not even counted, and a digit whose histogram met a single value is neither
// scanned nor scattered.  The per-pass buffer selector then stays put.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "tcr_scan.cuh"

namespace tcr {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // 2048 keys per tile (1024 measured slower)
constexpr int kBins = 256;
static_assert(kSortThreads == kBins, "the scatter scans one digit per thread");

template <typename K>
struct SortStateT {
    K key_min, key_max;   // reduced by the producer of the keys
    int32_t sel[9];       // sel[p]: which buffer (0/1) holds the input of pass p
    int32_t pad;
    int64_t n_dev;        // >= 0: sort only the first n_dev keys (a count known on the device only)
    uint32_t seen[8][8];  // per pass: bitmap of the digit values the histogram met
    unsigned bar;         // arrivals at the one-launch sort's barrier
};
using SortState32 = SortStateT<uint32_t>;
using SortState64 = SortStateT<unsigned long long>;

template <typename K>
__host__ __device__ constexpr int key_passes() { return (int)sizeof(K); }

__device__ __forceinline__ int top_bit(uint32_t x) { return 31 - __clz(x); }
__device__ __forceinline__ int top_bit(unsigned long long x) { return 63 - __clzll(x); }

// Producer-side reset (one thread): empty key range, input in buffer 0, no digits seen.
template <typename K>
__device__ __forceinline__ void sort_state_reset(SortStateT<K>* st) {
    st->key_min = ~(K)0;
    st->key_max = 0;
    st->sel[0] = 0;
    st->n_dev = -1;
    st->bar = 0u;
    for (int p = 0; p < 8; ++p)
        for (int i = 0; i < 8; ++i) st->seen[p][i] = 0u;
}

// Some key differs from another at or above bit `shift`.
template <typename K>
__device__ __forceinline__ bool pass_needed(const SortStateT<K>* st, int shift) {
    const K x = st->key_min ^ st->key_max;
    if (x == 0) return false;
    return top_bit(x) >= shift;
}

// The histogram of this pass met more than one digit value.
template <typename K>
__device__ __forceinline__ bool pass_varies(const SortStateT<K>* st, int pass) {
    int n = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) n += __popc(st->seen[pass][i]);
    return n > 1;
}

template <typename K>
__device__ __forceinline__ bool pass_runs(const SortStateT<K>* st, int shift, int pass) {
    return pass_needed(st, shift) && pass_varies(st, pass);
}

template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const K* keys0, const K* keys1, int64_t n, int shift,
                                                                  int pass, int64_t ntiles, SortStateT<K>* st,
                                                                  int32_t* hist) {
    if (!pass_needed(st, shift)) return;
    if (st->n_dev >= 0 && st->n_dev < n) n = st->n_dev;
    const K* keys = st->sel[pass] ? keys1 : keys0;
    __shared__ int32_t sh[kBins];
    for (int i = threadIdx.x; i < kBins; i += kSortThreads) sh[i] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        int64_t i = base + (int64_t)k * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&sh[(int)((keys[i] >> shift) & 0xff)], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kBins; d += kSortThreads) hist[(int64_t)d * ntiles + blockIdx.x] = sh[d];
    if (threadIdx.x < kBins / 32) {  // the digit values this tile met
        uint32_t bits = 0;
        for (int b = 0; b < 32; ++b) bits |= (sh[threadIdx.x * 32 + b] != 0 ? 1u : 0u) << b;
        if (bits && (bits & ~st->seen[pass][threadIdx.x])) atomicOr(&st->seen[pass][threadIdx.x], bits);
    }
}

// Stable scatter of one tile.  Warp w owns keys [w*R*32, (w+1)*R*32) of the tile (R = kSortItems),
// processed in R rounds of 32 consecutive keys, so (warp, round, lane) order is the input order.  The tile is
// first ordered by digit in shared memory (stable), then written out by consecutive threads over
// that order: the keys of one digit land in consecutive output slots, so the stores coalesce into
// runs instead of one sector per key.
template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(K* keys0, K* keys1, int32_t* vals0,
                                                                     int32_t* vals1, int64_t n, int shift, int pass,
                                                                     int64_t ntiles, SortStateT<K>* st,
                                                                     const int32_t* hist_scanned,
                                                                     const int32_t* digit_total) {
    const int s = st->sel[pass];
    if (!pass_runs(st, shift, pass)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) st->sel[pass + 1] = s;
        return;
    }
    if (st->n_dev >= 0 && st->n_dev < n) n = st->n_dev;
    const K* kin = s ? keys1 : keys0;
    const int32_t* vin = s ? vals1 : vals0;
    K* kout = s ? keys0 : keys1;
    int32_t* vout = s ? vals0 : vals1;
    constexpr int NW = kSortThreads / 32;
    __shared__ int32_t warp_hist[NW][kBins];
    __shared__ int32_t tile_base[kBins];   // first output slot of each digit of this tile
    __shared__ int32_t digit_start[kBins + 1];  // first slot of each digit in the tile's digit order
    __shared__ K sk[kSortTile];
    __shared__ int32_t sv[kSortTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < NW * kBins; i += kSortThreads) (&warp_hist[0][0])[i] = 0;
    {
        // first slot of digit d in the output: the keys of smaller digits, then this digit's keys in
        // earlier tiles (one digit per thread)
        __shared__ int32_t base_sm[kSortThreads / 32 + 1];
        int32_t total;
        const int d = threadIdx.x;
        const int32_t db = block_exclusive_scan<int32_t, kSortThreads>(digit_total[d], base_sm, total);
        tile_base[d] = db + hist_scanned[(int64_t)d * ntiles + blockIdx.x];
    }
    __syncthreads();
    const int64_t tile0 = (int64_t)blockIdx.x * kSortTile;
    const int64_t base = tile0 + (int64_t)warp * (kSortItems * 32);
    const unsigned lt = (1u << lane) - 1u;
    K key[kSortItems];
    int32_t val[kSortItems];
    int32_t rank[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        int64_t i = base + r * 32 + lane;
        bool valid = i < n;
        key[r] = valid ? kin[i] : (K)0;
        val[r] = valid ? vin[i] : 0;
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        int64_t i = base + r * 32 + lane;
        bool valid = i < n;
        uint32_t dig = valid ? (uint32_t)((key[r] >> shift) & 0xff) : 0x100u;  // invalid lanes: own group
        unsigned peers = __match_any_sync(0xffffffffu, dig);
        int before = __popc(peers & lt);
        int run = valid ? warp_hist[warp][dig] : 0;
        __syncwarp();
        if (valid && before == 0) warp_hist[warp][dig] = run + __popc(peers);
        __syncwarp();
        rank[r] = run + before;
    }
    __syncthreads();
    // per digit: exclusive scan over warps; the digit's total, scanned over digits, is its start
    // in the tile's digit order
    int32_t dtot = 0;
    const int d0 = threadIdx.x;  // kSortThreads == kBins: one digit per thread
    {
        int acc = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            int c = warp_hist[w][d0];
            warp_hist[w][d0] = acc;
            acc += c;
        }
        dtot = acc;
    }
    {
        __shared__ int32_t scan_sm[kSortThreads / 32 + 1];
        int32_t total;
        const int32_t ex = block_exclusive_scan<int32_t, kSortThreads>(dtot, scan_sm, total);
        digit_start[d0] = ex;
        if (d0 == 0) digit_start[kBins] = total;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        int64_t i = base + r * 32 + lane;
        if (i < n) {
            int dig = (int)((key[r] >> shift) & 0xff);
            const int loc = digit_start[dig] + warp_hist[warp][dig] + rank[r];
            sk[loc] = key[r];
            sv[loc] = val[r];
        }
    }
    __syncthreads();
    const int tn = digit_start[kBins];
    for (int i = threadIdx.x; i < tn; i += kSortThreads) {
        const K k = sk[i];
        const int dig = (int)((k >> shift) & 0xff);
        const int64_t pos = (int64_t)tile_base[dig] + (i - digit_start[dig]);
        kout[pos] = k;
        vout[pos] = sv[i];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) st->sel[pass + 1] = s ^ 1;
}

// Per digit (one block each): exclusive scan of the digit's tile counts in place, and the
// digit's total; the scatter adds the totals of the smaller digits.  Gated on the pass running.
template <typename K>
__global__ void __launch_bounds__(kScanThreads) hist_scan_digits(int32_t* hist, int64_t ntiles, int32_t* digit_total,
                                                                 const SortStateT<K>* st, int shift, int pass) {
    if (!pass_runs(st, shift, pass)) return;
    __shared__ int32_t sm[kScanThreads / 32 + 1];
    int32_t* row = hist + (int64_t)blockIdx.x * ntiles;
    int32_t carry = 0;
    for (int64_t b = 0; b < ntiles; b += kScanTile) {
        const int64_t i0 = b + (int64_t)threadIdx.x * kScanItems;
        int32_t v[kScanItems];
        int32_t sum = 0;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = i0 + k < ntiles ? row[i0 + k] : 0;
            sum += v[k];
        }
        int32_t total;
        int32_t ex = block_exclusive_scan<int32_t, kScanThreads>(sum, sm, total) + carry;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            if (i0 + k < ntiles) row[i0 + k] = ex;
            ex += v[k];
        }
        carry += total;
    }
    if (threadIdx.x == 0) digit_total[blockIdx.x] = carry;
}

template <typename K>
struct SortWorkspaceT {
    K* keys[2];
    int32_t* vals[2];
    int32_t* hist;          // kBins * ntiles
    int32_t* tile_sums;     // kBins digit totals of the running pass
    SortStateT<K>* state;   // device
};

inline int64_t sort_tiles(int64_t n) { return (n + kSortTile - 1) / kSortTile; }
inline int64_t sort_hist_elems(int64_t n) { return (int64_t)kBins * sort_tiles(n); }

// Sorts keys[sel0]/vals[sel0] (sel0 = state->sel[0], set by the producer, which also reduced the
// key range and cleared the digit bitmaps), n keys or state->n_dev when that is set and smaller.  The result lives in buffer state->sel[key_passes<K>()]
// after the call; consumers read the selector on the device.
template <typename K>
inline cudaError_t radix_sort_pairs(const SortWorkspaceT<K>& w, int64_t n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int64_t nt = sort_tiles(n);
    for (int p = 0; p < key_passes<K>(); ++p) {
        const int shift = 8 * p;
        radix_hist_kernel<K><<<(unsigned)nt, kSortThreads, 0, st>>>(w.keys[0], w.keys[1], n, shift, p, nt, w.state,
                                                                    w.hist);
        hist_scan_digits<K><<<kBins, kScanThreads, 0, st>>>(w.hist, nt, w.tile_sums, w.state, shift, p);
        radix_scatter_kernel<K><<<(unsigned)nt, kSortThreads, 0, st>>>(
            w.keys[0], w.keys[1], w.vals[0], w.vals[1], n, shift, p, nt, w.state, w.hist, w.tile_sums);
        note_launches(3);
    }
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------
// One launch: the whole sort, the placement of what was sorted, and the run starts.
//
// Every block owns a contiguous range of the keys.  Per digit: the blocks' histograms, a grid barrier, the
// stable scatter (each block adds the histograms of the blocks before it itself), a grid barrier.  Passes
// whose digit no two keys differ in cost nothing, where as launches (histogram, scan, scatter per
// pass, 12 for 32-bit and 24 for 64-bit keys) the unneeded ones alone took about 12 us of a search, and
// everything after the sort (placement, run-start scan, run records) four launches more.
//
// One block of 32 warps per SM: a launch is cooperative, so all blocks are resident, and each wait on
// the barrier is bounded: a block that gives up sets *failed and returns, and the others follow at their
// next wait.  What the sort should have written is then there in part: the kernels behind it check every index
// that they take from it, make no work units where the flag is set, and the host reports it.
constexpr int kCoopThreads = 1024;
constexpr int kCoopWarps = kCoopThreads / 32;
constexpr int kCoopRounds = 8;
constexpr int kCoopTile = kCoopThreads * kCoopRounds;
constexpr int64_t kCoopMinKeys = kSortTile;      // keys per block at least (the histograms' room follows the tiles)
constexpr unsigned kCoopSpins = 1u << 21;        // about a second and a half

template <typename K>
struct CoopSmem {
    int32_t warp_hist[kCoopWarps][kBins];
    K sk[kCoopTile];
    int32_t sv[kCoopTile];
    int32_t digit_start[kBins + 1];  // first slot of each digit in the tile's digit order
    int32_t next[kBins];             // next output slot of each digit of this block
    int32_t part[4][kBins], total[4][kBins];
    int32_t scan[kCoopWarps + 1];
    int32_t flag;
};

__device__ __forceinline__ bool coop_barrier(unsigned* bar, unsigned target, int32_t* failed, int32_t* flag) {
    __syncthreads();
    if (gridDim.x == 1) return true;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        int32_t bad = 0;
        unsigned spins = 0;
        while (*(volatile unsigned*)bar < target) {
            if (++spins > kCoopSpins || *(volatile int32_t*)failed) {
                atomicExch(failed, 1);
                bad = 1;
                break;
            }
        }
        __threadfence();
        *flag = bad;
    }
    __syncthreads();
    return *flag == 0;
}

// Tail: what to do with the sorted pairs.  kPlace: place(i, key, value) for every sorted position;
// kRuns: run(keys, i, r) for the first position i of run r (equal keys), starts[r] = i, starts[runs] = n.
struct NoTail {
    static constexpr bool kPlace = false, kRuns = false;
    int32_t* starts = nullptr;
    int32_t* num_runs = nullptr;
    template <typename K>
    __device__ void place(int64_t, K, int32_t) const {}
    template <typename K>
    __device__ void run(const K*, int64_t, int32_t) const {}
};

template <typename K, typename Tail>
__global__ void __launch_bounds__(kCoopThreads, 1)
    sort_coop_kernel(K* keys0, K* keys1, int32_t* vals0, int32_t* vals1, int64_t n_all, SortStateT<K>* st,
                     int32_t* hist, int32_t* failed, int chained, Tail tail) {
    extern __shared__ __align__(16) unsigned char coop_raw[];
    CoopSmem<K>& sm = *reinterpret_cast<CoopSmem<K>*>(coop_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = gridDim.x, b = blockIdx.x;
    // a sort before this one gave up: its pairs are not there
    const int32_t gone = chained ? *(volatile int32_t*)failed : 0;
    const int64_t n = (st->n_dev >= 0 && st->n_dev < n_all) ? st->n_dev : n_all;
    const int64_t per = ((n + G - 1) / G + 31) & ~int64_t(31);
    const int64_t lo = min(n, per * b), hi = min(n, lo + per);
    const unsigned lt = (1u << lane) - 1u;
    const bool single = per <= kCoopTile;
    const int rounds = (int)((min(per, (int64_t)kCoopTile) + kCoopThreads - 1) / kCoopThreads);
    const K differ = st->key_min ^ st->key_max;
    const int top = differ == 0 ? -1 : top_bit(differ);  // the highest bit in which two keys differ
    unsigned phase = 0;
    int sel = st->sel[0];
    if (gone) return;  // (here, so that the loads above are in flight together)
    bool placed = false;
    for (int pass = 0; pass < key_passes<K>(); ++pass) {
        const int shift = 8 * pass;
        if (top < shift) break;
        const K* kin = sel ? keys1 : keys0;
        const int32_t* vin = sel ? vals1 : vals0;
        K* kout = sel ? keys0 : keys1;
        int32_t* vout = sel ? vals0 : vals1;
        K key[kCoopRounds];
        int32_t val[kCoopRounds], rank[kCoopRounds];
        int32_t dtot = 0;  // (thread < 256) the tile's keys of digit tid
        // loads a tile of the range and ranks its keys: warp w owns keys [32 R w, 32 R (w + 1)); warp_hist
        // ends as the keys of a digit in the warps before
        auto rank_tile = [&](int64_t t0, int len, int R) {
            for (int i = tid; i < kCoopWarps * kBins; i += kCoopThreads) (&sm.warp_hist[0][0])[i] = 0;
#pragma unroll
            for (int r = 0; r < kCoopRounds; ++r) {
                const int i = warp * 32 * R + r * 32 + lane;
                const bool valid = r < R && i < len;
                key[r] = valid ? kin[t0 + i] : (K)0;
                val[r] = valid ? vin[t0 + i] : 0;
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < kCoopRounds; ++r) {
                if (r < R) {
                    const bool valid = warp * 32 * R + r * 32 + lane < len;
                    const uint32_t dig = valid ? (uint32_t)((key[r] >> shift) & 0xff) : 0x100u;
                    const unsigned peers = __match_any_sync(0xffffffffu, dig);
                    const int ahead = __popc(peers & lt);
                    const int run = valid ? sm.warp_hist[warp][dig] : 0;
                    __syncwarp();
                    if (valid && ahead == 0) sm.warp_hist[warp][dig] = run + __popc(peers);
                    __syncwarp();
                    rank[r] = run + ahead;
                }
            }
            __syncthreads();
            // exclusive over the warps, four groups of threads with eight warps each
            constexpr int kPer = kCoopWarps / (kCoopThreads / kBins);
            const int d = tid & (kBins - 1), grp = tid >> 8;
            int32_t c = 0;
#pragma unroll
            for (int w = 0; w < kPer; ++w) c += sm.warp_hist[grp * kPer + w][d];
            sm.part[grp][d] = c;
            __syncthreads();
            int32_t acc = 0;
            for (int g = 0; g < grp; ++g) acc += sm.part[g][d];
#pragma unroll
            for (int w = 0; w < kPer; ++w) {
                const int32_t x = sm.warp_hist[grp * kPer + w][d];
                sm.warp_hist[grp * kPer + w][d] = acc;
                acc += x;
            }
            dtot = 0;
            if (tid < kBins)
                for (int g = 0; g < kCoopThreads / kBins; ++g) dtot += sm.part[g][tid];
            __syncthreads();
        };
        // a range of one tile (up to 1.2M keys on 148 blocks) is ranked at once and stays in registers;
        // a longer one is counted first and ranked tile by tile
        if (single) {
            rank_tile(lo, (int)(hi - lo), rounds);
            if (tid < kBins) hist[(int64_t)b * kBins + tid] = dtot;
        } else {
            for (int i = tid; i < kCoopWarps * kBins; i += kCoopThreads) (&sm.warp_hist[0][0])[i] = 0;
            __syncthreads();
            for (int64_t i = lo + tid; i < hi; i += kCoopThreads)
                atomicAdd(&sm.warp_hist[warp][(int)((kin[i] >> shift) & 0xff)], 1);
            __syncthreads();
            if (tid < kBins) {
                int32_t c = 0;
#pragma unroll 8
                for (int w = 0; w < kCoopWarps; ++w) c += sm.warp_hist[w][tid];
                hist[(int64_t)b * kBins + tid] = c;
            }
        }
        if (!coop_barrier(&st->bar, (unsigned)G * ++phase, failed, &sm.flag)) return;
        // first output slot of every digit of this block: the smaller digits' keys, then this digit's of
        // the blocks before (four groups of 256 threads share the blocks)
        {
            const int d = tid & (kBins - 1), grp = tid >> 8;
            int32_t all = 0, before = 0;
            for (int j = grp; j < G; j += kCoopThreads / kBins) {
                const int32_t c = __ldcg(&hist[(int64_t)j * kBins + d]);
                all += c;
                if (j < b) before += c;
            }
            sm.total[grp][d] = all;
            sm.part[grp][d] = before;
            __syncthreads();
            int32_t tot = 0, bef = 0;
            if (tid < kBins)
                for (int g = 0; g < kCoopThreads / kBins; ++g) {
                    tot += sm.total[g][tid];
                    bef += sm.part[g][tid];
                }
            int32_t sum;
            const int32_t first = block_exclusive_scan<int32_t, kCoopThreads>(tot, sm.scan, sum);
            if (tid < kBins) sm.next[tid] = first + bef;
            // one digit holds every key: nothing moves
            if (__syncthreads_or(tid < kBins && tot == n)) {
                if (!coop_barrier(&st->bar, (unsigned)G * ++phase, failed, &sm.flag)) return;
                continue;
            }
        }
        const bool last = Tail::kPlace && top < shift + 8;
        for (int64_t t0 = lo; t0 < hi; t0 += kCoopTile) {
            const int len = (int)min((int64_t)kCoopTile, hi - t0);
            const int R = single ? rounds : (len + kCoopThreads - 1) / kCoopThreads;
            if (!single) rank_tile(t0, len, R);
            int32_t sum;
            const int32_t ex = block_exclusive_scan<int32_t, kCoopThreads>(dtot, sm.scan, sum);
            if (tid < kBins) sm.digit_start[tid] = ex;
            __syncthreads();
#pragma unroll
            for (int r = 0; r < kCoopRounds; ++r) {
                if (r < R && warp * 32 * R + r * 32 + lane < len) {
                    const int dig = (int)((key[r] >> shift) & 0xff);
                    const int loc = sm.digit_start[dig] + sm.warp_hist[warp][dig] + rank[r];
                    sm.sk[loc] = key[r];
                    sm.sv[loc] = val[r];
                }
            }
            __syncthreads();
            for (int i = tid; i < len; i += kCoopThreads) {
                const K k = sm.sk[i];
                const int dig = (int)((k >> shift) & 0xff);
                const int64_t pos = (int64_t)sm.next[dig] + (i - sm.digit_start[dig]);
                kout[pos] = k;
                if (last) tail.place(pos, k, sm.sv[i]);
                else vout[pos] = sm.sv[i];
            }
            __syncthreads();
            if (tid < kBins) sm.next[tid] += dtot;
        }
        sel ^= 1;
        placed = last;
        if (!coop_barrier(&st->bar, (unsigned)G * ++phase, failed, &sm.flag)) return;
    }
    if (b == 0 && tid == 0) st->sel[key_passes<K>()] = sel;
    const K* ks = sel ? keys1 : keys0;
    const int32_t* vs = sel ? vals1 : vals0;
    if (Tail::kPlace && !placed) {
        for (int64_t i = lo + tid; i < hi; i += kCoopThreads) tail.place(i, ks[i], vs[i]);
    }
    if (Tail::kRuns) {
        int32_t mine = 0;
        for (int64_t i = lo + tid; i < hi; i += kCoopThreads) mine += (i == 0 || ks[i] != ks[i - 1]) ? 1 : 0;
        int32_t runs;
        block_exclusive_scan<int32_t, kCoopThreads>(mine, sm.scan, runs);
        if (tid == 0) hist[b] = runs;
        // (the barrier also publishes what the blocks placed)
        if (!coop_barrier(&st->bar, (unsigned)G * ++phase, failed, &sm.flag)) return;
        int32_t before = 0;
        for (int j = tid; j < b; j += kCoopThreads) before += __ldcg(&hist[j]);
        int32_t r0;
        block_exclusive_scan<int32_t, kCoopThreads>(before, sm.scan, r0);
        int32_t r = r0;
        for (int64_t t0 = lo; t0 < hi; t0 += kCoopThreads) {
            const int64_t i = t0 + tid;
            const int32_t f = (i < hi && (i == 0 || ks[i] != ks[i - 1])) ? 1 : 0;
            int32_t sum;
            const int32_t ex = block_exclusive_scan<int32_t, kCoopThreads>(f, sm.scan, sum);
            if (f) tail.starts[r + ex] = (int32_t)i;
            r += sum;
        }
        if (b == G - 1 && tid == 0) {
            *tail.num_runs = r0 + runs;
            tail.starts[r0 + runs] = (int32_t)n;
        }
        __syncthreads();
        for (int32_t c = r0 + tid; c < r0 + runs; c += kCoopThreads) tail.run(ks, (int64_t)tail.starts[c], c);
    }
}

inline int coop_blocks(int64_t n, int sms) {
    if (n <= kCoopTile) return 1;  // one tile: no barriers to pay for (about 2 us each)
    const int64_t want = (n + kCoopMinKeys - 1) / kCoopMinKeys;
    return (int)(want < 1 ? 1 : (want < sms ? want : sms));
}

// Launches the one-launch sort of keys[0] / vals[0] (the selector and the key range as for
// radix_sort_pairs; the sorted keys end in buffer state->sel[key_passes<K>()]).  chained: the pairs come from
// a sort with the same flag.
template <typename K, typename Tail>
inline cudaError_t sort_coop(const SortWorkspaceT<K>& w, int64_t n, int32_t* failed, int chained, Tail tail,
                             cudaStream_t st) {
    int dev = 0, sms = 148;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    static uint64_t done_mask = 0;  // devices on which the kernel's shared memory limit is raised
    const uint64_t bit = 1ull << (dev & 63);
    if (!(__atomic_load_n(&done_mask, __ATOMIC_ACQUIRE) & bit)) {
        e = cudaFuncSetAttribute(sort_coop_kernel<K, Tail>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(CoopSmem<K>));
        if (e != cudaSuccess) return e;
        __atomic_fetch_or(&done_mask, bit, __ATOMIC_ACQ_REL);
    }
    K *k0 = w.keys[0], *k1 = w.keys[1];
    int32_t *v0 = w.vals[0], *v1 = w.vals[1], *hist = w.hist;
    SortStateT<K>* state = w.state;
    void* args[] = {&k0, &k1, &v0, &v1, &n, &state, &hist, &failed, &chained, &tail};
    // One block per SM is resident on the whole device; a stream that is given fewer SMs (a partition of
    // them) refuses that many.  Any number of blocks sorts, in longer ranges.
    for (int blocks = coop_blocks(n, sms);; blocks = (blocks + 1) / 2) {
        e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(sort_coop_kernel<K, Tail>), dim3((unsigned)blocks),
                                        dim3(kCoopThreads), args, sizeof(CoopSmem<K>), st);
        if (e != cudaErrorCooperativeLaunchTooLarge || blocks == 1) break;
        (void)cudaGetLastError();
    }
    note_launches(1);
    return e;
}

}  // namespace tcr
