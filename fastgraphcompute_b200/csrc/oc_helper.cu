// Object-condensation index matrices and the gather-with-default that consumes them (sm_100a).
//
//   M[k, :]     ids of the points of object k (points of one row split that share a
//               non-negative truth index), ascending, padded with -1
//   M_not[k, :] ids of all other points of the same row split, ascending, padded with -1
//   objects_per_split[e]
// as extensions/oc_helper.py:128-230 with extensions/oc_helper_cpu.cpp:14-83 and
// extensions/oc_helper_helper.cpp:31-93 of the reference.  The reference finds the objects
// with torch.unique on the host side of its wrapper and then lets every object scan its
// whole row split twice; here one radix sort of (truth index, point id) puts the members of
// every object next to each other, M is a copy of those runs, and M_not is computed
// element-wise: the j-th non-member of an object is  row start + j + t,  t = number of
// members m_0 < m_1 < ... with  m_i - row start - i <= j  (a binary search over the
// object's sorted members), so the big matrix is written once, coalesced, with no scan of
// the row split per object.
//
// The order of the objects (rows of M) is not defined by the reference ("not guaranteed to
// give the identical output in terms of index ordering", oc_helper.py:91-92); here it is
// ascending in (truth index, row split).
#include <cstring>

#include "fgc_common.cuh"
#include "scan.cuh"

namespace fgc {

struct OcHeader {
    int32_t status;     // FGC_STATUS_* bits (first word of the workspace)
    int32_t n_unique;   // number of objects
    int32_t n_maxuq;    // largest object
    int32_t n_maxrs;    // largest row split
    int32_t n_valid;    // points with a non-negative truth index
    int32_t keys_done;  // CTAs of k_oc_keys that have finished
    int32_t scan_ticket;
    int32_t active;     // bit p: pass p of the sort has work to do
    int32_t tile[8];    // tiles of a pass that have been taken
    unsigned long long none;     // key of the points without an object: the largest truth index + 1
};

constexpr size_t kOcHeaderBytes = 256;

// Positions are counted in 31 bits, by up to a scan tile of 2048 at a time.
constexpr int64_t kOcMostPoints = 0x7ffff000;

// The sort: eight passes of eight bits over 64-bit keys, one launch each, 4096 keys a CTA.
constexpr int kOcPasses = 8, kOcBins = 256, kOcWarps = 16, kOcRounds = 8, kOcSortTile = 32 * kOcWarps * kOcRounds;
inline int oc_sort_tiles(int64_t n) { return (int)((n + kOcSortTile - 1) / kOcSortTile); }

struct OcWorkspace {
    size_t header, keys_a, keys_b, vals_a, vals_b, flags, blocksums, obj_start, obj_split, bins, tiles, total;
};

inline OcWorkspace oc_workspace_layout(int64_t n_vert)
{
    OcWorkspace w;
    const size_t n = (size_t)n_vert;
    size_t off = 0;
    w.header = off; off += kOcHeaderBytes;
    w.keys_a = off; off = align_up(off + 8 * n, 256);
    w.keys_b = off; off = align_up(off + 8 * n, 256);
    w.vals_a = off; off = align_up(off + 4 * n, 256);
    w.vals_b = off; off = align_up(off + 4 * n, 256);
    w.flags = off; off = align_up(off + 4 * (n + 1), 256);
    w.blocksums = off; off = align_up(off + 4 * ((n + 1) / kScanTile + 2), 256);
    w.obj_start = off; off = align_up(off + 4 * (n + 1), 256);
    w.obj_split = off; off = align_up(off + 4 * (n + 1), 256);
    w.bins = off; off = align_up(off + 4 * (size_t)kOcPasses * kOcBins, 256);
    w.tiles = off; off = align_up(off + 8 * (size_t)kOcBins * oc_sort_tiles(n_vert), 256);
    w.total = off;
    return w;
}

// Clears what the sort and the counting add to, checks the row splits and finds the largest truth index.
__global__ void __launch_bounds__(256)
k_oc_first(const int64_t *__restrict__ asso, const int64_t *__restrict__ rs, int n_rs, int n_vert, unsigned long long *__restrict__ tiles,
           int64_t n_tiles, int *__restrict__ bins, unsigned long long *__restrict__ objects_per_split, OcHeader *h)
{
    chain_wait();
    chain_release();
    const int64_t t0 = (int64_t)blockIdx.x * 256 + threadIdx.x, stride = (int64_t)gridDim.x * 256;
    for (int64_t i = t0; i < n_tiles * kOcBins; i += stride) tiles[i] = 0;
    for (int64_t i = t0; i < kOcPasses * kOcBins; i += stride) bins[i] = 0;
    for (int64_t i = t0; i < n_rs - 1; i += stride) objects_per_split[i] = 0;
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        // row_splits must start at 0, end at n_vert and never decrease
        const int lane = threadIdx.x;
        int bad = 0, longest = 0;
        for (int i = 1 + lane; i < n_rs; i += 32) {
            const int64_t len = rs[i] - rs[i - 1];
            if (len < 0) bad = 1;
            else if (len > longest) longest = (int)(len > 0x7fffffff ? 0x7fffffff : len);
        }
        bad = __any_sync(FGC_FULL_MASK, bad);
        longest = __reduce_max_sync(FGC_FULL_MASK, longest);
        if (lane == 0) {
            if (bad || rs[0] != 0 || rs[n_rs - 1] != (int64_t)n_vert) atomicOr(&h->status, FGC_STATUS_BAD_ROW_SPLITS);
            h->n_maxrs = longest;
        }
    }
    unsigned long long most = 0;
#pragma unroll 4
    for (int64_t v = t0; v < n_vert; v += stride) {
        const int64_t a = asso[v];
        if (a >= 0) most = max(most, (unsigned long long)a + 1);
    }
    __shared__ unsigned long long s_most;
    if (threadIdx.x == 0) s_most = 0;
    __syncthreads();
    if (most) atomicMax(&s_most, most);
    __syncthreads();
    if (threadIdx.x == 0 && s_most) atomicMax(&h->none, s_most);
}

// Keys, and how often each value of their eight digits occurs; the last CTA turns that into the places where the values begin and
// finds the passes that would change nothing since all keys have one value there.
__global__ void __launch_bounds__(256)
k_oc_keys(const int64_t *__restrict__ asso, int n_vert, uint64_t *__restrict__ keys, int *__restrict__ vals, int *__restrict__ bins,
          OcHeader *h)
{
    chain_wait();
    chain_release();
    __shared__ int s_bins[kOcPasses * kOcBins];
    __shared__ int s_sum[8], s_last;
    const uint64_t none = h->none;
    const int passes = (64 - __clzll((long long)none) + 7) >> 3;         // all higher bits are 0
    for (int i = threadIdx.x; i < passes * kOcBins; i += 256) s_bins[i] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kOcSortTile;
#pragma unroll 4
    for (int r = 0; r < kOcSortTile / 256; r++) {
        const int64_t v = base + r * 256 + threadIdx.x;
        if (v >= n_vert) break;
        const int64_t a = asso[v];
        const uint64_t key = a < 0 ? none : (uint64_t)a;                  // points without an object sort to the end
        keys[v] = key;
        vals[v] = (int)v;
        for (int p = 0; p < passes; p++) atomicAdd(&s_bins[p * kOcBins + (int)(key >> (8 * p) & (kOcBins - 1))], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kOcBins; i += 256)
        if (s_bins[i]) atomicAdd(bins + i, s_bins[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&h->keys_done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int active = 0;
    for (int p = 0; p < passes; p++) {
        const int x = __ldcg(bins + p * kOcBins + threadIdx.x);
        int incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FGC_FULL_MASK, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_sum[w] = incl;
        const int one_value = __syncthreads_or(x == n_vert);
        for (int k = 0; k < w; k++) incl += s_sum[k];
        __stcg(bins + p * kOcBins + threadIdx.x, incl - x);
        active |= one_value ? 0 : 1 << p;
        __syncthreads();
    }
    if (threadIdx.x == 0) h->active = active;
}

__device__ __forceinline__ unsigned long long oc_load_tile(const unsigned long long *at)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(at) : "memory");
    return v;
}
__device__ __forceinline__ void oc_store_tile(unsigned long long *at, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(at), "l"(v) : "memory");
}

// One stable pass: CTAs take tiles in order; thread d finds how many keys with digit d the tiles before it have (decoupled
// look-back: Merrill and Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016), from words that hold the
// pass, whether the number is the tile's alone or that of all up to it, and the number.  Eight words are read at a time: one after
// another, 391 tiles that start together would wait for hundreds of round trips.  The keys go through shared memory in their new
// order, so that runs of equal digits are written together.
// Truth indexes below 256 take one of the eight passes, the others return at once: 1.6 M points with 200 values, whole preparation
// and M 0.35 -> 0.18 ms (CUB's sort always takes all eight, 0.14 ms); with 62-bit values 0.35 -> 0.30 ms.  Latency bounds a pass (a tile's
// ranks, three round trips to L2, the look-back): 16 warps with 8 rounds 67 / 226 us for the launches of 1.6 M keys of one / eight
// bytes; 8 with 16 67 / 235, 16 with 4 (half the tile) 67 / 266; words read 32 at a time 86 / 381 against 83 / 337 of eight (8 x 16, values
// read late).
constexpr int kOcLookBack = 8;
constexpr int kOcSpins = 1 << 20;        // polls without news before a pass gives up

__global__ void __launch_bounds__(kOcWarps * 32)
k_oc_pass(int p, int n_vert, uint64_t *keys_a, uint64_t *keys_b, int *vals_a, int *vals_b, const int *__restrict__ bins,
          unsigned long long *__restrict__ tiles, OcHeader *h)
{
    chain_wait();
    chain_release();
    const int active = h->active;
    if ((active >> p & 1) == 0) return;
    const bool from_b = __popc(active & ((1 << p) - 1)) & 1;
    const uint64_t *__restrict__ keys_in = from_b ? keys_b : keys_a;
    uint64_t *__restrict__ keys_out = from_b ? keys_a : keys_b;
    const int *__restrict__ vals_in = from_b ? vals_b : vals_a;
    int *__restrict__ vals_out = from_b ? vals_a : vals_b;
    __shared__ uint16_t s_cnt[kOcWarps][kOcBins];
    __shared__ int s_off[kOcBins], s_sum[8], s_tile;
    __shared__ __align__(8) uint64_t s_keys[kOcSortTile];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, shift = 8 * p;
    // (a status may be set by other CTAs of this pass: one thread looks, so that all of a CTA stay or leave)
    if (threadIdx.x == 0) s_tile = *(volatile int *)&h->status != 0 ? -1 : atomicAdd(&h->tile[p], 1);
    for (int i = threadIdx.x; i < kOcWarps * kOcBins / 2; i += kOcWarps * 32) ((uint32_t *)s_cnt)[i] = 0;
    __syncthreads();
    const int tile = s_tile;
    if (tile < 0) return;
    const int64_t first = (int64_t)tile * kOcSortTile, base = first + w * (kOcRounds * 32) + lane;
    const int n_here = (int)min((int64_t)kOcSortTile, n_vert - first);
    if (n_here <= 0) return;
    uint64_t key[kOcRounds];
    int val[kOcRounds];
    uint16_t at[kOcRounds];
#pragma unroll
    for (int r = 0; r < kOcRounds; r++) {
        key[r] = base + r * 32 < n_vert ? keys_in[base + r * 32] : 0;
        val[r] = base + r * 32 < n_vert ? vals_in[base + r * 32] : 0;
    }
#pragma unroll
    for (int r = 0; r < kOcRounds; r++) {
        const bool in = base + r * 32 < n_vert;
        const int d = in ? (int)(key[r] >> shift & (kOcBins - 1)) : kOcBins;
        const unsigned peers = __match_any_sync(FGC_FULL_MASK, d);
        const int before = in ? s_cnt[w][d] : 0;
        __syncwarp();
        if (in && (peers & lanemask_lt()) == 0) s_cnt[w][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        at[r] = (uint16_t)(before + __popc(peers & lanemask_lt()));
    }
    __syncthreads();
    // the tile's number of this thread's digit, published; where the digit begins in the tile
    const int d = threadIdx.x;
    unsigned long long *mine = tiles + (size_t)tile * kOcBins + d;
    const unsigned long long tag = (unsigned long long)(p + 1) << 56, all = 1ull << 48, number = all - 1;
    int count = 0, begin = 0;
    if (d < kOcBins) {
#pragma unroll
        for (int k = 0; k < kOcWarps; k++) {
            const int c = s_cnt[k][d];
            s_cnt[k][d] = (uint16_t)count;
            count += c;
        }
        oc_store_tile(mine, tag | (tile == 0 ? all : 0) | (unsigned long long)count);
        begin = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FGC_FULL_MASK, begin, o);
            if (lane >= o) begin += t;
        }
        if (lane == 31) s_sum[w] = begin;
    }
    __syncthreads();
    if (d < kOcBins) {
        for (int k = 0; k < w; k++) begin += s_sum[k];
        begin -= count;
#pragma unroll
        for (int k = 0; k < kOcWarps; k++) s_cnt[k][d] += (uint16_t)begin;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kOcRounds; r++) {
        if (base + r * 32 < n_vert) {
            at[r] += s_cnt[w][(int)(key[r] >> shift & (kOcBins - 1))];
            s_keys[at[r]] = key[r];
        }
    }
    int spins = 0;
    if (d < kOcBins) {
        const int start = bins[p * kOcBins + d];
        long long before = 0;
        for (int t = tile - 1; t >= 0;) {
            unsigned long long word[kOcLookBack];
#pragma unroll
            for (int k = 0; k < kOcLookBack; k++) word[k] = t - k >= 0 ? oc_load_tile(tiles + (size_t)(t - k) * kOcBins + d) : 0;
            bool open = true;
            int taken = 0;
#pragma unroll
            for (int k = 0; k < kOcLookBack; k++) {
                if (open && word[k] >> 56 == tag >> 56) {
                    before += (long long)(word[k] & number);
                    taken++;
                    if (word[k] & all) { open = false; t = -1; }
                } else {
                    open = false;
                }
            }
            if (t >= 0) t -= taken;
            spins = taken > 0 ? 0 : spins + 1;
            if (spins >= kOcSpins) break;
        }
        if (spins >= kOcSpins) atomicOr(&h->status, FGC_STATUS_INTERNAL);
        else if (tile > 0) oc_store_tile(mine, tag | all | (unsigned long long)(before + count));
        s_off[d] = (int)(start + before - begin);
    }
    if (__syncthreads_or(spins >= kOcSpins)) return;
    int to[kOcRounds];
#pragma unroll
    for (int r = 0; r < kOcRounds; r++) {
        const int i = r * (kOcWarps * 32) + threadIdx.x;
        to[r] = 0;
        if (i < n_here) {
            const uint64_t k = s_keys[i];
            to[r] = s_off[(int)(k >> shift & (kOcBins - 1))] + i;
            if (FGC_DBG_OK(to[r] >= 0 && to[r] < n_vert, &h->status)) keys_out[to[r]] = k;
            else to[r] = 0;
        }
    }
    __syncthreads();
    int *s_vals = (int *)s_keys;
#pragma unroll
    for (int r = 0; r < kOcRounds; r++)
        if (base + r * 32 < n_vert) s_vals[at[r]] = val[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kOcRounds; r++) {
        const int i = r * (kOcWarps * 32) + threadIdx.x;
        if (i < n_here) vals_out[to[r]] = s_vals[i];
    }
}

// Whether the sort ended in the second buffers.
__device__ __forceinline__ bool oc_in_b(const OcHeader *h) { return __popc(h->active) & 1; }

// Position p of the sorted list starts an object when its (truth index, row split) differs
// from its predecessor's: ids with one truth index ascend.
__global__ void __launch_bounds__(256)
k_oc_flags(const uint64_t *__restrict__ keys_a, const uint64_t *__restrict__ keys_b, const int *__restrict__ vals_a,
           const int *__restrict__ vals_b, const int64_t *__restrict__ rs, int n_rs, int n_vert, int *__restrict__ flags, OcHeader *h)
{
    chain_wait();
    chain_release();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (h->status != 0) return;
    if (p == n_vert) { flags[p] = 0; return; }
    if (p > n_vert) return;
    const uint64_t *__restrict__ keys = oc_in_b(h) ? keys_b : keys_a;
    const int *__restrict__ vals = oc_in_b(h) ? vals_b : vals_a;
    const uint64_t none = h->none, key = keys[p];
    bool head = key != none;
    if (head && p > 0 && keys[p - 1] == key) head = rs[row_split_of(rs, n_rs, vals[p])] > vals[p - 1];
    flags[p] = head ? 1 : 0;
    if (key != none && (p + 1 == n_vert || keys[p + 1] == none)) h->n_valid = p + 1;
}

__global__ void __launch_bounds__(256)
k_oc_objects(const int *__restrict__ vals_a, const int *__restrict__ vals_b, const int64_t *__restrict__ rs,
             int n_rs, int n_vert, const int *__restrict__ scanned, int *__restrict__ obj_start,
             int *__restrict__ obj_split, unsigned long long *__restrict__ objects_per_split, OcHeader *h)
{
    chain_wait();
    chain_release();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_vert || h->status != 0) return;
    if (p == 0) {
        const int n_unique = scanned[n_vert];
        h->n_unique = n_unique;
        obj_start[n_unique] = h->n_valid;
    }
    const int k = scanned[p];
    if (scanned[p + 1] != k) {
        const int split = row_split_of(rs, n_rs, (oc_in_b(h) ? vals_b : vals_a)[p]);
        obj_start[k] = p;
        obj_split[k] = split;
        atomicAdd(objects_per_split + split, 1ull);
    }
}

__global__ void __launch_bounds__(256)
k_oc_largest(const int *__restrict__ obj_start, int n_vert, OcHeader *h)
{
    chain_wait();
    chain_release();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (h->status != 0 || k >= h->n_unique) return;
    int c = obj_start[k + 1] - obj_start[k];
    c = __reduce_max_sync(__activemask(), c);
    if ((threadIdx.x & 31) == 0 || k == 0) atomicMax(&h->n_maxuq, c);
}

// M, one warp per row and kOcRowRun columns (a thread per element, with a division each, took 28 us for 12 MB).
constexpr int kOcRowRun = 512;

__global__ void __launch_bounds__(256)
k_oc_fill_m(const OcHeader *__restrict__ h, const int *__restrict__ vals_a, const int *__restrict__ vals_b,
            const int *__restrict__ obj_start, int64_t n_unique, int64_t n_maxuq, int64_t *__restrict__ M)
{
    const int lane = threadIdx.x & 31;
    const int *__restrict__ vals = oc_in_b(h) ? vals_b : vals_a;
    const int64_t runs_per_row = (n_maxuq + kOcRowRun - 1) / kOcRowRun, n_runs = n_unique * runs_per_row;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t run = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; run < n_runs; run += n_warps) {
        const int64_t k = run / runs_per_row, j0 = (run - k * runs_per_row) * kOcRowRun;
        const int beg = obj_start[k], cnt = obj_start[k + 1] - beg;
        const int64_t j_end = min(j0 + kOcRowRun, n_maxuq);
#pragma unroll 4
        for (int64_t j = j0 + lane; j < j_end; j += 32) M[k * n_maxuq + j] = j < cnt ? (int64_t)vals[beg + j] : (int64_t)-1;
    }
}

// M_not, one warp per run of kOcRun consecutive columns of one row, kOcStep at a time.  The j-th non-member is  row start + j + t(j),
// t(j) = number of members with at most j non-members before them, which is non-decreasing in j: the warp searches it once for
// the first column of its run and then walks the member list forward.  The lanes hold the next 32 members: a vote says how many of
// them fall into the step's columns, and each of those is compared with a lane's columns.  Where 32 members are not enough for
// a step (a dense object) every column searches instead.  VEC2: rows are 16-byte aligned (even row length, aligned base) and a
// lane stores two adjacent columns at once.
// Writing bounds it: 3200 rows of 100 000 columns 350 us = 7.3 TB/s (a plain fill of the matrix 339 us).  With every member compared
// with all columns of 512 and 64-bit sums it was 413 us, bound by its 34 instructions a column, with 64 columns a step 396; the search by
// 32 probes instead of halves, which a run waits for: 384 -> 350.  Runs of 2048 / 4096 / 8192 columns 358 / 369 / 382, 512 columns a
// step (runs of 2048) 353.
constexpr int kOcRun = 1024, kOcStep = 256;

template <bool VEC2>
__global__ void __launch_bounds__(256)
k_oc_fill_m_not(const OcHeader *__restrict__ h, const int *__restrict__ vals_a, const int *__restrict__ vals_b,
                const int *__restrict__ obj_start, const int *__restrict__ obj_split, const int64_t *__restrict__ rs, int64_t n_unique,
                int n_maxrs, int64_t *__restrict__ M_not)
{
    const int lane = threadIdx.x & 31;
    const int *__restrict__ vals = oc_in_b(h) ? vals_b : vals_a;
    const int runs_per_row = (int)(((int64_t)n_maxrs + kOcRun - 1) / kOcRun);
    const int64_t n_runs = n_unique * runs_per_row;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t run = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; run < n_runs; run += n_warps) {
        const int64_t k = run / runs_per_row;
        const int64_t run0 = (run - k * runs_per_row) * kOcRun;
        const int beg = obj_start[k], cnt = obj_start[k + 1] - beg;
        const int e = obj_split[k];
        const int row_start = (int)rs[e];                                 // ids have 31 bits
        const uint32_t n_non = (uint32_t)((int)rs[e + 1] - row_start - cnt);
        // member i (a global point id) has  members[i] - row_start - i  non-members before it
        const int *__restrict__ members = vals + beg;
        auto members_up_to = [&](uint32_t j, int lo, int hi) {
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if ((uint32_t)(members[mid] - row_start - mid) <= j) lo = mid + 1; else hi = mid;
            }
            return lo;
        };
        int64_t *__restrict__ row = M_not + k * (int64_t)n_maxrs;
        const uint32_t run_end = (uint32_t)min(run0 + kOcRun, (int64_t)n_maxrs);
        // members before the columns, found by 32 probes at a time
        int t = 0;
        for (int end = cnt; t < end;) {
            const int step = (end - t + 31) >> 5, at = t + lane * step;
            const bool up_to = at < end && members[at] - row_start - at < (int)run0;
            const int found = __popc(__ballot_sync(FGC_FULL_MASK, up_to));
            if (found == 0) break;
            if (step == 1) { t += found; break; }
            end = min(end, t + found * step);
            t += (found - 1) * step + 1;
        }
        int held = t;                                                     // the first member that a lane holds
        auto hold = [&]() { return held + lane < cnt ? (uint32_t)(members[held + lane] - row_start - held - lane) : 0x7fffffffu; };
        uint32_t next = hold();
        // (columns up to a step beyond the last: more than 31 bits)
        for (uint32_t j0 = (uint32_t)run0; j0 < run_end; j0 += kOcStep) {
            constexpr int PER = kOcStep / 32;                             // columns per lane
            const uint32_t j1 = run_end - j0 < kOcStep ? run_end : j0 + kOcStep;
            const uint32_t c0 = j0 + (VEC2 ? 2 * lane : lane);
            auto column = [&](int u) { return c0 + (VEC2 ? 64 * (u >> 1) + (u & 1) : 32 * u); };
            int in = __popc(__ballot_sync(FGC_FULL_MASK, next < j1));
            if (in == 32 && held < t) {
                held = t;
                next = hold();
                in = __popc(__ballot_sync(FGC_FULL_MASK, next < j1));
            }
            uint32_t id[PER];
#pragma unroll
            for (int u = 0; u < PER; u++) id[u] = row_start + t + column(u);
            if (in < 32) {
                for (int i = t - held; i < in; i++) {
                    const int b = (int)(__shfl_sync(FGC_FULL_MASK, next, i) - c0);
#pragma unroll
                    for (int u = 0; u < PER; u++) id[u] += (int)(column(u) - c0) >= b ? 1 : 0;
                }
                t = held + in;
            } else {
                const int t1 = members_up_to(j1 - 1, t, cnt);
#pragma unroll
                for (int u = 0; u < PER; u++) id[u] += members_up_to(column(u), t, t1) - t;
                held = t = t1;
                next = hold();
            }
            int64_t *__restrict__ out = row + c0;
            if (j0 + kOcStep <= min(run_end, n_non)) {
#pragma unroll
                for (int u = 0; u < PER; u += VEC2 ? 2 : 1) {
                    if (VEC2) *reinterpret_cast<uint4 *>(out + 32 * u) = make_uint4(id[u], 0u, id[u + 1], 0u);
                    else out[32 * u] = (int64_t)id[u];
                }
            } else {
#pragma unroll
                for (int u = 0; u < PER; u += VEC2 ? 2 : 1) {
                    const int64_t v = column(u) < n_non ? (int64_t)id[u] : (int64_t)-1;
                    if (column(u) >= j1) continue;
                    if (VEC2)                      // an even row length: the second column is in the row if the first is
                        *reinterpret_cast<longlong2 *>(out + 32 * u) =
                            make_longlong2(v, column(u + 1) < n_non ? (int64_t)id[u + 1] : (int64_t)-1);
                    else
                        out[32 * u] = v;
                }
            }
        }
    }
}

// out[(v*K + k)*F + f] = idx[v, k] == -1 ? default : feat[idx[v, k]*F + f], on raw words
template <typename W>
__global__ void __launch_bounds__(256)
k_select_with_default(const int64_t *__restrict__ idx, const W *__restrict__ feat, int64_t n_rows_feat,
                      int64_t n_idx, int64_t F, W default_word, W *__restrict__ out)
{
    const int64_t total = n_idx * F;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
        const int64_t e = t / F, f = t - e * F;
        const int64_t i = idx[e];
        out[t] = (i >= 0 && i < n_rows_feat) ? feat[i * F + f] : default_word;
    }
}

}  // namespace fgc

extern "C" size_t fgc_oc_workspace_bytes(int64_t n_vert)
{
    if (n_vert < 0 || n_vert > fgc::kOcMostPoints) return 0;
    return fgc::oc_workspace_layout(n_vert).total;
}

extern "C" int fgc_oc_prepare(const int64_t *asso_idx, int64_t n_vert, const int64_t *row_splits, int64_t n_rs,
                              void *workspace, size_t workspace_bytes, int64_t *objects_per_split,
                              fgc_stream_t stream)
{
    FGC_NVTX("fgc_oc_prepare");
    using namespace fgc;
    if (n_vert < 0 || n_rs < 1 || !row_splits || (!objects_per_split && n_rs > 1)) return FGC_ERR_BAD_ARGUMENT;
    if (n_vert > kOcMostPoints || n_rs > 0x7fffffff) return FGC_ERR_TOO_LARGE;
    const OcWorkspace L = oc_workspace_layout(n_vert);
    if (!workspace || workspace_bytes < L.total || ((uintptr_t)workspace & 255)) return FGC_ERR_WORKSPACE;
    cudaStream_t s = (cudaStream_t)stream;
    char *ws = (char *)workspace;
    OcHeader *h = (OcHeader *)(ws + L.header);
    FGC_RETURN_IF_CUDA(cudaMemsetAsync(h, 0, kOcHeaderBytes, s));
    if (n_vert > 0 && !asso_idx) return FGC_ERR_BAD_ARGUMENT;
    const int n = (int)n_vert, nr = (int)n_rs, tiles = oc_sort_tiles(n);
    const int blocks = (n + 255) / 256, first = blocks < sm_count() * 8 ? (blocks > 0 ? blocks : 1) : sm_count() * 8;
    uint64_t *keys_a = (uint64_t *)(ws + L.keys_a), *keys_b = (uint64_t *)(ws + L.keys_b);
    int *vals_a = (int *)(ws + L.vals_a), *vals_b = (int *)(ws + L.vals_b);
    int *flags = (int *)(ws + L.flags);
    int *blocksums = (int *)(ws + L.blocksums);
    int *obj_start = (int *)(ws + L.obj_start);
    int *obj_split = (int *)(ws + L.obj_split);
    int *bins = (int *)(ws + L.bins);
    unsigned long long *states = (unsigned long long *)(ws + L.tiles), *per_split = (unsigned long long *)objects_per_split;
    FGC_RETURN_IF_CUDA(launch_chained(k_oc_first, first, 256, 0, s, asso_idx, row_splits, nr, n, states, (int64_t)tiles, bins, per_split, h));
    if (n == 0) return FGC_OK;
    // stable radix sort: equal truth indices keep ascending point ids
    FGC_RETURN_IF_CUDA(launch_chained(k_oc_keys, tiles, 256, 0, s, asso_idx, n, keys_a, vals_a, bins, h));
    for (int p = 0; p < kOcPasses; p++)
        FGC_RETURN_IF_CUDA(launch_chained(k_oc_pass, tiles, kOcWarps * 32, 0, s, p, n, keys_a, keys_b, vals_a, vals_b, bins, states, h));
    FGC_RETURN_IF_CUDA(launch_chained(k_oc_flags, (n + 1 + 255) / 256, 256, 0, s, keys_a, keys_b, vals_a, vals_b, row_splits, nr, n, flags, h));
    const int scan_blocks = (int)ceil_div64((int64_t)n + 1, kScanTile);
    FGC_RETURN_IF_CUDA(launch_chained(k_scan_tile_sums_top, scan_blocks, 256, 0, s, flags, nullptr, n + 1, blocksums, &h->scan_ticket));
    FGC_RETURN_IF_CUDA(launch_chained(k_scan_apply, scan_blocks, 256, 0, s, flags, nullptr, n + 1, blocksums));
    FGC_RETURN_IF_CUDA(launch_chained(k_oc_objects, blocks, 256, 0, s, vals_a, vals_b, row_splits, nr, n, flags, obj_start, obj_split,
                                      per_split, h));
    FGC_RETURN_IF_CUDA(launch_chained(k_oc_largest, blocks, 256, 0, s, obj_start, n, h));
    return FGC_OK;
}

extern "C" int fgc_oc_read_sizes(const void *workspace, int32_t *status_host, int64_t sizes_host[3],
                                 fgc_stream_t stream)
{
    using namespace fgc;
    if (!workspace || !status_host || !sizes_host) return FGC_ERR_BAD_ARGUMENT;
    OcHeader h;
    cudaStream_t s = (cudaStream_t)stream;
    FGC_RETURN_IF_CUDA(cudaMemcpyAsync(&h, workspace, sizeof(OcHeader), cudaMemcpyDeviceToHost, s));
    FGC_RETURN_IF_CUDA(cudaStreamSynchronize(s));
    *status_host = h.status;
    sizes_host[0] = h.n_unique;
    sizes_host[1] = h.n_maxuq;
    sizes_host[2] = h.n_maxrs;
    return FGC_OK;
}

extern "C" int fgc_oc_fill(const void *workspace, size_t workspace_bytes, int64_t n_vert,
                           const int64_t *row_splits, int64_t n_unique, int64_t n_maxuq, int64_t n_maxrs,
                           int64_t *out_M, int64_t *out_M_not_or_null, fgc_stream_t stream)
{
    FGC_NVTX("fgc_oc_fill");
    using namespace fgc;
    if (n_vert < 0 || n_unique < 0 || n_maxuq < 0 || n_maxrs < 0 || !row_splits) return FGC_ERR_BAD_ARGUMENT;
    if (n_vert > kOcMostPoints) return FGC_ERR_TOO_LARGE;
    const OcWorkspace L = oc_workspace_layout(n_vert);
    if (!workspace || workspace_bytes < L.total || ((uintptr_t)workspace & 255)) return FGC_ERR_WORKSPACE;
    cudaStream_t s = (cudaStream_t)stream;
    const char *ws = (const char *)workspace;
    const OcHeader *h = (const OcHeader *)(ws + L.header);
    const int *vals_a = (const int *)(ws + L.vals_a), *vals_b = (const int *)(ws + L.vals_b);
    const int *obj_start = (const int *)(ws + L.obj_start);
    const int *obj_split = (const int *)(ws + L.obj_split);
    const int64_t m_total = n_unique * n_maxuq, mn_total = n_unique * n_maxrs;
    if (m_total > 0) {
        if (!out_M) return FGC_ERR_BAD_ARGUMENT;
        int64_t blocks = ceil_div64(n_unique * ceil_div64(n_maxuq, kOcRowRun), 8);
        if (blocks > fgc::sm_count() * 64) blocks = fgc::sm_count() * 64;
        k_oc_fill_m<<<(unsigned)blocks, 256, 0, s>>>(h, vals_a, vals_b, obj_start, n_unique, n_maxuq, out_M);
        FGC_CHECK_LAUNCH();
    }
    if (out_M_not_or_null && mn_total > 0) {
        if (n_maxrs > 0x7fffffff) return FGC_ERR_TOO_LARGE;
        const int64_t runs = n_unique * ceil_div64(n_maxrs, kOcRun);
        int64_t blocks = ceil_div64(runs, 8);           // 8 warps per CTA, one run per warp and pass
        if (blocks > 0x7fffffff) blocks = 0x7fffffff;
        if ((n_maxrs & 1) == 0 && ((uintptr_t)out_M_not_or_null & 15) == 0)
            k_oc_fill_m_not<true><<<(unsigned)blocks, 256, 0, s>>>(h, vals_a, vals_b, obj_start, obj_split, row_splits, n_unique,
                                                                   (int)n_maxrs, out_M_not_or_null);
        else
            k_oc_fill_m_not<false><<<(unsigned)blocks, 256, 0, s>>>(h, vals_a, vals_b, obj_start, obj_split, row_splits, n_unique,
                                                                    (int)n_maxrs, out_M_not_or_null);
        FGC_CHECK_LAUNCH();
    }
    return FGC_OK;
}

extern "C" int fgc_select_with_default(const int64_t *idx, int64_t n_idx, const void *feat, int64_t n_rows_feat,
                                       int64_t n_feat, int32_t word_bytes, const void *default_word_host,
                                       void *out, fgc_stream_t stream)
{
    FGC_NVTX("fgc_select_with_default");
    using namespace fgc;
    if (n_idx < 0 || n_rows_feat < 0 || n_feat < 0 || !default_word_host) return FGC_ERR_BAD_ARGUMENT;
    if (word_bytes != 4 && word_bytes != 8) return FGC_ERR_BAD_ARGUMENT;
    const int64_t total = n_idx * n_feat;
    if (total == 0) return FGC_OK;
    if (!idx || !out || (!feat && n_rows_feat > 0)) return FGC_ERR_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    int64_t blocks = ceil_div64(total, 256);
    if (blocks > fgc::sm_count() * 64) blocks = fgc::sm_count() * 64;
    if (word_bytes == 4) {
        uint32_t w;
        memcpy(&w, default_word_host, 4);
        k_select_with_default<uint32_t><<<(unsigned)blocks, 256, 0, s>>>(
            idx, (const uint32_t *)feat, n_rows_feat, n_idx, n_feat, w, (uint32_t *)out);
    } else {
        uint64_t w;
        memcpy(&w, default_word_host, 8);
        k_select_with_default<uint64_t><<<(unsigned)blocks, 256, 0, s>>>(
            idx, (const uint64_t *)feat, n_rows_feat, n_idx, n_feat, w, (uint64_t *)out);
    }
    FGC_CHECK_LAUNCH();
    return FGC_OK;
}
