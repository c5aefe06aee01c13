// binned_select_knn forward for sm_100a: the sort of a small search tree in one launch.
//
// For ten thousand points the thirteen launches of the sort (knn_tree.cu) cost several times their work.  Here a cluster of eight CTAs finds the
// extents, makes the keys and does two or three radix passes of 11 bits, with a hardware barrier between one and the next; the totals
// of the digits are read from the other CTAs' shared memory.  Keys have 22 or 32 bits -- cells of the curve are a sixteenth of the extent wide
// or narrower, which for so few points gives leaves as good as more bits would -- and the order among equal keys is the original one.
#include "cluster.cuh"
#include "knn_grid_build.cuh"
#include "knn_tree_build.cuh"

namespace fgc {

constexpr int kSmallRounds = (int)(kSmallTree / kClusterAll);
static_assert(kSmallRounds * kClusterAll == kSmallTree, "points do not fill the threads");

struct SmallTreePart {
    uint32_t min_key[kTreeKeyDims], max_key[kTreeKeyDims], bad;
};
constexpr int kPartWords = sizeof(SmallTreePart) / 4;

struct SmallTreeShared {
    uint16_t count[kClusterWarps][kRadixBins];
    int total[kRadixBins], base[kRadixBins];
};

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads)
k_tree_small(const float *coords, int n, int n_coords, int key_dims, int bits, int passes, const int64_t *row_splits, int n_rs, KnnGrid *g,
             KnnTree *tree, uint32_t *keys, int *ids, int *ids_last, volatile int32_t *info_mapped)
{
    chain_wait();
    chain_release();
    extern __shared__ __align__(16) char s_raw[];
    SmallTreeShared &s = *reinterpret_cast<SmallTreeShared *>(s_raw);
    __shared__ SmallTreePart s_mine;
    __shared__ uint32_t s_all[kClusterCtas][kPartWords];
    __shared__ int s_part[kClusterWarps];
    __shared__ KnnTree s_tree;
    __shared__ int s_status;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, cta = blockIdx.x, first = cta * kClusterThreads + t;
    if (cta == 0)
        for (int i = t; i < (int)((kGridHeaderBytes + kHardTicketBytes) / sizeof(int)); i += kClusterThreads) ((int *)g)[i] = 0;
    if (t < kPartWords) ((uint32_t *)&s_mine)[t] = 0;
    if (t < (int)(sizeof(KnnTree) / sizeof(int))) ((int *)&s_tree)[t] = 0;
    __syncthreads();
    {
        uint32_t lmin[kTreeKeyDims] = {}, lmax[kTreeKeyDims] = {}, bad = 0;
#pragma unroll
        for (int k = 0; k < kSmallRounds; k++) {
            const int v = first + k * kClusterAll;
            if (v < n) {
                const float *row = coords + (size_t)v * n_coords;
#pragma unroll
                for (int c = 0; c < kTreeKeyDims; c++) {
                    if (c < n_coords) {
                        const float x = __ldg(row + c);
                        if (!is_finite_bits(x)) bad |= 1;
                        const uint32_t key = float_to_ordered(x);
                        lmin[c] = max(lmin[c], ~key);
                        lmax[c] = max(lmax[c], key);
                    }
                }
                for (int c = kTreeKeyDims; c < n_coords; c++)
                    if (!is_finite_bits(__ldg(row + c))) bad |= 1;
            }
        }
        // row_splits must start at 0, end at n_vert and never decrease
        for (int i = first; i < n_rs; i += kClusterAll)
            if (i == 0 ? row_splits[0] != 0 : (row_splits[i] < row_splits[i - 1] || (i == n_rs - 1 && row_splits[i] != (int64_t)n))) bad |= 2;
        bad = __reduce_or_sync(FGC_FULL_MASK, bad);
        if (lane == 0 && bad) atomicOr(&s_mine.bad, bad);
#pragma unroll
        for (int c = 0; c < kTreeKeyDims; c++) {
            const uint32_t x = __reduce_max_sync(FGC_FULL_MASK, lmin[c]), y = __reduce_max_sync(FGC_FULL_MASK, lmax[c]);
            if (lane == 0) { atomicMax(&s_mine.min_key[c], x); atomicMax(&s_mine.max_key[c], y); }
        }
    }
    cluster_barrier();
    if (t < kClusterCtas * kPartWords) s_all[t / kPartWords][t % kPartWords] = cluster_word((uint32_t *)&s_mine + t % kPartWords, t / kPartWords);
    __syncthreads();
    // every CTA sets the curve up for itself
    if (t == 0) {
        uint32_t min_key[kTreeKeyDims], max_key[kTreeKeyDims], bad = 0;
        for (int k = 0; k < kClusterCtas; k++) bad |= s_all[k][2 * kTreeKeyDims];
#pragma unroll
        for (int c = 0; c < kTreeKeyDims; c++) {
            min_key[c] = max_key[c] = 0;
#pragma unroll
            for (int k = 0; k < kClusterCtas; k++) {
                min_key[c] = max(min_key[c], s_all[k][c]);
                max_key[c] = max(max_key[c], s_all[k][kTreeKeyDims + c]);
            }
        }
        tree_setup(&s_tree, min_key, max_key, key_dims, bits);
        s_status = (bad & 1 ? FGC_STATUS_NONFINITE : 0) | (bad & 2 ? FGC_STATUS_BAD_ROW_SPLITS : 0);
    }
    __syncthreads();
    const bool good = s_status == 0;
    if (cta == 0) {
        if (t < (int)(sizeof(KnnTree) / sizeof(int))) ((int *)tree)[t] = ((const int *)&s_tree)[t];
        if (t == 0) {
            g->n_events = n_rs - 1;
            g->status = s_status;
            if (info_mapped) store_info(info_mapped, s_status, 0);
        }
    }
    if (!good) {
        cluster_barrier();               // (a CTA that has left can not be read)
        return;
    }

    // A warp owns consecutive places, 32 a round: lanes with equal digits find one another by a match, the warp's counter of the digit
    // gives the rank.
    const int rounds = (n + kClusterAll - 1) / kClusterAll, mine = cta * kClusterThreads * rounds + w * 32 * rounds + lane;
    uint32_t key[kSmallRounds];
    int id[kSmallRounds], rank[kSmallRounds];
#pragma unroll
    for (int r = 0; r < kSmallRounds; r++) {
        const int v = mine + 32 * r;
        key[r] = 0;
        id[r] = v;
        if (r < rounds && v < n)
            key[r] = (bits * key_dims < 32 ? (uint32_t)row_split_of(row_splits, n_rs, v) << (bits * key_dims) : 0u) | tree_key(&s_tree, coords + (size_t)v * n_coords, key_dims, bits);
    }
    for (int pass = 0; pass < passes; pass++) {
        const int shift = pass * kRadixBits;
        for (int i = t; i < (int)sizeof(s.count) / 4; i += kClusterThreads) ((uint32_t *)s.count)[i] = 0;
        if (pass > 0) {
#pragma unroll
            for (int r = 0; r < kSmallRounds; r++) {
                const int at = mine + 32 * r;
                if (r < rounds && at < n) { key[r] = __ldcg(keys + at); id[r] = __ldcg(ids + at); }
            }
            cluster_barrier();           // (the places are written again below)
        } else {
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < kSmallRounds; r++) {
            const bool there = r < rounds && mine + 32 * r < n;
            const int d = there ? (int)(key[r] >> shift & (kRadixBins - 1)) : kRadixBins;
            const unsigned peers = __match_any_sync(FGC_FULL_MASK, d);
            const int before = there ? s.count[w][d] : 0;
            __syncwarp();
            if (there && (peers & lanemask_lt()) == 0) s.count[w][d] = (uint16_t)(before + __popc(peers));
            __syncwarp();
            rank[r] = before + __popc(peers & lanemask_lt());
        }
        __syncthreads();
        for (int d = t; d < kRadixBins; d += kClusterThreads) {
            int run = 0;
#pragma unroll
            for (int k = 0; k < kClusterWarps; k++) {
                const int c = s.count[k][d];
                s.count[k][d] = (uint16_t)run;
                run += c;
            }
            s.total[d] = run;
        }
        cluster_barrier();
        static_assert(kRadixBins == 4 * kClusterThreads, "four digits a thread");
        int4 all = make_int4(0, 0, 0, 0), lower = all;
#pragma unroll
        for (int k = 0; k < kClusterCtas; k++) {
            const int4 c = cluster_four(s.total + 4 * t, k);
            if (k == cta) lower = all;
            all.x += c.x; all.y += c.y; all.z += c.z; all.w += c.w;
        }
        int everything;
        const int begin = cta_scan(all.x + all.y + all.z + all.w, s_part, everything);
        *reinterpret_cast<int4 *>(s.base + 4 * t) = make_int4(begin + lower.x, begin + all.x + lower.y, begin + all.x + all.y + lower.z,
                                                              begin + all.x + all.y + all.z + lower.w);
        __syncthreads();
        const bool last = pass + 1 == passes;
#pragma unroll
        for (int r = 0; r < kSmallRounds; r++) {
            if (r < rounds && mine + 32 * r < n) {
                const int d = (int)(key[r] >> shift & (kRadixBins - 1)), to = s.base[d] + s.count[w][d] + rank[r];
                if (FGC_DBG_OK(to >= 0 && to < n, &g->status)) {
                    if (!last) keys[to] = key[r];
                    (last ? ids_last : ids)[to] = id[r];
                }
            }
        }
        cluster_barrier();
    }
}

bool small_tree_bits(int64_t n_vert, int n_coords, int64_t n_rs, int *key_dims, int *bits, int *passes)
{
    if (n_vert > kSmallTree) return false;
    int ebits = 0;
    while (((int64_t)1 << ebits) < n_rs - 1) ebits++;
    *key_dims = n_coords < kTreeKeyDims ? n_coords : kTreeKeyDims;
    const int enough = n_coords <= 3 ? 5 : 4;
    for (*passes = 2; *passes <= 3; ++*passes) {
        const int left = (*passes == 2 ? 2 * kRadixBits : 32) - ebits;
        *bits = left / *key_dims;
        if (*bits >= enough) return true;
    }
    return false;
}

cudaError_t launch_tree_small(const float *coords, int n, int n_coords, int key_dims, int bits, int passes, const int64_t *row_splits, int n_rs, KnnGrid *g,
                              KnnTree *tree, uint32_t *keys, int *ids, int *ids_last, volatile int32_t *info_mapped, cudaStream_t s)
{
    const cudaError_t e = cudaFuncSetAttribute(k_tree_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallTreeShared));
    if (e != cudaSuccess) return e;
    k_tree_small<<<kClusterCtas, kClusterThreads, sizeof(SmallTreeShared), s>>>(coords, n, n_coords, key_dims, bits, passes, row_splits, n_rs, g, tree, keys,
                                                                               ids, ids_last, info_mapped);
    return cudaGetLastError();
}

}  // namespace fgc
