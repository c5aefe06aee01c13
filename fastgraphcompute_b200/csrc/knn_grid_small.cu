// binned_select_knn forward for sm_100a: the search grid of a small batch in one launch.
//
// A chain of eleven short launches (knn_grid.cu) costs more than the work: for 10 k points the host spends 35 us on the launches and
// the device 45 us on their latencies; this kernel takes 24 us (extents 3, grid 4, histogram 6, scan 3, order 8).  Here a cluster of eight CTAs does the same passes one after the other with a hardware
// barrier between them; every thread keeps the cells and ranks of its points in registers.  What is computed -- the grid, the
// order of cells, points and ids -- is what the chain computes, by the same functions.  The words that the host waits for are
// written as soon as the checks are done and the form of the grid is known, and the cell order goes to the caller's array on the way.
#include <cstddef>

#include "cluster.cuh"
#include "knn_grid_build.cuh"

namespace fgc {

constexpr int kSmallPoints = (int)(kSmallBuild / kClusterAll);         // of a thread
static_assert(kSmallPoints * kClusterAll == kSmallBuild, "points do not fill the threads");
static_assert(kSortWarps == kClusterWarps, "large cells are sorted by the CTAs of the cluster");
constexpr int kSmallScan = 4;                                          // table entries of a thread per scan step
constexpr int kSmallSplits = kClusterThreads;                          // row splits that are kept in shared memory

// What a CTA has found, read by all others.
struct SmallPart {
    uint32_t min_key[4], max_key[4], bad, n_may;
    uint32_t sq[2][2];                   // density statistic of two passes, low and high word
    uint32_t entries;                    // points in the CTA's share of the table
};
constexpr int kSmallWords = sizeof(SmallPart) / 4;

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads)
k_build_small(const GridBuild a)
{
    chain_wait();
    chain_release();
    extern __shared__ int s_sort[];
    __shared__ SmallPart s_mine;
    __shared__ uint32_t s_all[kClusterCtas][kSmallWords];
    __shared__ unsigned long long s_sq;
    __shared__ int s_part[kSortWarps];
    __shared__ int s_splits[kSmallSplits];
    __shared__ KnnGrid s_grid;
    const int t = threadIdx.x, lane = t & 31, wib = t >> 5, cta = blockIdx.x, first = cta * kClusterThreads + t;
    const int n = a.n_vert;
    KnnGrid *g = a.grid;
    auto gather = [&]() {
        if (t < kClusterCtas * kSmallWords) s_all[t / kSmallWords][t % kSmallWords] = cluster_word((uint32_t *)&s_mine + t % kSmallWords, t / kSmallWords);
        __syncthreads();
    };

    // extents, checks and the number of possible neighbours; tickets and the first table cleared
    for (int i = first; i < (int)((kGridHeaderBytes + kHardTicketBytes) / sizeof(int)); i += kClusterAll) ((int *)g)[i] = 0;
    {
        const int n_counts = a.bins_cap_first * (a.n_rs - 1) * a.mirror + 1;
        for (int i = first; i < n_counts; i += kClusterAll) a.counts[i] = 0;
    }
    if (t < kSmallWords) ((uint32_t *)&s_mine)[t] = 0;
    if (t < (int)(sizeof(KnnGrid) / sizeof(int))) ((int *)&s_grid)[t] = 0;
    if (t == 0) s_sq = 0;
    __syncthreads();
    {
        uint32_t bad = 0, n_may = 0, lmin[4] = {0, 0, 0, 0}, lmax[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < kSmallPoints; k++) {
            const int v = first + k * kClusterAll;
            if (v < n) {
                const float *row = a.coords + (size_t)v * a.n_coords;
                if (a.mirror > 1) {
                    const int64_t d = a.direction[v];
                    n_may += d != 1 && d != 2;
                }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c < a.n_coords) {
                        const float x = __ldg(row + c);
                        if (!is_finite_bits(x)) bad |= 1;
                        if (c < a.n_bin_dims) {
                            const uint32_t key = float_to_ordered(x);
                            lmin[c] = max(lmin[c], ~key);
                            lmax[c] = max(lmax[c], key);
                        }
                    }
                }
                for (int c = 4; c < a.n_coords; c++)
                    if (!is_finite_bits(__ldg(row + c))) bad |= 1;
            }
        }
        // row_splits must start at 0, end at n_vert and never decrease
        if (t < a.n_rs && t < kSmallSplits) s_splits[t] = (int)min(max(a.row_splits[t], (int64_t)0), (int64_t)n);
        for (int i = first; i < a.n_rs; i += kClusterAll)
            if (i == 0 ? a.row_splits[0] != 0 : (a.row_splits[i] < a.row_splits[i - 1] || (i == a.n_rs - 1 && a.row_splits[i] != (int64_t)n))) bad |= 2;
        bad = __reduce_or_sync(FGC_FULL_MASK, bad);
        n_may = __reduce_add_sync(FGC_FULL_MASK, n_may);
        if (lane == 0) {
            if (bad) atomicOr(&s_mine.bad, bad);
            if (n_may) atomicAdd(&s_mine.n_may, n_may);
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint32_t x = __reduce_max_sync(FGC_FULL_MASK, lmin[c]), y = __reduce_max_sync(FGC_FULL_MASK, lmax[c]);
            if (lane == 0) { atomicMax(&s_mine.min_key[c], x); atomicMax(&s_mine.max_key[c], y); }
        }
    }
    cluster_barrier();
    // every CTA chooses the grid for itself
    gather();
    if (t == 0) {
        SmallPart p;
#pragma unroll
        for (int w = 0; w < 10; w++) {
            uint32_t x = s_all[0][w];
#pragma unroll
            for (int k = 1; k < kClusterCtas; k++) x = w < 8 ? max(x, s_all[k][w]) : (w == 8 ? x | s_all[k][w] : x + s_all[k][w]);
            ((uint32_t *)&p)[w] = x;
        }
        int mirror = a.mirror, bins_target = a.bins_target, bins_cap = a.bins_cap;
        if (mirror > 1) choose_sets(p.n_may, n, a.adaptive, mirror, bins_target, bins_cap);
        grid_setup(&s_grid, p.min_key, p.max_key, (p.bad & 1) != 0, a.n_rs, a.n_bin_dims, bins_target, a.bins_cap_first, bins_cap, (p.bad & 2) != 0, mirror);
    }
    __syncthreads();
    const bool good = s_grid.status == 0, late_words = good && a.allow_fallback;           // (its form may change)
    if (cta == 0 && t == 0 && a.info_mapped && !late_words) store_info(a.info_mapped, s_grid.status, s_grid.gdims);

    // histogram, density pass, and again on the grid that it chose
    int bin[kSmallPoints], rank[kSmallPoints];
    for (int pass = 0; pass < 3; pass++) {
        // (pass p follows the p-th density pass that changed the grid)
        const bool look = good && (pass == 0 ? a.adaptive != 0 : (pass == 1 && a.allow_fallback && s_grid.fallback3));
        if (pass > 0) {
            for (int i = first; i < s_grid.total_bins + 1; i += kClusterAll) a.counts[i] = 0;
            if (t == 0) s_sq = 0;
            cluster_barrier();
        }
        unsigned may = 0;                  // of the thread's points
#pragma unroll
        for (int k = 0; k < kSmallPoints; k++) {
            const int v = first + k * kClusterAll;
            bin[k] = -1;
            if (good && v < n) {
                int e;
                if (a.n_rs <= kSmallSplits) {
                    int lo = 1, hi = a.n_rs;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (s_splits[mid] > v) hi = mid; else lo = mid + 1;
                    }
                    e = lo - 1;
                } else {
                    e = row_split_of(a.row_splits, a.n_rs, v);
                }
                bin[k] = point_cell(&s_grid, a.coords + (size_t)v * a.n_coords, e);
                may |= 1u << k;
                if (s_grid.mirror > 1) {
                    const int64_t d = a.direction[v];
                    if (d == 1 || d == 2) {
                        bin[k] += s_grid.n_events * s_grid.B;
                        may &= ~(1u << k);
                    }
                }
                if (!FGC_DBG_OK(bin[k] >= 0 && bin[k] < s_grid.total_bins, &g->status)) bin[k] = 0;
            }
        }
        // warp-aggregated: one atomic per distinct cell in the warp; those of all points are on their way together
        unsigned peers[kSmallPoints];
#pragma unroll
        for (int k = 0; k < kSmallPoints; k++) {
            peers[k] = __match_any_sync(FGC_FULL_MASK, bin[k]);
            rank[k] = 0;
            if (bin[k] >= 0 && (peers[k] & lanemask_lt()) == 0) rank[k] = atomicAdd(a.counts + bin[k], __popc(peers[k]));
        }
        unsigned long long sq = 0;
#pragma unroll
        for (int k = 0; k < kSmallPoints; k++) {
            rank[k] = __shfl_sync(FGC_FULL_MASK, rank[k], __ffs(peers[k]) - 1) + __popc(peers[k] & lanemask_lt());
            if (may >> k & 1) sq += 2ull * (unsigned long long)rank[k] + 1ull;
        }
        if (look) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(FGC_FULL_MASK, sq, o);
            if (lane == 0 && sq) atomicAdd(&s_sq, sq);
            __syncthreads();
            if (t == 0) { s_mine.sq[pass][0] = (uint32_t)s_sq; s_mine.sq[pass][1] = (uint32_t)(s_sq >> 32); }
        }
        cluster_barrier();
        if (!look) break;
        gather();
        const int refined = s_grid.refined;
        __syncthreads();
        if (t == 0) {
            unsigned long long sum = 0;
#pragma unroll
            for (int k = 0; k < kClusterCtas; k++) sum += (unsigned long long)s_all[k][11 + 2 * pass] << 32 | s_all[k][10 + 2 * pass];
            grid_refine(&s_grid, sum, n, a.seen_target, a.seen_target3, a.bins_target, pass, pass == 0 && a.allow_fallback);
        }
        __syncthreads();
        if (s_grid.refined == refined) break;
    }
    // the grid for those who read it
    if (cta == 0) {
        // (the counts of large cells begin at zero, and the status may have bits of its own already)
        if (t < (int)(sizeof(KnnGrid) / sizeof(int)) && t != (int)(offsetof(KnnGrid, status) / 4) &&
            t != (int)(offsetof(KnnGrid, n_big_cells) / 4) && t != (int)(offsetof(KnnGrid, n_huge_cells) / 4))
            ((int *)g)[t] = ((const int *)&s_grid)[t];
        if (t == 0 && s_grid.status != 0) atomicOr(&g->status, s_grid.status);
        if (t == 0 && a.info_mapped && late_words) store_info(a.info_mapped, s_grid.status, s_grid.gdims + 16 * s_grid.fallback3);
    }
    if (!good) {
        for (int v = first; v < n; v += kClusterAll) {
            a.sorig[v] = v;
            if (a.out_order) a.out_order[v] = v;
        }
        cluster_barrier();               // (a CTA that has left can not be read)
        return;
    }

    // exclusive scan: a share of the table per CTA, in registers where it fits
    {
        const int entries = s_grid.total_bins + 1;
        const int share = ((entries + kClusterCtas - 1) / kClusterCtas + 3) & ~3, lo = min(entries, cta * share), hi = min(entries, lo + share);
        const bool once = share <= kClusterThreads * kSmallScan;
        int x[kSmallScan], sum = 0, all, before;
        if (once) {
#pragma unroll
            for (int k = 0; k < kSmallScan; k++) {
                const int at = lo + t * kSmallScan + k;
                x[k] = at < hi ? a.counts[at] : 0;
                sum += x[k];
            }
        } else {
            for (int i = lo + t; i < hi; i += kClusterThreads) sum += a.counts[i];
        }
        before = cta_scan(sum, s_part, all);
        if (t == 0) s_mine.entries = all;
        cluster_barrier();
        gather();
        int carry = 0;
        for (int k = 0; k < cta; k++) carry += s_all[k][14];
        for (int i0 = lo; i0 < hi; i0 += kClusterThreads * kSmallScan) {
            const int at = i0 + t * kSmallScan;
            if (!once) {
                sum = 0;
#pragma unroll
                for (int k = 0; k < kSmallScan; k++) {
                    x[k] = at + k < hi ? a.counts[at + k] : 0;
                    sum += x[k];
                }
                before = cta_scan(sum, s_part, all);
            }
            int run = carry + before;
#pragma unroll
            for (int k = 0; k < kSmallScan; k++) {
                if (at + k < hi) a.counts[at + k] = run;
                run += x[k];
            }
            carry += all;
        }
        cluster_barrier();
    }
    // ids in cell order, then in ascending order inside every cell
    const int *bounds = a.counts;
    int beg[kSmallPoints], len[kSmallPoints];
#pragma unroll
    for (int k = 0; k < kSmallPoints; k++) {
        beg[k] = bin[k] >= 0 ? bounds[bin[k]] : 0;
        len[k] = bin[k] >= 0 ? bounds[bin[k] + 1] - beg[k] : 0;
    }
#pragma unroll
    for (int k = 0; k < kSmallPoints; k++)
        if (bin[k] >= 0 && FGC_DBG_OK(beg[k] + rank[k] >= 0 && beg[k] + rank[k] < n, &g->status)) a.stmp[beg[k] + rank[k]] = first + k * kClusterAll;
    cluster_barrier();
    int smaller[kSmallPoints] = {}, most = 0;
#pragma unroll
    for (int k = 0; k < kSmallPoints; k++) most = max(most, len[k] <= kRankMax ? len[k] : 0);
    for (int i0 = 0; i0 < most; i0 += 4) {                     // (the reads of a step are on their way together)
#pragma unroll
        for (int k = 0; k < kSmallPoints; k++)
#pragma unroll
            for (int i = i0; i < i0 + 4; i++)
                if (i < len[k] && len[k] <= kRankMax) smaller[k] += a.stmp[beg[k] + i] < first + k * kClusterAll ? 1 : 0;
    }
#pragma unroll
    for (int k = 0; k < kSmallPoints; k++) {
        const int v = first + k * kClusterAll, at = beg[k] + smaller[k];
        if (bin[k] < 0) continue;
        if (len[k] <= kRankMax) {
            if (FGC_DBG_OK(beg[k] >= 0 && smaller[k] < len[k] && at < n, &g->status)) {
                place_point(at, v, grid_cell(&s_grid, bin[k]), a.coords, a.n_coords, a.nv, a.direction, a.sorig, a.scoords, a.sbin, a.sflag);
                if (a.out_order) a.out_order[at] = v;
            }
        } else {
            a.sorig[beg[k] + rank[k]] = v;
            if (rank[k] == 0) {
                if (len[k] <= kWarpSortMaxShared) a.biglist[atomicAdd(&g->n_big_cells, 1)] = bin[k];
                else a.hugelist[atomicAdd(&g->n_huge_cells, 1)] = bin[k];
            }
        }
    }
    cluster_barrier();
    const int n_big = __ldcg(&g->n_big_cells), n_huge = __ldcg(&g->n_huge_cells);
    for (int w = cta * kSortWarps + wib; w < n_big; w += kClusterCtas * kSortWarps) {
        const int cell = a.biglist[w], from = bounds[cell], many = bounds[cell + 1] - from;
        warp_sort_segment(a.sorig + from, many, s_sort + wib * kWarpSortMaxShared, lane);
        __syncwarp();
        for (int i = lane; i < many; i += 32) {
            const int v = a.sorig[from + i];
            place_point(from + i, v, grid_cell(&s_grid, cell), a.coords, a.n_coords, a.nv, a.direction, a.sorig, a.scoords, a.sbin, a.sflag);
            if (a.out_order) a.out_order[from + i] = v;
        }
        __syncwarp();
    }
    __syncthreads();
    for (int w = cta; w < n_huge; w += kClusterCtas) {
        const int cell = a.hugelist[w], from = bounds[cell], many = bounds[cell + 1] - from;
        sort_cell_by_cta(from, many, a.stmp, a.sorig, s_sort, kSortShared / 4, &g->status);
        for (int i = t; i < many; i += kClusterThreads) {
            const int v = a.sorig[from + i];
            place_point(from + i, v, grid_cell(&s_grid, cell), a.coords, a.n_coords, a.nv, a.direction, a.sorig, a.scoords, a.sbin, a.sflag);
            if (a.out_order) a.out_order[from + i] = v;
        }
        __syncthreads();
    }
}

cudaError_t launch_small_build(const GridBuild &b, cudaStream_t s)
{
    static_assert(kSortShared <= 48 * 1024, "needs an attribute");
    k_build_small<<<kClusterCtas, kClusterThreads, kSortShared, s>>>(b);
    return cudaGetLastError();
}

}  // namespace fgc
