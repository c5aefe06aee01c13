// binned_select_knn forward for sm_100a, part 1: the search grid (this file) --
// part 2, the search itself, is knn_search.cu.
//
// Pipeline (batches of up to kSmallBuild points take the same passes in one launch, knn_grid_small.cu; all on the
// caller's stream, no host synchronisation; 9 launches, 11 while the
// device still has to choose the grid's form for D = 4):
//   k_minmax_setup  fused finite check + min/max of the binned coordinates; clears the cell
//                 table; its last CTA validates the row splits and chooses cell width / grid
//                 shape from the extents and the point count (the grid spans the first
//                 min(D, 4) coordinates)
//   k_histogram   cell id per point, warp-aggregated atomic histogram; the value returned by
//                 the atomic is the point's rank inside its cell.  The ranks also give the
//                 density statistic sum_c c^2 for free, and the kernel's last CTA is the density
//                 pass: it shrinks the cells where the data is clustered; D = 4 data that is
//                 strongly clustered goes back to a grid over three coordinates and gets a
//                 second density pass there
//   k_zero_counts + k_histogram again, for the grid the density pass chose (return at once
//                 when it kept the first grid)
//   k_scan_tile_sums_top, k_scan_apply   exclusive scan of the histogram -> cell boundaries
//   k_fill_ids    counting-sort scatter of the original ids into cell order (arbitrary inside a cell)
//   k_rank_place  ids in ascending order inside every cell (the layout is the same on every
//                 run); coordinates (padded to float4), cell id and direction flag in that order
//   k_sort_large_cells  the same for the few cells too crowded for ranking
//   k_knn         one warp per query point: walks the neighbouring cells in
//                 expanding Chebyshev shells, evaluates 32 candidates per step
//                 (one per lane, 16-byte loads), keeps the K-1 best in registers
//                 and writes the row at its ORIGINAL position with ORIGINAL ids.
//
// What is computed is what the reference's CPU path computes
// (extensions/binned_knn_autograd_kernel.cpp:85-209 with
// extensions/binned_select_knn_cpu.cpp:56-208): per row split, the K-1 nearest
// other points (strict "<" replacement of the current worst, so among equal
// distances the first one visited stays), squared distances accumulated over the
// dimensions in order with one rounding per operation.  The visiting order, the
// grid and the stopping rule are this library's own; they never change which
// points are nearest, only which of several equidistant points is kept.
#include "knn_grid_build.cuh"
#include "knn_tree.cuh"
#include "shell_table.cuh"

namespace fgc {

// ---------------------------------------------------------------------------
// grid construction
// ---------------------------------------------------------------------------

// Before the grid of a second look: an empty header and tickets where there are rows to search again, else a
// status word that ends the kernels of the grid at once.
__global__ void __launch_bounds__(256)
k_tie_gate(KnnGrid *__restrict__ g, const KnnTree *__restrict__ t, int limit)
{
    chain_wait();
    chain_release();
    const int status = g->status;
    const long long tied = t->n_tied, both = tied + t->n_equal;
    __syncthreads();
    if (status != 0) return;
    if (both == 0 || tied > limit || (tied == 0 && both > limit)) {
        if (threadIdx.x == 0) g->status = kStatusNoGrid;
        return;
    }
    for (int i = threadIdx.x; i < (int)((kGridHeaderBytes + kHardTicketBytes) / sizeof(int)); i += 256) ((int *)g)[i] = 0;
    __syncthreads();
    if (threadIdx.x == 0) g->leave_equal = both > limit;
}

// Fused finite check + min/max of the binned coordinates; clears the cell table (all of its
// capacity: the grid that decides how much of it is used does not exist yet); counts the points that may
// be neighbours (mirror > 1); the CTA that finishes last (a ticket counter, no waiting) checks the row splits and
// chooses the grid.
__global__ void __launch_bounds__(256)
k_minmax_setup(const float *__restrict__ coords, int n_vert, int n_coords, int n_bin_dims,
               const int64_t *__restrict__ direction, KnnGrid *g, int *__restrict__ counts, long long n_counts,
               const int64_t *__restrict__ row_splits, int n_rs, int bins_target, int bins_cap_first, int bins_cap,
               int mirror, int adaptive, int gated)
{
    chain_wait();
    chain_release();
    if (gated && g->status != 0) return;           // (else zero until the last CTA sets it)
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_counts;
         i += (long long)gridDim.x * blockDim.x)
        counts[i] = 0;
    uint32_t lmin[4] = {0, 0, 0, 0}, lmax[4] = {0, 0, 0, 0};
    uint32_t bad = 0, n_cand = 0;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n_vert; v += gridDim.x * blockDim.x) {
        const float *row = coords + (size_t)v * n_coords;
        if (mirror > 1) {
            const int64_t d = direction[v];
            n_cand += d != 1 && d != 2;
        }
        for (int c = 0; c < n_coords; c++) {
            const float x = __ldg(row + c);
            if (!is_finite_bits(x)) bad = 1;
            if (c < n_bin_dims) {
                const uint32_t k = float_to_ordered(x);
#pragma unroll
                for (int cc = 0; cc < 4; cc++)
                    if (cc == c) { lmin[cc] = max(lmin[cc], ~k); lmax[cc] = max(lmax[cc], k); }
            }
        }
    }
    __shared__ uint32_t s_min[4], s_max[4], s_bad, s_cand;
    if (threadIdx.x < 4) { s_min[threadIdx.x] = 0; s_max[threadIdx.x] = 0; }
    if (threadIdx.x == 0) { s_bad = 0; s_cand = 0; }
    __syncthreads();
    if (mirror > 1) {
        n_cand = __reduce_add_sync(FGC_FULL_MASK, n_cand);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_cand, n_cand);
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint32_t a = __reduce_max_sync(FGC_FULL_MASK, lmin[c]);
        const uint32_t b = __reduce_max_sync(FGC_FULL_MASK, lmax[c]);
        if ((threadIdx.x & 31) == 0) { atomicMax(&s_min[c], a); atomicMax(&s_max[c], b); }
    }
    if (__any_sync(FGC_FULL_MASK, bad) && (threadIdx.x & 31) == 0) atomicOr(&s_bad, 1u);
    __syncthreads();
    if (threadIdx.x < 4) {
        atomicMax(&g->min_key[threadIdx.x], s_min[threadIdx.x]);
        atomicMax(&g->max_key[threadIdx.x], s_max[threadIdx.x]);
    }
    if (threadIdx.x == 0 && s_bad) atomicOr(&g->nonfinite, 1u);
    if (threadIdx.x == 0 && mirror > 1) atomicAdd(&g->sum_sq, (unsigned long long)s_cand);   // (free until the density pass)
    // the last CTA to arrive sees every CTA's extrema and sets the grid up
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&g->stat_blocks_done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // row_splits must start at 0, end at n_vert and never decrease
    int bad_rs = 0;
    for (int i = 1 + threadIdx.x; i < n_rs; i += blockDim.x)
        if (row_splits[i] < row_splits[i - 1]) bad_rs = 1;
    bad_rs = __syncthreads_or(bad_rs);
    if (threadIdx.x == 0) {
        g->stat_blocks_done = 0;       // the density pass counts its CTAs with the same ticket
        if (mirror > 1) choose_sets(atomicExch(&g->sum_sq, 0ull), n_vert, adaptive, mirror, bins_target, bins_cap);
        uint32_t min_key[4], max_key[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            min_key[c] = atomicMax(&g->min_key[c], 0u);
            max_key[c] = atomicMax(&g->max_key[c], 0u);
        }
        if (row_splits[0] != 0 || row_splits[n_rs - 1] != (int64_t)n_vert) bad_rs = 1;
        grid_setup(g, min_key, max_key, atomicOr(&g->nonfinite, 0u) != 0, n_rs, n_bin_dims, bins_target, bins_cap_first, bins_cap, bad_rs,
                   mirror);
    }
}

__global__ void __launch_bounds__(256)
k_zero_counts(int *__restrict__ counts, const KnnGrid *g, int stage)
{
    chain_wait();
    chain_release();
    if (g->refined < stage) return;      // stage s follows the s-th density pass that changed the grid
    const int n = g->total_bins + 1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        counts[i] = 0;
}

// refine_pass >= 0: the kernel is also the density pass of that number.  A point that arrives
// as the r-th of its cell adds 2r+1, so that a cell of c points adds c^2 in total: the sum over
// the cells of c^2 comes out of the histogram itself, with no second pass over the table.  The
// CTA that finishes last (a ticket counter, no waiting) decides about the finer grid.
__global__ void __launch_bounds__(256)
k_histogram(const float *__restrict__ coords, int n_vert, int n_coords,
            const int64_t *__restrict__ row_splits, int n_rs, const int64_t *__restrict__ direction,
            KnnGrid *__restrict__ g, int *__restrict__ counts, int *__restrict__ pbin, int *__restrict__ prank,
            int stage, int refine_pass, float seen_target, float seen_target3, int bins_target3,
            int allow_fallback)
{
    chain_wait();
    chain_release();
    if (g->refined < stage) return;
    if (refine_pass == 1 && !g->fallback3) refine_pass = -1;
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = v < n_vert && g->status == 0;
    int flat = 0;
    bool candidate = true;
    unsigned long long sq = 0;
    if (live) {
        flat = point_cell(g, coords + (size_t)v * n_coords, row_split_of(row_splits, n_rs, v));
        if (g->mirror > 1) {
            const int64_t d = direction[v];
            candidate = d != 1 && d != 2;
            if (!candidate) flat += g->n_events * g->B;
        }
    }
    const unsigned active = __ballot_sync(FGC_FULL_MASK, live && FGC_DBG_OK(flat >= 0 && flat < g->total_bins, &g->status));
    if (active >> (threadIdx.x & 31) & 1) {
        // warp-aggregated: one atomic per distinct cell in the warp
        const unsigned peers = __match_any_sync(active, flat);
        const int leader = __ffs(peers) - 1;
        int base = 0;
        if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(counts + flat, __popc(peers));
        base = __shfl_sync(peers, base, leader);
        pbin[v] = flat;
        const int rank = base + __popc(peers & lanemask_lt());
        prank[v] = rank;
        if (candidate) sq = 2ull * (unsigned long long)rank + 1ull;
    }
    if (refine_pass < 0 || g->status != 0) return;     // uniform over the grid
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(FGC_FULL_MASK, sq, o);
    __shared__ unsigned long long s_sq[8];
    if ((threadIdx.x & 31) == 0) s_sq[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int k = 0; k < 8; k++) t += s_sq[k];
        if (t) atomicAdd(&g->sum_sq, t);
        __threadfence();
        const int ticket = atomicAdd(&g->stat_blocks_done, 1);
        if (ticket == (int)gridDim.x - 1) {
            __threadfence();
            g->stat_blocks_done = 0;
            grid_refine(g, atomicAdd(&g->sum_sq, 0ull), n_vert, seen_target, seen_target3, bins_target3,
                        refine_pass, allow_fallback);
        }
    }
}

// Counting-sort scatter, step 1: original ids in cell order.  The position inside a cell is
// the rank the histogram's atomic handed out, i.e. arbitrary.
__global__ void __launch_bounds__(256)
k_fill_ids(int n_vert, const KnnGrid *__restrict__ g, const int *__restrict__ bounds,
           const int *__restrict__ pbin, const int *__restrict__ prank, int *__restrict__ stmp)
{
    chain_wait();
    chain_release();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_vert || g->status != 0) return;
    const int pos = bounds[pbin[v]] + prank[v];
    if (FGC_DBG_OK(pos >= 0 && pos < n_vert, &g->status)) stmp[pos] = v;
}

// Step 2: the ids inside every cell in ascending order, so that the cell-ordered layout --
// and with it the order in which the search visits candidates, its choice among equidistant
// candidates and the slot order of its output -- is the same on every run.  One thread per
// point: in a cell of up to kRankMax points the point's place is the number of smaller ids in
// the cell (read from the unordered list of step 1), and everything kept in cell order is
// written there at once.  Points of larger cells keep their arbitrary place for now and
// the cell goes to a work list (k_sort_large_cells).
__global__ void __launch_bounds__(256)
k_rank_place(const float *__restrict__ coords, int n_vert, int n_coords, int nv,
             const int64_t *__restrict__ direction, KnnGrid *__restrict__ g,
             const int *__restrict__ bounds, const int *__restrict__ pbin,
             const int *__restrict__ prank, const int *__restrict__ stmp,
             int *__restrict__ sorig, float4 *__restrict__ scoords, int *__restrict__ sbin,
             uint8_t *__restrict__ sflag, int *__restrict__ biglist, int *__restrict__ hugelist)
{
    chain_wait();
    chain_release();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_vert) return;
    const int status = g->status;
    if (status != 0) {
        if (status & kNotBuilt) sorig[v] = v;
        return;
    }
    const int bin = pbin[v];
    const int beg = bounds[bin], len = bounds[bin + 1] - beg;
    if (len <= kRankMax) {
        int rank = 0;
        for (int t = 0; t < len; t++) rank += stmp[beg + t] < v ? 1 : 0;
        if (FGC_DBG_OK(beg >= 0 && rank < len && beg + rank < n_vert, &g->status))
            place_point(beg + rank, v, grid_cell(g, bin), coords, n_coords, nv, direction, sorig, scoords, sbin, sflag);
    } else {
        const int r = prank[v];
        sorig[beg + r] = v;
        if (r == 0) {
            if (len <= kWarpSortMaxShared) biglist[atomicAdd(&g->n_big_cells, 1)] = bin;
            else hugelist[atomicAdd(&g->n_huge_cells, 1)] = bin;
        }
    }
}

// Bytes for the bits of n_vert ids (two CTAs an SM).
static int sort_shared_bytes(int64_t n_vert)
{
    const int64_t bytes = (n_vert < kSortMostBits ? n_vert + 31 : kSortMostBits) / 32 * 4;
    return bytes > kSortShared ? (int)bytes : kSortShared;
}

// Step 3: the cells of the work lists.  The first n_warp_blocks CTAs take the cells that one warp can sort (in registers /
// shared memory), the others those beyond kWarpSortMaxShared points, one CTA per cell.  After the sort the same warp / CTA
// places the cell's points.
__global__ void __launch_bounds__(kSortWarps * 32)
k_sort_large_cells(const float *__restrict__ coords, int n_coords, int nv,
                   const int64_t *__restrict__ direction, KnnGrid *__restrict__ g,
                   const int *__restrict__ bounds, const int *__restrict__ biglist,
                   const int *__restrict__ hugelist, int n_warp_blocks, const int *__restrict__ stmp, int n_words,
                   int *__restrict__ sorig, float4 *__restrict__ scoords, int *__restrict__ sbin,
                   uint8_t *__restrict__ sflag)
{
    chain_wait();
    chain_release();
    extern __shared__ int s_sort[];
    if (g->status != 0) return;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if ((int)blockIdx.x < n_warp_blocks) {
        const int n_big = g->n_big_cells;
        for (int w = blockIdx.x * kSortWarps + wib; w < n_big; w += n_warp_blocks * kSortWarps) {
            const int cell = biglist[w];
            const int beg = bounds[cell], n = bounds[cell + 1] - beg;
            warp_sort_segment(sorig + beg, n, s_sort + wib * kWarpSortMaxShared, lane);
            __syncwarp();
            for (int t = lane; t < n; t += 32)
                place_point(beg + t, sorig[beg + t], grid_cell(g, cell), coords, n_coords, nv, direction, sorig, scoords,
                            sbin, sflag);
            __syncwarp();
        }
        return;
    }
    const int n_huge = g->n_huge_cells;
    const int n_cta = gridDim.x - n_warp_blocks;
    for (int w = blockIdx.x - n_warp_blocks; w < n_huge; w += n_cta) {
        const int cell = hugelist[w];
        const int beg = bounds[cell], n = bounds[cell + 1] - beg;
        sort_cell_by_cta(beg, n, stmp, sorig, s_sort, n_words, &g->status);
        for (int t = threadIdx.x; t < n; t += blockDim.x)
            place_point(beg + t, sorig[beg + t], grid_cell(g, cell), coords, n_coords, nv, direction, sorig, scoords, sbin, sflag);
        __syncthreads();
    }
}

// Status word and the grid's form ((3 or 4) + 16 * fallback3) to memory the host can read.
__global__ void k_publish_grid_info(const KnnGrid *__restrict__ g, volatile int32_t *info_mapped)
{
    chain_wait();
    chain_release();
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        store_info(info_mapped, g->status, g->gdims + 16 * g->fallback3);
        __threadfence_system();
    }
}

// One store of the status word to memory the host can read (mapped pinned memory).
__global__ void k_publish_status(const int32_t *__restrict__ status_dev, volatile int32_t *status_mapped)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        *status_mapped = *status_dev;
        __threadfence_system();
    }
}

}  // namespace fgc

extern "C" size_t fgc_knn_workspace_bytes(int64_t n_vert, int32_t n_coords, int64_t n_rs, int32_t K)
{
    if (n_vert < 0 || n_vert > 0x7fffffff || n_coords < 1 || n_rs < 1 || K < 1) return 0;
    return fgc::knn_workspace_layout(n_vert, n_coords, n_rs, K).total;
}

extern "C" size_t fgc_knn_forward_workspace_bytes(int64_t n_vert, int32_t n_coords, int64_t n_rs, int32_t K, int32_t flags)
{
    const size_t grid = fgc_knn_workspace_bytes(n_vert, n_coords, n_rs, K);
    return grid == 0 || !(flags & FGC_FORWARD_TREE) ? grid : grid + fgc::tree_extra_bytes(n_vert, n_coords, n_rs);
}

extern "C" int fgc_read_status(const void *workspace_or_params, int32_t *status_host,
                               fgc_stream_t stream)
{
    if (!workspace_or_params || !status_host) return FGC_ERR_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    FGC_RETURN_IF_CUDA(cudaMemcpyAsync(status_host, workspace_or_params, sizeof(int32_t),
                                       cudaMemcpyDeviceToHost, s));
    FGC_RETURN_IF_CUDA(cudaStreamSynchronize(s));
    return FGC_OK;
}

extern "C" int fgc_publish_status(const void *workspace_or_params, int32_t *status_mapped,
                                  fgc_stream_t stream)
{
    if (!workspace_or_params || !status_mapped) return FGC_ERR_BAD_ARGUMENT;
    fgc::k_publish_status<<<1, 32, 0, (cudaStream_t)stream>>>((const int32_t *)workspace_or_params, status_mapped);
    FGC_CHECK_LAUNCH();
    return FGC_OK;
}

extern "C" int fgc_knn_publish_grid_info(const void *workspace, int32_t *info_mapped, fgc_stream_t stream)
{
    if (!workspace || !info_mapped) return FGC_ERR_BAD_ARGUMENT;
    FGC_RETURN_IF_CUDA(fgc::launch_chained(fgc::k_publish_grid_info, 1, 32, 0, (cudaStream_t)stream,
                                           (const fgc::KnnGrid *)workspace, info_mapped));
    return FGC_OK;
}

extern "C" int fgc_knn_build_grid(const float *coords, int64_t n_vert, int32_t n_coords,
                                  const int64_t *row_splits, int64_t n_rs, int32_t K,
                                  const int64_t *direction_or_null, float target_occupancy,
                                  void *workspace, size_t workspace_bytes, fgc_stream_t stream)
{
    return fgc_knn_build_grid_dims(coords, n_vert, n_coords, row_splits, n_rs, K, direction_or_null,
                                   target_occupancy, 0, workspace, workspace_bytes, stream);
}

namespace fgc {

static int knn_build_grid(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs,
                          int32_t K, const int64_t *direction_or_null, float target_occupancy, int32_t grid_dims,
                          bool only_for_ties, int32_t *info_mapped, int32_t *out_order, bool *done, void *workspace,
                          size_t workspace_bytes, fgc_stream_t stream)
{
    if (grid_dims != 0 && grid_dims != 3 && grid_dims != 4) return FGC_ERR_BAD_ARGUMENT;
    KnnWorkspace L;
    if (!row_splits) return FGC_ERR_BAD_ARGUMENT;
    const int rc = check_knn_args(n_vert, n_coords, n_rs, K, workspace, workspace_bytes, &L);
    if (rc != FGC_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    char *ws = (char *)workspace;
    KnnGrid *grid = (KnnGrid *)(ws + L.header);
    const bool small = !only_for_ties && n_vert > 0 && n_vert <= kSmallBuild;
    if (only_for_ties)
        FGC_RETURN_IF_CUDA(launch_chained(k_tie_gate, 1, 256, 0, s, grid, (const KnnTree *)(ws + L.tickets),
                                          (int)(n_vert / kTieShare)));
    else if (!small)
        FGC_RETURN_IF_CUDA(cudaMemsetAsync(grid, 0, kGridHeaderBytes + kHardTicketBytes, s));   // header and k_knn_hard's tickets
    if (n_vert == 0) return FGC_OK;
    if (!coords || n_rs < 2) return FGC_ERR_BAD_ARGUMENT;

    int *counts = (int *)(ws + L.counts);
    int *blocksums = (int *)(ws + L.blocksums);
    int *pbin = (int *)(ws + L.pbin);
    int *prank = (int *)(ws + L.prank);
    int *stmp = (int *)(ws + L.stmp);
    int *sorig = (int *)(ws + L.sorig);
    int *biglist = (int *)(ws + L.biglist);
    int *hugelist = (int *)(ws + L.hugelist);
    int *sbin = (int *)(ws + L.sbin);
    uint8_t *sflag = (uint8_t *)(ws + L.sflag);
    float4 *scoords = (float4 *)(ws + L.scoords);

    const int n = (int)n_vert;
    const int n_events = (int)n_rs - 1;
    // D = 4 lets the density pass choose between four and three binned coordinates unless the
    // caller fixes the choice (grid_dims 3 or 4; ignored for every other D)
    const int forced = n_coords == 4 ? grid_dims : 0;
    const int n_bin_dims = forced == 3 ? 3 : (n_coords < 4 ? n_coords : 4);
    // target_occupancy > 0: one fixed grid with that mean occupancy.  Otherwise: mean
    // occupancy K/21 within [1.5, 3] (measured on B200: K = 32 is fastest at 1 to 1.5, K = 64
    // at 3 to 4, K = 128 at 2 to 3; the optimum is flat, +-2 % over a factor of two), then
    // the density pass may shrink the cells so that a typical point sees about seen_target
    // points in its own cell.
    // With direction flags the points that may not be neighbours go to a second set of cells behind the
    // first: a walk then meets candidates only (B200, a third of the points candidates: ten row splits of
    // 100 k, K = 64: 2.34 -> 1.33 ms, 64 of 2900, K = 16: 0.250 -> 0.193; half of them: 4.56 -> 3.01, 0.386 -> 0.319).
    // One set where nearly all points are candidates (nine tenths: 3.2 -> 3.0 ms with two, but 1 M clustered points in four
    // coordinates, K = 20, 2.8 -> 4.1, for want of cells), and where the table could not hold two.
    const int mirror = direction_or_null && 2 * (int64_t)n_events <= L.cap_bins ? 2 : 1;
    const bool adaptive = !(target_occupancy > 0.f);
    if (adaptive) {
        target_occupancy = (float)K / 21.0f;
        if (target_occupancy < 1.5f) target_occupancy = 1.5f;
        if (target_occupancy > 3.0f) target_occupancy = 3.0f;
    }
    float seen_target = (float)K / 6.0f;
    if (seen_target < 4.f) seen_target = 4.f;
    const float seen_target3 = seen_target * 2.f;    // D = 4 binned in three coordinates
    if (n_coords > n_bin_dims) seen_target *= 2.f;   // coordinates that are not binned thin the cells out
    const int64_t bins_cap64 = L.cap_bins / n_events / mirror;
    const int bins_cap = (int)(bins_cap64 < 1 ? 1 : bins_cap64);
    const double bt = (double)n_vert / (double)n_events / (double)target_occupancy;
    int bins_target = bt >= (double)bins_cap ? bins_cap : (int)(bt + 0.5);
    if (bins_target < 1) bins_target = 1;

    const int pt_blocks = (n + 255) / 256;
    const int red_blocks = pt_blocks < fgc::sm_count() * 4 ? pt_blocks : fgc::sm_count() * 4;
    // The cell count is only known on the device.  The first grid may use up to four times the
    // wanted number of cells (its shape is rounded up per dimension): that part of the table is
    // cleared together with the extent reduction; a finer grid of the density pass clears what
    // it needs itself.  The scan grids are sized for the largest table (surplus blocks return
    // at once).
    const int64_t max_entries = (int64_t)bins_cap * n_events * mirror + 1;
    const int scan_blocks = (int)ceil_div64(max_entries, kScanTile);
    int bins_cap_first = bins_target > (bins_cap - 64) / 4 ? bins_cap : 4 * bins_target + 64;
    if (!adaptive) bins_cap_first = bins_cap;
    const int allow_fallback = adaptive && n_coords == 4 && forced == 0;
    if (small) {
        GridBuild b = {};
        b.coords = coords; b.row_splits = row_splits; b.direction = direction_or_null; b.grid = grid;
        b.counts = counts; b.stmp = stmp; b.sorig = sorig; b.sbin = sbin; b.biglist = biglist; b.hugelist = hugelist;
        b.sflag = sflag; b.scoords = scoords; b.n_vert = n; b.n_coords = n_coords; b.nv = L.nv; b.n_rs = (int)n_rs; b.n_bin_dims = n_bin_dims;
        b.mirror = mirror; b.bins_target = bins_target; b.bins_cap_first = bins_cap_first; b.bins_cap = bins_cap; b.adaptive = adaptive;
        b.allow_fallback = allow_fallback; b.seen_target = seen_target; b.seen_target3 = seen_target3; b.out_order = out_order;
        b.info_mapped = info_mapped;
        FGC_RETURN_IF_CUDA(launch_small_build(b, s));
        if (done) *done = true;
        return FGC_OK;
    }
    k_minmax_setup<<<red_blocks, 256, 0, s>>>(coords, n, n_coords, n_bin_dims, direction_or_null, grid, counts,
                                              (long long)bins_cap_first * n_events * mirror + 1, row_splits, (int)n_rs,
                                              bins_target, bins_cap_first, bins_cap, mirror, adaptive, only_for_ties);
    FGC_CHECK_LAUNCH();
    FGC_RETURN_IF_CUDA(launch_chained(k_histogram, pt_blocks, 256, 0, s, coords, n, n_coords, row_splits, (int)n_rs, direction_or_null,
                                      grid, counts, pbin, prank, 0, adaptive ? 0 : -1, seen_target, seen_target3,
                                      bins_target, allow_fallback));
    if (adaptive) {
        // the grid of the density pass, when it chose one (both kernels return at once otherwise)
        FGC_RETURN_IF_CUDA(launch_chained(k_zero_counts, fgc::sm_count() * 4, 256, 0, s, counts, grid, 1));
        FGC_RETURN_IF_CUDA(launch_chained(k_histogram, pt_blocks, 256, 0, s, coords, n, n_coords, row_splits, (int)n_rs,
                                          direction_or_null, grid, counts, pbin, prank, 1, allow_fallback ? 1 : -1, seen_target,
                                          seen_target3, bins_target, 0));
        if (allow_fallback) {
            // second density pass: ran only when the first one fell back to three coordinates
            FGC_RETURN_IF_CUDA(launch_chained(k_zero_counts, fgc::sm_count() * 4, 256, 0, s, counts, grid, 2));
            FGC_RETURN_IF_CUDA(launch_chained(k_histogram, pt_blocks, 256, 0, s, coords, n, n_coords, row_splits,
                                              (int)n_rs, direction_or_null, grid, counts, pbin, prank, 2, -1, seen_target, seen_target3,
                                              bins_target, 0));
        }
    }
    FGC_RETURN_IF_CUDA(launch_chained(k_scan_tile_sums_top, scan_blocks, 256, 0, s, counts, &grid->total_bins, 1,
                                      blocksums, &grid->scan_ticket));
    FGC_RETURN_IF_CUDA(launch_chained(k_scan_apply, scan_blocks, 256, 0, s, counts, &grid->total_bins, 1, blocksums));
    FGC_RETURN_IF_CUDA(launch_chained(k_fill_ids, pt_blocks, 256, 0, s, n, grid, counts, pbin, prank, stmp));
    FGC_RETURN_IF_CUDA(launch_chained(k_rank_place, pt_blocks, 256, 0, s, coords, n, n_coords, L.nv, direction_or_null,
                                      grid, counts, pbin, prank, stmp, sorig, scoords, sbin, sflag, biglist, hugelist));
    const int n_warp_blocks = fgc::sm_count(), sort_bytes = sort_shared_bytes(n_vert);
    if (sort_bytes > 48 * 1024)
        FGC_RETURN_IF_CUDA(cudaFuncSetAttribute(k_sort_large_cells, cudaFuncAttributeMaxDynamicSharedMemorySize, sort_bytes));
    FGC_RETURN_IF_CUDA(launch_chained(k_sort_large_cells, n_warp_blocks + fgc::sm_count() / 2, kSortWarps * 32, sort_bytes, s, coords,
                                      n_coords, L.nv, direction_or_null, grid, counts, biglist, hugelist, n_warp_blocks, stmp,
                                      sort_bytes / 4, sorig, scoords, sbin, sflag));
    return FGC_OK;
}

}  // namespace fgc

extern "C" int fgc_knn_build_grid_dims(const float *coords, int64_t n_vert, int32_t n_coords,
                                       const int64_t *row_splits, int64_t n_rs, int32_t K,
                                       const int64_t *direction_or_null, float target_occupancy,
                                       int32_t grid_dims, void *workspace, size_t workspace_bytes,
                                       fgc_stream_t stream)
{
    FGC_NVTX("fgc_knn_build_grid_dims");
    return fgc::knn_build_grid(coords, n_vert, n_coords, row_splits, n_rs, K, direction_or_null, target_occupancy, grid_dims,
                               false, nullptr, nullptr, nullptr, workspace, workspace_bytes, stream);
}

int fgc::knn_build_grid_forward(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs,
                                int32_t K, const int64_t *direction_or_null, float target_occupancy, int32_t grid_dims,
                                int32_t *info_mapped, int32_t *out_order, bool *done, void *workspace, size_t workspace_bytes,
                                fgc_stream_t stream)
{
    FGC_NVTX("fgc_knn_build_grid_dims");
    return knn_build_grid(coords, n_vert, n_coords, row_splits, n_rs, K, direction_or_null, target_occupancy, grid_dims, false,
                          info_mapped, out_order, done, workspace, workspace_bytes, stream);
}

int fgc::knn_build_grid_for_ties(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits,
                                 int64_t n_rs, int32_t K, const int64_t *direction_or_null, float target_occupancy,
                                 void *workspace, size_t workspace_bytes, fgc_stream_t stream)
{
    FGC_NVTX("fgc_knn_build_grid_for_ties");
    return knn_build_grid(coords, n_vert, n_coords, row_splits, n_rs, K, direction_or_null, target_occupancy, 0, true,
                          nullptr, nullptr, nullptr, workspace, workspace_bytes, stream);
}

extern "C" const int32_t *fgc_knn_cell_order(const void *workspace, int64_t n_vert, int32_t n_coords,
                                             int64_t n_rs, int32_t K)
{
    if (!workspace || n_vert < 0 || n_coords < 1 || n_rs < 1 || K < 1) return nullptr;
    const fgc::KnnWorkspace L = fgc::knn_workspace_layout(n_vert, n_coords, n_rs, K);
    return (const int32_t *)((const char *)workspace + L.sorig);
}

extern "C" int fgc_knn_read_counters(const void *workspace, uint64_t *counters_host,
                                     int32_t *grid_shape_host, float *cell_width_host,
                                     fgc_stream_t stream)
{
    using namespace fgc;
    if (!workspace) return FGC_ERR_BAD_ARGUMENT;
    KnnGrid h;
    cudaStream_t s = (cudaStream_t)stream;
    FGC_RETURN_IF_CUDA(cudaMemcpyAsync(&h, workspace, sizeof(KnnGrid), cudaMemcpyDeviceToHost, s));
    FGC_RETURN_IF_CUDA(cudaStreamSynchronize(s));
    if (counters_host) {
        for (int i = 0; i < 6; i++) counters_host[i] = h.counters[i];
        // facts about the grid build (always available, not only after a counting search)
        counters_host[6] = (uint64_t)h.n_hard;          // queries the last search handed to whole CTAs
        counters_host[7] = (uint64_t)h.n_huge_cells;    // cells above 512 points (sorted by one CTA each)
    }
    if (grid_shape_host) { grid_shape_host[0] = h.n[0]; grid_shape_host[1] = h.n[1]; grid_shape_host[2] = h.n[2] * h.n[3]; }
    if (cell_width_host) *cell_width_host = h.w;
    return FGC_OK;
}
