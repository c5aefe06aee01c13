// binned_select_knn forward for sm_100a: building the search tree (see knn_tree.cuh).
//
//   k_tree_extent   bounding box of the points, checks of coordinates and row splits (small batches take everything up to the
//                   sorted ids in one launch, knn_tree_small.cu)
//   k_tree_keys     64-bit key of every point (row split, place on the Hilbert curve) and the first
//                   radix histogram
//   k_tree_hist     histogram of a later pass;  scan.cuh: its exclusive scan
//   k_tree_scatter  stable scatter of a pass (three or four passes of 11 bits)
//   k_tree_leaves   gathers the points in curve order, boxes of leaves and nodes
//   k_tree_top      boxes of the top nodes
//
// The sort is stable and starts from the original order, so the tree is the same on every run.
// Launch latency bounds the build of small batches (0.15 ms for 200 k points), scattered writes that
// of large ones (0.31 ms for 1.6 M points, against 8 ms and more for their search).
#include "knn_tree_build.cuh"

namespace fgc {

__global__ void __launch_bounds__(256)
k_tree_extent(const float *__restrict__ coords, int n_vert, int n_coords, int key_dims, int bits,
              const int64_t *__restrict__ row_splits, int n_rs, KnnGrid *__restrict__ g, KnnTree *__restrict__ t)
{
    chain_wait();
    chain_release();
    uint32_t lmin[kTreeKeyDims], lmax[kTreeKeyDims], bad = 0;
#pragma unroll
    for (int c = 0; c < kTreeKeyDims; c++) { lmin[c] = 0; lmax[c] = 0; }
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n_vert; v += (int64_t)gridDim.x * blockDim.x) {
        const float *row = coords + (size_t)v * n_coords;
#pragma unroll
        for (int c = 0; c < kTreeKeyDims; c++) {
            if (c < n_coords) {
                const float x = __ldg(row + c);
                if (!is_finite_bits(x)) bad = 1;
                const uint32_t k = float_to_ordered(x);
                lmin[c] = max(lmin[c], ~k);
                lmax[c] = max(lmax[c], k);
            }
        }
        for (int c = kTreeKeyDims; c < n_coords; c++)
            if (!is_finite_bits(__ldg(row + c))) bad = 1;
    }
    __shared__ uint32_t s_min[kTreeKeyDims], s_max[kTreeKeyDims], s_bad;
    if (threadIdx.x < kTreeKeyDims) { s_min[threadIdx.x] = 0; s_max[threadIdx.x] = 0; }
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kTreeKeyDims; c++) {
        const uint32_t a = __reduce_max_sync(FGC_FULL_MASK, lmin[c]);
        const uint32_t b = __reduce_max_sync(FGC_FULL_MASK, lmax[c]);
        if ((threadIdx.x & 31) == 0) { atomicMax(&s_min[c], a); atomicMax(&s_max[c], b); }
    }
    if (__any_sync(FGC_FULL_MASK, bad) && (threadIdx.x & 31) == 0) atomicOr(&s_bad, 1u);
    __syncthreads();
    if (threadIdx.x < kTreeKeyDims) {
        atomicMax(&t->min_key[threadIdx.x], s_min[threadIdx.x]);
        atomicMax(&t->max_key[threadIdx.x], s_max[threadIdx.x]);
    }
    if (threadIdx.x == 0 && s_bad) atomicOr(&t->nonfinite, 1u);
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&t->blocks_done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // row_splits must start at 0, end at n_vert and never decrease
    int bad_rs = 0;
    for (int i = 1 + threadIdx.x; i < n_rs; i += blockDim.x)
        if (row_splits[i] < row_splits[i - 1]) bad_rs = 1;
    bad_rs = __syncthreads_or(bad_rs);
    if (threadIdx.x == 0) {
        if (row_splits[0] != 0 || row_splits[n_rs - 1] != (int64_t)n_vert) bad_rs = 1;
        int status = 0;
        if (__ldcg(&t->nonfinite)) status |= FGC_STATUS_NONFINITE;
        if (bad_rs) status |= FGC_STATUS_BAD_ROW_SPLITS;
        uint32_t min_key[kTreeKeyDims], max_key[kTreeKeyDims];
#pragma unroll
        for (int c = 0; c < kTreeKeyDims; c++) { min_key[c] = __ldcg(&t->min_key[c]); max_key[c] = __ldcg(&t->max_key[c]); }
        tree_setup(t, min_key, max_key, key_dims, bits);
        g->n_events = n_rs - 1;
        g->status = status;
    }
}

template <int ROUNDS>
__global__ void __launch_bounds__(256)
k_tree_keys(const float *__restrict__ coords, int n_vert, int n_coords, int key_dims, int bits,
            const int64_t *__restrict__ row_splits, int n_rs, const KnnGrid *__restrict__ g,
            const KnnTree *__restrict__ t, uint64_t *__restrict__ keys, int *__restrict__ hist, int n_tiles)
{
    chain_wait();
    chain_release();
    __shared__ int s_hist[kRadixBins];
    for (int i = threadIdx.x; i < kRadixBins; i += 256) s_hist[i] = 0;
    __syncthreads();
    if (g->status != 0) return;
    const int64_t base = (int64_t)blockIdx.x * (ROUNDS * 256);
    for (int k = threadIdx.x; k < ROUNDS * 256 && base + k < n_vert; k += 256) {
        const int64_t v = base + k;
        const uint64_t e = (uint64_t)row_split_of(row_splits, n_rs, v);
        const uint64_t key = (e << (bits * key_dims)) | tree_key(t, coords + (size_t)v * n_coords, key_dims, bits);
        keys[v] = key;
        atomicAdd(&s_hist[(int)(key & (kRadixBins - 1))], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kRadixBins; i += 256) hist[(size_t)i * n_tiles + blockIdx.x] = s_hist[i];
}

template <int ROUNDS>
__global__ void __launch_bounds__(256)
k_tree_hist(const uint64_t *__restrict__ keys, int n_vert, int shift, const KnnGrid *__restrict__ g,
            int *__restrict__ hist, int n_tiles)
{
    chain_wait();
    chain_release();
    __shared__ int s_hist[kRadixBins];
    for (int i = threadIdx.x; i < kRadixBins; i += 256) s_hist[i] = 0;
    __syncthreads();
    if (g->status != 0) return;
    const int64_t base = (int64_t)blockIdx.x * (ROUNDS * 256);
#pragma unroll 4
    for (int k = threadIdx.x; k < ROUNDS * 256; k += 256)
        if (base + k < n_vert) atomicAdd(&s_hist[(int)((keys[base + k] >> shift) & (kRadixBins - 1))], 1);
    __syncthreads();
    for (int i = threadIdx.x; i < kRadixBins; i += 256) hist[(size_t)i * n_tiles + blockIdx.x] = s_hist[i];
}

// One stable radix pass.  A warp owns an eighth of the tile's keys, consecutive ones, and goes
// through them 32 at a time: lanes with equal digits find one another by a match, the warp's counter
// of the digit gives the rank.  ids_in == nullptr: the first pass, the ids are the positions.
template <int ROUNDS>
__global__ void __launch_bounds__(256)
k_tree_scatter(const uint64_t *__restrict__ keys_in, const int *__restrict__ ids_in, int n_vert, int shift,
               KnnGrid *__restrict__ g, const int *__restrict__ hist, int n_tiles, uint64_t *__restrict__ keys_out,
               int *__restrict__ ids_out)
{
    chain_wait();
    chain_release();
    __shared__ uint16_t s_cnt[8][kRadixBins];
    __shared__ int s_base[kRadixBins];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < 8 * kRadixBins / 2; i += 256) ((uint32_t *)s_cnt)[i] = 0;
    __syncthreads();
    if (g->status != 0) return;
    const int64_t base = (int64_t)blockIdx.x * (ROUNDS * 256) + w * (ROUNDS * 32);
    uint64_t key[ROUNDS];
    uint16_t rank[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int64_t v = base + r * 32 + lane;
        key[r] = v < n_vert ? keys_in[v] : 0;
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int64_t v = base + r * 32 + lane;
        const int d = v < n_vert ? (int)((key[r] >> shift) & (kRadixBins - 1)) : kRadixBins;
        const unsigned peers = __match_any_sync(FGC_FULL_MASK, d);
        const int before = d < kRadixBins ? s_cnt[w][d] : 0;
        __syncwarp();
        if (d < kRadixBins && (peers & lanemask_lt()) == 0) s_cnt[w][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        rank[r] = (uint16_t)(before + __popc(peers & lanemask_lt()));
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kRadixBins; d += 256) {
        s_base[d] = hist[(size_t)d * n_tiles + blockIdx.x];
        int run = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int c = s_cnt[k][d];
            s_cnt[k][d] = (uint16_t)run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int64_t v = base + r * 32 + lane;
        if (v < n_vert) {
            const int d = (int)((key[r] >> shift) & (kRadixBins - 1));
            const int to = s_base[d] + s_cnt[w][d] + rank[r];
            if (FGC_DBG_OK(to >= 0 && to < n_vert, &g->status)) {
                if (keys_out) keys_out[to] = key[r];
                ids_out[to] = ids_in ? ids_in[v] : (int)v;
            }
        }
    }
}

// Row split of box slot s at a level: the largest e with tree_base(row_splits[e], e) <= s.
__device__ __forceinline__ int tree_event_of(const int64_t *__restrict__ rs, int n_rs, int64_t s, int shift)
{
    int lo = 0, hi = n_rs - 2;
    while (lo < hi) {
        const int mid = (int)(((int64_t)lo + hi + 1) >> 1);
        if (tree_base(rs[mid], mid, shift) <= s) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// What the search by groups reads beside the tree (TreeLayout); null: it is not taken.
struct LeafArrays {
    float4 *box_lo, *box_hi, *half_lo, *half_hi, *point_a;
    float2 *box_e, *half_e;
    float *point_e;
};

// One CTA per node slot (32 leaves): points in curve order, the boxes of the leaves and the node's.
template <int NV>
__global__ void __launch_bounds__(256)
k_tree_leaves(const float *__restrict__ coords, int n_vert, int n_coords, const int64_t *__restrict__ direction,
              const int64_t *__restrict__ row_splits, int n_rs, KnnGrid *__restrict__ g, const int *__restrict__ ids,
              int *__restrict__ sorig, float4 *__restrict__ scoords, uint8_t *__restrict__ sflag,
              float4 *__restrict__ leaf_box, float4 *__restrict__ node_box, const LeafArrays arrays, int *__restrict__ out_order)
{
    chain_wait();
    chain_release();
    if (g->status != 0) {                                   // kNotBuilt
        for (int v = blockIdx.x * 256 + threadIdx.x; v < n_vert; v += gridDim.x * 256) {
            sorig[v] = v;
            if (out_order) out_order[v] = v;
        }
        return;
    }
    __shared__ uint32_t s_lo[4 * NV], s_hi[4 * NV];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < 4 * NV) { s_lo[threadIdx.x] = 0xffffffffu; s_hi[threadIdx.x] = 0; }
    __syncthreads();
    const int e = tree_event_of(row_splits, n_rs, blockIdx.x, 10);
    const int64_t ev_begin = row_splits[e], ev_end = row_splits[e + 1];
    const int64_t node = (int64_t)blockIdx.x - tree_base(ev_begin, e, 10);
    const int64_t first = ev_begin + node * 1024;
    if (first >= ev_end) return;                              // a slot without points
    const int64_t leaf0 = tree_base(ev_begin, e, 5) + node * 32;
    for (int l = w; l < 32 && first + l * 32 < ev_end; l += 8) {
        const int64_t j = first + l * 32 + lane;
        const bool act = j < ev_end;
        int id = act ? ids[j] : 0;
        if (!FGC_DBG_OK(id >= 0 && id < n_vert, &g->status)) id = 0;
        float x[4 * NV];
#pragma unroll
        for (int c = 0; c < 4 * NV; c++) x[c] = act && c < n_coords ? __ldg(coords + (size_t)id * n_coords + c) : 0.f;
        if (act) {
            sorig[j] = id;
            if (out_order) out_order[j] = id;
#pragma unroll
            for (int v = 0; v < NV; v++)
                scoords[(size_t)j * NV + v] = make_float4(x[4 * v], x[4 * v + 1], x[4 * v + 2], x[4 * v + 3]);
            if (direction) {
                const int64_t d = direction[id];
                sflag[j] = d >= 0 && d <= 2 ? (uint8_t)d : (uint8_t)3;
            }
        }
        float lo[4 * NV], hi[4 * NV];
        float half_lo[4 * NV], half_hi[4 * NV];                // of the lane's half
#pragma unroll
        for (int c = 0; c < 4 * NV; c++) {
            const uint32_t k = float_to_ordered(x[c]);
            const bool low = lane < 16;
            const uint32_t a0 = __reduce_min_sync(FGC_FULL_MASK, act && low ? k : 0xffffffffu);
            const uint32_t b0 = __reduce_max_sync(FGC_FULL_MASK, act && low ? k : 0u);
            const uint32_t a1 = __reduce_min_sync(FGC_FULL_MASK, act && !low ? k : 0xffffffffu);
            const uint32_t b1 = __reduce_max_sync(FGC_FULL_MASK, act && !low ? k : 0u);
            const uint32_t a = min(a0, a1), b = max(b0, b1);
            lo[c] = ordered_to_float(a);
            hi[c] = ordered_to_float(b);
            // (a half without points is infinitely far from everything)
            half_lo[c] = low ? ordered_to_float(a0) : (a1 <= b1 ? ordered_to_float(a1) : __uint_as_float(0x7f800000u));
            half_hi[c] = low ? ordered_to_float(b0) : (a1 <= b1 ? ordered_to_float(b1) : __uint_as_float(0xff800000u));
            if (lane == 0) { atomicMin(&s_lo[c], a); atomicMax(&s_hi[c], b); }
        }
        if constexpr (NV == 2) {
            if (arrays.box_lo) {
                const size_t at = (size_t)(leaf0 + l), half = 2 * at + (lane >> 4);
                if (lane == 0) {
                    arrays.box_lo[at] = make_float4(lo[0], lo[1], lo[2], lo[3]);
                    arrays.box_hi[at] = make_float4(hi[0], hi[1], hi[2], hi[3]);
                    arrays.box_e[at] = make_float2(lo[4], hi[4]);
                }
                if ((lane & 15) == 0) {
                    arrays.half_lo[half] = make_float4(half_lo[0], half_lo[1], half_lo[2], half_lo[3]);
                    arrays.half_hi[half] = make_float4(half_hi[0], half_hi[1], half_hi[2], half_hi[3]);
                    arrays.half_e[half] = make_float2(half_lo[4], half_hi[4]);
                }
                if (act) {
                    arrays.point_a[j] = make_float4(x[0], x[1], x[2], x[3]);
                    arrays.point_e[j] = x[4];
                }
            }
        }
        if (lane == 0) {
            float4 *out = leaf_box + (size_t)(leaf0 + l) * 2 * NV;
#pragma unroll
            for (int v = 0; v < NV; v++) {
                out[v] = make_float4(lo[4 * v], lo[4 * v + 1], lo[4 * v + 2], lo[4 * v + 3]);
                out[NV + v] = make_float4(hi[4 * v], hi[4 * v + 1], hi[4 * v + 2], hi[4 * v + 3]);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 4 * NV) {
        float *out = (float *)(node_box + (size_t)blockIdx.x * 2 * NV);
        out[threadIdx.x] = ordered_to_float(s_lo[threadIdx.x]);
        out[4 * NV + threadIdx.x] = ordered_to_float(s_hi[threadIdx.x]);
    }
}

// One warp per top slot: the box over its up to 32 nodes.
template <int NV>
__global__ void __launch_bounds__(256)
k_tree_top(const int64_t *__restrict__ row_splits, int n_rs, const KnnGrid *__restrict__ g,
           const float4 *__restrict__ node_box, float4 *__restrict__ top_box, int64_t n_slots)
{
    chain_wait();
    chain_release();
    if (g->status != 0) return;
    const int lane = threadIdx.x & 31;
    const int64_t slot = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (slot >= n_slots) return;
    const int e = tree_event_of(row_splits, n_rs, slot, 15);
    const int64_t ev_begin = row_splits[e], ev_end = row_splits[e + 1];
    const int64_t top = slot - tree_base(ev_begin, e, 15);
    if (ev_begin + top * 32768 >= ev_end) return;
    const int64_t node = top * 32 + lane;
    const bool act = ev_begin + node * 1024 < ev_end;
    const float *in = (const float *)(node_box + (size_t)(tree_base(ev_begin, e, 10) + node) * 2 * NV);
    float *out = (float *)(top_box + (size_t)slot * 2 * NV);
#pragma unroll
    for (int c = 0; c < 4 * NV; c++) {
        const uint32_t a = __reduce_min_sync(FGC_FULL_MASK, act ? float_to_ordered(__ldg(in + c)) : 0xffffffffu);
        const uint32_t b = __reduce_max_sync(FGC_FULL_MASK, act ? float_to_ordered(__ldg(in + 4 * NV + c)) : 0u);
        if (lane == 0) { out[c] = ordered_to_float(a); out[4 * NV + c] = ordered_to_float(b); }
    }
}

#define FGC_TRY(expr)                                    \
    do {                                                 \
        const cudaError_t rc_ = (expr);                  \
        if (rc_ != cudaSuccess) return rc_;              \
    } while (0)

template <int ROUNDS>
static cudaError_t sort_points(const float *coords, int n, int n_coords, const int64_t *row_splits, int n_rs,
                               const KnnWorkspace &L, const TreeLayout &T, char *ws, cudaStream_t s)
{
    KnnGrid *g = (KnnGrid *)(ws + L.header);
    KnnTree *t = (KnnTree *)(ws + L.tickets);
    uint64_t *keys[2] = {(uint64_t *)(ws + T.keys[0]), (uint64_t *)(ws + T.keys[1])};
    int *ids[2] = {(int *)(ws + T.ids[0]), (int *)(ws + T.ids[1])};
    int *hist = (int *)(ws + T.hist), *sums = (int *)(ws + T.hist_sums);
    FGC_TRY(launch_chained(k_tree_keys<ROUNDS>, T.tiles, 256, 0, s, coords, n, n_coords, T.key_dims, T.bits, row_splits,
                           n_rs, g, t, keys[0], hist, T.tiles));
    const int entries = kRadixBins * T.tiles;
    const int scan_blocks = (entries + kScanTile - 1) / kScanTile;
    for (int p = 0; p < T.passes; p++) {
        const int shift = p * kRadixBits;
        if (p > 0) FGC_TRY(launch_chained(k_tree_hist<ROUNDS>, T.tiles, 256, 0, s, keys[p & 1], n, shift, g, hist, T.tiles));
        FGC_TRY(launch_chained(k_scan_tile_sums_top, scan_blocks, 256, 0, s, hist, nullptr, entries, sums, &t->scan_ticket));
        FGC_TRY(launch_chained(k_scan_apply, scan_blocks, 256, 0, s, hist, nullptr, entries, sums));
        FGC_TRY(launch_chained(k_tree_scatter<ROUNDS>, T.tiles, 256, 0, s, keys[p & 1], p > 0 ? ids[p & 1] : nullptr, n,
                               shift, g, hist, T.tiles, p + 1 < T.passes ? keys[(p + 1) & 1] : nullptr, ids[(p + 1) & 1]));
    }
    return cudaSuccess;
}

template <int NV>
static cudaError_t launch_boxes(const float *coords, int n, int n_coords, const int64_t *direction,
                                const int64_t *row_splits, int n_rs, const KnnWorkspace &L, const TreeLayout &T, const int *ids,
                                int *out_order, char *ws, cudaStream_t s)
{
    KnnGrid *g = (KnnGrid *)(ws + L.header);
    LeafArrays arrays = {};
    if (T.groups && n_coords == kApartDims) {
        arrays.box_lo = (float4 *)(ws + T.box_lo); arrays.box_hi = (float4 *)(ws + T.box_hi); arrays.box_e = (float2 *)(ws + T.box_e);
        arrays.half_lo = (float4 *)(ws + T.half_lo); arrays.half_hi = (float4 *)(ws + T.half_hi); arrays.half_e = (float2 *)(ws + T.half_e);
        arrays.point_a = (float4 *)(ws + T.point_a); arrays.point_e = (float *)(ws + T.point_e);
    }
    FGC_TRY(launch_chained(k_tree_leaves<NV>, (unsigned)T.n_box[1], 256, 0, s, coords, n, n_coords, direction,
                           row_splits, n_rs, g, ids, (int *)(ws + L.sorig),
                           (float4 *)(ws + L.scoords), (uint8_t *)(ws + L.sflag), (float4 *)(ws + T.box[0]),
                           (float4 *)(ws + T.box[1]), arrays, out_order));
    if (n <= 32768) return cudaSuccess;                  // no row split has more than one top node: never read
    return launch_chained(k_tree_top<NV>, (unsigned)((T.n_box[2] + 7) / 8), 256, 0, s, row_splits, n_rs, g,
                          (const float4 *)(ws + T.box[1]), (float4 *)(ws + T.box[2]), T.n_box[2]);
}

}  // namespace fgc

// Points per row split that the search by groups needs: with fewer a leaf's warp has few queries, and the grid takes whole
// row splits.  Time over the grid's, uniform points, splits of 100 / 200 / 256 / 300 / 400 points: three coordinates, K = 36, 800 k 1.43 / 0.89 / 0.76 /
// 0.68 / 0.57, K = 64, 200 k 1.76 / 1.19 / 1.05 / 0.95 / 0.76, K = 66 1.24 / 0.57 / 0.46, K = 128 1.78 / 0.73 / 0.52, K = 200 1.32 / 1.28 / 0.62, 20 k,
// K = 257 in splits of 256 1.32, 400 0.65; four, 200 k, K = 40 - / 1.20 / 1.04 / 0.96 / 0.79; five, 800 k, K = 66 1.07 / 0.54, in splits of 50 2.2.
static int64_t least_row_split(int64_t n_vert, int K)
{
    return K <= 65 ? (n_vert >= 800000 ? 256 : 300) : (K < 160 ? 200 : K + K / 4);
}

// Where the tree is the better search.  Neither search is ahead for all data: the figures are the time of the tree over that of
// the grid, whole forward, B200, for uniform points in a cube / normal ones / 50 clusters of width 0.02 ("mixture"); up to five
// coordinates they are of the search one query at a time (the forward's search by groups takes 0.6 to 0.9 of its time).
// Below 16384 points the sort's launches outweigh the search (10 k in three coordinates, K = 100: 0.110 / 0.112 ms); in up to
// five coordinates, where the forward searches by groups, so they do for tiny row splits (least_row_split).
//
// D = 3, K >= 96: the grid's list of four slots a lane (K > 65) is slow, and a dense cluster fits into one of its cells.  400 k
// points in two row splits, K = 96: 0.98 / 0.74 / 0.74, skewed clusters 0.41; K = 80: 1.06 / 0.70 / 0.67, K = 66: 1.20 / 0.78 /
// 0.69.  From 65536 points on (one of 20 k uniform, K = 96: 0.164 / 0.204 ms).
// D = 4: K = 100 uniform 1.08, one row split of 20 k 1.2: the grid (but see long_tails).
// D = 5 and more: the grid bins four of the coordinates, the tree's boxes have them all.  K > 65: D = 5, 800 k in eight row
// splits, K = 66: 0.69 / 0.87 / 0.69; D = 6, 400 k in twenty 0.57 / 0.91 / 0.60.  Shorter lists need the more coordinates the
// shorter they are; with one or two row splits the grid's last warps run on alone over sparse tails, and the tree is ahead earlier:
//   D = 5   100 k, K = 40: 0.86 / 0.72 / 0.97;  in twenty row splits 0.79 / 1.06 / 1.47;  K = 32: 0.92 / 1.05 / 1.25
//   D = 6   400 k, K = 24: 0.56 / 0.78 / 1.19;  in twenty 0.72 / 1.30 / 1.19, K = 48: 0.63 / 1.08 / 0.86
//   D = 7   400 k, K = 16: 0.51 / 0.89 / 1.30;  in twenty 0.62 / 1.24 / 1.21, K = 40: 0.51 / 1.06 / 0.93
//   D = 8   400 k, K = 16: 0.46 / 0.86 / 1.25;  in twenty 0.53 / 1.15 / 1.15, K = 24: 0.44 / 1.04 / 1.06
//   D = 9   100 k, K = 8: 0.50 / 0.85 / 0.87;  in five 0.55 / 0.91 / 0.94;  K = 2: 0.94 / 1.37 / 1.05
//   D = 12  100 k, K = 2: 0.50 / 0.99 / 0.88;  in five 0.49 / 0.95 / 0.93
// The tree's worst are small row splits of clusters with hardly more points than K: 5000 in 50 clusters, K = 65, D = 9: 1.55 (0.09
// uniform, 0.62 normal).
//
// long_tails: the caller expects coordinates with sparse tails, as the learned ones of a GravNet layer have (linear
// maps of many features; "learned" are normal points mapped from 64 to 4).  In four dimensions the grid's last warps then walk
// empty cells long after all others are done, unless many row splits hide them.  Learned, K = 32 / 40 / 64: one row split of 20 k
// to 400 k 0.64 to 0.88, four of 25 k 0.93 / 0.78 / 0.74, ten of 20 k 1.10 / 0.96 / 0.89, fifty of 8 k 1.27 / 1.10 / 1.00, K = 66
// there 0.75.  16 of 100 k: 8.28 / 9.18 (K = 40) and 10.7 / 11.0 ms (K = 64).  K = 16 has less to gain (four of 50 k:
// 0.92 / 0.95 ms), so have three dimensions (four of 50 k, K = 40: 0.67 / 0.78 ms); uniform points in a cube have no tails
// (100 k, K = 40: 0.41 / 0.53 ms).
extern "C" int fgc_knn_tree_preferred(int64_t n_vert, int32_t n_coords, int64_t n_rs, int32_t K, int32_t long_tails)
{
    using namespace fgc;
    if (n_vert < 16384 || n_vert > 0x7fffffff || n_coords < 2 || n_coords > FGC_MAX_KNN_DIMS || n_rs < 2 ||
        n_rs > 0x7fffffff || K < 1 || K > FGC_MAX_K)
        return 0;
    const int64_t n_events = n_rs - 1;
    int least = FGC_MAX_K + 1;                   // shortest list for the tree
    switch (n_coords) {
    case 2: break;
    case 3: if (n_vert >= 65536) least = 96; break;
    case 4: if (long_tails && n_vert <= 500000) least = n_events <= 4 ? 32 : (n_events <= 16 ? 40 : 66); break;
    case 5: least = n_events <= 2 ? 40 : 66; break;
    case 6: least = n_events <= 2 ? 24 : 48; break;
    case 7: least = n_events <= 2 ? 16 : 40; break;
    case 8: least = n_events <= 2 ? 16 : 24; break;
    case 9: case 10: case 11: least = 8; break;
    default: least = 1;
    }
    if (K < least || (K > 65 && n_coords <= kGroupDims && n_vert / n_events < least_row_split(n_vert, K))) return 0;
    return tree_layout(knn_workspace_layout(n_vert, n_coords, n_rs, K), n_vert, n_coords, n_rs).fits ? 1 : 0;
}

// Where the search by groups (knn_tree_group.cu) is ahead of the grid, beyond where the tree is taken anyway.  The figures are
// its time over that of the grid, whole forward with the second look at rows with equal distances (FGC_FORWARD_GRID_ORDER), B200,
// uniform / normal / mixture points, and in three coordinates skewed clusters:
//   three coordinates  K = 128: 20 k in four row splits 0.96 / 0.47 / 0.63 / 0.38;  K = 80: 50 k 0.83 / 0.60 / 0.66 / 0.64, K = 64: 1.21 /
//                      0.95 / 1.23 / 0.87;  K = 66: 150 k 0.89 / 0.46 / 0.68 / 0.46, K = 64: 1.11 / 0.62 / 0.97 / 0.60, 200 k 1.05 / 0.67 /
//                      0.89 / 0.49, 300 k in six 0.96 / 0.75 / 0.88 / 0.57, K = 48: 400 k in eight 1.00 / 0.80 / 0.91 / 0.56;  K = 36: 800 k
//                      0.95 / 0.50 / 0.83 / 0.33, K = 32: 1.03 / 0.52 / 0.97 / 0.37
//   four               K = 128: 20 k in four 0.49 / 0.46 / 0.58;  K = 72: 50 k 0.94 / 0.44 / 0.71, K = 40: 1.26 / 0.60 / 1.04, 200 k in
//                      eight 1.04 / 0.82 / 0.91, 13 1.00 / 0.91 / 0.98, K = 24: 1.09 / 0.96 / 1.13;  800 k, K = 24: 1.09 / 0.51 / 0.62, in 16 0.99 / 0.94 /
//                      0.80, K = 16: 1.13 / 0.49 / 0.67, in 16 1.04 / 1.00 / 0.84, K = 8 1.30 / 1.03 / 0.75
//   five               K = 40: 60 k in four 0.87 / 0.89 / 1.22, 200 k in four 0.69 / 0.98 / 0.96, 600 k in five 0.67 / 0.98 / 0.84, 20 k 0.83 /
//                      0.72 / 1.20;  K = 66: in three or more 0.60 / 0.77 / 0.53
// The worst are row splits of 5000 points in 50 clusters, for which the grid's cells are right (1.05 to 1.3 with K <= 65), and lattices
// (1.0 to 1.2: a million points, K = 64, on 40 x 40 x 40 places).
// Short lists in four coordinates: K = 16 in splits of 1500 0.90 / 1.12 / 1.47, of 5000 0.89 / 1.08 / 1.09, K = 24 of 1500 0.82 / 1.03 / 1.24,
// K = 32 0.79 / 0.99 / 0.77.
// Whether distances get gradients plays no part: the same call takes the same search with and without, and gives the
// same neighbours in the same slots.
// long_tails: learned coordinates as in fgc_knn_tree_preferred, no second look: three coordinates, row splits of 15 k or more 0.60
// to 0.80 at K = 16, of 10 k 0.95 at K = 24, of 2000 0.99 at K = 40 and 0.86 at 64; four, 0.56 to 0.95 at K = 8, 0.91 to 0.94 at K = 24, 0.81
// to 0.85 at K = 40.
extern "C" int fgc_knn_groups_preferred(int64_t n_vert, int32_t n_coords, int64_t n_rs, int32_t K, int32_t long_tails)
{
    using namespace fgc;
    if (n_vert < 16384 || n_vert > 0x7fffffff || n_coords < 3 || n_coords > kGroupDims || n_rs < 2 || n_rs > 0x7fffffff || K < 1 ||
        K > FGC_MAX_K)
        return 0;
    const int64_t n_events = n_rs - 1, mean = n_vert / n_events;
    int least = FGC_MAX_K + 1;                   // shortest list
    if (long_tails && n_coords <= 4) {
        const bool four = n_coords == 4;
        if (mean >= 15000) least = four ? 8 : 16;
        else if (mean >= 8000) least = 24;
        else if (mean >= 1500) least = four ? 40 : 48;
    } else if (n_coords == 5) {
        if (n_vert >= 60000 && mean >= 15000) least = 40;
    } else if (n_coords == 4) {
        least = n_vert >= 50000 ? 72 : 128;
        if (n_vert >= 200000 && n_events >= 8) least = 40;
        if (n_vert >= 800000) least = mean >= 5000 ? 16 : 32;
    } else {
        least = n_vert >= 800000 ? 36 : (n_vert >= 200000 ? 64 : (n_vert >= 150000 ? 66 : (n_vert >= 50000 ? 80 : 128)));
    }
    if (K < least || mean < least_row_split(n_vert, K)) return 0;
    return tree_layout(knn_workspace_layout(n_vert, n_coords, n_rs, K), n_vert, n_coords, n_rs).fits ? 1 : 0;
}

// What the search by groups has won since: with lists for eight queries it takes 0.6 to 0.8 of the time that the figures above are of.
// Time over that of the grid, as above, in one row split / eight (mean size in brackets where it matters):
//   three coordinates  K = 12: 1.6 M in 16 0.95 / 0.82 / 0.90 / 0.43, K = 8 1.10;  K = 16: 800 k 0.94 / 0.78 / 0.93 / 0.44, in 160 0.93 / 0.90 / 1.10 /
//                      0.54;  K = 32: 400 k 0.93 / 0.46 / 0.90 / 0.40 and 0.92 / 0.74 / 0.99 / 0.48, K = 24 1.00; K = 40, in 80 0.82 / 0.76 / 1.05 / 0.18;
//                      K = 48: 200 k 0.98 / 0.52 / 0.86 / 0.53 and 0.97 / 0.74 / 0.95 / 0.64, K = 40 1.01;  K = 64: 100 k 0.99 / 0.55 / 0.93 / 0.61 and
//                      0.97 / 0.63 / 1.06 / 0.60;  K = 66: 50 k 0.83 / 0.59 / 0.82 / 0.63
//   four               K = 12: 1.6 M in 16 0.85 / 0.74 / 0.61, K = 8 1.03;  K = 16: 400 k 0.95 / 0.43 / 0.61 and 0.90 / 0.75 / 0.76;  K = 24: 400 k in 80
//                      0.74 / 0.78 / 1.12, 200 k 1.00 / 0.51 / 0.72 and 0.97 / 0.78 / 0.96;  K = 32: 200 k in 40 0.85 / 0.84 / 1.30 (not taken);  K = 40: 100 k 0.94 /
//                      0.48 / 0.81 and 0.89 / 0.74 / 1.01;  K = 66: 50 k 0.85 / 0.38 / 0.51
//   five               K = 4: 800 k 0.75 / 0.42 / 0.58 and 0.77 / 0.65 / 0.72;  K = 8: 200 k in eight 0.88 / 0.70 / 1.06, 800 k in 160 0.70 / 0.79 / 1.07;  K = 24:
//                      50 k in one 0.65 / 0.57 / 1.12;  not taken, since clusters lose more than a tenth: K = 16 there 0.84 / 0.52 / 1.18, 50 k in
//                      five, K = 40 0.65 / 0.65 / 1.24, in twelve 0.62 / 0.75 / 1.50;  200 k in 40 0.45 / 0.64 / 1.25;  20 k in four 0.74 / 0.59 / 1.55
//   learned, three     K = 8: 50 k in one 0.84;  K = 16: 50 k in ten 0.78, 200 k in 40 0.96;  K = 24: 50 k in 25 0.84
//   learned, four      K = 8: 50 k in ten 0.87, 200 k in 40 0.97;  K = 16: 50 k in 25 0.84
//   learned, sorted in one launch (up to kSmallTree points; three / four)  K = 10: 3 k in one row split 0.63 / 0.64, 5 k in five 0.90 / 0.90, 10 k in
//                      thirty 0.92 / 0.98, 16 k in fifty 0.84 / 0.89;  K = 40: 10 k in ten 0.76 / 0.68, 20 k in one 0.69 / 0.38;  K = 16: 1000 in one 0.88 / 0.91
// The ranges weigh uniform, normal and skewed points most.  Clusters of about as many points as K, for which the grid's cells are right, lose:
// uniform / normal / mixture / skewed again, three coordinates, 800 k in 200, K = 16 0.91 / 0.90 / 1.11 / 0.81; four, 200 k in 20, K = 32 0.88 / 0.80 /
// 1.12 / 0.20, 400 k in 100, K = 24 and 31 0.72 / 0.79 / 1.19 / 0.44 and 0.71 / 0.84 / 1.24 / 0.26; five, 50 k in two, K = 24 0.72 / 0.54 / 1.28 / 0.25, 100 k in five
// 0.61 / 0.62 / 1.15 / 0.19, 800 k in 200, K = 8 0.70 / 0.80 / 1.12 / 0.80.  So do layers whose coordinates are not what long_tails says, learned / mixture /
// uniform: three, 5000 in one, K = 8 0.94 / 1.18 / 1.46, 50 k in one, K = 8 0.97 / 1.34 / 1.57; four, 5000 in one 0.67 / 1.10 / 1.65, 50 k in 33, K = 16 0.86 /
// 1.43 / 1.02.
extern "C" int fgc_knn_groups_ahead(int64_t n_vert, int32_t n_coords, int64_t n_rs, int32_t K, int32_t long_tails)
{
    using namespace fgc;
    if (n_vert < 1000 || n_vert > 0x7fffffff || n_coords < 3 || n_coords > kGroupDims || n_rs < 2 || n_rs > 0x7fffffff || K < 1 ||
        K > FGC_MAX_K)
        return 0;
    const int64_t mean = n_vert / (n_rs - 1);
    const bool large = mean >= 10000;
    int least = FGC_MAX_K + 1;                   // shortest list
    if (long_tails && n_coords <= 4) {
        if (n_vert <= kSmallTree) least = n_vert >= 3000 ? 8 : (mean >= 1000 ? 16 : least);
        else if (n_coords == 4) least = mean >= 4000 ? 8 : (mean >= 1500 ? 16 : least);
        else least = mean >= 15000 ? 8 : (mean >= 4000 ? 16 : (mean >= 1500 ? 24 : least));
    } else if (n_coords == 5) {
        if (n_vert >= 50000 && mean >= 20000) least = n_vert >= 200000 ? 8 : 24;
        if (n_vert >= 800000 && mean >= 4000) least = large ? 4 : 8;
    } else if (n_coords == 4) {
        if (n_vert >= 50000) least = 66;
        if (n_vert >= 100000 && large) least = 40;
        if (n_vert >= 200000 && large) least = mean >= 20000 ? 24 : 32;
        if (n_vert >= 400000 && mean >= 4000) least = mean >= 20000 ? 16 : 24;
        if (n_vert >= 800000 && mean >= 4000) least = 16;
        if (n_vert >= 1500000 && large) least = 12;
    } else {
        if (n_vert >= 50000) least = 66;
        if (n_vert >= 100000 && large) least = 64;
        if (n_vert >= 200000 && large) least = 48;
        if (n_vert >= 400000 && mean >= 4000) least = large ? 32 : 40;
        if (n_vert >= 800000 && mean >= 4000) least = 16;
        if (n_vert >= 1500000 && large) least = 12;
    }
    if (K < least || mean < least_row_split(n_vert, K)) return 0;
    return tree_layout(knn_workspace_layout(n_vert, n_coords, n_rs, K), n_vert, n_coords, n_rs).groups ? 1 : 0;
}

namespace fgc {

int knn_build_tree_forward(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K,
                           const int64_t *direction_or_null, int32_t *info_mapped, int32_t *out_order, bool *words, void *workspace,
                           size_t workspace_bytes, fgc_stream_t stream)
{
    FGC_NVTX("fgc_knn_build_tree");
    KnnWorkspace L;
    if (!row_splits) return FGC_ERR_BAD_ARGUMENT;
    const int rc = check_knn_args(n_vert, n_coords, n_rs, K, workspace, workspace_bytes, &L);
    if (rc != FGC_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    char *ws = (char *)workspace;
    KnnGrid *g = (KnnGrid *)(ws + L.header);
    KnnTree *t = (KnnTree *)(ws + L.tickets);
    int key_dims, bits, passes;
    const bool small = n_vert > 0 && small_tree_bits(n_vert, n_coords, n_rs, &key_dims, &bits, &passes);
    if (!small) FGC_RETURN_IF_CUDA(cudaMemsetAsync(g, 0, kGridHeaderBytes + kHardTicketBytes, s));
    if (n_vert == 0) return FGC_OK;
    if (!coords || n_rs < 2) return FGC_ERR_BAD_ARGUMENT;
    const TreeLayout T = tree_layout(L, n_vert, n_coords, n_rs);
    if (!T.fits) return FGC_ERR_TOO_LARGE;
    const int n = (int)n_vert, nrs = (int)n_rs;
    const int *ids = (const int *)(ws + T.ids[small ? 1 : T.passes & 1]);
    if (small) {
        FGC_RETURN_IF_CUDA(launch_tree_small(coords, n, n_coords, key_dims, bits, passes, row_splits, nrs, g, t, (uint32_t *)(ws + T.keys[0]),
                                             (int *)(ws + T.ids[0]), (int *)(ws + T.ids[1]), info_mapped, s));
        if (words) *words = true;
    } else {
        const int64_t pt_blocks = (n_vert + 255) / 256;
        const int red_blocks = pt_blocks < sm_count() * 4 ? (int)pt_blocks : sm_count() * 4;
        k_tree_extent<<<red_blocks, 256, 0, s>>>(coords, n, n_coords, T.key_dims, T.bits, row_splits, nrs, g, t);
        FGC_CHECK_LAUNCH();
        FGC_RETURN_IF_CUDA(T.rounds == 16 ? sort_points<16>(coords, n, n_coords, row_splits, nrs, L, T, ws, s)
                                          : sort_points<4>(coords, n, n_coords, row_splits, nrs, L, T, ws, s));
    }
    auto boxes = L.nv == 1 ? launch_boxes<1> : (L.nv == 2 ? launch_boxes<2> : (L.nv == 3 ? launch_boxes<3> : launch_boxes<4>));
    FGC_RETURN_IF_CUDA(boxes(coords, n, n_coords, direction_or_null, row_splits, nrs, L, T, ids, out_order, ws, s));
    return FGC_OK;
}

}  // namespace fgc

extern "C" int fgc_knn_build_tree(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits,
                                  int64_t n_rs, int32_t K, const int64_t *direction_or_null, void *workspace,
                                  size_t workspace_bytes, fgc_stream_t stream)
{
    return fgc::knn_build_tree_forward(coords, n_vert, n_coords, row_splits, n_rs, K, direction_or_null, nullptr, nullptr, nullptr, workspace,
                                       workspace_bytes, stream);
}
