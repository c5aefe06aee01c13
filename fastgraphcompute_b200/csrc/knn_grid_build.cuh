// Parts shared by the two builds of the search grid (knn_grid.cu in a chain of launches, knn_grid_small.cu in one).
#pragma once
#include "knn_grid.cuh"
#include "segsort.cuh"

namespace fgc {

// Cells per dimension for a wanted cell width; widens the cells until the table fits.
__device__ inline void fit_shape(const float (&ext)[4], double wd, int bins_cap, int (&n)[4], float &w)
{
    for (int iter = 0; iter < 400; iter++) {
        w = (float)wd;
        const float inv = __fdiv_rn(1.0f, w);
        double prod = 1.0;
        for (int gd = 0; gd < 4; gd++) {
            n[gd] = ext[gd] > 0.f ? (int)floorf(__fmul_rn(ext[gd], inv)) + 1 : 1;
            prod *= (double)n[gd];
        }
        if (prod <= (double)bins_cap) break;
        wd *= 1.05;
    }
}

// One thread.  Chooses the cell width so that a row split of average size gets
// about bins_target cells, bounded by bins_cap cells per row split.
static __device__ void grid_setup(KnnGrid *g, const uint32_t (&min_key)[4], const uint32_t (&max_key)[4], bool nonfinite, int n_rs,
                           int n_bin_dims, int bins_target, int bins_cap_first, int bins_cap, int bad_rs, int mirror)
{
    int status = 0;
    if (nonfinite) status |= FGC_STATUS_NONFINITE;
    if (bad_rs) status |= FGC_STATUS_BAD_ROW_SPLITS;
    const int n_events = n_rs - 1;
    const int G = n_bin_dims >= 4 ? 4 : 3;      // grid dimensions in use
    const int sh = G - n_bin_dims;
    float ext[4];
    double vol = 1.0;
    int nz = 0;
    float ext_max = 0.f;
    for (int gd = 0; gd < 4; gd++) {
        if (gd >= G) {
            g->cdim[gd] = -1;
            g->origin[gd] = 0.f;
            ext[gd] = 0.f;
        } else if (gd < sh || (status & FGC_STATUS_NONFINITE)) {
            g->cdim[gd] = gd < sh ? -1 : gd - sh;
            g->origin[gd] = 0.f;
            ext[gd] = 0.f;
        } else {
            const int c = gd - sh;
            const float lo = ordered_to_float(~min_key[c]), hi = ordered_to_float(max_key[c]);
            g->cdim[gd] = c;
            g->origin[gd] = lo;
            ext[gd] = __fsub_rn(hi, lo);
            if (!(ext[gd] >= 0.f) || !is_finite_bits(ext[gd])) ext[gd] = 0.f;
        }
        if (ext[gd] > 0.f) { vol *= (double)ext[gd]; nz++; }
        ext_max = fmaxf(ext_max, ext[gd]);
    }
    int n[4] = {1, 1, 1, 1};
    float w = 1.f;
    if (nz > 0) {
        if (bins_target < 1) bins_target = 1;
        double wd = pow(vol / (double)bins_target, 1.0 / (double)nz);
        // a degenerate extent ratio can make the width underflow: keep it representable
        if (!(wd > (double)ext_max * 1e-6)) wd = (double)ext_max * 1e-6;
        fit_shape(ext, wd, bins_cap_first, n, w);
    }
    long long B = (long long)n[0] * n[1] * n[2] * n[3];
    if (B > bins_cap_first) {  // cannot happen after the loop above unless the extents are absurd
        n[0] = n[1] = n[2] = n[3] = 1; B = 1; w = fmaxf(ext_max, 1.f) * 2.f;
        status |= FGC_STATUS_INTERNAL;
    }
    g->n[0] = n[0]; g->n[1] = n[1]; g->n[2] = n[2]; g->n[3] = n[3];
    g->gdims = G;
    g->B = (int)B;
    g->n_events = n_events;
    g->mirror = mirror;
    g->total_bins = (int)(B * n_events * mirror);
    grid_set_divisors(g);
    g->w = w;
    g->inv_w = __fdiv_rn(1.0f, w);
    g->slack = 4e-6f * fmaxf(ext_max, w);
    g->ext[0] = ext[0]; g->ext[1] = ext[1]; g->ext[2] = ext[2]; g->ext[3] = ext[3];
    g->bins_cap = bins_cap;
    g->status = status;
}

// Density pass.  The first grid is sized from the bounding box, i.e. from the MEAN density.
// Clustered data puts most points into cells far above that mean, and the cost of a query
// grows with the occupancy of the cells around it.  sum_c c^2 / N is the occupancy a typical
// point sees in its own cell; when it is well above the wanted value the grid is rebuilt
// with cells shrunk by the cube root of the ratio (occupancy scales with the cell volume
// where the density is locally smooth).
// pass 0: the density pass on the first grid.  pass 1: a second one, only after pass 0 fell
// back from a grid over four coordinates to one over three (D = 4 only): a dense cell table
// over the four-dimensional bounding box cannot follow strongly clustered data -- the wanted
// cell size would need far more cells than the table holds -- so data that asks for cells more
// than 2.8x finer than the mean density suggests is binned in three coordinates, where the
// same table reaches the wanted size.
static __device__ void grid_refine(KnnGrid *g, unsigned long long sum_sq, int n_vert, float seen_target,
                            float seen_target3, int bins_target3, int pass, int allow_fallback)
{
    const float target = pass == 0 ? seen_target : seen_target3;
    const double seen = (double)sum_sq / (double)(n_vert > 0 ? n_vert : 1);
    if (!(seen > 1.5 * (double)target)) return;
    int nz = 0;
    float ext[4], ext_max = 0.f;
    for (int gd = 0; gd < 4; gd++) {
        ext[gd] = g->ext[gd];
        if (ext[gd] > 0.f) nz++;
        ext_max = fmaxf(ext_max, ext[gd]);
    }
    if (nz == 0) return;
    double shrink = pow((double)target / seen, 1.0 / (double)nz);
    int n[4] = {1, 1, 1, 1};
    float w = g->w;
    if (pass == 0 && allow_fallback && g->gdims == 4 && shrink < 0.36) {
        g->gdims = 3;
        g->cdim[3] = -1; g->origin[3] = 0.f; g->ext[3] = 0.f;
        ext[3] = 0.f;
        double vol = 1.0;
        nz = 0; ext_max = 0.f;
        for (int gd = 0; gd < 3; gd++) {
            if (ext[gd] > 0.f) { vol *= (double)ext[gd]; nz++; }
            ext_max = fmaxf(ext_max, ext[gd]);
        }
        if (nz > 0) {
            double wd = pow(vol / (double)(bins_target3 < 1 ? 1 : bins_target3), 1.0 / (double)nz);
            if (!(wd > (double)ext_max * 1e-6)) wd = (double)ext_max * 1e-6;
            fit_shape(ext, wd, g->bins_cap, n, w);
        } else {
            w = 1.f;
        }
        const long long B3 = (long long)n[0] * n[1] * n[2];
        g->n[0] = n[0]; g->n[1] = n[1]; g->n[2] = n[2]; g->n[3] = 1;
        g->B = (int)B3;
        g->total_bins = (int)(B3 * g->n_events * g->mirror);
        grid_set_divisors(g);
        g->w = w;
        g->inv_w = __fdiv_rn(1.0f, w);
        g->slack = 4e-6f * fmaxf(ext_max, w);
        g->fallback3 = 1;
        g->refined = 1;
        g->sum_sq = 0;              // the second density pass starts from scratch
        g->stat_blocks_done = 0;
        return;
    }
    // Never more than 2.2x: data that mixes very dense clusters with a thin background
    // would otherwise pay with long walks through empty cells for the background queries.
    if (shrink < 1.0 / 2.2) shrink = 1.0 / 2.2;
    double wd = (double)g->w * shrink;
    if (!(wd > (double)ext_max * 1e-6)) wd = (double)ext_max * 1e-6;
    fit_shape(ext, wd, g->bins_cap, n, w);
    const long long B = (long long)n[0] * n[1] * n[2] * n[3];
    if (B > g->bins_cap || !(w < g->w)) return;
    g->n[0] = n[0]; g->n[1] = n[1]; g->n[2] = n[2]; g->n[3] = n[3];
    g->B = (int)B;
    g->total_bins = (int)(B * g->n_events * g->mirror);
    grid_set_divisors(g);
    g->w = w;
    g->inv_w = __fdiv_rn(1.0f, w);
    g->slack = 4e-6f * fmaxf(ext_max, w);
    g->refined = pass + 1;
}

// Cell coordinate of a shifted coordinate; identical in every kernel that needs it.
__device__ __forceinline__ int cell_of(float x, float origin, float inv_w, int n)
{
    const float t = __fsub_rn(x, origin);
    int b = (int)floorf(__fmul_rn(t, inv_w));
    b = b < 0 ? 0 : b;
    return b >= n ? n - 1 : b;
}

// Flat id of a point's cell in the first set; row: its coordinates, e: its row split.
__device__ __forceinline__ int point_cell(const KnnGrid *g, const float *__restrict__ row, int e)
{
    int b[4];
#pragma unroll
    for (int gd = 0; gd < 4; gd++) {
        const int c = g->cdim[gd];
        b[gd] = c < 0 ? 0 : cell_of(__ldg(row + c), g->origin[gd], g->inv_w, g->n[gd]);
    }
    // the fourth dimension has one cell (b[3] = 0) in a grid over three coordinates
    return e * g->B + ((b[0] * g->n[1] + b[1]) * g->n[2] + b[2]) * g->n[3] + b[3];
}

// With direction flags: one or two sets of cells, and for how many points they are sized (n_may of n_vert may be neighbours).
static __device__ void choose_sets(unsigned long long n_may, int n_vert, int adaptive, int &mirror, int &bins_target, int &bins_cap)
{
    if (8 * n_may >= 7 * (unsigned long long)n_vert) {
        // (nearly) all points: one set, which may have twice the cells
        mirror = 1;
        bins_cap *= 2;
    } else if (adaptive) {
        // cells sized for the points that are met in a walk; not below a third of the points, so that the cells of
        // the others stay small enough to be put in order
        bins_target = (int)(bins_target * fmax((double)n_may / (double)n_vert, 1.0 / 3.0) + 0.5);
    }
}

// Everything that is kept per point in cell order: original id, coordinates padded to
// float4, cell id, direction flag.
__device__ __forceinline__ void place_point(int pos, int v, int bin, const float *__restrict__ coords,
                                            int n_coords, int nv, const int64_t *__restrict__ direction,
                                            int *__restrict__ sorig, float4 *__restrict__ scoords,
                                            int *__restrict__ sbin, uint8_t *__restrict__ sflag)
{
    const float *row = coords + (size_t)v * n_coords;
    for (int q = 0; q < nv; q++) {
        float4 o;
        o.x = 4 * q + 0 < n_coords ? __ldg(row + 4 * q + 0) : 0.f;
        o.y = 4 * q + 1 < n_coords ? __ldg(row + 4 * q + 1) : 0.f;
        o.z = 4 * q + 2 < n_coords ? __ldg(row + 4 * q + 2) : 0.f;
        o.w = 4 * q + 3 < n_coords ? __ldg(row + 4 * q + 3) : 0.f;
        scoords[(size_t)pos * nv + q] = o;
    }
    sorig[pos] = v;
    sbin[pos] = bin;
    if (direction) {
        const int64_t d = direction[v];
        sflag[pos] = (d >= 0 && d <= 2) ? (uint8_t)d : (uint8_t)3;
    }
}

constexpr int kSortWarps = 16;
constexpr int kSortShared = kSortWarps * kWarpSortMaxShared * (int)sizeof(int);       // of the warps
constexpr int kSortMostBits = 96 * 1024 * 8;

// The ids of a cell beyond kWarpSortMaxShared points from stmp to sorig, in ascending order, by a CTA of kSortWarps warps.  They are different numbers of one
// row split: a bit for each in shared memory (n_words words), and the place of an id is the number of bits before it -- three passes over
// the cell whatever its size, where a sorting network in global memory took hundreds (a second look at 800 k skewed points whose
// largest cell holds some 50 k: 1.36 -> 0.1 ms).  Ids that span more than the bits go through them a window at a time.
__device__ __forceinline__ void sort_cell_by_cta(int beg, int n, const int *stmp, int *sorig, int *s_bits, int n_words, int *status)
{
    __shared__ int s_part[kSortWarps], s_low, s_high;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (threadIdx.x == 0) { s_low = 0x7fffffff; s_high = 0; }
    __syncthreads();
    int low = 0x7fffffff, high = 0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const int v = stmp[beg + t];
        low = min(low, v);
        high = max(high, v);
    }
    low = __reduce_min_sync(FGC_FULL_MASK, low);
    high = __reduce_max_sync(FGC_FULL_MASK, high);
    if (lane == 0) { atomicMin(&s_low, low); atomicMax(&s_high, high); }
    __syncthreads();
    low = s_low;
    high = s_high;
    int done = 0;                                          // ids of earlier windows
    for (long long first = low; first <= high; first += 32ll * n_words) {
        const int words = (int)min((long long)n_words, (high - first) / 32 + 1);
        for (int i = threadIdx.x; i < words; i += blockDim.x) s_bits[i] = 0;
        __syncthreads();
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const long long off = (long long)stmp[beg + t] - first;
            if (off >= 0 && off < 32ll * words) atomicOr(s_bits + (int)(off >> 5), 1 << (int)(off & 31));
        }
        __syncthreads();
        // a run of words per thread, an exclusive scan of their counts, then the ids of the run in order
        const int run = (words + (int)blockDim.x - 1) / (int)blockDim.x;
        const int i0 = min(words, (int)threadIdx.x * run), i1 = min(words, i0 + run);
        int count = 0;
        for (int i = i0; i < i1; i++) count += __popc(s_bits[i]);
        int before = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(FGC_FULL_MASK, before, o);
            if (lane >= o) before += x;
        }
        if (lane == 31) s_part[wib] = before;
        before -= count;
        __syncthreads();
        int total = 0;
#pragma unroll
        for (int k = 0; k < kSortWarps; k++) {
            if (k == wib) before += total;
            total += s_part[k];
        }
        int at = done + before;
        for (int i = i0; i < i1; i++) {
            for (uint32_t bits = (uint32_t)s_bits[i]; bits; bits &= bits - 1, at++) {
                if (FGC_DBG_OK(at >= 0 && at < n, status)) sorig[beg + at] = (int)(first + 32ll * i + __ffs(bits) - 1);
            }
        }
        done += total;
        __syncthreads();
    }
}

// The two words for the host: in one store where they lie so, since the host may be looking for them.
__device__ __forceinline__ void store_info(volatile int32_t *info_mapped, int32_t status, int32_t form)
{
    if (((uintptr_t)info_mapped & 7) == 0) {
        *(volatile int64_t *)info_mapped = (int64_t)(uint32_t)status | (int64_t)form << 32;
    } else {
        info_mapped[0] = status;
        info_mapped[1] = form;
    }
}

// What a build on the device needs to know.
struct GridBuild {
    const float *coords;
    const int64_t *row_splits, *direction;
    KnnGrid *grid;
    int *counts, *stmp, *sorig, *sbin, *biglist, *hugelist;
    uint8_t *sflag;
    float4 *scoords;
    int n_vert, n_coords, nv, n_rs, n_bin_dims, mirror;
    int bins_target, bins_cap_first, bins_cap;
    int adaptive, allow_fallback;
    float seen_target, seen_target3;
    int *out_order;                        // original ids in cell order, or null
    volatile int32_t *info_mapped;         // two words that the host reads (fgc_knn_publish_grid_info), or null
};

// Up to so many points the grid is built by one launch.  Forward, K = 16 in three coordinates, chain / one launch, us: uniform points, 1000
// 131 / 65, 10 k 119 / 78, 16 k 121 / 90, 32 k 137 / 126; with sparse tails 10 k in ten row splits 117 / 113, 16 k 186 / 194, 32 k 202 / 230 (its
// crowded cells are put in order by eight SMs).
constexpr int64_t kSmallBuild = 16384;
cudaError_t launch_small_build(const GridBuild &b, cudaStream_t s);

}  // namespace fgc
