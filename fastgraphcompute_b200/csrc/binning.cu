// bin_by_coordinates for sm_100a: fused finite/min/max pass, device-side
// derivation of the binning parameters, per-point bin assignment with a
// warp-aggregated histogram.
//
// Semantics follow the reference's CPU implementation bit for bit:
//   host derivation  extensions/bin_by_coordinates.cpp:51-120
//   per-point kernel extensions/bin_by_coordinates_cpu.cpp:7-99
// All float steps use explicit round-to-nearest intrinsics (no contraction, no
// fast division) so that bin indices agree with the x86-64 build.
#include "fgc_common.cuh"

namespace fgc {

constexpr int kReduceThreads = 256;

// One thread: the D-element derivation of shift, dmax, n_bins and bin_width from a copy of the scratch words.
__device__ void bin_derive(fgc_bin_params *prm, const uint32_t *found, int64_t n_vert, int n_coords, int pre_normalized,
                           const float *__restrict__ bin_width_in, const int64_t *__restrict__ n_bins_in,
                           int n_bins_len)
{
    int status = 0;
    if (found[2 * FGC_MAX_BIN_DIMS]) status |= FGC_STATUS_NONFINITE;
    float bw_max = -INFINITY;
    const bool have_bw = bin_width_in != nullptr;
    const bool have_nb = n_bins_in != nullptr;
    for (int c = 0; c < FGC_MAX_BIN_DIMS; c++) { prm->shift[c] = 0.f; prm->n_bins[c] = 1; }
    for (int c = 0; c < n_coords; c++) {
        float lo = n_vert > 0 ? ordered_to_float(~found[c]) : 0.f;
        float hi = n_vert > 0 ? ordered_to_float(found[FGC_MAX_BIN_DIMS + c]) : 0.f;
        float shift = 0.f;
        if (!pre_normalized) {
            shift = lo;
            hi = __fsub_rn(hi, lo);  // max of the shifted column (x - lo is monotone in x)
            lo = __fsub_rn(lo, lo);
        }
        prm->shift[c] = shift;
        float dmax = hi;
        if (lo == hi) dmax = __fadd_rn(dmax, 1.0f);
        dmax = __fadd_rn(dmax, (float)1e-3);
        if (!is_finite_bits(dmax)) dmax = 1.0f;
        if (!(dmax > 0.f)) status |= FGC_STATUS_BAD_DMAX;
        if (have_bw) {
            if (have_nb)
                prm->n_bins[c] = n_bins_in[n_bins_len == 1 ? 0 : c];
            else
                prm->n_bins[c] = (int64_t)__fdiv_rn(dmax, bin_width_in[0]) + 1;
        } else {
            const int64_t nb = n_bins_in[n_bins_len == 1 ? 0 : c];
            prm->n_bins[c] = nb;
            const float bw = __fdiv_rn(dmax, (float)nb);
            if (bw > bw_max) bw_max = bw;
        }
    }
    const float bw = have_bw ? bin_width_in[0] : bw_max;
    prm->bin_width = bw;
    for (int c = 0; c < n_coords; c++)
        if (!(prm->n_bins[c] > 0)) status |= FGC_STATUS_BAD_NBINS;
    if (!(bw > 0.f)) status |= FGC_STATUS_BAD_BINWIDTH;
    prm->n_coords = n_coords;
    prm->status = status;
}

// scratch layout inside fgc_bin_params: [0..7] ~ordered(min), [8..15] ordered(max),
// [16] non-finite flag, [17] CTAs that are done.  All start at zero, so one memset initialises them and
// both extremes are maintained with atomicMax.
//
// Flat pass over the array: the stride is a multiple of n_coords, so that a thread stays in its columns
// and needs neither a division nor the extremes of the others.  WIDE: 16 bytes a load, four columns a thread (an aligned array); the
// few round trips that a thread waits for bound it (3 M points in four dimensions 45.7 -> 17.7 us, 1 M 12.3 -> 10.2; 5000 in three, where the
// derivation by the last CTA is most of it, 5.3 -> 4.5 since its words are read at once).
template <bool WIDE>
__global__ void __launch_bounds__(kReduceThreads)
k_bin_minmax(const float *__restrict__ coords, int64_t n_vert, int n_coords, int pre_normalized,
             const float *__restrict__ bin_width_in, const int64_t *__restrict__ n_bins_in, int n_bins_len,
             fgc_bin_params *prm)
{
    constexpr int PER = WIDE ? 4 : 1;
    __shared__ uint32_t s_min[FGC_MAX_BIN_DIMS], s_max[FGC_MAX_BIN_DIMS], s_bad;
    if (threadIdx.x < FGC_MAX_BIN_DIMS) { s_min[threadIdx.x] = 0; s_max[threadIdx.x] = 0; }
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    const int64_t total = n_vert * (int64_t)n_coords;
    const int64_t all = (int64_t)gridDim.x * blockDim.x;
    const int64_t stride = all - all % n_coords;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t bad = 0, lmin[PER], lmax[PER];
#pragma unroll
    for (int k = 0; k < PER; k++) lmin[k] = lmax[k] = 0;
    auto take = [&](float v, int k) {
        if (!is_finite_bits(v)) bad = 1;
        const uint32_t key = float_to_ordered(v);
        lmin[k] = max(lmin[k], ~key);
        lmax[k] = max(lmax[k], key);
    };
    if (tid < stride) {
#pragma unroll 4
        for (int64_t e = tid; e < total / PER; e += stride) {
            if constexpr (WIDE) {
                const float4 v = __ldg((const float4 *)coords + e);
                take(v.x, 0); take(v.y, 1); take(v.z, 2); take(v.w, 3);
            } else {
                take(__ldg(coords + e), 0);
            }
        }
        // up to three numbers behind the last four
        if (WIDE && tid == total / PER % stride)
            for (int k = 0; k < (int)(total % PER); k++) {
                const float v = __ldg(coords + total / PER * PER + k);
                if (k == 0) take(v, 0);
                else if (k == 1) take(v, 1 % PER);
                else take(v, 2 % PER);
            }
    }
    const int first = (int)(tid * PER % n_coords);
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int c = (first + k) % n_coords;
        if (PER % n_coords == 0) {                            // one column for all lanes
            lmin[k] = __reduce_max_sync(FGC_FULL_MASK, lmin[k]);
            lmax[k] = __reduce_max_sync(FGC_FULL_MASK, lmax[k]);
            if ((threadIdx.x & 31) == 0) { atomicMax(&s_min[c], lmin[k]); atomicMax(&s_max[c], lmax[k]); }
        } else if (lmax[k] | lmin[k]) {
            atomicMax(&s_min[c], lmin[k]);
            atomicMax(&s_max[c], lmax[k]);
        }
    }
    if (bad) s_bad = 1u;
    __syncthreads();
    if (threadIdx.x < n_coords) {
        atomicMax(&prm->scratch[threadIdx.x], s_min[threadIdx.x]);
        atomicMax(&prm->scratch[FGC_MAX_BIN_DIMS + threadIdx.x], s_max[threadIdx.x]);
    }
    if (threadIdx.x == 0 && s_bad) atomicOr(&prm->scratch[2 * FGC_MAX_BIN_DIMS], 1u);
    __threadfence();
    __syncthreads();
    if (threadIdx.x >= 32) return;
    int last = 0;
    if (threadIdx.x == 0) last = atomicAdd(&prm->scratch[2 * FGC_MAX_BIN_DIMS + 1], 1u) == gridDim.x - 1;
    if (!__shfl_sync(FGC_FULL_MASK, last, 0)) return;
    __threadfence();
    __shared__ uint32_t s_found[2 * FGC_MAX_BIN_DIMS + 1];
    if (threadIdx.x <= 2 * FGC_MAX_BIN_DIMS) s_found[threadIdx.x] = __ldcg(&prm->scratch[threadIdx.x]);
    __syncwarp();
    if (threadIdx.x == 0)
        bin_derive(prm, s_found, n_vert, n_coords, pre_normalized, bin_width_in, n_bins_in, n_bins_len);
}

// kBinPoints points per thread (one after the other where indexes have 64 bits).  Every output is written, so none has to be cleared first; the rows of the bin
// indices go through shared memory and leave in one contiguous run per CTA.  A point whose flat bin lies beyond the table
// (malformed row splits) gets zeros and is not counted.  Tables whose indexes have 32 bits (whatever their row split) are
// counted in 32 bits, a warp's row splits are found by one vote where there are at most 32 (an event's end among its points: a
// search).  Conversions to 64 bits, matches of 64-bit indexes and the rows of 64 bits in shared memory bounded it (issue slots 0.39, most
// of the stalls on them): 1 M points in four dimensions 25.4 -> 17.0 us (without the table 13.7 -> 11.4), 3 M 82.0 -> 69.5; one point
// per thread 17.9.  With the table its atomics bound it (1 M normal points in three dimensions 10.1 us without, 29.2 with it).
constexpr int kBinPoints = 2;

template <int D, int PTS, typename INT>
__device__ __forceinline__ void bin_assign(const float *__restrict__ coords, int64_t n_vert, int64_t first,
                                           const int64_t *__restrict__ row_splits, int n_rs, bool vote, int64_t split_end,
                                           const fgc_bin_params *__restrict__ prm, const int64_t (&nb)[D], int calc_n_per_bin, int64_t n_total_bins,
                                           int64_t *__restrict__ out_bin_idx, int64_t *__restrict__ out_flat,
                                           unsigned long long *__restrict__ out_n_per_bin, INT *s_row)
{
    constexpr int ROW = D + 1, PITCH = ROW | 1;          // odd pitch: threads in different banks
    const int lane = threadIdx.x & 31;
    const float bw = prm->bin_width;
    float x[PTS][D];
#pragma unroll
    for (int r = 0; r < PTS; r++) {
        const int64_t v = first + r * 256 + threadIdx.x;
        if (v >= n_vert) continue;
#pragma unroll
        for (int c = 0; c < D; c++) x[r][c] = __ldg(coords + v * D + c);
    }
    INT flat[PTS];
    bool counts[PTS];
#pragma unroll
    for (int r = 0; r < PTS; r++) {
        const int64_t v = first + r * 256 + threadIdx.x;
        counts[r] = false;
        // splits that end at or before the warp's first point, and whether one ends before this point
        int rs = __popc(__ballot_sync(FGC_FULL_MASK, split_end <= v - lane));
        const int64_t end = __shfl_sync(FGC_FULL_MASK, split_end, rs & 31);
        if (v >= n_vert) continue;
        if (!vote || (rs < 32 && v >= end)) rs = row_split_of(row_splits, n_rs, v);
        INT stride = 1, f = 0, cidx[D];
#pragma unroll
        for (int c = D - 1; c >= 0; c--) {
            const float q = __fadd_rn(__fdiv_rn(__fsub_rn(x[r][c], prm->shift[c]), bw), 1e-3f);
            const INT n = (INT)nb[c];
            INT b;
            if constexpr (sizeof(INT) == 4) {
                const int at = __float2int_rd(q);         // saturates; (not a number: 0)
                b = (INT)max(at, 0);
                if (b >= n) b = n - 1;
            } else {
                b = (INT)floorf(q);
                if (b < 0) b = 0;
                else if (b >= n) b = n - 1;
            }
            cidx[c] = b;
            f += b * stride;
            stride *= n;
        }
        f += (INT)rs * stride;
        counts[r] = sizeof(INT) == 4 ? (int64_t)f < n_total_bins : f < (INT)n_total_bins && f >= 0;
        flat[r] = counts[r] ? f : 0;
        INT *row = s_row + (r * 256 + threadIdx.x) * PITCH;
        row[0] = counts[r] ? (INT)rs : 0;
#pragma unroll
        for (int c = 0; c < D; c++) row[c + 1] = counts[r] ? cidx[c] : 0;
        out_flat[v] = (int64_t)flat[r];
    }
    __syncthreads();
    const int n_here = (int)max((int64_t)0, n_vert - first < 256 * PTS ? n_vert - first : 256 * PTS) * ROW;
    int64_t *out = out_bin_idx + first * ROW;
#pragma unroll 4
    for (int i = threadIdx.x; i < n_here; i += 256) out[i] = (int64_t)s_row[PITCH == ROW ? i : (i / ROW) * PITCH + i % ROW];
    if (!calc_n_per_bin) return;
#pragma unroll
    for (int r = 0; r < PTS; r++) {
        // warp-aggregated histogram: one atomic per distinct bin per warp
        const unsigned active = __ballot_sync(FGC_FULL_MASK, counts[r]);
        if (counts[r]) {
            const unsigned peers = __match_any_sync(active, flat[r]);
            if ((peers & lanemask_lt()) == 0) atomicAdd(out_n_per_bin + flat[r], (unsigned long long)__popc(peers));
        }
    }
}

template <int D>
__global__ void __launch_bounds__(256)
k_bin_assign(const float *__restrict__ coords, int64_t n_vert, const int64_t *__restrict__ row_splits, int n_rs,
             const fgc_bin_params *__restrict__ prm, int calc_n_per_bin, int64_t n_total_bins,
             int64_t *__restrict__ out_bin_idx, int64_t *__restrict__ out_flat,
             unsigned long long *__restrict__ out_n_per_bin)
{
    static_assert(kBinPoints <= 2, "rows of 32 bits take as much room as 256 of 64");
    __shared__ int64_t s_row[256 * ((D + 1) | 1)];
    int64_t nb[D], table = 1;
    bool narrow = true;
#pragma unroll
    for (int c = 0; c < D; c++) {
        nb[c] = prm->n_bins[c];
        narrow = narrow && nb[c] > 0 && nb[c] < 0x7fffffff && table <= 0xffffffff;
        table *= narrow ? nb[c] : 1;
    }
    narrow = narrow && table <= 0xffffffff / (uint32_t)n_rs;
    // a warp's vote needs row splits that never decrease
    const int lane = threadIdx.x & 31;
    const int64_t split_end = n_rs <= 33 && 1 + lane < n_rs ? row_splits[1 + lane] : INT64_MAX;
    const int64_t next_end = __shfl_down_sync(FGC_FULL_MASK, split_end, 1);             // (lane 31: its own)
    const bool ascend = __all_sync(FGC_FULL_MASK, split_end <= next_end), vote = n_rs <= 33 && ascend;
    const int64_t first = (int64_t)blockIdx.x * (256 * kBinPoints);
    if (narrow) {
        bin_assign<D, kBinPoints, uint32_t>(coords, n_vert, first, row_splits, n_rs, vote, split_end, prm, nb, calc_n_per_bin, n_total_bins,
                                            out_bin_idx, out_flat, out_n_per_bin, (uint32_t *)s_row);
    } else {
        for (int r = 0; r < kBinPoints; r++) {
            bin_assign<D, 1, int64_t>(coords, n_vert, first + r * 256, row_splits, n_rs, vote, split_end, prm, nb, calc_n_per_bin,
                                      n_total_bins, out_bin_idx, out_flat, out_n_per_bin, s_row);
            __syncthreads();
        }
    }
}

}  // namespace fgc

extern "C" int fgc_bin_prepare(const float *coords, int64_t n_vert, int32_t n_coords,
                               int32_t pre_normalized, const float *bin_width_or_null,
                               const int64_t *n_bins_or_null, int32_t n_bins_len,
                               fgc_bin_params *out_params, fgc_stream_t stream)
{
    FGC_NVTX("fgc_bin_prepare");
    if (!out_params || n_vert < 0 || n_coords < 1 || n_coords > FGC_MAX_BIN_DIMS)
        return FGC_ERR_BAD_ARGUMENT;
    if (n_vert > 0 && !coords) return FGC_ERR_BAD_ARGUMENT;
    if (!bin_width_or_null && !n_bins_or_null) return FGC_ERR_BAD_ARGUMENT;
    if (n_bins_or_null && n_bins_len != 1 && n_bins_len != n_coords) return FGC_ERR_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    FGC_RETURN_IF_CUDA(cudaMemsetAsync(out_params, 0, sizeof(fgc_bin_params), s));
    const int64_t total = n_vert * n_coords;
    int blocks = (int)(fgc::ceil_div64(total, (int64_t)fgc::kReduceThreads * 8) < fgc::sm_count() * 8
                           ? fgc::ceil_div64(total, (int64_t)fgc::kReduceThreads * 8) : fgc::sm_count() * 8);
    if (blocks < 1) blocks = 1;
    if (((uintptr_t)coords & 15) == 0)
        fgc::k_bin_minmax<true><<<blocks, fgc::kReduceThreads, 0, s>>>(coords, n_vert, n_coords, pre_normalized, bin_width_or_null,
                                                                       n_bins_or_null, n_bins_len, out_params);
    else
        fgc::k_bin_minmax<false><<<blocks, fgc::kReduceThreads, 0, s>>>(coords, n_vert, n_coords, pre_normalized, bin_width_or_null,
                                                                        n_bins_or_null, n_bins_len, out_params);
    FGC_CHECK_LAUNCH();
    return FGC_OK;
}

extern "C" int fgc_bin_assign(const float *coords, int64_t n_vert, int32_t n_coords,
                              const int64_t *row_splits, int64_t n_rs,
                              const fgc_bin_params *params, int32_t calc_n_per_bin,
                              int64_t n_total_bins, int64_t *out_bin_idx, int64_t *out_flat,
                              int64_t *out_n_per_bin, fgc_stream_t stream)
{
    FGC_NVTX("fgc_bin_assign");
    if (!params || n_vert < 0 || n_coords < 1 || n_coords > FGC_MAX_BIN_DIMS || n_rs < 1 ||
        n_rs > 0x7fffffff || !row_splits)
        return FGC_ERR_BAD_ARGUMENT;
    if (n_vert == 0) return FGC_OK;
    if (!coords || !out_bin_idx || !out_flat || (calc_n_per_bin && !out_n_per_bin))
        return FGC_ERR_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    if (fgc::ceil_div64(n_vert, 256) > 0x7fffffff) return FGC_ERR_TOO_LARGE;
    const int64_t blocks = fgc::ceil_div64(n_vert, 256 * fgc::kBinPoints);
#define FGC_BIN_ASSIGN(D)                                                                                   \
    case D:                                                                                                 \
        fgc::k_bin_assign<D><<<(unsigned)blocks, 256, 0, s>>>(coords, n_vert, row_splits, (int)n_rs, params, \
                                                              calc_n_per_bin, n_total_bins, out_bin_idx, out_flat, \
                                                              (unsigned long long *)out_n_per_bin);          \
        break
    switch (n_coords) {
        FGC_BIN_ASSIGN(1);
        FGC_BIN_ASSIGN(2);
        FGC_BIN_ASSIGN(3);
        FGC_BIN_ASSIGN(4);
        FGC_BIN_ASSIGN(5);
        FGC_BIN_ASSIGN(6);
        FGC_BIN_ASSIGN(7);
        FGC_BIN_ASSIGN(8);
    }
#undef FGC_BIN_ASSIGN
    FGC_CHECK_LAUNCH();
    return FGC_OK;
}
