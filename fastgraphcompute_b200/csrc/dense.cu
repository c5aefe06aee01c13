// Dense layers around the message passing for sm_100a: bias and ReLU of a layer's output in one pass,
// and the backward of bias, weight and ReLU in one pass over the incoming gradient.
//
// The products with the weight matrix itself (forward and input gradient) stay with the library GEMMs.
// The weight gradient dW[o, c] = sum over rows of dY[row, o] * x[row, c] is the shape a general GEMM
// is worst at -- hundreds of thousands of rows summed into a 128 x 128 result -- and the ReLU mask and the
// bias gradient read the same dY again:
//
//   k_dense_bwd     a CTA owns one tile of dW (up to 128 x 128) and a range of rows.  Rows are natural
//                   outer-product operands (both sides are contiguous in a row), so tiles go to shared
//                   memory as they are, 16 rows at a time, double-buffered through registers; on the way dY is
//                   masked by the layer's output, written out for the input-gradient GEMM and summed
//                   for the bias.  Scalar fp32 multiply-adds, 8 x 8 per thread.
//   k_dense_reduce  adds the CTAs' partial results in a fixed order: the result is the same on
//                   every run.
//
// Bound by latency between the fp32 multiply-adds: two CTAs of eight warps on an SM fill 0.56 of the issue slots, 400 k rows,
// 128 to 128, 0.46 ms, i.e. 28 of 72 TFLOP/s and 1.7 TB/s.  Forward and backward of one layer with ReLU,
// library only -> with these kernels (B200, ms): 200 k rows, 128 to 128: 1.02 -> 0.64; 64 to 128: 0.88 ->
// 0.44; 128 to 10: 0.385 -> 0.281; 800 k rows, 128 to 64: 1.70 -> 1.20; where they lose (launches, narrow and wide
// weights) the caller keeps the modules.  Relative error of dW against 64 bits at 200 k rows,
// 128 to 128: 1.1e-6 (library) -> 3.5e-7.
#include "fgc_common.cuh"

namespace fgc {

constexpr int kDenseThreads = 256;
constexpr int kDenseRows = 16;       // rows per step

// y = act(y + b), in place.  VEC: four columns at a time (n_out % 4 == 0, 16-byte aligned).
template <bool VEC>
__global__ void __launch_bounds__(256)
k_bias_act(float *__restrict__ y, const float *__restrict__ b, long long n_rows, int n_out, int relu)
{
    constexpr int V = VEC ? 4 : 1;
    const int cols = n_out / V;
    const long long total = n_rows * cols;
    const long long step = (long long)gridDim.x * blockDim.x;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int c = (int)(i % cols);
    const int dc = (int)(step % cols);
    for (; i < total; i += step) {
        if constexpr (VEC) {
            float4 v = ((float4 *)y)[i];
            const float4 w = __ldg((const float4 *)b + c);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
            // (NaN stays NaN, as in torch.relu)
            if (relu) { v.x = v.x < 0.f ? 0.f : v.x; v.y = v.y < 0.f ? 0.f : v.y; v.z = v.z < 0.f ? 0.f : v.z; v.w = v.w < 0.f ? 0.f : v.w; }
            ((float4 *)y)[i] = v;
        } else {
            const float v = y[i] + __ldg(b + c);
            y[i] = relu && v < 0.f ? 0.f : v;
        }
        c += dc;
        if (c >= cols) c -= cols;
    }
}

// Four consecutive columns of a row, zero beyond the matrix.
template <bool VEC>
__device__ __forceinline__ float4 dense_load4(const float *__restrict__ m, long long row, long long row_end, int col, int n_cols)
{
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < row_end && col < n_cols) {
        const float *p = m + (size_t)row * n_cols + col;
        if constexpr (VEC) v = __ldg((const float4 *)p);
        else {
            v.x = __ldg(p);
            if (col + 1 < n_cols) v.y = __ldg(p + 1);
            if (col + 2 < n_cols) v.z = __ldg(p + 2);
            if (col + 3 < n_cols) v.w = __ldg(p + 3);
        }
    }
    return v;
}

// BO x BC: tile of dW.  Thread (ty, tx) owns outputs 4 ty + 64 k + {0..3} and inputs 4 tx + 64 j + {0..3}.
template <int BO, int BC, bool VEC>
__global__ void __launch_bounds__(kDenseThreads, 2)
k_dense_bwd(const float *__restrict__ x, const float *__restrict__ dy, const float *__restrict__ y, long long n_rows,
            int n_in, int n_out, long long rows_per_cta, float *__restrict__ dy_masked, float *__restrict__ part_w,
            float *__restrict__ part_b)
{
    constexpr int MO = BO / 16, MC = BC / 16;
    constexpr int LO = kDenseRows * BO / 4 / kDenseThreads, LC = kDenseRows * BC / 4 / kDenseThreads;   // float4 loads per thread
    __shared__ float4 s_y[2][kDenseRows][BO / 4];
    __shared__ float4 s_x[2][kDenseRows][BC / 4];
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const int o0 = blockIdx.z * BO, c0 = blockIdx.y * BC;
    const long long first = (long long)blockIdx.x * rows_per_cta;
    const long long last = min(n_rows, first + rows_per_cta);
    const int oc = (t % (BO / 4)) * 4, orow = t / (BO / 4);
    const int xc = (t % (BC / 4)) * 4, xrow = t / (BC / 4);
    const bool owner = blockIdx.y == 0;          // of the mask and the bias sum
    float acc[MO][MC];
#pragma unroll
    for (int i = 0; i < MO; i++)
#pragma unroll
        for (int j = 0; j < MC; j++) acc[i][j] = 0.f;
    // two levels, so that a thread never adds thousands of rows one to another
    float4 bsum = make_float4(0.f, 0.f, 0.f, 0.f), btotal = bsum;
    auto fold = [&]() {
        btotal.x += bsum.x; btotal.y += bsum.y; btotal.z += bsum.z; btotal.w += bsum.w;
        bsum = make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float4 ry[LO], rx[LC];
    auto fetch = [&](long long row0) {
#pragma unroll
        for (int k = 0; k < LO; k++) {
            const long long row = row0 + orow + k * (kDenseThreads / (BO / 4));
            ry[k] = dense_load4<VEC>(dy, row, last, o0 + oc, n_out);
            if (y) {
                const float4 a = dense_load4<VEC>(y, row, last, o0 + oc, n_out);
                // the gradient passes unless the output is at or below zero (a NaN lets it pass, as in torch)
                if (a.x <= 0.f) ry[k].x = 0.f;
                if (a.y <= 0.f) ry[k].y = 0.f;
                if (a.z <= 0.f) ry[k].z = 0.f;
                if (a.w <= 0.f) ry[k].w = 0.f;
                if (owner && dy_masked && row < last && o0 + oc < n_out) {
                    float *p = dy_masked + (size_t)row * n_out + o0 + oc;
                    if constexpr (VEC) *(float4 *)p = ry[k];
                    else {
                        const int left = n_out - o0 - oc;
                        p[0] = ry[k].x;
                        if (left > 1) p[1] = ry[k].y;
                        if (left > 2) p[2] = ry[k].z;
                        if (left > 3) p[3] = ry[k].w;
                    }
                }
            }
            bsum.x += ry[k].x; bsum.y += ry[k].y; bsum.z += ry[k].z; bsum.w += ry[k].w;
        }
#pragma unroll
        for (int k = 0; k < LC; k++)
            rx[k] = dense_load4<VEC>(x, row0 + xrow + k * (kDenseThreads / (BC / 4)), last, c0 + xc, n_in);
    };
    auto stage = [&](int b) {
#pragma unroll
        for (int k = 0; k < LO; k++) s_y[b][orow + k * (kDenseThreads / (BO / 4))][oc >> 2] = ry[k];
#pragma unroll
        for (int k = 0; k < LC; k++) s_x[b][xrow + k * (kDenseThreads / (BC / 4))][xc >> 2] = rx[k];
    };
    int b = 0, steps = 0;
    if (first < last) {
        fetch(first);
        stage(0);
    }
    __syncthreads();
    for (long long row0 = first; row0 < last; row0 += kDenseRows) {
        const bool more = row0 + kDenseRows < last;
        if ((++steps & 15) == 0) fold();
        if (more) fetch(row0 + kDenseRows);
#pragma unroll
        for (int r = 0; r < kDenseRows; r++) {
            float a[MO], v[MC];
#pragma unroll
            for (int k = 0; k < MO / 4; k++) {
                const float4 f = s_y[b][r][ty + 16 * k];
                a[4 * k] = f.x; a[4 * k + 1] = f.y; a[4 * k + 2] = f.z; a[4 * k + 3] = f.w;
            }
#pragma unroll
            for (int k = 0; k < MC / 4; k++) {
                const float4 f = s_x[b][r][tx + 16 * k];
                v[4 * k] = f.x; v[4 * k + 1] = f.y; v[4 * k + 2] = f.z; v[4 * k + 3] = f.w;
            }
#pragma unroll
            for (int i = 0; i < MO; i++)
#pragma unroll
                for (int j = 0; j < MC; j++) acc[i][j] = fmaf(a[i], v[j], acc[i][j]);
        }
        if (more) stage(b ^ 1);
        b ^= 1;
        __syncthreads();
    }
    float *pw = part_w + (size_t)blockIdx.x * n_out * n_in;
#pragma unroll
    for (int i = 0; i < MO; i++) {
        const int o = o0 + 4 * ty + 64 * (i >> 2) + (i & 3);
#pragma unroll
        for (int j = 0; j < MC; j++) {
            const int c = c0 + 4 * tx + 64 * (j >> 2) + (j & 3);
            if (o < n_out && c < n_in) pw[(size_t)o * n_in + c] = acc[i][j];
        }
    }
    if (owner) {
        // threads that loaded the same four columns, added in a fixed order
        float4 *sb = &s_x[0][0][0];
        fold();
        sb[t] = btotal;
        __syncthreads();
        if (t < BO) {
            float s = 0.f;
            for (int k = 0; k < kDenseThreads / (BO / 4); k++) s += ((const float *)(sb + k * (BO / 4) + (t >> 2)))[t & 3];
            if (o0 + t < n_out) part_b[(size_t)blockIdx.x * n_out + o0 + t] = s;
        }
    }
}

// out[i] = sum over the parts of part[p][i]: 32 entries per CTA, eight threads each, every thread an
// interleaved eighth of the parts.  Entries 0..n_w-1 are the weight's, the others the bias'.
__global__ void __launch_bounds__(256)
k_dense_reduce(const float *__restrict__ part_w, const float *__restrict__ part_b, int n_parts, long long n_w, int n_b,
               float *__restrict__ dw, float *__restrict__ db)
{
    __shared__ float s[8][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const long long i = (long long)blockIdx.x * 32 + lane;
    const bool is_w = i < n_w;
    const float *p = is_w ? part_w + i : part_b + (i - n_w);
    const size_t ld = is_w ? (size_t)n_w : (size_t)n_b;
    float v = 0.f;
    if (i < n_w + n_b) {
#pragma unroll 4
        for (int k = g; k < n_parts; k += 8) v += __ldg(p + (size_t)k * ld);
    }
    s[g][lane] = v;
    __syncthreads();
    if (g == 0 && i < n_w + n_b) {
        float sum = s[0][lane];
#pragma unroll
        for (int k = 1; k < 8; k++) sum += s[k][lane];
        if (is_w) dw[i] = sum; else db[i - n_w] = sum;
    }
}

struct DenseSplit {
    int bo, bc, tiles_o, tiles_c, parts;
    long long rows;
};

// Tiles of 64 or 128 per dimension, whichever covers it with less padding; as many row ranges as keep
// two CTAs on every SM, but at least 64 rows each.
static DenseSplit dense_split(int64_t n_rows, int n_in, int n_out)
{
    DenseSplit d;
    d.bo = n_out <= 64 ? 64 : 128;
    d.bc = n_in <= 64 || (n_in > 128 && n_in <= 192) ? 64 : 128;
    d.tiles_o = (n_out + d.bo - 1) / d.bo;
    d.tiles_c = (n_in + d.bc - 1) / d.bc;
    const int64_t tiles = (int64_t)d.tiles_o * d.tiles_c;
    int64_t parts = 296 / tiles;
    if (parts < 1) parts = 1;
    const int64_t most = (n_rows + 63) / 64;
    if (parts > most) parts = most < 1 ? 1 : most;
    d.rows = ((n_rows + parts - 1) / parts + kDenseRows - 1) / kDenseRows * kDenseRows;
    d.parts = d.rows > 0 ? (int)((n_rows + d.rows - 1) / d.rows) : 0;
    if (d.parts < 1) d.parts = 1;
    return d;
}

static bool dense_args_ok(int64_t n_rows, int32_t n_in, int32_t n_out)
{
    return n_rows >= 0 && n_in >= 1 && n_out >= 1 && n_in <= 65535 && n_out <= 65535;
}

template <int BO, int BC>
static void launch_dense_bwd(const DenseSplit &d, bool vec, cudaStream_t s, const float *x, const float *dy, const float *y,
                             int64_t n_rows, int n_in, int n_out, float *dy_masked, float *part_w, float *part_b)
{
    const dim3 grid((unsigned)d.parts, (unsigned)d.tiles_c, (unsigned)d.tiles_o);
    if (vec) k_dense_bwd<BO, BC, true><<<grid, kDenseThreads, 0, s>>>(x, dy, y, n_rows, n_in, n_out, d.rows, dy_masked, part_w, part_b);
    else k_dense_bwd<BO, BC, false><<<grid, kDenseThreads, 0, s>>>(x, dy, y, n_rows, n_in, n_out, d.rows, dy_masked, part_w, part_b);
}

}  // namespace fgc

extern "C" int fgc_bias_act(float *y, const float *bias, int64_t n_rows, int32_t n_out, int32_t relu, fgc_stream_t stream)
{
    FGC_NVTX("fgc_bias_act");
    using namespace fgc;
    if (n_rows < 0 || n_out < 1) return FGC_ERR_BAD_ARGUMENT;
    if (n_rows == 0) return FGC_OK;
    if (!y || !bias) return FGC_ERR_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    const bool vec = n_out % 4 == 0 && (((uintptr_t)y | (uintptr_t)bias) & 15) == 0;
    const int64_t items = n_rows * (vec ? n_out / 4 : n_out);
    int64_t blocks = (items + 255) / 256;
    if (blocks > sm_count() * 16) blocks = sm_count() * 16;
    if (vec) k_bias_act<true><<<(unsigned)blocks, 256, 0, s>>>(y, bias, n_rows, n_out, relu);
    else k_bias_act<false><<<(unsigned)blocks, 256, 0, s>>>(y, bias, n_rows, n_out, relu);
    return (int)cudaGetLastError();
}

extern "C" size_t fgc_dense_backward_bytes(int64_t n_rows, int32_t n_in, int32_t n_out)
{
    using namespace fgc;
    if (!dense_args_ok(n_rows, n_in, n_out)) return 0;
    const DenseSplit d = dense_split(n_rows, n_in, n_out);
    return sizeof(float) * (size_t)d.parts * ((size_t)n_in * n_out + n_out);
}

extern "C" int fgc_dense_backward(const float *x, const float *dy, const float *y_or_null, int64_t n_rows, int32_t n_in,
                                  int32_t n_out, float *dy_masked_or_null, float *dw, float *db, void *workspace,
                                  size_t workspace_bytes, fgc_stream_t stream)
{
    FGC_NVTX("fgc_dense_backward");
    using namespace fgc;
    if (!dense_args_ok(n_rows, n_in, n_out) || !dw || !db || (dy_masked_or_null && !y_or_null)) return FGC_ERR_BAD_ARGUMENT;
    if (n_rows > 0 && (!x || !dy)) return FGC_ERR_BAD_ARGUMENT;
    if (!workspace || workspace_bytes < fgc_dense_backward_bytes(n_rows, n_in, n_out) || ((uintptr_t)workspace & 15))
        return FGC_ERR_WORKSPACE;
    const DenseSplit d = dense_split(n_rows, n_in, n_out);
    cudaStream_t s = (cudaStream_t)stream;
    float *part_w = (float *)workspace;
    float *part_b = part_w + (size_t)d.parts * n_in * n_out;
    const bool vec = n_in % 4 == 0 && n_out % 4 == 0 &&
                     (((uintptr_t)x | (uintptr_t)dy | (uintptr_t)y_or_null | (uintptr_t)dy_masked_or_null) & 15) == 0;
    if (d.bo == 64 && d.bc == 64)
        launch_dense_bwd<64, 64>(d, vec, s, x, dy, y_or_null, n_rows, n_in, n_out, dy_masked_or_null, part_w, part_b);
    else if (d.bo == 64)
        launch_dense_bwd<64, 128>(d, vec, s, x, dy, y_or_null, n_rows, n_in, n_out, dy_masked_or_null, part_w, part_b);
    else if (d.bc == 64)
        launch_dense_bwd<128, 64>(d, vec, s, x, dy, y_or_null, n_rows, n_in, n_out, dy_masked_or_null, part_w, part_b);
    else
        launch_dense_bwd<128, 128>(d, vec, s, x, dy, y_or_null, n_rows, n_in, n_out, dy_masked_or_null, part_w, part_b);
    FGC_CHECK_LAUNCH();
    const long long n_w = (long long)n_in * n_out;
    k_dense_reduce<<<(unsigned)((n_w + n_out + 31) / 32), 256, 0, s>>>(part_w, part_b, d.parts, n_w, n_out, dw, db);
    return (int)cudaGetLastError();
}
