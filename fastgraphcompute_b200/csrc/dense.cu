// Dense layers around the message passing for sm_100a, on the tensor cores at fp32 accuracy (tensor_core.cuh).
//
// Tall matrices against a small weight: hundreds of thousands of rows, up to a few hundred columns.  The scalar fp32
// products of a library take several times what it takes to read the rows, and bias, ReLU and its mask cost passes of their own.
//
//   k_dense_rows    out = act(A W + b) for 128 rows at a time: a forward, or an input gradient with A the incoming gradient, masked
//                   by the layer's output on the way.  A CTA keeps the weight, split into three parts, in shared memory and
//                   goes through tiles of rows, 64 columns a step: sixteen warps load one or two steps ahead into registers, split and write
//                   to one of three buffers, one thread issues the products of a step, eight warps write the results of a tile
//                   while the next one is formed (two sets of accumulators in TMEM).
//   k_dense_weight  dW = dY^T x and db: a CTA goes through a range of rows, 64 at a time, which are M- and N-major operands as
//                   they are.  The accumulators of every 64 rows are added to fp32 registers, so that no sum is
//                   rounded by the tensor core more than a few times.
//   k_dense_reduce  adds the CTAs' partial results in a fixed order: the result is the same on
//                   every run.
//
// Tiles of rows, and sixteens of the weight's columns, with numbers that cannot be split (infinities, 2^43 and more) are computed by scalar
// operations: 200 k rows, 128 to 128 with ReLU, forward and backward 0.25 ms without such numbers, 0.51 with one in x, 1.06 with one in the weight,
// 4.4 with all of x (every result summed on its own 2.0, 43 and 27; modules 0.99).  NaN costs nothing.
//
// Kernels with ReLU, us (read and written once): 200 k rows, 128 to 128: forward 59 (31), input gradient 71 (47), dW 106 (47); 1.6 M rows, 128 to
// 64: 270 (188), 391 (250), 476 (250).  Forward and backward of the first, modules / library products with passes of our own for bias,
// mask and dW / now: 1018 / 640 / 270.  Relative error against 64 bits, library / now: forward 2.0e-7 / 1.2e-7, input gradient 1.4e-7 / 0.8e-7,
// dW 1.1e-6 (3.5e-7 summed in fp32 by 148 CTAs) / 1.4e-7.
//
// What bounds them is the latency of the splitting warps between loads and buffers (400 k rows, 128 to 128: 0.38 to 0.43 of the issue slots, tensor pipe 0.21 to 0.36).  With four warps instead of
// eight to write results a forward took 80 instead of 59 us (they read, added and wrote one sixteen of columns after the other); with
// loads of a whole step issued when the last one had been split dW took 126 instead of 106, and 105 instead of 60 for 64 to 64,
// where half of the threads had no columns.
#include "tensor_core.cuh"

namespace fgc {

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


// Eight columns from `at` on, zero where fewer are left; `at` is 16-byte aligned if VEC.
template <bool VEC>
__device__ __forceinline__ void dense_load8_at(const float *__restrict__ at, int left, float4 (&v)[2])
{
    v[0] = v[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (VEC) {
        if (left > 0) v[0] = __ldg((const float4 *)at);
        if (left > 4) v[1] = __ldg((const float4 *)at + 1);
    } else {
        float *o = reinterpret_cast<float *>(v);
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (i < left) o[i] = __ldg(at + i);
    }
}
// The gradient passes unless the output is at or below zero (a NaN lets it pass, as in torch).
__device__ __forceinline__ void mask8(float4 (&g)[2], const float4 (&y)[2])
{
#pragma unroll
    for (int i = 0; i < 2; i++) {
        if (y[i].x <= 0.f) g[i].x = 0.f;
        if (y[i].y <= 0.f) g[i].y = 0.f;
        if (y[i].z <= 0.f) g[i].z = 0.f;
        if (y[i].w <= 0.f) g[i].w = 0.f;
    }
}
__device__ __forceinline__ float split_to(char *operand, int part_bytes, int row, int unit, const float4 (&v)[2])
{
    const float f[8] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w};
    uint4 part[3];
    const float most = split8(f, part);
    char *to = operand + operand_at(row, unit);
#pragma unroll
    for (int k = 0; k < 3; k++) *reinterpret_cast<uint4 *>(to + k * part_bytes) = part[k];
    return most;
}

// ----------------------------------------------------------------------------- rows times a weight

struct DenseRows {
    const float *a, *mask, *w, *bias;      // [n_rows, n_sum], the same or null, weight, [n_cols] or null
    float *out;                            // [n_rows, n_cols]
    long long n_rows;
    int n_sum, n_cols;
    int w_sum, w_col;                      // steps of the weight along what is summed over, and from column to column
    int relu;
    int chunks, tile_cols, buffers;        // 64 numbers of the sum each; columns of a CTA; steps that are split ahead
};
// Warps of a CTA: 16 load and split, eight write results, one issues products.
constexpr int kRowsSplit = 16, kRowsWrite = 8, kRowsThreads = 32 * (kRowsSplit + kRowsWrite + 1), kRowsTile = 128;
constexpr int kRowsBuffer = 3 * kRowsTile * 128, kRowsStage = 32 * 20 * 4;
constexpr int kRowsBad = 8;                // tiles that splitting may be ahead of writing: five
inline size_t dense_rows_smem(int buffers, int chunks, int tile_cols)
{
    return 1024 + buffers * (size_t)kRowsBuffer + 3 * (size_t)chunks * tile_cols * 128 + kRowsWrite * (size_t)kRowsStage + 128 * 4 + 256;
}

template <bool VEC, bool MASK>
__global__ void __launch_bounds__(kRowsThreads, 1)
k_dense_rows(const DenseRows g)
{
    extern __shared__ char s_raw[];
    char *s = s_raw + ((1024 - (smem_at(s_raw) & 1023)) & 1023);
    char *s_a = s, *s_w = s + g.buffers * kRowsBuffer;
    const int w_part = g.chunks * g.tile_cols * 128;
    float *s_stage = reinterpret_cast<float *>(s_w + 3 * w_part);
    float *s_bias = s_stage + kRowsWrite * (kRowsStage / 4);                               // of the CTA's columns
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(s_bias + 128);
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 10);
    volatile int *s_late = reinterpret_cast<int *>(s_tmem + 1), *s_bad = s_late + 1;       // a wait that gave up; tiles not to be split,
    int *s_bad_cols = const_cast<int *>(s_bad) + kRowsBad;                                 // sixteens of columns, a bit each
    const uint32_t bar = smem_at(s_bar), full = bar, empty = bar + 24, done = bar + 48, read = bar + 64;
    const int t = threadIdx.x, lane = t & 31, w = __shfl_sync(FGC_FULL_MASK, t >> 5, 0);
    const int col0 = blockIdx.y * g.tile_cols, NT = g.tile_cols;
    const uint32_t columns = tmem_columns(4 * NT);
    if (w == 0) tmem_alloc(smem_at(s_tmem), columns);
    if (t == 0) {
        for (int i = 0; i < 3; i++) {
            mbar_init(full + 8 * i, kRowsSplit);
            mbar_init(empty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(done + 8 * i, 1);
            mbar_init(read + 8 * i, kRowsWrite);
        }
        *s_late = *s_bad_cols = 0;
        for (int i = 0; i < kRowsBad; i++) s_bad[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (t < NT) s_bias[t] = g.bias && col0 + t < g.n_cols ? __ldg(g.bias + col0 + t) : 0.f;
    // the weight: row n of the operand is output column col0 + n
    for (int i = t; i < g.chunks * NT * 8; i += kRowsThreads) {
        const int unit = i & 7, n = (i >> 3) % NT, chunk = (i >> 3) / NT;
        float4 v[2];
        float *f = reinterpret_cast<float *>(v);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int at = chunk * 64 + unit * 8 + k;
            f[k] = col0 + n < g.n_cols && at < g.n_sum ? __ldg(g.w + (size_t)at * g.w_sum + (size_t)(col0 + n) * g.w_col) : 0.f;
        }
        if (split_to(s_w + chunk * NT * 128, w_part, n, unit, v) >= kUnsplit) atomicOr(s_bad_cols, 1 << (n >> 4));
    }
    smem_to_tensor_core();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *s_tmem;
    const long long n_tiles = (g.n_rows + kRowsTile - 1) / kRowsTile;
    const int my_tiles = (int)((n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
    const int steps = my_tiles * g.chunks;

    if (w < kRowsSplit) {
        const int row_in = t >> 3, unit = t & 7;               // of the two passes of 64 rows over a tile
        long long row = (long long)blockIdx.x * kRowsTile + row_in;          // of the next load
        int col = unit * 8;
        auto fetch = [&](int i, float4 (&a)[2][2], float4 (&m)[2][2]) {
            const size_t at = (size_t)(row + 64 * i) * g.n_sum + col;
            const int left = row + 64 * i < g.n_rows ? g.n_sum - col : 0;
            dense_load8_at<VEC>(g.a + at, left, a[i]);
            if constexpr (MASK) dense_load8_at<VEC>(g.mask + at, left, m[i]);
        };
        auto advance = [&]() {
            col += 64;
            if (col >= 64 * g.chunks) {
                col = unit * 8;
                row += (long long)gridDim.x * kRowsTile;
            }
        };
        int b = 0, round = 0, chunk = 0, tile = 0;
        // (a register is loaded again as soon as it has been split; beyond the last row nothing is read)
        auto split_step = [&](float4 (&a)[2][2], float4 (&m)[2][2]) {
            if (round > 0 && !__all_sync(FGC_FULL_MASK, wait_unless(empty + 8 * b, (round - 1) & 1, s_late))) return;
            float top = 0.f;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if constexpr (MASK) mask8(a[i], m[i]);
                top = fmaxf(top, split_to(s_a + b * kRowsBuffer, kRowsTile * 128, row_in + 64 * i, unit, a[i]));
                fetch(i, a, m);
            }
            advance();
            if (top >= kUnsplit) s_bad[tile & (kRowsBad - 1)] = 1;
            smem_to_tensor_core();
            __syncwarp();
            if (lane == 0) mbar_arrive(full + 8 * b);
            if (++b == g.buffers) { b = 0; round++; }
            if (++chunk == g.chunks) { chunk = 0; tile++; }
        };
        // loads two steps ahead, or one with a mask, for want of registers
        constexpr int AHEAD = MASK ? 1 : 2;
        float4 va[AHEAD][2][2], vm[AHEAD][2][2];
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            fetch(0, va[k], vm[k]);
            fetch(1, va[k], vm[k]);
            advance();
        }
        for (int step = 0; step < steps; step += AHEAD) {
#pragma unroll
            for (int k = 0; k < AHEAD; k++)
                if (step + k < steps) split_step(va[k], vm[k]);
        }
    } else if (w == kRowsSplit + kRowsWrite) {
        if (lane == 0) {
            const uint32_t desc = product_desc(NT, false), a_at = smem_at(s_a), w_at = smem_at(s_w);
            int b = 0, round = 0, chunk = 0, tile = 0;
            for (int step = 0; step < steps; step++) {
                if (chunk == 0 && tile >= 2) {
                    if (!wait_unless(read + 8 * (tile & 1), ((tile >> 1) - 1) & 1, s_late)) break;
                    s_bad[(tile - 2) & (kRowsBad - 1)] = 0;
                }
                if (!wait_unless(full + 8 * b, round & 1, s_late)) break;
                tc_after_sync();
                const uint32_t acc = tmem + (uint32_t)((tile & 1) * 2 * NT);
                const int left = g.n_sum - chunk * 64, parts = left >= 64 ? 4 : (left + 15) / 16;
                tc_steps(acc, acc + NT, operand_desc(a_at + b * kRowsBuffer, 16), kRowsTile * 128, operand_desc(w_at + chunk * NT * 128, 16), w_part, 32,
                         desc, parts, chunk > 0);
                tc_commit(empty + 8 * b);
                if (++b == g.buffers) { b = 0; round++; }
                if (++chunk == g.chunks) {
                    tc_commit(done + 8 * (tile & 1));
                    chunk = 0;
                    tile++;
                }
            }
        }
    } else {
        // Results of the warp's 32 rows, 16 columns at a time, of two warps one takes the even sixteens and one the odd ones; through
        // shared memory, so that four lanes write 64 bytes of a row.  The next sixteen are read while these are written.
        const int quarter = w & 3, odd = (w - kRowsSplit) >> 2;
        float *stage = s_stage + (w - kRowsSplit) * (kRowsStage / 4);
        for (int tile = 0; tile < my_tiles; tile++) {
            const long long row0 = ((long long)blockIdx.x + (long long)tile * gridDim.x) * kRowsTile + 32 * quarter;
            const uint32_t acc = tmem + (uint32_t)((tile & 1) * 2 * NT) + ((uint32_t)(32 * quarter) << 16);
            bool plain = !__all_sync(FGC_FULL_MASK, wait_unless(done + 8 * (tile & 1), (tile >> 1) & 1, s_late));
            plain = plain || s_bad[tile & (kRowsBad - 1)];
            const int scalar = __any_sync(FGC_FULL_MASK, plain) ? 0xff : *s_bad_cols;      // sixteens that the tensor core has not formed
            tc_after_sync();
            uint32_t big[16], small[16];
            auto read16 = [&](int c) {
                if (c >= NT || (scalar >> (c >> 4) & 1)) return;
                tmem_read16(acc + c, big);
                tmem_read16(acc + NT + c, small);
            };
            read16(16 * odd);
            for (int c = 16 * odd; c < NT; c += 32) {
                float v[16];
                if (!(scalar >> (c >> 4) & 1)) {
                    tmem_wait_read();
#pragma unroll
                    for (int k = 0; k < 16; k++) v[k] = (__uint_as_float(big[k]) + __uint_as_float(small[k])) * kSplitUndo;
                } else {
                    // A row a lane, its 16 columns side by side; rows and columns beyond the last are read as the last and not written.  Two
                    // numbers of the sum at a time, the next two on their way: the lanes hold their 32 of the weight.
                    const size_t row = (size_t)min(row0 + lane, g.n_rows - 1) * g.n_sum;
                    const int col = min(col0 + c + (lane & 15), g.n_cols - 1), mine = lane >> 4;
                    const float *w = g.w + (size_t)col * g.w_col + (size_t)mine * g.w_sum;
                    float a[2], b, next_a[2], next_b;
                    auto load = [&](int i) {
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            next_a[j] = i + j < g.n_sum ? __ldg(g.a + row + i + j) : 0.f;
                            if (MASK && i + j < g.n_sum && __ldg(g.mask + row + i + j) <= 0.f) next_a[j] = 0.f;
                        }
                        next_b = i + mine < g.n_sum ? __ldg(w + (size_t)i * g.w_sum) : 0.f;
                    };
#pragma unroll
                    for (int k = 0; k < 16; k++) v[k] = 0.f;
                    load(0);
                    for (int i = 0; i < g.n_sum; i += 2) {
                        a[0] = next_a[0];
                        a[1] = next_a[1];
                        b = next_b;
                        load(i + 2);
#pragma unroll
                        for (int k = 0; k < 16; k++) v[k] = fmaf(a[0], __shfl_sync(FGC_FULL_MASK, b, k), v[k]);
                        if (i + 1 >= g.n_sum) break;
#pragma unroll
                        for (int k = 0; k < 16; k++) v[k] = fmaf(a[1], __shfl_sync(FGC_FULL_MASK, b, 16 + k), v[k]);
                    }
                }
                read16(c + 32);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const float4 bias = *reinterpret_cast<const float4 *>(s_bias + c + 4 * k);
                    float4 o = make_float4(v[4 * k] + bias.x, v[4 * k + 1] + bias.y, v[4 * k + 2] + bias.z, v[4 * k + 3] + bias.w);
                    if (g.relu) {                                                         // (NaN stays NaN, as in torch.relu)
                        o.x = o.x < 0.f ? 0.f : o.x;
                        o.y = o.y < 0.f ? 0.f : o.y;
                        o.z = o.z < 0.f ? 0.f : o.z;
                        o.w = o.w < 0.f ? 0.f : o.w;
                    }
                    *reinterpret_cast<float4 *>(stage + lane * 20 + 4 * k) = o;
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = 8 * i + (lane >> 2), cc = 4 * (lane & 3), col = col0 + c + cc;
                    const float4 o = *reinterpret_cast<const float4 *>(stage + r * 20 + cc);
                    if (row0 + r < g.n_rows && col < g.n_cols) {
                        float *to = g.out + (size_t)(row0 + r) * g.n_cols + col;
                        if (VEC && (g.n_cols & 3) == 0) *reinterpret_cast<float4 *>(to) = o;
                        else {
                            to[0] = o.x;
                            if (col + 1 < g.n_cols) to[1] = o.y;
                            if (col + 2 < g.n_cols) to[2] = o.z;
                            if (col + 3 < g.n_cols) to[3] = o.w;
                        }
                    }
                }
                __syncwarp();
            }
            tc_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(read + 8 * (tile & 1));
        }
    }
    tc_before_sync();
    __syncthreads();
    if (w == 0) {
        tc_after_sync();
        tmem_free(tmem, columns);
    }
}

// Columns of a CTA: as many as fit beside the buffers, in equal shares.
static int dense_tile_cols(int chunks, int n_cols)
{
    int most = (int)((227 * 1024 - dense_rows_smem(2, chunks, 0)) / (3 * chunks * 128)) / 16 * 16;
    if (most > 128) most = 128;
    if (most < 16) return 0;
    const int padded = (n_cols + 15) / 16 * 16, shares = (padded + most - 1) / most;
    return ((padded + shares - 1) / shares + 15) / 16 * 16;
}

template <bool VEC, bool MASK>
static cudaError_t launch_rows(const DenseRows &g, cudaStream_t s)
{
    const size_t smem = dense_rows_smem(g.buffers, g.chunks, g.tile_cols);
    const cudaError_t e = cudaFuncSetAttribute(k_dense_rows<VEC, MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const unsigned shares = (unsigned)((g.n_cols + g.tile_cols - 1) / g.tile_cols);
    const long long tiles = (g.n_rows + kRowsTile - 1) / kRowsTile;
    long long ctas = sm_count() / shares;
    if (ctas < 1) ctas = 1;
    if (ctas > tiles) ctas = tiles;
    k_dense_rows<VEC, MASK><<<dim3((unsigned)ctas, shares), kRowsThreads, smem, s>>>(g);
    return cudaGetLastError();
}

static int dense_rows(DenseRows g, cudaStream_t s)
{
    g.chunks = (g.n_sum + 63) / 64;
    g.tile_cols = g.chunks <= FGC_DENSE_MAX_SUM / 64 ? dense_tile_cols(g.chunks, g.n_cols) : 0;
    if (g.tile_cols == 0) return FGC_ERR_TOO_LARGE;
    g.buffers = dense_rows_smem(3, g.chunks, g.tile_cols) <= 227 * 1024 ? 3 : 2;
    const bool vec = g.n_sum % 4 == 0 && (((uintptr_t)g.a | (uintptr_t)g.mask | (uintptr_t)g.out) & 15) == 0;
    if (g.mask) return (int)(vec ? launch_rows<true, true>(g, s) : launch_rows<false, true>(g, s));
    return (int)(vec ? launch_rows<true, false>(g, s) : launch_rows<false, false>(g, s));
}

// ----------------------------------------------------------------------------- sums over rows

// Warps of a CTA: 16 load and split, eight add up, one issues products.
constexpr int kWeightSplit = 16, kWeightAdd = 8, kWeightThreads = 32 * (kWeightSplit + kWeightAdd + 1), kWeightRows = 64;
constexpr int kWeightChunk = 3 * kWeightRows * 128;                    // the three parts of 64 columns
constexpr int kWeightBuffer = 4 * kWeightChunk;                        // two of the matrix with 128 columns, two of the other
constexpr int kWeightBias = 32 * 128 * 4;                              // a thread's sums of dY
constexpr size_t kWeightSmem = 1024 + 2 * (size_t)kWeightBuffer + kWeightBias + 128;
static_assert(kWeightSmem <= 227 * 1024, "buffers too large");

struct DenseWeight {
    const float *x, *dy, *y;               // [n_rows, n_in], [n_rows, n_out], the same as dy or null
    long long n_rows, rows_per_cta;
    int n_in, n_out;
    int tile_in, tile_out;                 // columns of a CTA, of x and of dy
    int swap;                              // the accumulators' rows are inputs (else outputs)
    float *dy_masked, *part_w, *part_b;
};

template <bool VEC>
__global__ void __launch_bounds__(kWeightThreads, 1)
k_dense_weight(const DenseWeight g)
{
    extern __shared__ char s_raw[];
    char *s = s_raw + ((1024 - (smem_at(s_raw) & 1023)) & 1023);
    float *s_bias = reinterpret_cast<float *>(s + 2 * kWeightBuffer);
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(s + 2 * kWeightBuffer + kWeightBias);
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 6);
    volatile int *s_late = reinterpret_cast<int *>(s_tmem + 1), *s_bad = s_late + 1;       // a wait that gave up; steps not to be split
    const uint32_t full = smem_at(s_bar), done = full + 16, read = full + 32;              // two each
    const int t = threadIdx.x, lane = t & 31, w = __shfl_sync(FGC_FULL_MASK, t >> 5, 0);
    const int c0 = blockIdx.y * g.tile_in, o0 = blockIdx.z * g.tile_out;
    const long long first = (long long)blockIdx.x * g.rows_per_cta, last = min(g.n_rows, first + g.rows_per_cta);
    const int steps = first < last ? (int)((last - first + kWeightRows - 1) / kWeightRows) : 0;
    const bool owner = blockIdx.y == 0;                        // of the mask and the bias sum
    const int NT = ((g.swap ? g.tile_out : g.tile_in) + 15) / 16 * 16;
    const uint32_t columns = tmem_columns(4 * NT);
    const int n_in = min(g.n_in, c0 + g.tile_in), n_out = min(g.n_out, o0 + g.tile_out);
    if (w == 0) tmem_alloc(smem_at(s_tmem), columns);
    if (t == 0) {
        for (int i = 0; i < 2; i++) {
            mbar_init(full + 8 * i, kWeightSplit);
            mbar_init(done + 8 * i, 1);
            mbar_init(read + 8 * i, kWeightAdd);
        }
        *s_late = 0;
        for (int i = 0; i < kRowsBad; i++) s_bad[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *s_tmem;

    if (w < kWeightSplit) {
        // The matrix whose columns are rows of the result comes first in a buffer.  Columns beyond a tile are not written: what is
        // there makes rows and columns of the result that are not read.
        // Units of eight columns: eight or 16 to a row, so that 64 rows take one pass or two.  A register is loaded again as soon as it
        // has been split: the loads of a step are on their way during the rest of the one before.
        const int wide_x = g.tile_in > 64 ? 1 : 0, wide_y = g.tile_out > 64 ? 1 : 0;
        const int unit_x = t & (7 + 8 * wide_x), row_x = t >> (3 + wide_x), unit_y = t & (7 + 8 * wide_y), row_y = t >> (3 + wide_y);
        char *s_x = s + (g.swap ? 0 : 2 * kWeightChunk) + (unit_x >> 3) * kWeightChunk;
        char *s_y = s + (g.swap ? 2 * kWeightChunk : 0) + (unit_y >> 3) * kWeightChunk;
        const int x_left = n_in - c0 - unit_x * 8, y_left = n_out - o0 - unit_y * 8;
        const float *px = g.x + (size_t)(first + row_x) * g.n_in + c0 + unit_x * 8;
        size_t at_y = (size_t)(first + row_y) * g.n_out + o0 + unit_y * 8;
        long long row0 = first;                                // of the step
        float4 vx[2][2], vy[2][2], vm[2][2];
        float sum[8] = {};
        float *total = s_bias + row_y * (64 + 64 * wide_y) + unit_y * 8;         // two levels, so that a thread never adds thousands of rows one to another
        auto fold = [&]() {
#pragma unroll
            for (int k = 0; k < 8; k++) { total[k] += sum[k]; sum[k] = 0.f; }
        };
#pragma unroll
        for (int k = 0; k < 8; k++) total[k] = 0.f;
        auto fetch_x = [&](int i) { dense_load8_at<VEC>(px + (size_t)(32 * i) * g.n_in, row0 + row_x + 32 * i < last ? x_left : 0, vx[i]); };
        auto fetch_y = [&](int i) {
            const int left = row0 + row_y + 32 * i < last ? y_left : 0;
            dense_load8_at<VEC>(g.dy + at_y + (size_t)(32 * i) * g.n_out, left, vy[i]);
            if (g.y) dense_load8_at<VEC>(g.y + at_y + (size_t)(32 * i) * g.n_out, left, vm[i]);
        };
        if (steps > 0) {
            fetch_x(0);
            if (wide_x) fetch_x(1);
            fetch_y(0);
            if (wide_y) fetch_y(1);
        }
        for (int step = 0; step < steps; step++) {
            const int b = step & 1;
            float top = 0.f;
            if (step >= 2 && !__all_sync(FGC_FULL_MASK, wait_unless(done + 8 * b, ((step >> 1) - 1) & 1, s_late))) top = kUnsplit;
            // (the rows of the next step from here on; beyond the last nothing is read)
            const long long row_now = row0;
            const size_t y_now = at_y;
            row0 += kWeightRows;
            px += (size_t)kWeightRows * g.n_in;
            at_y += (size_t)kWeightRows * g.n_out;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if (i == 0 || wide_x) {
                    top = fmaxf(top, split_to(s_x + b * kWeightBuffer, kWeightRows * 128, row_x + 32 * i, unit_x & 7, vx[i]));
                    fetch_x(i);
                }
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if (i == 0 || wide_y) {
                    if (g.y) mask8(vy[i], vm[i]);
                    const float *v = reinterpret_cast<const float *>(vy[i]);
                    if (owner && g.dy_masked && row_now + row_y + 32 * i < last) {
#pragma unroll
                        for (int k = 0; k < 8; k++)
                            if (k < y_left) g.dy_masked[y_now + (size_t)(32 * i) * g.n_out + k] = v[k];
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++) sum[k] += v[k];
                    top = fmaxf(top, split_to(s_y + b * kWeightBuffer, kWeightRows * 128, row_y + 32 * i, unit_y & 7, vy[i]));
                    fetch_y(i);
                }
            }
            if (top >= kUnsplit) s_bad[step & (kRowsBad - 1)] = 1;
            smem_to_tensor_core();
            __syncwarp();
            if (lane == 0) mbar_arrive(full + 8 * b);
            if ((step & 15) == 15) fold();
        }
        fold();
    } else if (w == kWeightSplit + kWeightAdd) {
        if (lane == 0) {
            const uint32_t desc = product_desc(NT, true), s_at = smem_at(s);
            for (int step = 0; step < steps; step++) {
                const int b = step & 1;
                if (step >= 2) {
                    if (!wait_unless(read + 8 * b, ((step >> 1) - 1) & 1, s_late)) break;
                    s_bad[(step - 2) & (kRowsBad - 1)] = 0;
                }
                if (!wait_unless(full + 8 * b, (step >> 1) & 1, s_late)) break;
                tc_after_sync();
                const uint32_t acc = tmem + (uint32_t)(b * 2 * NT), at = s_at + b * kWeightBuffer;
                tc_steps(acc, acc + NT, operand_desc(at, kWeightChunk), kWeightRows * 128, operand_desc(at + 2 * kWeightChunk, kWeightChunk),
                         kWeightRows * 128, 2048, desc, kWeightRows / 16, false);
                tc_commit(done + 8 * b);
            }
        }
    } else {
        // sums of 64 rows into registers: 32 rows of the result a warp, half of the columns, one row a lane
        float total[64] = {};
        const int half = (w - kWeightSplit) >> 2, n_half = 64 * half;
        const int m = 32 * (w & 3) + lane + (g.swap ? c0 : o0), n0 = n_half + (g.swap ? o0 : c0);
        auto masked_dy = [&](long long row, int o) {
            const float d = __ldg(g.dy + (size_t)row * g.n_out + o);
            return g.y && __ldg(g.y + (size_t)row * g.n_out + o) <= 0.f ? 0.f : d;
        };
        for (int step = 0; step < steps; step++) {
            const int b = step & 1;
            bool plain = !wait_unless(done + 8 * b, (step >> 1) & 1, s_late) || s_bad[step & (kRowsBad - 1)];
            plain = __any_sync(FGC_FULL_MASK, plain);
            tc_after_sync();
            if (!plain) {
                const uint32_t acc = tmem + (uint32_t)(b * 2 * NT) + ((uint32_t)(32 * (w & 3)) << 16);
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    if (n_half + 16 * h < NT) {
                        uint32_t big[16], small[16];
                        tmem_read16(acc + n_half + 16 * h, big);
                        tmem_read16(acc + NT + n_half + 16 * h, small);
                        tmem_wait_read();
#pragma unroll
                        for (int k = 0; k < 16; k++) total[16 * h + k] = fmaf(__uint_as_float(big[k]) + __uint_as_float(small[k]), kSplitUndo, total[16 * h + k]);
                    }
                }
            } else {
                // a row of the matrices at a time, the next one on its way: the lanes hold its 64 numbers of the one, and theirs of the other
                const long long row0 = first + (long long)step * kWeightRows, end = min(last, row0 + kWeightRows);
                float a, v[2], next_a, next_v[2];
                auto load = [&](long long row) {
                    next_a = row >= end ? 0.f : (g.swap ? (m < n_in ? __ldg(g.x + (size_t)row * g.n_in + m) : 0.f) : (m < n_out ? masked_dy(row, m) : 0.f));
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int n = n0 + 32 * j + lane;
                        next_v[j] = row >= end ? 0.f : (g.swap ? (n < n_out ? masked_dy(row, n) : 0.f) : (n < n_in ? __ldg(g.x + (size_t)row * g.n_in + n) : 0.f));
                    }
                };
                load(row0);
                for (long long row = row0; row < end; row++) {
                    a = next_a;
                    v[0] = next_v[0];
                    v[1] = next_v[1];
                    load(row + 1);
#pragma unroll
                    for (int k = 0; k < 64; k++) total[k] = fmaf(a, __shfl_sync(FGC_FULL_MASK, v[k >> 5], k & 31), total[k]);
                }
            }
            tc_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(read + 8 * b);
        }
        float *pw = g.part_w + (size_t)blockIdx.x * g.n_out * g.n_in;
#pragma unroll
        for (int k = 0; k < 64; k++) {
            if (g.swap) {
                if (m < n_in && n0 + k < n_out) pw[(size_t)(n0 + k) * g.n_in + m] = total[k];
            } else {
                if (m < n_out && n0 + k < n_in) pw[(size_t)m * g.n_in + n0 + k] = total[k];
            }
        }
    }
    tc_before_sync();
    __syncthreads();
    if (w == 0) {
        tc_after_sync();
        tmem_free(tmem, columns);
    }
    // threads that loaded the same columns, added in a fixed order
    if (owner && t < g.tile_out && o0 + t < n_out) {
        float sum = 0.f;
        const int length = g.tile_out > 64 ? 128 : 64, rows = kWeightBias / 4 / length;
        for (int k = 0; k < rows; k++) sum += s_bias[k * length + t];
        g.part_b[(size_t)blockIdx.x * g.n_out + o0 + t] = sum;
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
    int tile_out, tile_in, tiles_out, tiles_in, parts;
    long long rows;
};

// Tiles of up to 128 columns, in equal shares of whole units; as many row ranges as there are SMs for, at least 64 rows each.
static DenseSplit dense_split(int64_t n_rows, int n_in, int n_out)
{
    DenseSplit d;
    auto share = [](int n, int &tiles) {
        tiles = (n + 127) / 128;
        return ((n + tiles - 1) / tiles + 7) / 8 * 8;
    };
    d.tile_out = share(n_out, d.tiles_out);
    d.tile_in = share(n_in, d.tiles_in);
    const int64_t tiles = (int64_t)d.tiles_out * d.tiles_in;
    int64_t parts = sm_count() / tiles;
    if (parts < 1) parts = 1;
    const int64_t most = (n_rows + kWeightRows - 1) / kWeightRows;
    if (parts > most) parts = most < 1 ? 1 : most;
    d.rows = ((n_rows + parts - 1) / parts + kWeightRows - 1) / kWeightRows * kWeightRows;
    d.parts = d.rows > 0 ? (int)((n_rows + d.rows - 1) / d.rows) : 0;
    if (d.parts < 1) d.parts = 1;
    return d;
}

static bool dense_args_ok(int64_t n_rows, int32_t n_in, int32_t n_out)
{
    return n_rows >= 0 && n_in >= 1 && n_out >= 1 && n_in <= 65535 && n_out <= 65535;
}

}  // namespace fgc

extern "C" int fgc_dense_forward(const float *x, const float *weight, const float *bias_or_null, int64_t n_rows, int32_t n_in,
                                 int32_t n_out, int32_t relu, float *out, fgc_stream_t stream)
{
    FGC_NVTX("fgc_dense_forward");
    using namespace fgc;
    if (!dense_args_ok(n_rows, n_in, n_out)) return FGC_ERR_BAD_ARGUMENT;
    if (n_in > FGC_DENSE_MAX_SUM) return FGC_ERR_TOO_LARGE;
    if (n_rows == 0) return FGC_OK;
    if (!x || !weight || !out) return FGC_ERR_BAD_ARGUMENT;
    DenseRows g = {};
    g.a = x; g.w = weight; g.bias = bias_or_null; g.out = out; g.n_rows = n_rows;
    g.n_sum = n_in; g.n_cols = n_out; g.w_sum = 1; g.w_col = n_in; g.relu = relu;
    return dense_rows(g, (cudaStream_t)stream);
}

extern "C" int fgc_dense_input_gradient(const float *dy, const float *y_or_null, const float *weight, int64_t n_rows, int32_t n_in,
                                        int32_t n_out, float *dx, fgc_stream_t stream)
{
    FGC_NVTX("fgc_dense_input_gradient");
    using namespace fgc;
    if (!dense_args_ok(n_rows, n_in, n_out)) return FGC_ERR_BAD_ARGUMENT;
    if (n_out > FGC_DENSE_MAX_SUM) return FGC_ERR_TOO_LARGE;
    if (n_rows == 0) return FGC_OK;
    if (!dy || !weight || !dx) return FGC_ERR_BAD_ARGUMENT;
    DenseRows g = {};
    g.a = dy; g.mask = y_or_null; g.w = weight; g.out = dx; g.n_rows = n_rows;
    g.n_sum = n_out; g.n_cols = n_in; g.w_sum = n_in; g.w_col = 1;
    return dense_rows(g, (cudaStream_t)stream);
}

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
    DenseWeight g = {};
    g.x = x; g.dy = dy; g.y = y_or_null; g.n_rows = n_rows; g.rows_per_cta = d.rows; g.n_in = n_in; g.n_out = n_out;
    g.tile_in = d.tile_in; g.tile_out = d.tile_out; g.swap = d.tile_out <= 64 && d.tile_in > d.tile_out;
    g.dy_masked = dy_masked_or_null; g.part_w = (float *)workspace; g.part_b = g.part_w + (size_t)d.parts * n_in * n_out;
    const bool vec = n_in % 4 == 0 && n_out % 4 == 0 && (((uintptr_t)x | (uintptr_t)dy | (uintptr_t)y_or_null) & 15) == 0;
    auto *const kernel = vec ? k_dense_weight<true> : k_dense_weight<false>;
    FGC_RETURN_IF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWeightSmem));
    kernel<<<dim3((unsigned)d.parts, (unsigned)d.tiles_in, (unsigned)d.tiles_out), kWeightThreads, kWeightSmem, s>>>(g);
    FGC_CHECK_LAUNCH();
    const long long n_w = (long long)n_in * n_out;
    k_dense_reduce<<<(unsigned)((n_w + n_out + 31) / 32), 256, 0, s>>>(g.part_w, g.part_b, d.parts, n_w, n_out, dw, db);
    return (int)cudaGetLastError();
}
