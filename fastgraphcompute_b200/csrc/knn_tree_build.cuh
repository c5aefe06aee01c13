// Parts shared by the two sorts of the search tree (knn_tree.cu in a chain of launches, knn_tree_small.cu in one).
#pragma once
#include "knn_tree.cuh"

namespace fgc {

// The curve's cells: equal in all dimensions; an extent of zero or one that overflows puts every point into cell 0 (any order gives a
// valid tree).  min_key, max_key: ~ordered(min) and ordered(max) per coordinate.
static __device__ void tree_setup(KnnTree *t, const uint32_t (&min_key)[kTreeKeyDims], const uint32_t (&max_key)[kTreeKeyDims], int key_dims, int bits)
{
    float ext = 0.f;
#pragma unroll
    for (int c = 0; c < kTreeKeyDims; c++) {
        if (c < key_dims) {
            const float lo = ordered_to_float(~min_key[c]), hi = ordered_to_float(max_key[c]);
            t->origin[c] = lo;
            ext = fmaxf(ext, hi - lo);
        }
    }
    const float s = (float)(1u << bits) / ext;
    t->scale = ext > 0.f && is_finite_bits(s) ? s : 0.f;
    t->magic = kTreeMagic;
}

// Place of a cell on the Hilbert curve over ND dimensions of `bits` bits: J. Skilling, "Programming
// the Hilbert curve", AIP Conf. Proc. 707 (2004), the transform from axes to the transposed index,
// whose bits are then interleaved.
template <int ND>
__device__ __forceinline__ uint32_t hilbert_index(uint32_t (&x)[kTreeKeyDims], int bits)
{
    for (uint32_t q = 1u << (bits - 1); q > 1; q >>= 1) {
        const uint32_t p = q - 1;
#pragma unroll
        for (int i = 0; i < ND; i++) {
            if (x[i] & q) x[0] ^= p;
            else { const uint32_t d = (x[0] ^ x[i]) & p; x[0] ^= d; x[i] ^= d; }
        }
    }
#pragma unroll
    for (int i = 1; i < ND; i++) x[i] ^= x[i - 1];
    uint32_t e = 0;
    for (uint32_t q = 1u << (bits - 1); q > 1; q >>= 1)
        if (x[ND - 1] & q) e ^= q - 1;
    uint32_t key = 0;
    for (int b = bits - 1; b >= 0; b--)
#pragma unroll
        for (int i = 0; i < ND; i++) key = (key << 1) | (((x[i] ^ e) >> b) & 1u);
    return key;
}

__device__ __forceinline__ uint32_t tree_key(const KnnTree *__restrict__ t, const float *__restrict__ row, int key_dims, int bits)
{
    const uint32_t top = (1u << bits) - 1;
    uint32_t x[kTreeKeyDims];
    const float scale = t->scale;
#pragma unroll
    for (int c = 0; c < kTreeKeyDims; c++)
        x[c] = c < key_dims ? min(__float2uint_rz((__ldg(row + c) - t->origin[c]) * scale), top) : 0u;
    switch (key_dims) {
    case 2: return hilbert_index<2>(x, bits);
    case 3: return hilbert_index<3>(x, bits);
    case 4: return hilbert_index<4>(x, bits);
    case 5: return hilbert_index<5>(x, bits);
    default: return hilbert_index<6>(x, bits);
    }
}

// Up to so many points the sort is one launch.  Forward of learned coordinates in three dimensions, K = 40, sort in a chain / one launch, us:
// 10 k in ten row splits 137 / 94, 20 k 146 / 115, 32 k 158 / 138; in four, K = 10, 32 k in eighty 144 / 159.
constexpr int64_t kSmallTree = 24576;
// Whether it takes these points, and its keys: dimensions, bits per dimension, radix passes.
bool small_tree_bits(int64_t n_vert, int n_coords, int64_t n_rs, int *key_dims, int *bits, int *passes);
// ids_last: original ids in curve order; keys, ids: scratch; info_mapped: two words that the host reads, or null.
cudaError_t launch_tree_small(const float *coords, int n, int n_coords, int key_dims, int bits, int passes, const int64_t *row_splits, int n_rs, KnnGrid *g,
                              KnnTree *tree, uint32_t *keys, int *ids, int *ids_last, volatile int32_t *info_mapped, cudaStream_t s);

}  // namespace fgc
