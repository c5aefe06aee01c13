// Parts shared by the kernels that search the tree: one query at a time (knn_tree_search.cu) and all queries of a leaf
// (knn_tree_group.cu).
#pragma once
#include "knn_tree.cuh"

namespace fgc {

// Boxes of up to five coordinates: corners of the first four, both of the fifth.
struct BoxArrays {
    const float4 *lo, *hi;
    const float2 *e;
};

struct TreeArgs {
    const float4 *scoords;
    const int *sorig;
    const uint8_t *sflag;      // nullptr: no direction restriction
    const float4 *box[3];      // leaves, nodes, top nodes
    // in five coordinates: boxes of leaves and of their halves (16 points), points in curve order
    BoxArrays leaves, halves;
    const float4 *point_a;
    const float *point_e;
    const int64_t *row_splits;
    KnnGrid *grid;
    KnnTree *tree;
    int64_t *out_idx;
    float *out_dist;
    int n_vert;
    int n_rs;
    int K;
    int tf_compat;
    TieMarks mark_ties;        // which rows get kTieRow in slot 0
    // the search by groups only
    int slot0, n_slots;        // leaf slots of this launch: from the one up to the other
    int list_cap, list_room;
    int *listed;               // queries that are searched one by one instead (places in curve order)
    int *list, *list_n;        // leaves [slots of this launch][list_room] that a leaf's queries may need; their number (-1: no points)
    int4 *leaf_info;           // per leaf slot: first point of the leaf in its row split, begin and size of the row split
    int2 *leaf_part;           // per eight queries of a leaf slot: begin and length of their part of the list
    float *bound;              // per query of this launch: at least K - 1 candidates are this near (kNoQuery, kListedQuery)
};

constexpr uint32_t kNoBox = 0xffffffffu;
constexpr float kNoQuery = -1.f;         // bound of a query that may not have neighbours
constexpr float kListedQuery = -2.f;     // bound of a listed query

// Whether two of the kn nearest in an ascending list (entry r * 32 + lane, id -1: empty) have the same distance.
template <int R>
__device__ __forceinline__ bool equal_in_list(const float (&d)[R], const int (&id)[R], int kn, int lane)
{
    bool same = false;
#pragma unroll
    for (int r = 0; r < R; r++) {
        float next = __shfl_down_sync(FGC_FULL_MASK, d[r], 1);
        if (r + 1 < R) {
            const float first = __shfl_sync(FGC_FULL_MASK, d[r + 1 < R ? r + 1 : r], 0);
            if (lane == 31) next = first;
        }
        same = same || (r * 32 + lane + 1 < kn && id[r] >= 0 && d[r] == next);
    }
    return __any_sync(FGC_FULL_MASK, same);
}

// Slot 0 of a row: the point itself, or the mark.  tie: a choice at the K-th distance; same: equal distances in the list.
__device__ __forceinline__ int64_t mark_row(const TreeArgs &a, bool tie, bool same, int orig_q)
{
    if (a.mark_ties == TieMarks::kNone || !(tie || same)) return orig_q;
    atomicAdd(tie ? &a.tree->n_tied : &a.tree->n_equal, 1);
    return tie ? kTieRow : kEqualRow;
}

// Checks of the arguments of a search, and what every kernel needs of them.
int tree_args(int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K, int32_t has_direction,
              int32_t tf_compat, TieMarks mark_ties, int64_t *out_idx, float *out_distsq, void *workspace, size_t workspace_bytes,
              TreeArgs *a, KnnWorkspace *L, TreeLayout *T);
// One query per warp, for the listed ones.
int launch_tree_listed(const TreeArgs &a, int nv, cudaStream_t s);

#define FGC_TRY(expr)                                    \
    do {                                                 \
        const cudaError_t rc_ = (expr);                  \
        if (rc_ != cudaSuccess) return rc_;              \
    } while (0)

}  // namespace fgc
