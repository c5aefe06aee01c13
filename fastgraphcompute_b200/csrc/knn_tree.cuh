// Search tree of the kNN: points in Hilbert order, boxes over runs of 32, 1024 and 32768 points.
//
// The points of a row split are sorted along a Hilbert curve; 32 consecutive ones form a leaf, 32
// leaves a node, 32 nodes a top node, each with the bounding box of its points over all
// coordinates.  One lane tests one box, so a warp tests all children of a node at once.  Unlike
// the cells of a grid the boxes follow the density: every leaf holds 32 points whether the data is
// uniform, normally distributed or clustered.
//
// Two searches: one query at a time (knn_tree_search.cu), and in up to five coordinates all queries of a leaf at once
// (knn_tree_group.cu).
//
// The tree lives in the workspace of the grid (knn_grid.cuh): sorted coordinates, original ids and
// flags in the same sections, everything else in the space of the cell table.  Its record lies
// in the section behind the grid's header, of which it uses only the status word.
#pragma once
#include <cstddef>

#include "knn_grid.cuh"

namespace fgc {

constexpr int kTreeKeyDims = 6;         // coordinates that enter the Hilbert key (boxes cover all)
constexpr uint32_t kTreeMagic = 0x74726565u;

struct KnnTree {
    uint32_t magic;
    uint32_t nonfinite;
    int32_t blocks_done;
    int32_t scan_ticket;
    uint32_t min_key[kTreeKeyDims];     // ~ordered(min) (atomicMax)
    uint32_t max_key[kTreeKeyDims];     // ordered(max)
    float origin[kTreeKeyDims];
    float scale;                        // cells of the Hilbert curve per unit length
    int32_t n_tied;                     // rows marked kTieRow by the search
    int32_t n_equal;                    // rows marked kEqualRow
    int32_t n_listed;                   // queries that the search by groups leaves to the search one by one
    int32_t next_listed;                // of those, taken so far
};
static_assert(sizeof(KnnTree) <= kHardTicketBytes, "tree record too large");
static_assert(offsetof(KnnTree, n_listed) == 100, "read there by tests/test_gpu_tree_groups.py");

constexpr int kRadixBits = 11;
constexpr int kRadixBins = 1 << kRadixBits;

// First box of row split e at each level (a row split of n points has ceil(n / 2^shift) boxes there):
// unique and increasing in e without a prefix sum over the row splits, at the price of at most
// one unused box per row split.
__host__ __device__ inline int64_t tree_base(int64_t ev_begin, int64_t e, int shift) { return (ev_begin >> shift) + e; }

constexpr int kGroupDims = 5;          // searches by groups take up to so many coordinates,
constexpr int kApartDims = 5;          // and in so many they look at boxes of 16 points, and read from arrays apart

struct TreeLayout {
    size_t keys[2], ids[2], hist, hist_sums, box[3], end;
    size_t listed, leaf_info;                // of the search by groups, in the place of the keys when they are sorted
    // in five coordinates the boxes of leaves and of their halves and the points once more, lower corners, upper corners and what is fifth
    // apart: a warp that reads 32 in a row touches a quarter of the lines
    size_t box_lo, box_hi, box_e, half_lo, half_hi, half_e, point_a, point_e;
    int64_t n_box[3];      // slots per level: leaves, nodes, top nodes
    int rounds;            // a CTA of a radix pass takes 256 * rounds keys
    int tiles;
    int key_dims, bits;    // Hilbert curve: dimensions and bits per dimension
    int passes;
    bool fits;
    bool groups;           // room for these: row splits of thirty points or more, or few of them
};

inline TreeLayout tree_layout(const KnnWorkspace &w, int64_t n_vert, int n_coords, int64_t n_rs)
{
    TreeLayout t;
    const int64_t n_events = n_rs > 1 ? n_rs - 1 : 1;
    int ebits = 0;
    while (((int64_t)1 << ebits) < n_events) ebits++;
    // Key = row split, then the place on the curve, sorted 11 bits a pass.  Three passes while
    // they leave 24 bits or more for the curve, else four.
    t.passes = 3;
    if (t.passes * kRadixBits - ebits < 24) t.passes = 4;
    t.key_dims = n_coords < kTreeKeyDims ? n_coords : kTreeKeyDims;
    int hb = t.passes * kRadixBits - ebits;
    if (hb > 32) hb = 32;
    t.bits = hb / t.key_dims;
    // small batches: more CTAs with less work each (50 k points: build 0.164 -> 0.089 ms)
    t.rounds = n_vert >= 1000000 ? 16 : 4;
    t.tiles = (int)ceil_div64(n_vert, 256 * t.rounds);
    size_t off = w.counts;
    for (int i = 0; i < 2; i++) { t.keys[i] = off; off = align_up(off + 8 * (size_t)n_vert, 256); }
    for (int i = 0; i < 2; i++) { t.ids[i] = off; off = align_up(off + 4 * (size_t)n_vert, 256); }
    const size_t entries = (size_t)kRadixBins * t.tiles;
    t.hist = off; off = align_up(off + 4 * entries, 256);
    t.hist_sums = off; off = align_up(off + 4 * (entries / kScanTile + 2), 256);
    for (int l = 0; l < 3; l++) {
        t.n_box[l] = (n_vert >> (5 * (l + 1))) + n_events + 1;
        t.box[l] = off;
        off = align_up(off + sizeof(float4) * 2 * w.nv * (size_t)t.n_box[l], 256);
    }
    t.end = off;
    // the sections from the cell table up to the original ids are the tree's to use
    t.fits = t.end <= w.sorig && t.bits >= 1 && entries < ((size_t)1 << 31);
    t.listed = t.keys[0];
    t.leaf_info = align_up(t.listed + 4 * (size_t)n_vert, 256);
    const size_t leaves = n_coords == kApartDims ? (size_t)t.n_box[0] : 0, halves = 2 * leaves, points = n_coords == kApartDims ? (size_t)n_vert : 0;
    off = t.end;
    auto section = [&](size_t bytes) { const size_t at = off; off = align_up(off + bytes, 256); return at; };
    t.box_lo = section(sizeof(float4) * leaves);
    t.box_hi = section(sizeof(float4) * leaves);
    t.box_e = section(sizeof(float2) * leaves);
    t.half_lo = section(sizeof(float4) * halves);
    t.half_hi = section(sizeof(float4) * halves);
    t.half_e = section(sizeof(float2) * halves);
    t.point_a = section(sizeof(float4) * points);
    t.point_e = section(sizeof(float) * points);
    t.groups = n_coords <= kGroupDims && t.fits && off <= w.sorig &&
               t.leaf_info + (sizeof(int4) + 4 * sizeof(int2)) * (size_t)t.n_box[0] <= t.ids[0];
    return t;
}

// List length class of a search: K - 1 <= 32 R.
inline int tree_list_rows(int K) { return K <= 33 ? 1 : (K <= 65 ? 2 : (K <= 129 ? 4 : 8)); }

// Scratch of a search by groups: what k_tree_groups leaves for the queries of `slots` leaf slots.
struct TreeScratch {
    int slots, list_cap, list_room;
    int *list, *list_n;
    float *bound;
};
// Leaves that a leaf's queries may need (mean over uniform, normal and clustered points, K = 16 to 200: 36 to 110 in three
// coordinates, 140 to 350 in four, 1000 in five); with more they are searched one by one.  A million normal points in five
// coordinates, K = 40, with 768 / 1536 / 2304 / 3072 of them: 17.2 / 15.0 / 15.2 / 15.3 ms (77 / 16 / 7 / 4 % listed); 600 k uniform ones, K =
// 200: 12.0 / 11.0 / 11.0 / 10.9.  A leaf of 32 points takes 2180 / 4228 / 6276 bytes in three / four / five.
__host__ __device__ constexpr int tree_list_cap(int n_coords) { return n_coords <= 3 ? 512 : (n_coords == 4 ? 1024 : 1536); }
// The four lists of eight queries each that are made of it (knn_tree_group.cu) may take twice that in five coordinates (a million
// normal points, K = 40: with as much as the one list 0.24 of all leaves have room for four).
__host__ __device__ constexpr int tree_list_room(int n_coords) { return n_coords <= 4 ? 1 : 2; }
// Larger searches take several rounds (6.4 M points in three coordinates 13.54 ms, with half of it 13.59; 3 M in five 43.4 and 43.6).
constexpr size_t kTreeScratchBytes = (size_t)256 << 20;
inline size_t tree_slot_bytes(int n_coords) { return 4 * ((size_t)tree_list_cap(n_coords) + 1 + 32); }
// What a workspace for searches by groups holds behind the sections of the grid.
inline size_t tree_extra_bytes(int64_t n_vert, int n_coords, int64_t n_rs)
{
    if (n_coords > kGroupDims) return 0;
    const size_t most = kTreeScratchBytes / tree_slot_bytes(n_coords), slots = tree_list_room(n_coords) * (size_t)(n_vert / 32 + n_rs + 1);
    return (slots < most ? slots : most) * tree_slot_bytes(n_coords);
}
inline bool tree_scratch(const KnnWorkspace &w, int n_coords, char *ws, size_t bytes, TreeScratch *out)
{
    const int room = tree_list_room(n_coords);
    if (n_coords > kGroupDims || bytes < w.total + room * tree_slot_bytes(n_coords)) return false;
    size_t slots = (bytes - w.total) / tree_slot_bytes(n_coords);
    const size_t most = kTreeScratchBytes / tree_slot_bytes(n_coords);
    if (slots > most) slots = most;
    out->slots = (int)(slots / room);
    out->list_cap = tree_list_cap(n_coords);
    out->list_room = room * out->list_cap;
    out->list = (int *)(ws + w.total);
    out->list_n = out->list + slots * out->list_cap;
    out->bound = (float *)(out->list_n + slots);
    return true;
}

// Marks in slot 0 of a row that is to be searched again on a grid: several points share its K-th distance and some are left out;
// or only its order would be another one, since it holds equal distances.
constexpr int64_t kTieRow = INT64_MIN, kEqualRow = INT64_MIN + 1;
// Which rows are marked: none; kTieRow only; both, with sorted lists (K <= 65).
enum class TieMarks : int { kNone, kKth, kAny };
// Rows that may be marked and searched again, as a share of all rows (if both kinds together are more, those marked kTieRow): see
// knn_forward_launch.
constexpr int kTieShare = 16;
// Status word between the tree search and the end of the second look when there is nothing to search again:
// the kernels of the grid return at once.
constexpr int32_t kStatusNoGrid = 1 << 30;

// fgc_knn_build_tree; out_order: original ids in curve order, or null; small batches write the two words that the host reads on the way
// (*words is set then).
int knn_build_tree_forward(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K,
                           const int64_t *direction_or_null, int32_t *info_mapped, int32_t *out_order, bool *words, void *workspace,
                           size_t workspace_bytes, fgc_stream_t stream);
// fgc_knn_search_tree; mark_ties: such rows are marked (and have to be searched again on a grid).
int knn_search_tree(int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K,
                    int32_t has_direction, int32_t tf_compat, TieMarks mark_ties, int64_t *out_idx, float *out_distsq,
                    void *workspace, size_t workspace_bytes, fgc_stream_t stream);
// The same for all queries of a leaf at once, directly behind fgc_knn_build_tree, in a workspace with the scratch that
// fgc_knn_forward_workspace_bytes counts in (tree_scratch).
int knn_search_tree_groups(int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K,
                           int32_t has_direction, int32_t tf_compat, TieMarks mark_ties, int64_t *out_idx, float *out_distsq,
                           void *workspace, size_t workspace_bytes, fgc_stream_t stream);
// fgc_knn_build_grid_dims behind a search with mark_ties: builds nothing (kStatusNoGrid) where no row is marked,
// or more than a kTieShare-th of them are (see k_tie_gate).
int knn_build_grid_for_ties(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs,
                            int32_t K, const int64_t *direction_or_null, float target_occupancy, void *workspace,
                            size_t workspace_bytes, fgc_stream_t stream);
// fgc_knn_search; only_marked: rows marked by knn_search_tree only (without a grid the marks are taken off).
int knn_search_grid(int64_t n_vert, int32_t n_coords, int64_t n_rs, int32_t K, int32_t has_direction, int32_t tf_compat,
                    int32_t flags, bool only_marked, int64_t *out_idx, float *out_distsq, void *workspace,
                    size_t workspace_bytes, fgc_stream_t stream);

}  // namespace fgc
