// binned_select_knn forward for sm_100a: the neighbour search on a tree of boxes (knn_tree.cuh).
//
// One warp per query, queries in curve order, so that the warps of a CTA visit the same boxes.
// Top nodes, nodes and leaves are visited nearest box first: 32 lanes compute the distance to 32
// boxes, a warp minimum picks the next one, and a level ends with the first box that is not
// nearer than the current bound on the K-th distance.  A leaf is one step: 32 points, one per lane;
// those below the bound are appended to an array of the warp, which is cut back to the K - 1 nearest
// (and the bound renewed) when it has grown.  The query's own node gives the first bound; all
// other leaves within it are collected first and then visited nearest first, so that few are visited
// that the final bound would have ruled out.
//
// The distance of a box is computed with the operations of dist_sq in the same order.  Rounding is
// monotone, so it never exceeds the computed distance of a point inside: pruning needs no margin and
// the result is exactly the K-1 smallest computed distances, whatever the tree.  Boxes and points at exactly the
// bound are taken until a candidate there has been left out, so that one that equals the K-th distance is always noticed.
//
// In up to five coordinates the forward takes it only for what the search by groups (knn_tree_group.cu) leaves, and in workspaces
// without its scratch; from six on, and in fgc_knn_search_tree, for every query.
//
// What bounds it: issue slots (0.88 of them used; compares, minima and logic run at half rate).  A
// query of 500 k uniform points in three coordinates with K = 64 takes 3350 warp instructions, the 500 k of them 1.67 ms; one of
// 200 k normal points in five with K = 40 takes 11 500, at 0.61 of the issue slots (the last warps run on alone).  Against
// the grid (whole forward without the second look at tied rows): a million normal points in five coordinates, K = 40 26.4 ->
// 18.2 ms; 60 k uniform in eight, K = 20: 3.40 -> 1.5; 400 k normal in six, K = 24 0.78 of its time; 6.4 M uniform in three, K = 64: 18.3 -> 21.5.
//
// Other forms measured: candidates merged into a sorted list 32 at a time instead of selected by
// bisection (28.8 against 22.3 ms, 6.4 M uniform points, K = 64); one query per lane with a column of
// candidates each in shared memory (52 ms: 0.31 of the issue slots, few resident warps); probes of the
// bisection placed by a power law (5.8 against 5.0 ms, 1.6 M points).
#include <type_traits>

#include "knn_list.cuh"
#include "knn_tree_args.cuh"

namespace fgc {

constexpr int kTreeWarps = 8;

// Parameters of the search, measured on B200 (800 k skewed points in three coordinates, K = 128 / 1.6 M
// normal ones in four, K = 40 / 500 k normal ones in five, K = 40; ms):
//  kFirstExtra  candidates beyond the list before the first bound is taken (24: 5.7 / 10.2 / 11.0,
//               64: 5.5 / 9.6 / 10.6)
//  kMoreExtra   candidates beyond the list before the bound is renewed (40: 4.7 / 8.7 / 8.2,
//               64: 4.1 / 8.8 / 8.8)
//  kSpare       entries that may stay above the K-th when the bound is renewed
//  kMaxList     leaves that are collected before the nearest ones are visited (8: 5.8 / 9.4 / 8.4, 16:
//               4.3 / 9.2 / 8.8, 32: 4.1 / 8.8 / 8.8)
constexpr int kFirstExtra = 64, kMoreExtra = 64, kSpare = 8, kMaxList = 32;
// resident CTAs per SM asked of the compiler (1: 5.7 / 10.2 / 11.0; 5 and 6 within 3 %; 6 spills with
// more than four coordinates or K > 129: 1.14 against 0.90 ms for 100 k points, K = 200)
constexpr int tree_ctas(int nv, int r) { return nv > 1 || r > 4 ? 5 : 6; }

// Row split of a position in curve order (positions of a row split are its original range): 32 pivots
// at a time.
__device__ __forceinline__ int warp_row_split_of(const int64_t *__restrict__ rs, int n_rs, int64_t v, int lane)
{
    int lo = 1, hi = n_rs - 1;          // the first index in [lo, hi] with rs[index] > v
    while (lo < hi) {
        const int step = (hi - lo + 31) >> 5;
        const long long p = lo + (long long)lane * step;
        const bool above = p < hi ? __ldg(rs + p) > v : true;
        const unsigned m = __ballot_sync(FGC_FULL_MASK, above);
        const int f = m ? __ffs(m) - 1 : 32;
        const long long nhi = lo + (long long)f * step;
        if (f > 0) lo += (f - 1) * step + 1;
        if (f < 32 && nhi < hi) hi = (int)nhi;
    }
    return lo - 1;
}

// Squared distance to a box (0 inside), rounded like dist_sq.
template <int NV>
__device__ __forceinline__ float box_sq(const float4 (&q)[NV], const float4 *__restrict__ b)
{
    float acc = 0.f;
#pragma unroll
    for (int v = 0; v < NV; v++) {
        const float4 lo = __ldg(b + v), hi = __ldg(b + NV + v);
        const float g0 = fmaxf(fmaxf(__fsub_rn(lo.x, q[v].x), __fsub_rn(q[v].x, hi.x)), 0.f);
        const float g1 = fmaxf(fmaxf(__fsub_rn(lo.y, q[v].y), __fsub_rn(q[v].y, hi.y)), 0.f);
        const float g2 = fmaxf(fmaxf(__fsub_rn(lo.z, q[v].z), __fsub_rn(q[v].z, hi.z)), 0.f);
        const float g3 = fmaxf(fmaxf(__fsub_rn(lo.w, q[v].w), __fsub_rn(q[v].w, hi.w)), 0.f);
        acc = v == 0 ? __fmul_rn(g0, g0) : __fadd_rn(acc, __fmul_rn(g0, g0));
        acc = __fadd_rn(acc, __fmul_rn(g1, g1));
        acc = __fadd_rn(acc, __fmul_rn(g2, g2));
        acc = __fadd_rn(acc, __fmul_rn(g3, g3));
    }
    return acc;
}

// Sort key of box `lane` among 32: its distance with the lane in the low bits (cleared first, so the
// key never exceeds the distance).
__device__ __forceinline__ uint32_t box_key(float d, int lane) { return (__float_as_uint(d) & ~31u) | (uint32_t)lane; }

// The nearest of the 32 boxes that have not been taken yet, or -1 when none is nearer than `beyond`.
__device__ __forceinline__ int next_box(uint32_t &key, uint32_t beyond, int lane)
{
    const uint32_t m = __reduce_min_sync(FGC_FULL_MASK, key);
    if ((m & ~31u) >= beyond) return -1;
    const int src = (int)(m & 31u);
    if (lane == src) key = kNoBox;
    return src;
}

// Candidates of a warp: one unordered array in shared memory.  select() finds the kn-th smallest
// distance by bisection over the bit patterns (each lane holds CAP / 32 entries) and drops the
// entries above it.  R: rows of 32 list entries (kn <= 32 R).
template <int R>
struct BisectSelect {
    static constexpr int CAP = R <= 2 ? 32 * (R + 3) : 64 * R;
    // a leaf is appended as a whole: what may be there before it, plus 32, has to fit
    static_assert(32 * R + kFirstExtra + 31 <= CAP, "array too short for the first bound");
    uint32_t left_out;         // the last distance at which a candidate was left out that equals the bound
    // Points and boxes nearer than this are wanted: everything up to the bound, and once a candidate at the bound has been left
    // out only what is nearer.  Others at it change nothing then, and where many points are equal they would be all that
    // is visited (half of 100 k in three coordinates, K = 64, listed by the search by groups: 10.3 -> 0.34 ms, grid 13.7).
    uint32_t beyond;
    int n;
    // At least kn of the smallest entries stay, at most kn + spare.
    __device__ __forceinline__ void select(float *bd, int *bj, int lane, int kn, int spare)
    {
        constexpr int S = CAP / 32;
        uint32_t v[S];
        int id[S];
        __syncwarp();
        uint32_t lo = kNoBox, hi = 0;
#pragma unroll
        for (int r = 0; r < S; r++) {
            const bool in = r * 32 + lane < n;
            v[r] = in ? __float_as_uint(bd[r * 32 + lane]) : kNoBox;
            id[r] = in ? bj[r * 32 + lane] : -1;
            lo = min(lo, v[r]);
            hi = max(hi, in ? v[r] : 0u);
        }
        lo = __reduce_min_sync(FGC_FULL_MASK, lo);
        hi = __reduce_max_sync(FGC_FULL_MASK, hi);
        int at_most = n;                 // entries <= hi
        while (lo < hi && at_most > kn + spare) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            int c = 0;
#pragma unroll
            for (int r = 0; r < S; r++) c += v[r] <= mid ? 1 : 0;
            c = __reduce_add_sync(FGC_FULL_MASK, c);
            if (c >= kn) { hi = mid; at_most = c; } else lo = mid + 1;
        }
        int equal = CAP;                 // entries equal to hi that may stay
        if (at_most > kn + spare) {
            int below = 0;
#pragma unroll
            for (int r = 0; r < S; r++) below += v[r] < hi ? 1 : 0;
            equal = kn - __reduce_add_sync(FGC_FULL_MASK, below);
            left_out = hi;
        }
        beyond = hi + (equal < CAP ? 0u : 1u);
        int to = 0;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < S; r++) {
            bool keep = v[r] <= hi;
            if (equal < CAP) {
                const unsigned same = __ballot_sync(FGC_FULL_MASK, v[r] == hi);
                keep = v[r] < hi || (v[r] == hi && __popc(same & lanemask_lt()) < equal);
                equal -= min(equal, __popc(same));
            }
            const unsigned m = __ballot_sync(FGC_FULL_MASK, keep);
            if (keep) {
                const int at = to + __popc(m & lanemask_lt());
                bd[at] = __uint_as_float(v[r]);
                bj[at] = id[r];
            }
            to += __popc(m);
        }
        n = to;
        __syncwarp();
    }
    __device__ __forceinline__ void add(float *bd, int *bj, int lane, unsigned m, float d, int j)
    {
        if (m >> lane & 1) {
            const int at = n + __popc(m & lanemask_lt());
            bd[at] = d;
            bj[at] = j;
        }
        n += __popc(m);
    }
};

// Ascending order of one key per lane, and of two ascending runs of 32 as one of 64.
__device__ __forceinline__ void sort_keys(uint32_t &k, int lane)
{
#pragma unroll
    for (int m = 2; m <= 32; m <<= 1)
#pragma unroll
        for (int jj = m >> 1; jj > 0; jj >>= 1) {
            const uint32_t o = __shfl_xor_sync(FGC_FULL_MASK, k, jj);
            const bool smaller = m == 32 ? (lane & jj) == 0 : ((lane & jj) != 0) == ((lane & m) != 0);
            k = smaller ? min(k, o) : max(k, o);
        }
}
__device__ __forceinline__ void merge_keys(uint32_t &a, uint32_t &b, int lane)
{
    const uint32_t r = __shfl_sync(FGC_FULL_MASK, b, 31 - lane);
    b = max(a, r);
    a = min(a, r);
#pragma unroll
    for (int jj = 16; jj > 0; jj >>= 1) {
        const uint32_t oa = __shfl_xor_sync(FGC_FULL_MASK, a, jj), ob = __shfl_xor_sync(FGC_FULL_MASK, b, jj);
        a = (lane & jj) == 0 ? min(a, oa) : max(a, oa);
        b = (lane & jj) == 0 ? min(b, ob) : max(b, ob);
    }
}

// Rows of points without neighbours: bad input, no tree was built.
__device__ __forceinline__ void default_row(const TreeArgs &a, int qi)
{
    const int64_t pad = a.tf_compat ? (int64_t)qi : (int64_t)-1;
    for (int s = threadIdx.x & 31; s < a.K; s += 32) {
        a.out_idx[(size_t)qi * a.K + s] = s == 0 ? (int64_t)qi : pad;
        a.out_dist[(size_t)qi * a.K + s] = 0.f;
    }
}

// One query by one warp.
template <int NV, int R>
__device__ __forceinline__ void tree_query(const TreeArgs &a, int qi)
{
    using Select = BisectSelect<R>;
    __shared__ float s_d[kTreeWarps][Select::CAP];
    __shared__ int s_j[kTreeWarps][Select::CAP];
    __shared__ int s_leaf[kTreeWarps][64];
    __shared__ uint32_t s_key[kTreeWarps][64];
    static_assert(kMaxList + 32 <= 64, "leaf list too short");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int K = a.K, kn = K - 1;
    const int orig_q = __ldg(a.sorig + qi);
    if (!FGC_DBG_OK(orig_q >= 0 && orig_q < a.n_vert, &a.grid->status)) return;
    const uint8_t *__restrict__ sflag = a.sflag;
    float *bd = s_d[w];
    int *bj = s_j[w];
    int *lleaf = s_leaf[w];
    uint32_t *lkey = s_key[w];
    Select sel;
    sel.beyond = kInfBits;
    sel.left_out = kNoBox;
    sel.n = 0;
    if (kn > 0 && !(sflag && (sflag[qi] == 0 || sflag[qi] == 2))) {
        float4 q[NV];
#pragma unroll
        for (int v = 0; v < NV; v++) q[v] = __ldg(a.scoords + (size_t)qi * NV + v);
        const int e = warp_row_split_of(a.row_splits, a.n_rs, qi, lane);
        const int ev_begin = (int)__ldg(a.row_splits + e), n_e = (int)__ldg(a.row_splits + e + 1) - ev_begin;
        const int n_leaf = (n_e + 31) >> 5, n_node = (n_e + 1023) >> 10, n_top = (n_e + 32767) >> 15;
        const float4 *leaf_box = a.box[0] + (size_t)tree_base(ev_begin, e, 5) * (2 * NV);
        const float4 *node_box = a.box[1] + (size_t)tree_base(ev_begin, e, 10) * (2 * NV);
        const float4 *top_box = a.box[2] + (size_t)tree_base(ev_begin, e, 15) * (2 * NV);
        auto visit = [&](int leaf) {
            const int rel = leaf * 32 + lane;
            const int j = ev_begin + rel;
            float dc = __uint_as_float(kInfBits);
            if (rel < n_e && j != qi) {
                float4 c[NV];
#pragma unroll
                for (int v = 0; v < NV; v++) c[v] = __ldg(a.scoords + (size_t)j * NV + v);
                dc = dist_sq<NV>(q, c, 0);
                if (sflag) { const uint8_t f = sflag[j]; if (f == 1 || f == 2) dc = __uint_as_float(kInfBits); }
            }
            const unsigned m = __ballot_sync(FGC_FULL_MASK, __float_as_uint(dc) < sel.beyond);
            if (m) sel.add(bd, bj, lane, m, dc, j);
        };
        // First bound: the nearest leaves of the query's own node, until there are kFirstExtra
        // candidates more than the list needs.
        const int own = (qi - ev_begin) >> 10;
        unsigned seen = 0;
        {
            uint32_t key0 = kNoBox;
            const int mine = own * 32 + lane;
            if (mine < n_leaf) key0 = box_key(box_sq<NV>(q, leaf_box + (size_t)mine * (2 * NV)), lane);
            for (int c0; sel.n < kn + kFirstExtra && (c0 = next_box(key0, kInfBits, lane)) >= 0;) {
                seen |= 1u << c0;
                visit(own * 32 + c0);
            }
            if (sel.n > kn) sel.select(bd, bj, lane, kn, kSpare);
        }
        // Then all other leaves that the bound reaches: collected node by node, visited nearest first.
        int n_list = 0;
        auto flush = [&]() {
            __syncwarp();
            uint32_t k0 = lane < n_list ? lkey[lane] : kNoBox, k1 = kNoBox;
            sort_keys(k0, lane);
            if (n_list > 32) {
                k1 = 32 + lane < n_list ? lkey[32 + lane] : kNoBox;
                sort_keys(k1, lane);
                merge_keys(k0, k1, lane);
            }
            for (int i = 0; i < n_list; i++) {
                const uint32_t k = __shfl_sync(FGC_FULL_MASK, i < 32 ? k0 : k1, i & 31);
                if ((k & ~63u) >= sel.beyond) break;
                visit(lleaf[k & 63u]);
                if (sel.n > Select::CAP - 32 || sel.n > kn + kMoreExtra) sel.select(bd, bj, lane, kn, kSpare);
            }
            n_list = 0;
            __syncwarp();
        };
        // top nodes 32 at a time, first the 32 (a million points) around the query
        const int n_group = (n_top + 31) >> 5, own_group = own >> 10;
        for (int gi = 0; gi < n_group; gi++) {
            const int group = gi == 0 ? own_group : (gi <= own_group ? gi - 1 : gi);
            uint32_t key2 = kNoBox;
            const int mine2 = group * 32 + lane;
            if (mine2 < n_top) key2 = n_top == 1 ? (uint32_t)lane : box_key(box_sq<NV>(q, top_box + (size_t)mine2 * (2 * NV)), lane);
            for (int c2; (c2 = next_box(key2, sel.beyond, lane)) >= 0;) {
                const int mine1 = (group * 32 + c2) * 32 + lane;
                uint32_t key1 = kNoBox;
                if (mine1 < n_node) key1 = n_node == 1 ? (uint32_t)lane : box_key(box_sq<NV>(q, node_box + (size_t)mine1 * (2 * NV)), lane);
                for (int c1; (c1 = next_box(key1, sel.beyond, lane)) >= 0;) {
                    const int node = (group * 32 + c2) * 32 + c1;
                    const int leaf = node * 32 + lane;
                    uint32_t d0 = kNoBox;
                    if (leaf < n_leaf && !(node == own && (seen >> lane & 1)))
                        d0 = __float_as_uint(box_sq<NV>(q, leaf_box + (size_t)leaf * (2 * NV)));
                    const bool want = d0 < sel.beyond;
                    const unsigned m = __ballot_sync(FGC_FULL_MASK, want);
                    if (want) {
                        const int at = n_list + __popc(m & lanemask_lt());
                        lleaf[at] = leaf;
                        lkey[at] = (d0 & ~63u) | (uint32_t)at;
                    }
                    n_list += __popc(m);
                    if (n_list > kMaxList) flush();
                }
            }
        }
        if (n_list > 0) flush();
        if (sel.n > (R <= 2 ? 32 * R : kn)) sel.select(bd, bj, lane, kn, R <= 2 ? 32 * R - kn : 0);
        __syncwarp();
    }
    int64_t *__restrict__ out_i = a.out_idx + (size_t)orig_q * K;
    float *__restrict__ out_d = a.out_dist + (size_t)orig_q * K;
    uint32_t last = 0;                       // the K-th distance (0: the list is not full)
    bool tie = false, same = false;
    const int64_t pad = a.tf_compat ? (int64_t)orig_q : (int64_t)-1;
    if constexpr (R <= 2) {
        // ascending distances
        SortedList<R> list;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int s = r * 32 + lane;
            list.d[r] = s < sel.n ? bd[s] : __uint_as_float(kInfBits);
            list.id[r] = s < sel.n ? bj[s] : -1;
            if (r * 32 < sel.n) sort32(list.d[r], list.id[r], lane);
        }
        if (R == 2 && sel.n > 32) list.merge_halves(lane);
        if (sel.n >= kn && kn > 0) {
            last = __float_as_uint(__shfl_sync(FGC_FULL_MASK, kn > 32 ? list.d[R - 1] : list.d[0], (kn - 1) & 31));
            // an entry behind the list that equals its last one
#pragma unroll
            for (int r = 0; r < R; r++)
                tie = tie || __any_sync(FGC_FULL_MASK, r * 32 + lane >= kn && __float_as_uint(list.d[r]) == last && list.id[r] >= 0);
        }
        if (a.mark_ties == TieMarks::kAny) same = equal_in_list<R>(list.d, list.id, kn, lane);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int s = r * 32 + lane;
            if (s < kn) {
                const bool filled = list.id[r] >= 0;
                out_i[1 + s] = filled ? (int64_t)__ldg(a.sorig + list.id[r]) : pad;
                out_d[1 + s] = filled ? list.d[r] : 0.f;
            }
        }
    } else {
        for (int s = lane; s < kn; s += 32) {
            const bool filled = s < sel.n;
            out_i[1 + s] = filled ? (int64_t)__ldg(a.sorig + bj[s]) : pad;
            out_d[1 + s] = filled ? bd[s] : 0.f;
            if (filled) last = max(last, __float_as_uint(bd[s]));
        }
        last = __reduce_max_sync(FGC_FULL_MASK, last);
        if (sel.n < kn) last = 0;
    }
    tie = tie || (kn > 0 && sel.n >= kn && last == sel.left_out);
    if (lane == 0) {
        out_i[0] = mark_row(a, tie, same, orig_q);
        out_d[0] = 0.f;
    }
}

template <int NV, int R>
__global__ void __launch_bounds__(kTreeWarps * 32, tree_ctas(NV, R))
k_knn_tree(const TreeArgs a)
{
    chain_wait();
    chain_release();
    const int64_t qi = (int64_t)blockIdx.x * kTreeWarps + (threadIdx.x >> 5);          // position in curve order
    if (qi >= a.n_vert) return;
    if (a.tree->magic != kTreeMagic) {                                    // not a tree: nothing is walked
        if (qi == 0 && threadIdx.x == 0) atomicOr(&a.grid->status, FGC_STATUS_INTERNAL);
        return;
    }
    if (a.grid->status != 0) default_row(a, (int)qi);
    else tree_query<NV, R>(a, (int)qi);
}

// The listed queries, usually few.  A warp takes the next one when it has finished its last: they differ by orders of
// magnitude (half of 400 k points in a cloud a millionth as wide as the rest, three coordinates, K = 64: 157 -> 95 ms, the search one
// query at a time for all of them 104).
template <int NV, int R>
__global__ void __launch_bounds__(kTreeWarps * 32, tree_ctas(NV, R))
k_knn_tree_listed(const TreeArgs a)
{
    chain_wait();
    chain_release();
    if (a.grid->status != 0) return;
    const int n = min(a.tree->n_listed, a.n_vert);
    if (n == 0) return;
    for (;;) {
        int i = 0;
        if ((threadIdx.x & 31) == 0) i = atomicAdd(&a.tree->next_listed, 1);
        i = __shfl_sync(FGC_FULL_MASK, i, 0);
        if (i >= n) return;
        const int qi = a.listed[i];
        if (FGC_DBG_OK(qi >= 0 && qi < a.n_vert, &a.grid->status)) tree_query<NV, R>(a, qi);
        __syncwarp();
    }
}

template <int NV>
static cudaError_t launch_listed(const TreeArgs &a, cudaStream_t s)
{
    const int rows = tree_list_rows(a.K), T = kTreeWarps * 32;
    const unsigned blocks = (unsigned)(sm_count() * tree_ctas(NV, rows));
    switch (rows) {
    case 1: return launch_chained(k_knn_tree_listed<NV, 1>, blocks, T, 0, s, a);
    case 2: return launch_chained(k_knn_tree_listed<NV, 2>, blocks, T, 0, s, a);
    case 4: return launch_chained(k_knn_tree_listed<NV, 4>, blocks, T, 0, s, a);
    default: return launch_chained(k_knn_tree_listed<NV, 8>, blocks, T, 0, s, a);
    }
}

int launch_tree_listed(const TreeArgs &a, int nv, cudaStream_t s)
{
    return (int)(nv == 1 ? launch_listed<1>(a, s) : launch_listed<2>(a, s));
}

template <int NV>
static cudaError_t launch_tree(const TreeArgs &a, cudaStream_t s)
{
    const unsigned blocks = (unsigned)(((int64_t)a.n_vert + kTreeWarps - 1) / kTreeWarps);
    const int kn = a.K - 1, T = kTreeWarps * 32;
    if (kn <= 32) return launch_chained(k_knn_tree<NV, 1>, blocks, T, 0, s, a);
    if (kn <= 64) return launch_chained(k_knn_tree<NV, 2>, blocks, T, 0, s, a);
    if (kn <= 128) return launch_chained(k_knn_tree<NV, 4>, blocks, T, 0, s, a);
    return launch_chained(k_knn_tree<NV, 8>, blocks, T, 0, s, a);
}

int tree_args(int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K, int32_t has_direction,
              int32_t tf_compat, TieMarks mark_ties, int64_t *out_idx, float *out_distsq, void *workspace, size_t workspace_bytes,
              TreeArgs *a, KnnWorkspace *L, TreeLayout *T)
{
    const int rc = check_knn_args(n_vert, n_coords, n_rs, K, workspace, workspace_bytes, L);
    if (rc != FGC_OK) return rc;
    if (n_vert == 0) return FGC_OK;
    if (!row_splits || n_rs < 2 || !out_idx || !out_distsq) return FGC_ERR_BAD_ARGUMENT;
    *T = tree_layout(*L, n_vert, n_coords, n_rs);
    if (!T->fits) return FGC_ERR_TOO_LARGE;
    char *ws = (char *)workspace;
    *a = TreeArgs();
    a->scoords = (const float4 *)(ws + L->scoords);
    a->sorig = (const int *)(ws + L->sorig);
    a->sflag = has_direction ? (const uint8_t *)(ws + L->sflag) : nullptr;
    for (int l = 0; l < 3; l++) a->box[l] = (const float4 *)(ws + T->box[l]);
    a->row_splits = row_splits;
    a->grid = (KnnGrid *)(ws + L->header);
    a->tree = (KnnTree *)(ws + L->tickets);
    a->out_idx = out_idx;
    a->out_dist = out_distsq;
    a->n_vert = (int)n_vert;
    a->n_rs = (int)n_rs;
    a->K = K;
    a->tf_compat = tf_compat;
    a->mark_ties = mark_ties;
    return FGC_OK;
}

}  // namespace fgc

extern "C" int fgc_knn_search_tree(int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K,
                                   int32_t has_direction, int32_t tf_compat, int64_t *out_idx, float *out_distsq,
                                   void *workspace, size_t workspace_bytes, fgc_stream_t stream)
{
    return fgc::knn_search_tree(n_vert, n_coords, row_splits, n_rs, K, has_direction, tf_compat, fgc::TieMarks::kNone, out_idx, out_distsq,
                                workspace, workspace_bytes, stream);
}

int fgc::knn_search_tree(int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K,
                         int32_t has_direction, int32_t tf_compat, TieMarks mark_ties, int64_t *out_idx, float *out_distsq,
                         void *workspace, size_t workspace_bytes, fgc_stream_t stream)
{
    FGC_NVTX("fgc_knn_search_tree");
    using namespace fgc;
    TreeArgs a;
    KnnWorkspace L;
    TreeLayout T;
    const int rc = tree_args(n_vert, n_coords, row_splits, n_rs, K, has_direction, tf_compat, mark_ties, out_idx, out_distsq, workspace,
                             workspace_bytes, &a, &L, &T);
    if (rc != FGC_OK || n_vert == 0) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (L.nv == 1) FGC_RETURN_IF_CUDA(launch_tree<1>(a, s));
    else if (L.nv == 2) FGC_RETURN_IF_CUDA(launch_tree<2>(a, s));
    else if (L.nv == 3) FGC_RETURN_IF_CUDA(launch_tree<3>(a, s));
    else FGC_RETURN_IF_CUDA(launch_tree<4>(a, s));
    return FGC_OK;
}
