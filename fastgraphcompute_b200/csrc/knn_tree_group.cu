// binned_select_knn forward for sm_100a: the search on a tree of boxes (knn_tree.cuh) in two kernels, the first of which
// works for the 32 queries of a leaf at once.  They are neighbours on the curve and have nearly the same candidates, so
// what one query per warp spends most of its instructions on (knn_tree_search.cu: finding its bound by repeated
// selection, and walking the levels of the tree) is paid once for 32.
//
//  k_tree_groups  One warp per leaf.  The points of the leaves nearest to its own are counted by distance for every query
//                 (32 classes, eight to a factor of two); the class in which the K-th falls gives an upper bound on its K-th
//                 distance.  |c|^2 - 2 c.q + |q|^2, with coordinates relative to the leaf, is a product of 32 queries x 32 points
//                 over two more places than there are coordinates: a few matrix instructions in tf32, |c|^2 in two parts.
//                 The bound is widened by what rounding can add, so it stays an upper bound.  Then the leaves whose box is
//                 within the largest of the bounds are listed.
//  k_tree_rows    One warp per query.  It compares its own bound with the boxes of the list, visits those within it, keeps
//                 the points within it -- distances by dist_sq, which is what is returned -- and sorts them (K <= 65)
//                 or selects the K - 1 smallest.  On uniform data a quarter more points than K pass.
//
// The distance of two boxes, or of a point and a box, is computed with the operations of dist_sq in the same order.  Rounding is
// monotone, so it never exceeds the computed distance of two points inside: pruning needs no margin and
// the result is exactly the K-1 smallest computed distances, whatever the tree.  Boxes and points at exactly the bound
// are taken until a candidate equal to it has been left out, so that one that equals the K-th distance is always noticed.
//
// What bounds them (a million uniform points in ten row splits, three coordinates, K = 64, ncu): k_tree_rows issue slots (0.79 of them
// used, 1490 warp instructions a query, arithmetic pipe 0.70; 46 registers, 57 % of the warps resident), k_tree_groups the shared-memory
// pipe (0.93; the counting's atomics meet in banks; 190 instructions a query; 72 registers and 60 bytes of them spilled, 28 one-warp CTAs
// an SM).  Whole forward / one query at a time / the grid, ms, without a second look in the first two: 6.4 M uniform points in three
// coordinates, K = 64 13.5 / 21.5 / 18.3; 1.6 M learned ones in four, K = 40 6.6 / 9.4 / 8.4; 800 k skewed in three, K = 128 3.0 / 4.6 / 18.8; a
// million normal ones in five, K = 40 15.0 / 18.2 / 26.4.  The second look adds 0.85, 0.4, 1.5 and 0.4.
//
// Other splits of the work, measured on the first and the third of these (then 13.9 and 3.2): one kernel, a lane per query, the points of a leaf read from
// shared memory by all 32 lanes (15.5; broadcast 16-byte loads write 512 bytes back each, four cycles an SM); candidates of all
// 32 queries filtered by the matrix product and kept in the workspace, a second kernel for the rows (15.7 and 7.8: leaves that
// visit thousands of others run on alone).
//
// A leaf far larger than the distances of its neighbours (points far apart that happen to follow one another on the curve)
// would list too many leaves: its queries are searched one by one (knn_tree_search.cu).
#include "knn_list.cuh"
#include "knn_tree_args.cuh"

namespace fgc {

// Row split of leaf slot s: the largest e with tree_base(row_splits[e], e, 5) <= s, 32 pivots at a time.
__device__ __forceinline__ int warp_event_of_leaf(const int64_t *__restrict__ rs, int n_rs, int64_t s, int lane)
{
    int lo = 1, hi = n_rs - 1;          // the first index in [lo, hi] that begins behind s (n_rs - 1: none before it)
    while (lo < hi) {
        const int step = (hi - lo + 31) >> 5;
        const long long p = lo + (long long)lane * step;
        const bool behind = p < hi ? tree_base(__ldg(rs + p), p, 5) > s : true;
        const unsigned m = __ballot_sync(FGC_FULL_MASK, behind);
        const int f = m ? __ffs(m) - 1 : 32;
        const long long nhi = lo + (long long)f * step;
        if (f > 0) lo += (f - 1) * step + 1;
        if (f < 32 && nhi < hi) hi = (int)nhi;
    }
    return lo - 1;
}

// Squared distance between two boxes (0 where they touch), rounded like dist_sq.  A point is a box without extent.
template <int NV>
__device__ __forceinline__ float box_box_sq(const float4 (&lo)[NV], const float4 (&hi)[NV], const float4 *__restrict__ box)
{
    float acc = 0.f;
#pragma unroll
    for (int v = 0; v < NV; v++) {
        const float4 bl = __ldg(box + v), bh = __ldg(box + NV + v);
        const float g0 = fmaxf(fmaxf(__fsub_rn(bl.x, hi[v].x), __fsub_rn(lo[v].x, bh.x)), 0.f);
        const float g1 = fmaxf(fmaxf(__fsub_rn(bl.y, hi[v].y), __fsub_rn(lo[v].y, bh.y)), 0.f);
        const float g2 = fmaxf(fmaxf(__fsub_rn(bl.z, hi[v].z), __fsub_rn(lo[v].z, bh.z)), 0.f);
        const float g3 = fmaxf(fmaxf(__fsub_rn(bl.w, hi[v].w), __fsub_rn(lo[v].w, bh.w)), 0.f);
        acc = v == 0 ? __fmul_rn(g0, g0) : __fadd_rn(acc, __fmul_rn(g0, g0));
        acc = __fadd_rn(acc, __fmul_rn(g1, g1));
        acc = __fadd_rn(acc, __fmul_rn(g2, g2));
        acc = __fadd_rn(acc, __fmul_rn(g3, g3));
    }
    return acc;
}

// ----------------------------------------------------------------------------- bounds and lists

constexpr int kHistClasses = 32;
// Leaves that the bound is taken from: more make it tighter.
// Measured with 5 / 8 / 12 / 16 / 24 / 36 of them (400 k points, whole forward, ms): uniform in three coordinates, K = 16 0.67 / 0.67 /
// 0.69 / 0.71 / 0.76 / 0.82, K = 64 1.15 / 1.07 / 1.04 / 1.05 / 1.09 / 1.18, K = 200 6.3 / 2.6 / 2.3 / 2.23 / 2.18 / 2.22; four learned
// coordinates, K = 40 2.06 / 1.94 / 1.89 / 1.88 / 1.93 / 1.98; five, normal, K = 40 8.4 / 7.8 / 7.3 / 7.2 / 7.1 / 7.1.
constexpr int kSeedNodes = 4;
__device__ __forceinline__ int seed_leaves(int kn, int dims)
{
    return min(4 + kn / 6, 28) + (dims >= 4 ? 6 : 0) + (dims >= 5 ? 6 : 0);
}

// An upper bound on the distance d of a point c from q whose |c|^2 - 2 c.q + |q|^2 comes out as t or less (coordinates relative to
// some centre, |q|^2 = q2).  |c| is at most |q| + sqrt(d).  Both operands are rounded to tf32, 2^-11 of their size: e(d) = 2^-9 |q| (|q| +
// sqrt(d)) on 2 c.q.  Everything else is in single precision or split in two: at most 50 operations that are off by 2^-23 of
// (|q| + |c|)^2.  So d <= t + e(d).  The sum T below has sqrt(t) in the place of sqrt(d): |q| + sqrt(T) is at most 1.057 (|q| + sqrt(t)),
// since T - t is 0.0032 |q| (|q| + sqrt(t)) and a little, so e(T) <= 0.0021 |q| (|q| + sqrt(t)) is less than T - t, and beyond T e grows
// by less than a fiftieth of d: no larger d fits.  The last term is for squares that underflow.
__device__ __forceinline__ float widened(float t, float q2)
{
    const float q = sqrtf(q2), c = q + sqrtf(t), s = q + c;
    return t + 0.0032f * q * c + 6e-6f * s * s + 1e-36f;
}

// |c|^2 of what is no candidate; with cross terms of up to 2e36 (coordinates up to 1e18) still above 0x7e900000 = 9.6e37.
constexpr float kNotThere = 1e38f;

// d = a * b + d for a tile of 16 x 8 over 8 places, tf32
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int NV, int DC>
__device__ __forceinline__ void bound_leaf(const TreeArgs &a, const int slot)
{
    static_assert(DC + 2 <= 8, "one matrix product over coordinates and |c|^2 twice");
    constexpr int CHUNKS = (DC + 3) / 4;
    __shared__ __align__(16) int s_hist[32 * (kHistClasses + 1)];
    const int lane = threadIdx.x & 31;
    const int kn = a.K - 1;
    const uint8_t *__restrict__ sflag = a.sflag;
    const int place = slot - a.slot0;                                       // of the leaf in the scratch

    const int e = warp_event_of_leaf(a.row_splits, a.n_rs, slot, lane);
    const int ev_begin = (int)__ldg(a.row_splits + e), n_e = (int)__ldg(a.row_splits + e + 1) - ev_begin;
    const int own_leaf = slot - (int)tree_base(ev_begin, e, 5);
    if (own_leaf < 0 || (long long)own_leaf * 32 >= n_e) {                    // a slot without points
        if (lane == 0) a.list_n[place] = -1;
        return;
    }
    const int n_leaf = (n_e + 31) >> 5, n_node = (n_e + 1023) >> 10, n_top = (n_e + 32767) >> 15;
    const float4 *leaf_box = a.box[0] + (size_t)tree_base(ev_begin, e, 5) * (2 * NV);
    const float4 *node_box = a.box[1] + (size_t)tree_base(ev_begin, e, 10) * (2 * NV);
    const float4 *top_box = a.box[2] + (size_t)tree_base(ev_begin, e, 15) * (2 * NV);
    const int rel_q = own_leaf * 32 + lane;
    const bool valid = rel_q < n_e;
    const int qi = ev_begin + (valid ? rel_q : n_e - 1);
    bool active = valid && kn > 0;
    if (sflag && (sflag[qi] == 0 || sflag[qi] == 2)) active = false;
    if (!__any_sync(FGC_FULL_MASK, active)) {            // no query of the leaf may have neighbours
        a.bound[place * 32 + lane] = kNoQuery;
        if (lane == 0) a.list_n[place] = 0;
        return;
    }

    float4 glo[NV], ghi[NV];
    float t = __uint_as_float(kInfBits);         // bound: at least kn candidates are this near
#pragma unroll
    for (int v = 0; v < NV; v++) {
        glo[v] = __ldg(leaf_box + (size_t)own_leaf * (2 * NV) + v);
        ghi[v] = __ldg(leaf_box + (size_t)own_leaf * (2 * NV) + NV + v);
    }
    if (n_e - 1 > kn) {
        float4 q[NV], mid[NV];
        float diag = 0.f;
#pragma unroll
        for (int v = 0; v < NV; v++) {
            q[v] = __ldg(a.scoords + (size_t)qi * NV + v);
            mid[v] = make_float4(0.5f * glo[v].x + 0.5f * ghi[v].x, 0.5f * glo[v].y + 0.5f * ghi[v].y,
                                 0.5f * glo[v].z + 0.5f * ghi[v].z, 0.5f * glo[v].w + 0.5f * ghi[v].w);
            const float dx = ghi[v].x - glo[v].x, dy = ghi[v].y - glo[v].y, dz = ghi[v].z - glo[v].z, dw = ghi[v].w - glo[v].w;
            diag += dx * dx + dy * dy + dz * dz + dw * dw;
        }
        // Tiles of 32 queries x 32 points.  Lane 4 g + p holds, of the queries, rows g, g + 8, g + 16 and g + 24 at places p
        // and p + 4, of the points column g of four tiles at the same places, and of the result the same rows at columns 2 p
        // and 2 p + 1.  Places: the coordinates, then |c|^2 in two parts.
        const int g4 = lane >> 2, p4 = lane & 3;
        float mid_p[CHUNKS], q2 = 0.f;
#pragma unroll
        for (int i = 0; i < CHUNKS; i++) mid_p[i] = p4 == 0 ? mid[i].x : (p4 == 1 ? mid[i].y : (p4 == 2 ? mid[i].z : mid[i].w));
        uint32_t qa[2][4];
        {
            float *sq = reinterpret_cast<float *>(s_hist);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                float y = k < DC + 2 ? 1.f : 0.f;
                if (k < DC) {
                    const float4 &x = q[k < DC ? k / 4 : 0], &o = mid[k < DC ? k / 4 : 0];
                    y = k % 4 == 0 ? x.x - o.x : (k % 4 == 1 ? x.y - o.y : (k % 4 == 2 ? x.z - o.z : x.w - o.w));
                    q2 = fmaf(y, y, q2);
                    y *= -2.f;
                }
                sq[k * 32 + lane] = y;
            }
            __syncwarp();
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int r = 0; r < 4; r++)
                    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(qa[m][r]) : "f"(sq[(p4 + 4 * (r >> 1)) * 32 + 16 * m + g4 + 8 * (r & 1)]));
            __syncwarp();
        }
        for (int i = lane; i < 32 * (kHistClasses + 1); i += 32) s_hist[i] = 0;
        // Classes are the upper bits of a distance: eight to a factor of two, the last one and what is beyond it without an
        // end.  The K-th distance of a point in a leaf of 32 is a tenth to a half of the leaf's squared diagonal at K =
        // 16 to 128 and more at a border: four factors of two up to twice it, less for short lists.  The last class begins below
        // kNotThere, so that what is no candidate is never counted below it, however large the leaf.
        const float share = kn >= 63 ? 2.f : 2.f * powf((float)(kn + 1) * (1.f / 64.f), 2.f / DC);
        const int last = (int)min(__float_as_uint(share * diag), 0x7e800000u) >> 20;
        const int first = max(last - (kHistClasses - 1), 0);
        // the nearest leaves of the nearest nodes
        const int own_node = own_leaf >> 5, node0 = own_node & ~31;
        uint32_t nkey = kNoBox, lkey[kSeedNodes];
        int node_of[kSeedNodes];
        if (node0 + lane < n_node)
            nkey = node0 + lane == own_node ? (uint32_t)lane
                   : ((__float_as_uint(box_box_sq<NV>(mid, mid, node_box + (size_t)(node0 + lane) * (2 * NV))) & ~31u) | (uint32_t)lane);
#pragma unroll
        for (int k = 0; k < kSeedNodes; k++) {
            const uint32_t m = __reduce_min_sync(FGC_FULL_MASK, nkey);
            lkey[k] = kNoBox;
            node_of[k] = node0 + (int)(m & 31u);
            if (m != kNoBox) {
                if (lane == (int)(m & 31u)) nkey = kNoBox;
                const int leaf = node_of[k] * 32 + lane;
                if (leaf < n_leaf)
                    lkey[k] = (__float_as_uint(box_box_sq<NV>(mid, mid, leaf_box + (size_t)leaf * (2 * NV))) & ~127u) |
                              (uint32_t)(k << 5 | lane);
            }
        }
        __syncwarp();
        auto next_seed = [&]() -> int {
            uint32_t m = lkey[0];
#pragma unroll
            for (int k = 1; k < kSeedNodes; k++) m = min(m, lkey[k]);
            m = __reduce_min_sync(FGC_FULL_MASK, m);
            if (m == kNoBox) return -1;
            const int src = (int)(m & 31u), from = (int)(m >> 5 & 3u);
            int node = node_of[0];
#pragma unroll
            for (int k = 0; k < kSeedNodes; k++) {
                if (k == from) {
                    if (lane == src) lkey[k] = kNoBox;
                    node = node_of[k];
                }
            }
            return node * 32 + src;
        };
        const float *points = reinterpret_cast<const float *>(a.scoords + (size_t)ev_begin * NV);
        auto load = [&](int leaf, float (&c)[4][CHUNKS]) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int rel = min(leaf * 32 + 8 * j + g4, n_e - 1);
                if (!FGC_DBG_OK(rel >= 0 && ev_begin + rel < a.n_vert, &a.grid->status)) continue;
#pragma unroll
                for (int i = 0; i < CHUNKS; i++) c[j][i] = __ldg(points + (size_t)rel * (4 * NV) + 4 * i + p4);
            }
        };
        float h[4], c[4][CHUNKS] = {};
#pragma unroll
        for (int i = 0; i < 4; i++) h[i] = __shfl_sync(FGC_FULL_MASK, q2, g4 + 8 * i);
        int *mine = s_hist + g4 * (kHistClasses + 1) - first;
        const int lo_bits = first << 20, hi_bits = (first + kHistClasses - 1) << 20;
        const int n_seed = seed_leaves(kn, DC);
        int leaf = next_seed();
        if (leaf >= 0) load(leaf, c);
        for (int i = 0; i < n_seed && leaf >= 0; i++) {
            const int left = n_e - leaf * 32;
            unsigned there = left >= 32 ? FGC_FULL_MASK : (1u << left) - 1u;
            if (sflag) {
                const uint8_t f = lane < left ? sflag[ev_begin + leaf * 32 + lane] : (uint8_t)1;
                there = __ballot_sync(FGC_FULL_MASK, f != 1 && f != 2);
            }
            float f[2][4][4];
            bool wide = false;                   // a point too far away to be squared
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float y[CHUNKS], c2 = 0.f;
#pragma unroll
                for (int i4 = 0; i4 < CHUNKS; i4++) {
                    y[i4] = c[j][i4] - mid_p[i4];
                    c2 = fmaf(y[i4], y[i4], c2);
                }
                c2 += __shfl_xor_sync(FGC_FULL_MASK, c2, 1);
                c2 += __shfl_xor_sync(FGC_FULL_MASK, c2, 2);
                wide = wide || !(c2 <= 1e36f);
                if (!(there >> (8 * j + g4) & 1)) c2 = kNotThere;
                const float c2_high = __uint_as_float(__float_as_uint(c2) & 0xffffe000u), c2_low = c2 - c2_high;
                uint32_t b[2];
#pragma unroll
                for (int i4 = 0; i4 < 2; i4++) {
                    float z = 4 * i4 + p4 == DC ? c2_high : (4 * i4 + p4 == DC + 1 ? c2_low : 0.f);
                    if (i4 < CHUNKS && 4 * i4 + p4 < DC) z = y[i4 < CHUNKS ? i4 : 0];
                    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(b[i4]) : "f"(z));
                }
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    f[m][j][0] = f[m][j][1] = h[2 * m];
                    f[m][j][2] = f[m][j][3] = h[2 * m + 1];
                    mma_tf32(f[m][j], qa[m], b[0], b[1]);
                }
            }
            const bool usable = !__any_sync(FGC_FULL_MASK, wide);
            leaf = next_seed();
            if (leaf >= 0) load(leaf, c);
            if (!usable) continue;
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int b = min(max(__float_as_int(f[m][j][k]), lo_bits), hi_bits) >> 20;
                        atomicAdd(mine + (16 * m + 8 * (k >> 1)) * (kHistClasses + 1) + b, 1);
                    }
        }
        __syncwarp();
        // the query itself is among those counted, or the bound is a place too far
        int below = 0, classes = 0;
#pragma unroll 16
        for (int b = 0; b < kHistClasses; b++) {
            below += s_hist[lane * (kHistClasses + 1) + b];
            classes += below <= kn ? 1 : 0;
        }
        if (classes < kHistClasses - 1 && q2 <= 1e36f) {
            t = widened(__uint_as_float((uint32_t)(first + classes + 1) << 20), q2);
            if (!is_finite_bits(t)) t = __uint_as_float(kInfBits);
        }
    }

    // the leaves within the largest bound, the own node's first
    if (!active) t = kNoQuery;
    a.bound[place * 32 + lane] = t;
    const float tmax = __uint_as_float(__reduce_max_sync(FGC_FULL_MASK, __float_as_uint(fmaxf(t, 0.f))));
    int *__restrict__ list = a.list + (size_t)place * a.list_cap;
    const int own_node = own_leaf >> 5;
    int n = 0;
    auto take_node = [&](int node) {
        const int leaf = node * 32 + lane;
        bool want = false;
        if (leaf < n_leaf) want = box_box_sq<NV>(glo, ghi, leaf_box + (size_t)leaf * (2 * NV)) <= tmax;
        const unsigned m = __ballot_sync(FGC_FULL_MASK, want);
        const int at = n + __popc(m & lanemask_lt());
        if (want && at < a.list_cap) list[at] = leaf;
        n += __popc(m);
    };
    take_node(own_node);
    for (int g0 = 0; g0 < n_top && n <= a.list_cap; g0 += 32) {
        bool want = false;
        if (g0 + lane < n_top)
            want = n_top == 1 || box_box_sq<NV>(glo, ghi, top_box + (size_t)(g0 + lane) * (2 * NV)) <= tmax;
        unsigned tops = __ballot_sync(FGC_FULL_MASK, want);
        while (tops && n <= a.list_cap) {
            const int node0 = (g0 + __ffs(tops) - 1) * 32;
            tops &= tops - 1;
            want = false;
            if (node0 + lane < n_node && node0 + lane != own_node)
                want = box_box_sq<NV>(glo, ghi, node_box + (size_t)(node0 + lane) * (2 * NV)) <= tmax;
            unsigned nodes = __ballot_sync(FGC_FULL_MASK, want);
            while (nodes && n <= a.list_cap) {
                take_node(node0 + __ffs(nodes) - 1);
                nodes &= nodes - 1;
            }
        }
    }
    if (n > a.list_cap) {
        int at = 0;
        const unsigned who = __ballot_sync(FGC_FULL_MASK, active);
        if (lane == 0) at = atomicAdd(&a.tree->n_listed, __popc(who));
        at = __shfl_sync(FGC_FULL_MASK, at, 0) + __popc(who & lanemask_lt());
        if (active && FGC_DBG_OK(at >= 0 && at < a.n_vert, &a.grid->status)) a.listed[at] = qi;
        if (active) a.bound[place * 32 + lane] = kListedQuery;       // (the others still get their default rows)
        n = 0;
    }
    if (lane == 0) a.list_n[place] = n;
}

template <int NV, int DC>
__global__ void __launch_bounds__(32, NV == 1 ? 28 : 20)
k_tree_groups(const TreeArgs a)
{
    chain_wait();
    chain_release();
    if (a.tree->magic != kTreeMagic) {                                    // not a tree: nothing is walked
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&a.grid->status, FGC_STATUS_INTERNAL);
        return;
    }
    const int slot = a.slot0 + (int)blockIdx.x;
    if (a.grid->status == 0 && slot < a.n_slots) bound_leaf<NV, DC>(a, slot);
}

// ----------------------------------------------------------------------------- rows

// Sorting of one key per lane and row, ascending over the lanes.  Every merge starts with reversed partners, so a
// stage's direction is one lane bit.
template <int S>
__device__ __forceinline__ void key_stage(uint32_t (&k)[S], int x, bool low)
{
#pragma unroll
    for (int r = 0; r < S; r++) {
        const uint32_t o = __shfl_xor_sync(FGC_FULL_MASK, k[r], x);
        k[r] = low ? min(k[r], o) : max(k[r], o);
    }
}
template <int S>
__device__ __forceinline__ void key_sort32(uint32_t (&k)[S], int lane)
{
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        key_stage<S>(k, 2 * m - 1, (lane & m) == 0);
#pragma unroll
        for (int bit = m >> 1; bit > 0; bit >>= 1) key_stage<S>(k, bit, (lane & bit) == 0);
    }
}
// a bitonic sequence per row into ascending order
template <int S>
__device__ __forceinline__ void key_merge32(uint32_t (&k)[S], int lane)
{
#pragma unroll
    for (int bit = 16; bit > 0; bit >>= 1) key_stage<S>(k, bit, (lane & bit) == 0);
}
// two ascending rows into one ascending sequence of 64
__device__ __forceinline__ void key_merge64(uint32_t (&k)[2], int lane)
{
    const uint32_t r = __shfl_xor_sync(FGC_FULL_MASK, k[1], 31);
    k[1] = max(k[0], r);
    k[0] = min(k[0], r);
    key_merge32<2>(k, lane);
}

// The 32 R smallest of S rows, ascending.  Returns the smallest key that is left out (kNoBox: none).
template <int S, int R>
__device__ __forceinline__ uint32_t key_select(uint32_t (&k)[S], uint32_t (&out)[R], int lane)
{
    static_assert(R <= 2, "longer lists are not sorted");
    uint32_t dropped = kNoBox;
    key_sort32<S>(k, lane);
    if constexpr (R == 1) {
        uint32_t a[1] = {k[0]};
#pragma unroll
        for (int r = 1; r < S; r++) {
            const uint32_t o = __shfl_xor_sync(FGC_FULL_MASK, k[r], 31);
            dropped = min(dropped, max(a[0], o));
            a[0] = min(a[0], o);
            key_merge32<1>(a, lane);
        }
        out[0] = a[0];
    } else {
        uint32_t a[2] = {k[0], k[1]};
        key_merge64(a, lane);
#pragma unroll
        for (int r = 2; r < S; r += 2) {
            uint32_t o[2] = {kNoBox, kNoBox};
            if (r + 1 < S) {
                uint32_t b[2] = {k[r], k[r + 1 < S ? r + 1 : r]};
                key_merge64(b, lane);
                o[0] = __shfl_xor_sync(FGC_FULL_MASK, b[1], 31);
                o[1] = __shfl_xor_sync(FGC_FULL_MASK, b[0], 31);
            } else {
                o[1] = __shfl_xor_sync(FGC_FULL_MASK, k[r], 31);
            }
            // the element-wise minimum with the reversed other one is a bitonic sequence of the 64 smallest
            dropped = min(dropped, min(max(a[0], o[0]), max(a[1], o[1])));
            const uint32_t l = min(a[0], o[0]), h = min(a[1], o[1]);
            a[0] = min(l, h);
            a[1] = max(l, h);
            key_merge32<2>(a, lane);
        }
        out[0] = a[0];
        out[1] = a[1];
    }
    return dropped;
}

// Points kept for a query, in shared memory: ROWS times 32; cut back to the nearest when they are full.
constexpr int kRowWarps = 8;
template <int R>
struct RowShape {
    static constexpr int ROWS = R == 1 ? 4 : (R == 2 ? 6 : (R == 4 ? 8 : 12));
    static constexpr int SLOT_BITS = ROWS <= 4 ? 7 : 8;
    static_assert(32 * R + 8 + 64 <= ROWS * 32, "no room for two leaves behind what a cut leaves");
};

// The keys of the 32 R nearest in ascending order: the distance as a fixed-point fraction of the largest, then the place.
template <int R, int S>
__device__ __forceinline__ uint32_t sort_entries(const float2 *pairs, int m, uint32_t (&out)[R], int lane)
{
    constexpr int SLOT_BITS = RowShape<R>::SLOT_BITS;
    static_assert(S * 32 <= 1 << SLOT_BITS, "places do not fit the keys");
    constexpr float TOP = (float)(1u << (32 - SLOT_BITS)) - 4.f;
    uint32_t v[S], key[S], top = 0;
#pragma unroll
    for (int r = 0; r < S; r++) {
        v[r] = r * 32 + lane < m ? __float_as_uint(pairs[r * 32 + lane].x) : 0u;
        top = max(top, v[r]);
    }
    top = __reduce_max_sync(FGC_FULL_MASK, top);
    const float scale = __fdividef(TOP, fmaxf(__uint_as_float(top), 1e-30f));
#pragma unroll
    for (int r = 0; r < S; r++)
        key[r] = r * 32 + lane >= m ? kNoBox
                 : (min(__float2uint_rz(__uint_as_float(v[r]) * scale), (uint32_t)TOP) << SLOT_BITS | (uint32_t)(r * 32 + lane));
    return key_select<S, R>(key, out, lane);
}

// The kn smallest of v (kNoBox: nothing there), or up to spare more, by bisection over the bit patterns: entries up to hi, of
// those equal to it the first `equal` ones.  at_most: how many there are, then how many are up to hi.  Returns whether some
// that equal hi are left out.
template <int S>
__device__ __forceinline__ bool bisect(const uint32_t (&v)[S], int kn, int spare, int &at_most, uint32_t &hi, int &equal)
{
    uint32_t lo = kNoBox;
    hi = 0;
#pragma unroll
    for (int r = 0; r < S; r++) {
        lo = min(lo, v[r]);
        hi = max(hi, v[r] == kNoBox ? 0u : v[r]);
    }
    lo = __reduce_min_sync(FGC_FULL_MASK, lo);
    hi = __reduce_max_sync(FGC_FULL_MASK, hi);
    while (lo < hi && at_most > kn + spare) {
        const uint32_t half = lo + ((hi - lo) >> 1);
        int c = 0;
#pragma unroll
        for (int r = 0; r < S; r++) c += v[r] <= half ? 1 : 0;
        c = __reduce_add_sync(FGC_FULL_MASK, c);
        if (c >= kn) { hi = half; at_most = c; } else lo = half + 1;
    }
    equal = S * 32;
    if (at_most <= kn + spare) return false;
    int below = 0;
#pragma unroll
    for (int r = 0; r < S; r++) below += v[r] < hi ? 1 : 0;
    equal = kn - __reduce_add_sync(FGC_FULL_MASK, below);
    return true;
}
// the lanes whose entry of one row stays
__device__ __forceinline__ unsigned staying(uint32_t v, uint32_t hi, int most, int &equal)
{
    bool keep = v <= hi && v != kNoBox;
    if (equal < most) {
        const unsigned same = __ballot_sync(FGC_FULL_MASK, v == hi);
        keep = v < hi || (v == hi && __popc(same & lanemask_lt()) < equal);
        equal -= min(equal, __popc(same));
    }
    return __ballot_sync(FGC_FULL_MASK, keep);
}

template <int NV, int R>
__global__ void __launch_bounds__(kRowWarps * 32, R == 8 ? 3 : (R == 4 || NV == 2 ? 4 : 5))
k_tree_rows(const TreeArgs a)
{
    chain_wait();
    chain_release();
    constexpr int ROWS = RowShape<R>::ROWS, MOST = ROWS * 32;
    __shared__ float2 s_pairs[kRowWarps][MOST];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int K = a.K, kn = K - 1;
    if (a.grid->status != 0) {
        // rows of points without neighbours: bad input, no tree was built
        if (a.slot0 > 0) return;
        for (int64_t qi = (int64_t)blockIdx.x * kRowWarps + w; qi < a.n_vert; qi += (int64_t)gridDim.x * kRowWarps) {
            const int64_t pad = a.tf_compat ? qi : (int64_t)-1;
            for (int s = lane; s < K; s += 32) {
                a.out_idx[(size_t)qi * K + s] = s == 0 ? qi : pad;
                a.out_dist[(size_t)qi * K + s] = 0.f;
            }
        }
        return;
    }
    // queries of this launch, in curve order: the eight of a CTA are of one leaf
    const int64_t row = (int64_t)blockIdx.x * kRowWarps + w;
    const int64_t slot = a.slot0 + (row >> 5);
    if (slot >= a.n_slots) return;
    const int n_list = __ldg(a.list_n + (row >> 5));
    if (n_list < 0) return;
    float t = __ldg(a.bound + row);
    const int e = warp_event_of_leaf(a.row_splits, a.n_rs, slot, lane);
    const int ev_begin = (int)__ldg(a.row_splits + e);
    const int n_e = (int)__ldg(a.row_splits + e + 1) - ev_begin;
    const int64_t leaf0 = tree_base(ev_begin, e, 5);
    const int rel_q = (int)(slot - leaf0) * 32 + (int)(row & 31);
    const bool writes = rel_q < n_e && t != kListedQuery;
    // (an open bound as the largest number: distances that overflow are no candidates)
    t = writes ? fminf(t, 3.402823466e38f) : kNoQuery;
    const int qi = ev_begin + min(rel_q, n_e - 1);
    const float4 *__restrict__ leaf_box = a.box[0] + (size_t)leaf0 * (2 * NV);
    const int *__restrict__ list = a.list + (size_t)(row >> 5) * a.list_cap;
    const uint8_t *__restrict__ sflag = a.sflag;
    float2 *pairs = s_pairs[w];
    float4 x[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) x[v] = __ldg(a.scoords + (size_t)qi * NV + v);
    int m = 0;                               // points kept
    uint32_t left_out = kNoBox;              // the last distance at which a point was left out that equals the bound
    auto load = [&](int leaf, float4 (&c)[NV], int &j) {
        const int rel = leaf * 32 + lane;
        j = rel < n_e ? ev_begin + rel : -1;
        if (!FGC_DBG_OK(j < a.n_vert, &a.grid->status)) j = -1;
#pragma unroll
        for (int v = 0; v < NV; v++) c[v] = __ldg(a.scoords + (size_t)(j < 0 ? qi : j) * NV + v);
    };
    auto keep = [&](const float4 (&c)[NV], int j) {
        const float d = dist_sq<NV>(x, c, 0);
        bool in = d <= t && j >= 0 && j != qi;
        if (sflag && in) { const uint8_t f = sflag[j]; in = f != 1 && f != 2; }
        const unsigned mask = __ballot_sync(FGC_FULL_MASK, in);
        if (in) pairs[m + __popc(mask & lanemask_lt())] = make_float2(d, __int_as_float(j));
        m += __popc(mask);
    };
    // down to the kn nearest or a few more, and the bound with them
    auto cut = [&]() {
        uint32_t v[ROWS], hi;
        int equal, at_most = m, to = 0;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < ROWS; r++) v[r] = r * 32 + lane < m ? __float_as_uint(pairs[r * 32 + lane].x) : kNoBox;
        const bool left = bisect<ROWS>(v, kn, 8, at_most, hi, equal);
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const unsigned kept = staying(v[r], hi, MOST, equal);
            const int j = __float_as_int(pairs[r * 32 + lane].y);
            __syncwarp();                    // (entries move to lower places only, row by row)
            if (kept >> lane & 1) pairs[to + __popc(kept & lanemask_lt())] = make_float2(__uint_as_float(v[r]), __int_as_float(j));
            to += __popc(kept);
        }
        __syncwarp();
        m = to;
        // Once one that equals the bound has been left out, others there change nothing: only what is nearer is wanted (0 gives
        // not a number: nothing is within that), or many equal points force a cut every two leaves.  Half of the points equal, ms: 20 k in three
        // coordinates, K = 64 0.70 -> 0.17 (grid 1.06), 100 k in five, K = 40 12.6 -> 0.82 (21.8).
        if (left) left_out = hi;
        t = __uint_as_float(hi - (left ? 1u : 0u));
    };
    // the leaves of `todo`, two at a time
    auto visit = [&](unsigned todo, auto leaf_at) {
        while (todo) {
            const int b0 = __ffs(todo) - 1;
            todo &= todo - 1;
            const int b1 = todo ? __ffs(todo) - 1 : -1;
            todo &= todo - 1;
            float4 c0[NV], c1[NV];
            int j0, j1;
            load(leaf_at(b0), c0, j0);
            load(leaf_at(b1 < 0 ? b0 : b1), c1, j1);
            if (b1 < 0) j1 = -1;
            keep(c0, j0);
            keep(c1, j1);
            if (m > MOST - 64) cut();
        }
    };
    if constexpr (NV == 1) {
        for (int base = 0; base < n_list && t >= 0.f; base += 32) {
            int leaf = 0;
            bool want = false;
            if (base + lane < n_list) {
                leaf = __ldg(list + base + lane);
                want = box_box_sq<NV>(x, x, leaf_box + (size_t)leaf * (2 * NV)) <= t;
            }
            visit(__ballot_sync(FGC_FULL_MASK, want), [&](int b) { return __shfl_sync(FGC_FULL_MASK, leaf, b); });
        }
    } else {
        // In five coordinates the boxes of a list are 64 KB, which every warp would read for itself: the eight of a CTA read them
        // once, and leave those near enough to some of their queries in shared memory (a million normal points, K = 40, lists of up to
        // 3072: 18.4 -> 15.6 ms).  With up to four, where a list is one or two steps long, waiting for one another costs more
        // than it saves (6.4 M uniform points in three, K = 64: 13.9 -> 15.2 ms).
        constexpr int NC = kGroupDims;
        __shared__ float s_box[2 * NC][kRowWarps * 32];
        __shared__ int s_leaf[kRowWarps * 32];
        __shared__ float s_query[kRowWarps][4 * NV], s_eight[2][NC], s_bound[kRowWarps];
        __shared__ int s_count[kRowWarps];
        float xc[4 * NV];
#pragma unroll
        for (int v = 0; v < NV; v++) { xc[4 * v] = x[v].x; xc[4 * v + 1] = x[v].y; xc[4 * v + 2] = x[v].z; xc[4 * v + 3] = x[v].w; }
        if (lane == 0) {
            s_bound[w] = t;
#pragma unroll
            for (int v = 0; v < NV; v++) {
                s_query[w][4 * v] = x[v].x; s_query[w][4 * v + 1] = x[v].y;
                s_query[w][4 * v + 2] = x[v].z; s_query[w][4 * v + 3] = x[v].w;
            }
        }
        __syncthreads();
        if (threadIdx.x < NC) {
            float lo = __uint_as_float(kInfBits), hi = -__uint_as_float(kInfBits);
#pragma unroll
            for (int k = 0; k < kRowWarps; k++)
                if (s_bound[k] >= 0.f) { lo = fminf(lo, s_query[k][threadIdx.x]); hi = fmaxf(hi, s_query[k][threadIdx.x]); }
            s_eight[0][threadIdx.x] = lo;
            s_eight[1][threadIdx.x] = hi;
        }
        float tmax = s_bound[0];
#pragma unroll
        for (int k = 1; k < kRowWarps; k++) tmax = fmaxf(tmax, s_bound[k]);
        __syncthreads();
        for (int base = 0; base < n_list && tmax >= 0.f; base += kRowWarps * 32) {
            int leaf = 0;
            bool want = false;
            float box[8 * NV];
            if (base + (int)threadIdx.x < n_list) {
                leaf = __ldg(list + base + threadIdx.x);
#pragma unroll
                for (int v = 0; v < 2 * NV; v++) {
                    const float4 b = __ldg(leaf_box + (size_t)leaf * (2 * NV) + v);
                    box[4 * v] = b.x; box[4 * v + 1] = b.y; box[4 * v + 2] = b.z; box[4 * v + 3] = b.w;
                }
                float acc = 0.f;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const float g = fmaxf(fmaxf(__fsub_rn(box[c], s_eight[1][c]), __fsub_rn(s_eight[0][c], box[4 * NV + c])), 0.f);
                    acc = c == 0 ? __fmul_rn(g, g) : __fadd_rn(acc, __fmul_rn(g, g));
                }
                want = acc <= tmax;
            }
            const unsigned mine = __ballot_sync(FGC_FULL_MASK, want);
            if (lane == 0) s_count[w] = __popc(mine);
            __syncthreads();
            int at = __popc(mine & lanemask_lt()), total = 0;
#pragma unroll
            for (int k = 0; k < kRowWarps; k++) {
                if (k == w) at += total;
                total += s_count[k];
            }
            if (want) {
                s_leaf[at] = leaf;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    s_box[c][at] = box[c];
                    s_box[NC + c][at] = box[4 * NV + c];
                }
            }
            __syncthreads();
            for (int i0 = 0; i0 < total && t >= 0.f; i0 += 32) {
                const int i = i0 + lane;
                float acc = 0.f;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const float g = fmaxf(fmaxf(__fsub_rn(s_box[c][i], xc[c]), __fsub_rn(xc[c], s_box[NC + c][i])), 0.f);
                    acc = c == 0 ? __fmul_rn(g, g) : __fadd_rn(acc, __fmul_rn(g, g));
                }
                visit(__ballot_sync(FGC_FULL_MASK, i < total && acc <= t), [&](int b) { return s_leaf[i0 + b]; });
            }
            __syncthreads();
        }
    }
    if (!writes) return;
    __syncwarp();
    const int orig_q = __ldg(a.sorig + qi);
    if (!FGC_DBG_OK(orig_q >= 0 && orig_q < a.n_vert, &a.grid->status)) return;
    int64_t *row_i = a.out_idx + (size_t)orig_q * K;
    float *row_d = a.out_dist + (size_t)orig_q * K;
    const int64_t pad = a.tf_compat ? (int64_t)orig_q : (int64_t)-1;
    bool tie = false, same = false, full;
    uint32_t kth = 0;
    if constexpr (R <= 2) {
        constexpr int SLOT_BITS = RowShape<R>::SLOT_BITS;
        uint32_t key[R], drop;
        if (R == 1 && m <= 32) drop = sort_entries<R, R>(pairs, m, key, lane);
        else if (m <= 64) drop = sort_entries<R, 2>(pairs, m, key, lane);
        else if (m <= 96) drop = sort_entries<R, 3>(pairs, m, key, lane);
        else if (m <= 128) drop = sort_entries<R, 4>(pairs, m, key, lane);
        else drop = sort_entries<R, ROWS>(pairs, m, key, lane);
        float d[R];
        int j[R];
        const uint32_t edge = __shfl_sync(FGC_FULL_MASK, kn > 32 ? key[R - 1] : key[0], (kn - 1) & 31);
        full = kn > 0 && edge != kNoBox;
        bool unclear = full && drop >> SLOT_BITS == edge >> SLOT_BITS, look = false;
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 p = make_float2(__uint_as_float(0x7fffffffu), __int_as_float(-1));      // (empty: compares as false)
            if (key[r] != kNoBox) p = pairs[key[r] & ((1u << SLOT_BITS) - 1)];
            d[r] = p.x;
            j[r] = __float_as_int(p.y);
            unclear = unclear || (full && r * 32 + lane >= kn && key[r] >> SLOT_BITS == edge >> SLOT_BITS);
            const float nd = __shfl_down_sync(FGC_FULL_MASK, d[r], 1);
            look = look || (lane < 31 && d[r] >= nd);
        }
        if (R == 2) {
            const float nd = __shfl_sync(FGC_FULL_MASK, d[R - 1], 0);
            look = look || (lane == 31 && d[0] >= nd);
        }
        bool again = false;
        if (__any_sync(FGC_FULL_MASK, unclear || look)) {
            // few rows come here: some are equal or in the wrong order
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float nd = __shfl_down_sync(FGC_FULL_MASK, d[r], 1), next = __shfl_sync(FGC_FULL_MASK, d[R - 1], 0);
                unclear = unclear || (lane < 31 ? d[r] > nd : (r + 1 < R && d[r] > next));
            }
            again = __any_sync(FGC_FULL_MASK, unclear);
            if (again) {
                // distances that differ by less than the keys tell: sorted as they are
                SortedList<R> near;
                near.init(lane, kn);
#pragma unroll 1
                for (int i = lane; i - lane < m; i += 32) near.merge32(lane, kn, i < m ? pairs[i].x : __uint_as_float(kInfBits), i);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    d[r] = near.d[r];
                    j[r] = __float_as_uint(near.d[r]) < kInfBits ? __float_as_int(pairs[near.id[r]].y) : -1;
                }
            }
            if (a.mark_ties == TieMarks::kAny) same = equal_in_list<R>(d, j, kn, lane);
        }
        kth = __float_as_uint(__shfl_sync(FGC_FULL_MASK, kn > 32 ? d[R - 1] : d[0], (kn - 1) & 31));
        if (again) {
            int within = 0;
#pragma unroll 1
            for (int i = lane; i - lane < m; i += 32)
                within += __popc(__ballot_sync(FGC_FULL_MASK, i < m && __float_as_uint(pairs[i].x) <= kth));
            tie = full && within > kn;
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int s = r * 32 + lane;
            if (s < kn) {
                row_i[1 + s] = j[r] < 0 ? pad : (int64_t)__ldg(a.sorig + j[r]);
                row_d[1 + s] = j[r] < 0 ? 0.f : d[r];
            }
        }
    } else {
        uint32_t v[ROWS], hi;
        int equal, at_most = m, to = 0;
#pragma unroll
        for (int r = 0; r < ROWS; r++) v[r] = r * 32 + lane < m ? __float_as_uint(pairs[r * 32 + lane].x) : kNoBox;
        full = m >= kn;
        tie = bisect<ROWS>(v, kn, 0, at_most, hi, equal);
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            if (r * 32 >= m) break;
            const unsigned kept = staying(v[r], hi, MOST, equal);
            if (kept >> lane & 1) {
                const int at = 1 + to + __popc(kept & lanemask_lt());
                row_i[at] = (int64_t)__ldg(a.sorig + __float_as_int(pairs[r * 32 + lane].y));
                row_d[at] = __uint_as_float(v[r]);
                kth = max(kth, v[r]);
            }
            to += __popc(kept);
        }
        for (int s = to + lane; s < kn; s += 32) {
            row_i[1 + s] = pad;
            row_d[1 + s] = 0.f;
        }
        kth = __reduce_max_sync(FGC_FULL_MASK, kth);
    }
    if (lane == 0) {
        row_i[0] = mark_row(a, full && (tie || kth == left_out), same, orig_q);
        row_d[0] = 0.f;
    }
}

template <int NV, int DC>
static cudaError_t launch_tree(TreeArgs a, const TreeScratch &scratch, cudaStream_t s)
{
    a.list = scratch.list;
    a.list_n = scratch.list_n;
    a.list_cap = scratch.list_cap;
    a.bound = scratch.bound;
    const int n_slots = a.n_slots;
    for (int slot = 0; slot < n_slots; slot = a.n_slots) {
        a.slot0 = slot;
        a.n_slots = n_slots - slot < scratch.slots ? n_slots : slot + scratch.slots;      // the end of this round
        const unsigned count = (unsigned)(a.n_slots - slot), rows = count * (32 / kRowWarps);
        FGC_TRY(launch_chained(k_tree_groups<NV, DC>, count, 32, 0, s, a));
        switch (tree_list_rows(a.K)) {
        case 1: FGC_TRY(launch_chained(k_tree_rows<NV, 1>, rows, kRowWarps * 32, 0, s, a)); break;
        case 2: FGC_TRY(launch_chained(k_tree_rows<NV, 2>, rows, kRowWarps * 32, 0, s, a)); break;
        case 4: FGC_TRY(launch_chained(k_tree_rows<NV, 4>, rows, kRowWarps * 32, 0, s, a)); break;
        default: FGC_TRY(launch_chained(k_tree_rows<NV, 8>, rows, kRowWarps * 32, 0, s, a));
        }
    }
    return cudaSuccess;
}

}  // namespace fgc

int fgc::knn_search_tree_groups(int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs, int32_t K,
                                int32_t has_direction, int32_t tf_compat, TieMarks mark_ties, int64_t *out_idx, float *out_distsq,
                                void *workspace, size_t workspace_bytes, fgc_stream_t stream)
{
    FGC_NVTX("fgc_knn_search_tree_groups");
    using namespace fgc;
    TreeArgs a;
    KnnWorkspace L;
    TreeLayout T;
    const int rc = tree_args(n_vert, n_coords, row_splits, n_rs, K, has_direction, tf_compat, mark_ties, out_idx, out_distsq, workspace,
                             workspace_bytes, &a, &L, &T);
    if (rc != FGC_OK || n_vert == 0) return rc;
    TreeScratch scratch;
    if (!tree_scratch(L, n_coords, (char *)workspace, workspace_bytes, &scratch)) return FGC_ERR_WORKSPACE;
    cudaStream_t s = (cudaStream_t)stream;
    a.n_slots = (int)T.n_box[0];
    a.listed = (int *)((char *)workspace + T.keys[0]);           // free since the build
    if (n_coords <= 3) FGC_RETURN_IF_CUDA((launch_tree<1, 3>(a, scratch, s)));
    else if (n_coords == 4) FGC_RETURN_IF_CUDA((launch_tree<1, 4>(a, scratch, s)));
    else FGC_RETURN_IF_CUDA((launch_tree<2, 5>(a, scratch, s)));
    return launch_tree_listed(a, L.nv, s);
}
