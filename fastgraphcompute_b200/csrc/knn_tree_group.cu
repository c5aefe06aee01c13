// binned_select_knn forward for sm_100a: the search on a tree of boxes (knn_tree.cuh) in two kernels, the first of which
// works for the 32 queries of a leaf at once.  They are neighbours on the curve and have nearly the same candidates, so
// what one query per warp spends most of its instructions on (knn_tree_search.cu: finding its bound by repeated
// selection, and walking the levels of the tree) is paid once for 32.
//
//  k_tree_groups  One warp per leaf.  The points of the leaves nearest to its own are counted by distance for every query
//                 (40 classes, eight to a factor of two); the class in which the K-th falls gives an upper bound on its K-th
//                 distance.  |c|^2 - 2 c.q + |q|^2, with coordinates relative to the leaf, is a product of 32 queries x 32 points
//                 over two more places than there are coordinates: a few matrix instructions in tf32, |c|^2 in two parts.
//                 The bound is widened by what rounding can add, so it stays an upper bound.  Then the leaves whose box is
//                 within the largest of the bounds are listed, and of those again, for every eight of the queries, the leaves within theirs.
//  k_tree_rows    One warp per query.  It compares its own bound with the boxes of its list, visits those within it, keeps
//                 the points within it -- distances by dist_sq, which is what is returned -- and sorts them (K <= 65)
//                 or selects the K - 1 smallest.  On uniform data a quarter more points than K pass.
//
// The distance of two boxes, or of a point and a box, is computed with the operations of dist_sq in the same order.  Rounding is
// monotone, so it never exceeds the computed distance of two points inside: pruning needs no margin and
// the result is exactly the K-1 smallest computed distances, whatever the tree.  Boxes and points at exactly the bound
// are taken until a candidate equal to it has been left out, so that one that equals the K-th distance is always noticed.
//
// What bounds them (a million uniform points in ten row splits, three coordinates, K = 64, ncu): k_tree_rows issue slots (1000 warp
// instructions a query: some 250 for its list and its boxes, 350 for 16 leaves, 400 for the sort and the row) and the latency of list, box and
// point one after the other, hence the many warps; k_tree_groups the shared-memory pipe (0.83; the counting's atomics) and issue slots
// (0.71; 240 instructions a query; 72 registers, some of them spilled, 28 one-warp CTAs an SM).
// In five coordinates k_tree_rows was bound by the lines that its reads touch (shared-memory and L1 pipe 0.97, issue slots 0.40): boxes of 64 bytes and
// points of 32, of which 40 and 20 are used.  Boxes, halves and points in arrays apart: a million normal points, K = 40 12.0 -> 7.7 ms.
// Whole forward in ms, before the lists for eight queries / now / one query at a time / the grid, without a second look in the
// first three: 6.4 M uniform points in three coordinates, K = 64 13.5 / 10.1 / 21.5 / 18.3; 1.6 M learned ones in four, K = 40 6.6 / 4.5 / 9.4 /
// 8.4; 800 k skewed in three, K = 128 3.0 / 2.2 / 4.6 / 18.8; a million normal ones in five, K = 40 15.0 / 7.5 / 18.2 / 26.4.  The second look adds
// 0.85, 0.4, 1.0 and 0.4.
//
// Other splits of the work, measured on the first and the third of these when they took 13.9 and 3.2: one kernel, a lane per query, the points of a leaf read from
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

// The same for a leaf; in five coordinates from the arrays apart.
template <int NV, int DC>
__device__ __forceinline__ float leaf_box_sq(const float4 (&lo)[NV], const float4 (&hi)[NV], const TreeArgs &a, int64_t at)
{
    if constexpr (DC < kApartDims) {
        return box_box_sq<NV>(lo, hi, a.box[0] + 2 * at);
    } else {
        const float4 bl = __ldg(a.leaves.lo + at), bh = __ldg(a.leaves.hi + at);
        const float2 e = __ldg(a.leaves.e + at);
        const float g0 = fmaxf(fmaxf(__fsub_rn(bl.x, hi[0].x), __fsub_rn(lo[0].x, bh.x)), 0.f);
        const float g1 = fmaxf(fmaxf(__fsub_rn(bl.y, hi[0].y), __fsub_rn(lo[0].y, bh.y)), 0.f);
        const float g2 = fmaxf(fmaxf(__fsub_rn(bl.z, hi[0].z), __fsub_rn(lo[0].z, bh.z)), 0.f);
        const float g3 = fmaxf(fmaxf(__fsub_rn(bl.w, hi[0].w), __fsub_rn(lo[0].w, bh.w)), 0.f);
        const float g4 = fmaxf(fmaxf(__fsub_rn(e.x, hi[NV - 1].x), __fsub_rn(lo[NV - 1].x, e.y)), 0.f);
        float acc = __fadd_rn(__fadd_rn(__fmul_rn(g0, g0), __fmul_rn(g1, g1)), __fmul_rn(g2, g2));
        acc = __fadd_rn(acc, __fmul_rn(g3, g3));
        return __fadd_rn(acc, __fmul_rn(g4, g4));
    }
}

// ----------------------------------------------------------------------------- bounds and lists

constexpr int kHistClasses = 40;
// Leaves that the bound is taken from: more make it tighter.
// Measured with 5 / 8 / 12 / 16 / 24 / 36 of them (400 k points, whole forward, ms): uniform in three coordinates, K = 16 0.67 / 0.67 /
// 0.69 / 0.71 / 0.76 / 0.82, K = 64 1.15 / 1.07 / 1.04 / 1.05 / 1.09 / 1.18, K = 200 6.3 / 2.6 / 2.3 / 2.23 / 2.18 / 2.22; four learned
// coordinates, K = 40 2.06 / 1.94 / 1.89 / 1.88 / 1.93 / 1.98; five, normal, K = 40 8.4 / 7.8 / 7.3 / 7.2 / 7.1 / 7.1.
// They are looked for in so many nodes: with eight instead of four 1.6 M learned points in four coordinates, K = 40 take 4.8 instead of 5.0 ms, a million
// normal ones in five 12.3 instead of 13.2, with twelve leaves more 12.0; in three 6.4 M uniform ones, K = 64 10.6 instead of 10.3.
__host__ __device__ constexpr int seed_nodes(int dims) { return dims <= 3 ? 4 : 8; }
__device__ __forceinline__ int seed_leaves(int kn, int dims)
{
    return min(6 + kn / 6, 26) + (dims >= 4 ? 8 : 0) + (dims >= 5 ? 12 : 0);
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
    constexpr int CHUNKS = (DC + 3) / 4, NODES = seed_nodes(DC);
    static_assert(NODES <= 8, "three bits of a key");
    // classes of the counting, then the list of leaves
    __shared__ __align__(16) int s_hist[tree_list_cap(DC) > 32 * (kHistClasses + 1) ? tree_list_cap(DC) : 32 * (kHistClasses + 1)];
    __shared__ float s_part[4][2 * 4 * NV + 1];                 // boxes of eight queries, the largest bound among them
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
    const int64_t leaf0 = tree_base(ev_begin, e, 5);
    const float4 *leaf_box = a.box[0] + (size_t)leaf0 * (2 * NV);
    const float4 *node_box = a.box[1] + (size_t)tree_base(ev_begin, e, 10) * (2 * NV);
    const float4 *top_box = a.box[2] + (size_t)tree_base(ev_begin, e, 15) * (2 * NV);
    const int rel_q = own_leaf * 32 + lane;
    const bool valid = rel_q < n_e;
    const int qi = ev_begin + (valid ? rel_q : n_e - 1);
    bool active = valid && kn > 0;
    if (sflag && (sflag[qi] == 0 || sflag[qi] == 2)) active = false;
    if (!__any_sync(FGC_FULL_MASK, active)) {            // no query of the leaf may have neighbours
        a.bound[place * 32 + lane] = kNoQuery;
        if (lane == 0) { a.list_n[place] = 0; a.leaf_info[slot] = make_int4(own_leaf * 32, ev_begin, n_e, 0); }
        if (lane < 4) a.leaf_part[slot * 4 + lane] = make_int2(0, 0);
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
        // 16 to 128, less in more coordinates and more at a border: five factors of two up to twice it, less for short lists (with four the
        // first class was the K-th's for most points in five coordinates: a million normal ones, K = 40 13.7 -> 13.2 ms).  The last class begins below
        // kNotThere, so that what is no candidate is never counted below it, however large the leaf.
        const float share = kn >= 63 ? 2.f : 2.f * powf((float)(kn + 1) * (1.f / 64.f), 2.f / DC);
        const int last = (int)min(__float_as_uint(share * diag), 0x7e800000u) >> 20;
        const int first = max(last - (kHistClasses - 1), 0);
        // the nearest leaves of the nearest nodes
        const int own_node = own_leaf >> 5, node0 = own_node & ~31;
        uint32_t nkey = kNoBox, lkey[NODES];
        int node_of[NODES];
        if (node0 + lane < n_node)
            nkey = node0 + lane == own_node ? (uint32_t)lane
                   : ((__float_as_uint(box_box_sq<NV>(mid, mid, node_box + (size_t)(node0 + lane) * (2 * NV))) & ~31u) | (uint32_t)lane);
#pragma unroll
        for (int k = 0; k < NODES; k++) {
            const uint32_t m = __reduce_min_sync(FGC_FULL_MASK, nkey);
            lkey[k] = kNoBox;
            node_of[k] = node0 + (int)(m & 31u);
            if (m != kNoBox) {
                if (lane == (int)(m & 31u)) nkey = kNoBox;
                const int leaf = node_of[k] * 32 + lane;
                if (leaf < n_leaf)
                    lkey[k] = (__float_as_uint(leaf_box_sq<NV, DC>(mid, mid, a, leaf0 + leaf)) & ~255u) |
                              (uint32_t)(k << 5 | lane);
            }
        }
        __syncwarp();
        auto next_seed = [&]() -> int {
            uint32_t m = lkey[0];
#pragma unroll
            for (int k = 1; k < NODES; k++) m = min(m, lkey[k]);
            m = __reduce_min_sync(FGC_FULL_MASK, m);
            if (m == kNoBox) return -1;
            const int src = (int)(m & 31u), from = (int)(m >> 5 & 7u);
            int node = node_of[0];
#pragma unroll
            for (int k = 0; k < NODES; k++) {
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
        // Once K points are below the end of some class, what is beyond it is counted in the next class: it changes nothing there, and
        // the counts of a row that all go to one place do not meet those of other rows in a bank.
        auto classes_below = [&]() {             // classes whose end has fewer than K + 1 points before it (the query itself is counted)
            __syncwarp();
            int below = 0, classes = 0;
#pragma unroll 16
            for (int b = 0; b < kHistClasses; b++) {
                below += s_hist[lane * (kHistClasses + 1) + b];
                classes += below <= kn ? 1 : 0;
            }
            return classes;
        };
        int next_look = kn / 32 + 4, end[4];
#pragma unroll
        for (int k = 0; k < 4; k++) end[k] = hi_bits;
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
            if (i == next_look) {
                const int classes = classes_below();
                const int open = min((first + classes + 1) << 20, hi_bits);
#pragma unroll
                for (int k = 0; k < 4; k++) end[k] = __shfl_sync(FGC_FULL_MASK, open, g4 + 8 * k);
                next_look += 8;
            }
            if (!usable) continue;
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int b = min(max(__float_as_int(f[m][j][k]), lo_bits), end[2 * m + (k >> 1)]) >> 20;
                        atomicAdd(mine + (16 * m + 8 * (k >> 1)) * (kHistClasses + 1) + b, 1);
                    }
        }
        const int classes = classes_below();
        if (classes < kHistClasses - 1 && q2 <= 1e36f) {
            t = widened(__uint_as_float((uint32_t)(first + classes + 1) << 20), q2);
            if (!is_finite_bits(t)) t = __uint_as_float(kInfBits);
        }
    }

    // the leaves within the largest bound, the own node's first
    if (!active) t = kNoQuery;
    a.bound[place * 32 + lane] = t;
    const float tmax = __uint_as_float(__reduce_max_sync(FGC_FULL_MASK, __float_as_uint(fmaxf(t, 0.f))));
    int *list = s_hist;
    __syncwarp();
    const int own_node = own_leaf >> 5;
    int n = 0;
    auto take_node = [&](int node) {
        const int leaf = node * 32 + lane;
        bool want = false;
        if (leaf < n_leaf) want = leaf_box_sq<NV, DC>(glo, ghi, a, leaf0 + leaf) <= tmax;
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
    // The same for eight queries at a time: what a query has to look through is a third (four coordinates) to two thirds (three) of
    // the list for 32.  A leaf is kept with four bits, one for each eight; then the four lists are written one behind the other.
    if (n > 0) {
        float lo[4 * NV], hi[4 * NV], most = t;
        const float inf = __uint_as_float(kInfBits);
#pragma unroll
        for (int v = 0; v < NV; v++) {
            const float4 q = __ldg(a.scoords + (size_t)qi * NV + v);
            lo[4 * v] = hi[4 * v] = q.x; lo[4 * v + 1] = hi[4 * v + 1] = q.y;
            lo[4 * v + 2] = hi[4 * v + 2] = q.z; lo[4 * v + 3] = hi[4 * v + 3] = q.w;
        }
#pragma unroll
        for (int c = 0; c < DC; c++) {
            if (!active) { lo[c] = inf; hi[c] = -inf; }
#pragma unroll
            for (int x = 4; x > 0; x >>= 1) {
                lo[c] = fminf(lo[c], __shfl_xor_sync(FGC_FULL_MASK, lo[c], x));
                hi[c] = fmaxf(hi[c], __shfl_xor_sync(FGC_FULL_MASK, hi[c], x));
            }
            if ((lane & 7) == 0) { s_part[lane >> 3][c] = lo[c]; s_part[lane >> 3][DC + c] = hi[c]; }
        }
#pragma unroll
        for (int x = 4; x > 0; x >>= 1) most = fmaxf(most, __shfl_xor_sync(FGC_FULL_MASK, most, x));
        if ((lane & 7) == 0) s_part[lane >> 3][2 * DC] = most;
        __syncwarp();
        int count[4] = {0, 0, 0, 0};
        for (int i0 = 0; i0 < n; i0 += 32) {
            const bool in = i0 + lane < n;
            const int leaf = in ? list[i0 + lane] : 0;
            float4 bl, bh;
            float2 be = make_float2(0.f, 0.f);
            if constexpr (DC < kApartDims) {
                bl = __ldg(leaf_box + 2 * (size_t)leaf);
                bh = __ldg(leaf_box + 2 * (size_t)leaf + 1);
            } else {
                bl = __ldg(a.leaves.lo + leaf0 + leaf);
                bh = __ldg(a.leaves.hi + leaf0 + leaf);
                be = __ldg(a.leaves.e + leaf0 + leaf);
            }
            const float box_lo[5] = {bl.x, bl.y, bl.z, bl.w, be.x}, box_hi[5] = {bh.x, bh.y, bh.z, bh.w, be.y};
            int bits = 0;
#pragma unroll
            for (int p = 0; p < 4; p++) {
                float acc = 0.f;
#pragma unroll
                for (int c = 0; c < DC; c++) {
                    const float g = fmaxf(fmaxf(__fsub_rn(box_lo[c], s_part[p][DC + c]), __fsub_rn(s_part[p][c], box_hi[c])), 0.f);
                    acc = c == 0 ? __fmul_rn(g, g) : __fadd_rn(acc, __fmul_rn(g, g));
                }
                const bool want = in && acc <= s_part[p][2 * DC];
                bits |= want ? 1 << p : 0;
                count[p] += __popc(__ballot_sync(FGC_FULL_MASK, want));
            }
            if (in) list[i0 + lane] = leaf | bits << 28;
        }
        __syncwarp();
        const bool apart = count[0] + count[1] + count[2] + count[3] <= a.list_room;      // (else all have the one list)
        int *__restrict__ out = a.list + (size_t)place * a.list_room;
        int at = 0;
        for (int p = 0; p < (apart ? 4 : 1); p++) {
            if (lane == p) a.leaf_part[slot * 4 + p] = make_int2(at, count[p]);
            for (int i0 = 0; i0 < n; i0 += 32) {
                const int leaf = i0 + lane < n ? list[i0 + lane] : 0;
                const bool want = i0 + lane < n && (!apart || (leaf >> 28 & 1 << p));
                const unsigned m = __ballot_sync(FGC_FULL_MASK, want);
                if (want) out[at + __popc(m & lanemask_lt())] = leaf & 0xfffffff;
                at += __popc(m);
            }
        }
        if (!apart && lane < 4) a.leaf_part[slot * 4 + lane] = make_int2(0, n);
    } else if (lane < 4) {
        a.leaf_part[slot * 4 + lane] = make_int2(0, 0);
    }
    if (lane == 0) { a.list_n[place] = n; a.leaf_info[slot] = make_int4(own_leaf * 32, ev_begin, n_e, 0); }
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

// 16 bytes of coordinates in one read, used or not (left to itself the compiler reads three of four in two pieces).
__device__ __forceinline__ float4 read_four(const float4 *p)
{
    float4 v;
    asm("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
// Coordinates of a point, and its squared distance: the operations of dist_sq in the same order without the coordinates that
// are 0 on both sides.
template <int DC>
struct RowPoint {
    float4 a;
    float e;              // the fifth
};
template <int DC>
__device__ __forceinline__ RowPoint<DC> row_point(const TreeArgs &a, int j)
{
    RowPoint<DC> p;
    p.e = 0.f;
    if constexpr (DC < kApartDims) {
        p.a = read_four(a.scoords + j);
    } else {
        p.a = read_four(a.point_a + j);
        p.e = __ldg(a.point_e + j);
    }
    return p;
}
template <int DC>
__device__ __forceinline__ float row_dist(const RowPoint<DC> &q, const RowPoint<DC> &c)
{
    float s0, s1, s2, s3 = 0.f;
    sq_diff_f32x2(q.a.x, q.a.y, c.a.x, c.a.y, s0, s1);
    if constexpr (DC == 3) {
        const float z = __fsub_rn(q.a.z, c.a.z);
        s2 = __fmul_rn(z, z);
    } else {
        sq_diff_f32x2(q.a.z, q.a.w, c.a.z, c.a.w, s2, s3);
    }
    float acc = __fadd_rn(__fadd_rn(s0, s1), s2);
    if constexpr (DC >= 4) acc = __fadd_rn(acc, s3);
    if constexpr (DC >= 5) {
        const float e = __fsub_rn(q.e, c.e);
        acc = __fadd_rn(acc, __fmul_rn(e, e));
    }
    return acc;
}
// The squared distance to a box, likewise.
__device__ __forceinline__ float gap_sq(float lo, float hi, float x)
{
    const float g = fmaxf(fmaxf(__fsub_rn(lo, x), __fsub_rn(x, hi)), 0.f);
    return __fmul_rn(g, g);
}
template <int DC>
__device__ __forceinline__ float row_gap(const RowPoint<DC> &q, const float4 &lo, const float4 &hi)
{
    float acc = __fadd_rn(__fadd_rn(gap_sq(lo.x, hi.x, q.a.x), gap_sq(lo.y, hi.y, q.a.y)), gap_sq(lo.z, hi.z, q.a.z));
    if constexpr (DC >= 4) acc = __fadd_rn(acc, gap_sq(lo.w, hi.w, q.a.w));
    return acc;
}
// (with up to four coordinates the corners of a box lie side by side: one address; apart they cost a register, 7.15 -> 8.0 ms for 6.4 M
// uniform points in three, K = 64)
template <int DC>
__device__ __forceinline__ float row_box(const RowPoint<DC> &q, const float4 *__restrict__ box)
{
    return row_gap<DC>(q, read_four(box), read_four(box + 1));
}
template <int DC>
__device__ __forceinline__ float row_box(const RowPoint<DC> &q, const BoxArrays &box, int64_t at)
{
    const float2 e = __ldg(box.e + at);
    return __fadd_rn(row_gap<DC>(q, read_four(box.lo + at), read_four(box.hi + at)), gap_sq(e.x, e.y, q.e));
}

// A store, or a count, in shared memory under a predicate (as a branch it takes three instructions more).
__device__ __forceinline__ void store_if(bool p, uint32_t at, float d, int j)
{
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %0, 0; @q st.shared.v2.b32 [%1], {%2, %3}; }"
                 :: "r"((uint32_t)p), "r"(at), "r"(__float_as_uint(d)), "r"(j) : "memory");
}

// Leaves (halves of them, even ones and then odd ones) wanted by a query and not yet visited: what one step of boxes finds behind
// what is left of the steps before, and up to three (seven) behind the last one that fill four steps.
constexpr int kWanted = 32 + 32 + 8;
// Resident CTAs an SM asked of the compiler: the chain from a list to its boxes to the points is hidden by other warps, and a few
// spilled registers cost less than warps that are not there.  Time of the rows in ms with 4 / 5 / 6 / 7 CTAs: 6.4 M uniform points in three
// coordinates, K = 64 8.8 / 7.7 / 7.2 / 8.1, 800 k, K = 16 0.73 / 0.64 / 0.57 / 0.53; 1.6 M learned ones in four, K = 40 4.1 / 3.8 / 3.6 / 3.6; 800 k
// skewed in three, K = 128 1.74 / 1.61 / 1.50 / 1.53; 400 k uniform in four, K = 200 1.81 / 1.66 / 1.74 / -.
constexpr int row_ctas(int r) { return r == 1 ? 7 : (r == 8 ? 5 : 6); }

template <int DC, int R, bool FLAGS>
__global__ void __launch_bounds__(kRowWarps * 32, row_ctas(R))
k_tree_rows(const TreeArgs a)
{
    chain_wait();
    chain_release();
    constexpr int ROWS = RowShape<R>::ROWS, MOST = ROWS * 32;
    constexpr bool HALVES = DC >= kApartDims;
    constexpr int STEP = HALVES ? 8 : 4;
    __shared__ float2 s_pairs[kRowWarps][MOST];
    __shared__ __align__(16) int s_wanted[kRowWarps][kWanted];
    __shared__ int s_near[HALVES ? kRowWarps : 1][64];
    const int lane = threadIdx.x & 31, w = __shfl_sync(FGC_FULL_MASK, (int)threadIdx.x >> 5, 0);      // (known to be the same in a warp)
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
    // queries of this launch, in curve order: the eight of a CTA are those of one list
    const int row = (int)blockIdx.x * kRowWarps + w;
    const int slot = a.slot0 + (row >> 5);
    if (slot >= a.n_slots) return;
    if (__ldg(a.list_n + (row >> 5)) < 0) return;
    const int4 info = __ldg(a.leaf_info + slot);
    const int2 part = __ldg(a.leaf_part + slot * 4 + (row >> 3 & 3));
    float t = __ldg(a.bound + row);
    const int ev_begin = info.y, n_e = info.z, ev_end = ev_begin + n_e, n_list = part.y;
    const int rel_q = info.x + (row & 31);
    const bool writes = rel_q < n_e && t != kListedQuery;
    // (an open bound as the largest number: distances that overflow are no candidates)
    t = writes ? fminf(t, 3.402823466e38f) : kNoQuery;
    const int qi = ev_begin + min(rel_q, n_e - 1);
    const int *__restrict__ list = a.list + (size_t)(row >> 5) * a.list_room + part.x;
    const int64_t leaf0 = slot - (info.x >> 5);                  // first of the row split
    const float4 *__restrict__ leaf_box = a.box[0] + 2 * leaf0;  // (not in five coordinates)
    float2 *pairs = s_pairs[w];
    const uint32_t pairs_at = (uint32_t)__cvta_generic_to_shared(pairs);
    int *wanted = s_wanted[w], *near = s_near[HALVES ? w : 0];
    const RowPoint<DC> x = row_point<DC>(a, qi);
    int m = 0;                               // points kept
    uint32_t left_out = kNoBox;              // the last distance at which a point was left out that equals the bound
    auto keep = [&](const RowPoint<DC> &c, int j) {
        const float d = row_dist<DC>(x, c);
        const bool in = (d <= t) & (j != qi);
        const unsigned mask = __ballot_sync(FGC_FULL_MASK, in);
        store_if(in, pairs_at + 8 * (m + __popc(mask & lanemask_lt())), d, j);
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
    // Visits.  Lanes whose leaf is wanted write its first point down; then four leaves a step, whose points are on their way
    // together: one 16-byte read gives the four, where picking them out of a ballot took five instructions each.  In five
    // coordinates only the halves within the bound are visited, two side by side (a million normal points, K = 40: 9.5 -> 8.8 ms; with
    // fewer coordinates the boxes of the halves cost more than they save: 6.4 M uniform points in three, K = 64 8.6 against 7.7).
    int n_wanted = 0, n_near = 0, near0 = 0;
    const int *mine = HALVES ? wanted + (lane >> 4) * (kWanted / 2) : wanted;
    auto fetch = [&](int first, int &j, RowPoint<DC> &c) {
        j = first + (HALVES ? lane & 15 : lane);
        j = j < ev_end ? j : qi;
        if (!FGC_DBG_OK(j >= ev_begin && j < a.n_vert, &a.grid->status)) j = qi;
        c = row_point<DC>(a, j);
        if constexpr (FLAGS) { const uint8_t f = a.sflag[j]; if (f == 1 || f == 2) j = qi; }
    };
    auto visit_wanted = [&]() {
        if (lane < STEP - 1)                     // (no points there)
            wanted[HALVES ? ((n_wanted + lane) & 1) * (kWanted / 2) + ((n_wanted + lane) >> 1) : n_wanted + lane] = ev_end;
        __syncwarp();
        for (int i = 0; i < n_wanted && t >= 0.f; i += STEP) {
            const int4 first = *reinterpret_cast<const int4 *>(mine + (HALVES ? i >> 1 : i));
            int j0, j1, j2, j3;
            RowPoint<DC> c0, c1, c2, c3;
            fetch(first.x, j0, c0);
            fetch(first.y, j1, c1);
            fetch(first.z, j2, c2);
            fetch(first.w, j3, c3);
            keep(c0, j0);
            keep(c1, j1);
            if (m > MOST - 64) cut();
            if (i + STEP / 2 < n_wanted) {
                keep(c2, j2);
                keep(c3, j3);
                if (m > MOST - 64) cut();
            }
        }
        n_wanted = 0;
        __syncwarp();
    };
    // the halves of the next up to 16 near leaves
    auto halves = [&]() {
        __syncwarp();
        const int i = lane >> 1;
        int first = 0;
        bool want = false;
        if (i < n_near) {
            const int half = near[(near0 + i) & 63] * 2 + (lane & 1);
            first = ev_begin + half * 16;
            if constexpr (HALVES) want = row_box<DC>(x, a.halves, 2 * leaf0 + half) <= t;
        }
        const unsigned mask = __ballot_sync(FGC_FULL_MASK, want);
        const int at = n_wanted + __popc(mask & lanemask_lt());
        if (want) wanted[(at & 1) * (kWanted / 2) + (at >> 1)] = first;
        n_wanted += __popc(mask);
        near0 += 16;
        n_near -= 16;
        if (n_wanted > 32) visit_wanted();
    };
    for (int base = 0; base < n_list && t >= 0.f; base += 32) {
        int leaf = 0;
        bool want = false;
        if (base + lane < n_list) {
            leaf = __ldg(list + base + lane);
            if constexpr (DC < kApartDims) want = row_box<DC>(x, leaf_box + 2 * (size_t)leaf) <= t;
            else want = row_box<DC>(x, a.leaves, leaf0 + leaf) <= t;
        }
        const unsigned mask = __ballot_sync(FGC_FULL_MASK, want);
        if constexpr (HALVES) {
            if (want) near[(near0 + n_near + __popc(mask & lanemask_lt())) & 63] = leaf;
            n_near += __popc(mask);
            while (n_near >= 16 && t >= 0.f) halves();
        } else {
            if (want) wanted[n_wanted + __popc(mask & lanemask_lt())] = ev_begin + leaf * 32;
            n_wanted += __popc(mask);
            if (n_wanted > 32) visit_wanted();
        }
    }
    while (n_near > 0 && t >= 0.f) halves();
    if (n_wanted > 0) visit_wanted();
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

template <int DC, int R>
static cudaError_t launch_rows(const TreeArgs &a, unsigned blocks, cudaStream_t s)
{
    return a.sflag ? launch_chained(k_tree_rows<DC, R, true>, blocks, kRowWarps * 32, 0, s, a)
                   : launch_chained(k_tree_rows<DC, R, false>, blocks, kRowWarps * 32, 0, s, a);
}

template <int NV, int DC>
static cudaError_t launch_tree(TreeArgs a, const TreeScratch &scratch, cudaStream_t s)
{
    a.list = scratch.list;
    a.list_n = scratch.list_n;
    a.list_cap = scratch.list_cap;
    a.list_room = scratch.list_room;
    a.bound = scratch.bound;
    const int n_slots = a.n_slots;
    for (int slot = 0; slot < n_slots; slot = a.n_slots) {
        a.slot0 = slot;
        a.n_slots = n_slots - slot < scratch.slots ? n_slots : slot + scratch.slots;      // the end of this round
        const unsigned count = (unsigned)(a.n_slots - slot), rows = count * (32 / kRowWarps);
        FGC_TRY(launch_chained(k_tree_groups<NV, DC>, count, 32, 0, s, a));
        switch (tree_list_rows(a.K)) {
        case 1: FGC_TRY((launch_rows<DC, 1>(a, rows, s))); break;
        case 2: FGC_TRY((launch_rows<DC, 2>(a, rows, s))); break;
        case 4: FGC_TRY((launch_rows<DC, 4>(a, rows, s))); break;
        default: FGC_TRY((launch_rows<DC, 8>(a, rows, s)));
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
    if (!T.groups) return FGC_ERR_WORKSPACE;
    a.listed = (int *)((char *)workspace + T.listed);
    const char *ws = (const char *)workspace;                    // (empty with up to four coordinates)
    a.leaves = {(const float4 *)(ws + T.box_lo), (const float4 *)(ws + T.box_hi), (const float2 *)(ws + T.box_e)};
    a.halves = {(const float4 *)(ws + T.half_lo), (const float4 *)(ws + T.half_hi), (const float2 *)(ws + T.half_e)};
    a.point_a = (const float4 *)(ws + T.point_a);
    a.point_e = (const float *)(ws + T.point_e);
    a.leaf_info = (int4 *)((char *)workspace + T.leaf_info);
    a.leaf_part = (int2 *)(a.leaf_info + T.n_box[0]);
    if (n_coords <= 3) FGC_RETURN_IF_CUDA((launch_tree<1, 3>(a, scratch, s)));
    else if (n_coords == 4) FGC_RETURN_IF_CUDA((launch_tree<1, 4>(a, scratch, s)));
    else FGC_RETURN_IF_CUDA((launch_tree<2, 5>(a, scratch, s)));
    return launch_tree_listed(a, L.nv, s);
}
