// A cluster of eight CTAs that does the passes of a small build one after the other (knn_grid_small.cu, knn_tree_small.cu).
#pragma once
#include "fgc_common.cuh"

namespace fgc {

constexpr int kClusterCtas = 8, kClusterWarps = 16, kClusterThreads = kClusterWarps * 32, kClusterAll = kClusterCtas * kClusterThreads;

// All threads of the cluster; what was written before, to global memory or a CTA's shared memory, can be read by all after it.
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Address of a CTA's shared memory, for the two below.
__device__ __forceinline__ uint32_t cluster_at(const void *mine, int cta)
{
    uint32_t at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(cta));
    return at;
}
__device__ __forceinline__ uint32_t cluster_word(const void *mine, int cta)
{
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_at(mine, cta)) : "memory");
    return v;
}
__device__ __forceinline__ int4 cluster_four(const void *mine, int cta)
{
    int4 v;
    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(cluster_at(mine, cta)) : "memory");
    return v;
}

// Exclusive scan over the threads of a CTA; total: of all of them.
__device__ __forceinline__ int cta_scan(int x, int *s_part, int &total)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FGC_FULL_MASK, incl, o);
        if (lane >= o) incl += y;
    }
    __syncthreads();
    if (lane == 31) s_part[wib] = incl;
    __syncthreads();
    int before = incl - x;
    total = 0;
#pragma unroll
    for (int k = 0; k < kClusterWarps; k++) {
        if (k == wib) before += total;
        total += s_part[k];
    }
    return before;
}

}  // namespace fgc
