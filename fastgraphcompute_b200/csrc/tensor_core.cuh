// Tensor-core products of fp32 matrices at fp32 accuracy (sm_100a: tcgen05.mma, accumulators in TMEM).
//
// An fp32 number is the sum of three bfloat16 numbers: each takes the eight leading bits of what is left.  The third of a number below
// 2^-110 would have bits below bfloat16's smallest, 2^-133, so numbers are multiplied by 2^16 first: then the smallest fp32 number, 2^-149, is
// that one, and the three parts are exact for all of them (the tensor core keeps subnormal operands and sums: 2^-133 times 2^40, and
// 2^-126 + 2^-140 from two products, came out exactly).  Results are divided by 2^32.  Of the nine
// products of two such sums the six with the first part of either, or the second of both, are formed; the other three are below
// 2^-24 of the result.  Products of bfloat16 numbers are exact in the fp32 accumulators.  The product of the two first parts has an
// accumulator of its own, so that it is rounded only as often as it is added to.
// (Sums of bfloat16 numbers for fp32 products: Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for
// higher-precision computations", 2019.)
//
// Operands lie in shared memory as rows of 64 numbers (128 bytes) in the 128-byte swizzle: eight rows make an atom of 1024 bytes,
// 16-byte unit u of row r is at u ^ (r & 7).  The same bytes are a K-major operand (a row is a row or column of the result) and an
// M- or N-major one (a row is one of the numbers that are summed over): a pass over the rows and a sum over the rows
// take the same tiles.
#pragma once
#include <cuda_bf16.h>

#include "fgc_common.cuh"

namespace fgc {

constexpr float kSplitScale = 65536.f, kSplitUndo = 1.f / 65536.f / 65536.f;
// From here on (2^43 before the scaling; infinities among it) a number is not split: sums of 512 products could overflow where
// the result does not, and an infinity times a part that is 0 is not a number.  What holds one is computed by scalar operations.  NaN is split
// like any number: its parts are NaN, and so is what it is multiplied with or added to.
constexpr float kUnsplit = 5.764607523034235e17f;          // 2^59

// Eight numbers into three units of eight parts; returns the largest size of the scaled numbers, NaN left out.
// (Two at a time: the scaling costs nothing beside the differences one by one.)
__device__ __forceinline__ float split8(const float (&v)[8], uint4 (&part)[3])
{
    uint32_t p[3][4];
    float most = 0.f;
    const unsigned long long scale = pack_f32x2(kSplitScale, kSplitScale);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        unsigned long long ab;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(ab) : "l"(pack_f32x2(v[2 * i], v[2 * i + 1])), "l"(scale));
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float a, b;
            unpack_f32x2(ab, a, b);
            const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
            const uint32_t u = *reinterpret_cast<const uint32_t *>(&h);
            p[k][i] = u;
            if (k == 0) most = fmaxf(most, fmaxf(fabsf(a), fabsf(b)));
            if (k < 2)
                asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(ab) : "l"(ab), "l"(pack_f32x2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u))));
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) part[k] = make_uint4(p[k][0], p[k][1], p[k][2], p[k][3]);
    return most;
}

// Byte offset of 16-byte unit u (0..7) of row r of an operand.
__device__ __forceinline__ uint32_t operand_at(int r, int u) { return (uint32_t)(r * 128 + ((u ^ (r & 7)) << 4)); }

__device__ __forceinline__ uint32_t smem_at(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Descriptor of an operand at a shared-memory address: 128-byte swizzle, atoms of eight rows 1024 bytes apart; next_64: bytes from
// 64 numbers of a row to the next 64 (M- and N-major operands only).
__device__ __forceinline__ uint64_t operand_desc(uint32_t at, uint32_t next_64)
{
    return (uint64_t)((at >> 4) & 0x3fff) | (uint64_t)((next_64 >> 4) & 0x3fff) << 16 | (uint64_t)(1024 >> 4) << 32 | 1ull << 46 | 2ull << 61;
}
// Instruction descriptor: bfloat16 operands, fp32 accumulators, 128 rows, n columns.
__device__ __forceinline__ uint32_t product_desc(int n, bool rows_summed)
{
    return 1u << 4 | 1u << 7 | 1u << 10 | (rows_summed ? 3u << 15 : 0u) | (uint32_t)(n >> 3) << 17 | (128u >> 4) << 24;
}
// by one thread: accumulators (+)= a * b over 16 numbers
__device__ __forceinline__ void tc_mma(uint32_t acc, uint64_t a, uint64_t b, uint32_t desc, bool add)
{
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
                 :: "r"(acc), "l"(a), "l"(b), "r"(desc), "r"((uint32_t)add) : "memory");
}
// Steps of 16 numbers, six products each.  Part k of an operand is part_bytes behind part k - 1, a step step_bytes behind the one before
// (addresses are the low 14 bits of a descriptor, in units of 16 bytes: sums of them stay there).
__device__ __forceinline__ void tc_steps(uint32_t big, uint32_t small, uint64_t a, uint32_t a_part, uint64_t b, uint32_t b_part, uint32_t step_bytes,
                                         uint32_t desc, int steps, bool add)
{
    a_part >>= 4;
    b_part >>= 4;
    step_bytes >>= 4;
#pragma unroll 1
    for (int k = 0; k < steps; k++, a += step_bytes, b += step_bytes, add = true) {
        tc_mma(small, a, b + 2 * b_part, desc, add);
        tc_mma(small, a + 2 * a_part, b, desc, true);
        tc_mma(small, a + a_part, b + b_part, desc, true);
        tc_mma(small, a, b + b_part, desc, true);
        tc_mma(small, a + a_part, b, desc, true);
        tc_mma(big, a, b, desc, add);
    }
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t arrivals)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("{ .reg .b64 s; mbarrier.arrive.shared::cta.b64 s, [%0]; }" :: "r"(bar) : "memory");
}
// the barrier's phase ends when all products issued so far by this thread have been formed
__device__ __forceinline__ void tc_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
// Waits for the end of a phase, but not for ever: false after some seconds (the caller computes without the product then).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    for (int i = 0; i < 1 << 20; i++) {
        uint32_t done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// The same for warps that wait for one another: one that gives up says so, and the others do not wait any more.
__device__ __forceinline__ bool wait_unless(uint32_t bar, uint32_t parity, volatile int *late)
{
    for (int i = 0; i < 1 << 20; i++) {
        uint32_t done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if (*late) return false;
    }
    *late = 1;
    return false;
}

// by one warp: columns (a power of two, 32 or more) of TMEM; their address is written to shared memory
__device__ __forceinline__ void tmem_alloc(uint32_t to, uint32_t columns)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(to), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t at, uint32_t columns)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(at), "r"(columns) : "memory");
}
// 16 columns of the warp's 32 rows (rows 32 (warp & 3) and on), one row a lane; no wait
__device__ __forceinline__ void tmem_read16(uint32_t at, uint32_t (&v)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                   "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(at) : "memory");
}
__device__ __forceinline__ void tmem_wait_read() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// stores to shared memory become visible to the tensor core (each writer, before the barrier)
__device__ __forceinline__ void smem_to_tensor_core() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__host__ __device__ inline uint32_t tmem_columns(int n)
{
    uint32_t c = 32;
    while ((int)c < n) c <<= 1;
    return c;
}

}  // namespace fgc
