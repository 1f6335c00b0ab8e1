// fp32 products on the 5th-generation tensor cores: every fp32 number is split into three bf16 numbers
// whose sum is the number itself (3 x 8 significand bits with signs cover the 24 of fp32), and of the nine
// products of parts the six largest are formed,
//     x*y = x1*y1 + (x1*y2 + x2*y1) + (x1*y3 + x2*y2 + x3*y1) + 2^-26 |x*y| or less,
// by tcgen05.mma with fp32 accumulators in tensor memory.  Each part is rounded to nearest, so x2 and x3 are
// at most 2^-9 and 2^-18 of x and the three products left out are below the rounding of one fp32 multiply.
// Limits, which the kernels test for: |x| >= 2^-100 or zero (below that the third part would lose bits to
// the range of bf16), and finite numbers whose first part does not round to infinity.
//
// This file holds the split, the instruction wrappers and the shared-memory operand descriptors.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "barrier.cuh"
#include "launch.cuh"

namespace dlspm {

// ---- split ------------------------------------------------------------------------------------------

// Running minimum of the magnitude bits of nonzero numbers (doubled, minus one; zero counts as large).
__device__ __forceinline__ unsigned split_magnitude(float x, unsigned least)
{
    return __viaddmin_u32(__float_as_uint(x) << 1, 0xffffffffu, least);
}
constexpr unsigned kSplitLeast = (27u << 24) - 1u;  // of 2^-100: smaller values of split_magnitude are too small to split

// Smallest magnitude of three numbers (one instruction, NaN ignored): below 2^-100, zeros are told from small numbers
// by split_magnitude.
__device__ __forceinline__ float min3_magnitude(float a, float b, float c)
{
    float r;
    asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
constexpr float kSplitSmall = 7.888609052210118e-31f;  // 2^-100

__device__ __forceinline__ uint32_t bf16x2_bits(float lo, float hi)
{
    const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&t);
}

// x minus the low (high) half of a packed pair, exact where the half is x rounded to bf16.  One instruction that takes the
// half as it is: 7 instructions for a pair instead of 9 (with the halves widened first, two subtractions packed into one
// instruction); a batch of 256 SpMMs 5690 -> 5540 us, whose operand warps are bound by instruction issue.
__device__ __forceinline__ float minus_low(uint32_t pair, float x)
{
    float r;
    asm("{\n .reg .b16 lo, hi, m;\n mov.b32 {lo, hi}, %1;\n mov.b16 m, 0xbf80;\n fma.rn.f32.bf16 %0, lo, m, %2;\n}\n" : "=f"(r) : "r"(pair), "f"(x));
    return r;
}
__device__ __forceinline__ float minus_high(uint32_t pair, float x)
{
    float r;
    asm("{\n .reg .b16 lo, hi, m;\n mov.b32 {lo, hi}, %1;\n mov.b16 m, 0xbf80;\n fma.rn.f32.bf16 %0, hi, m, %2;\n}\n" : "=f"(r) : "r"(pair), "f"(x));
    return r;
}

// (x, y) -> the packed first, second and third parts.
__device__ __forceinline__ void split_pair(float x, float y, uint32_t &p1, uint32_t &p2, uint32_t &p3)
{
    p1 = bf16x2_bits(x, y);
    x = minus_low(p1, x);
    y = minus_high(p1, y);
    p2 = bf16x2_bits(x, y);
    x = minus_low(p2, x);
    y = minus_high(p2, y);
    p3 = bf16x2_bits(x, y);
}
// One number alone, parts in the low halves.
__device__ __forceinline__ void split_one(float x, uint32_t &p1, uint32_t &p2, uint32_t &p3)
{
    p1 = bf16x2_bits(x, 0.f);
    x = minus_low(p1, x);
    p2 = bf16x2_bits(x, 0.f);
    x = minus_low(p2, x);
    p3 = bf16x2_bits(x, 0.f);
}

// Stores by shared-memory address.
__device__ __forceinline__ void store_shared(uint32_t at, uint32_t x, uint32_t y)
{
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void store_shared_half(uint32_t at, uint32_t x)
{
    asm volatile("{\n .reg .b16 lo, hi;\n mov.b32 {lo, hi}, %1;\n st.shared.b16 [%0], lo;\n}\n" ::"r"(at), "r"(x) : "memory");
}
__device__ __forceinline__ void store_shared_zero(uint32_t at)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(0u) : "memory");
}

// ---- clusters ---------------------------------------------------------------------------------------

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
// Without an ordering of memory accesses: where only the blocks' lifetimes matter.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Address of the same shared-memory object in another block of the cluster.
__device__ __forceinline__ uint32_t cluster_map(uint32_t smem, unsigned rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem), "r"(rank));
    return r;
}
__device__ __forceinline__ float cluster_load(uint32_t addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ unsigned cluster_load_u32(uint32_t addr)
{
    unsigned v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
// Sets bits of a word that both blocks of a pair keep a copy of.  The readers of either block find them by way of barriers:
// this block's own (whose arrivals name no scope, which orders within the block only), a relay to the other block's, and
// the multiplies' completion.  The fence puts the remote write in front of all of these; where this is called is rare.
__device__ __forceinline__ void mark_in_pair(unsigned *word, unsigned bits, unsigned rank)
{
    atomicOr(word, bits);
    const uint32_t other = cluster_map(smem_u32(word), rank ^ 1u);
    asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;" ::"r"(other), "r"(bits) : "memory");
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
}
// Arrives on a barrier of another block (address from cluster_map).  What it passes on lies in its own block's shared
// memory already, written and fenced by others; remote writes are fenced where they are made (mark_in_pair).  With
// .release.cluster it would order those too, at 1 to 2 % of the SpMM kernel's time (1024 x 4096, N = 1024, and a batch of 256 problems).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait (a second or so) that gives up when `abort` is raised.  The warp is suspended inside the instruction
// until the phase completes or the hint, 20 us, has passed: polling instead cost the other warps of the SM a third
// of their issue slots.
__device__ __forceinline__ bool mbar_wait_suspended(unsigned long long *bar, unsigned parity, volatile int *abort)
{
    const uint32_t a = smem_u32(bar);
    for (unsigned i = 0; i < (1u << 16); i++) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity), "r"(20000u)
            : "memory");
        if (ok) return true;
        if (*abort) return false;
    }
    return false;
}

// True on one lane of a converged warp.
__device__ __forceinline__ bool elect_one()
{
    unsigned p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}

// ---- tensor memory and the multiply ------------------------------------------------------------------
// PAIR: two blocks of a cluster (ranks 2i and 2i + 1) work on one tile of 256 rows; the even one issues.

template <bool PAIR>
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, unsigned columns)
{
    if constexpr (PAIR) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
}
template <bool PAIR>
__device__ __forceinline__ void tmem_free(uint32_t base, unsigned columns)
{
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns));
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns));
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Sixteen columns of this warp's 32 tensor-memory lanes; tmem_load_wait before the values are used.
__device__ __forceinline__ void tmem_load16(uint32_t addr, float (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr));
}
// Ties the loaded values to the wait, so that no use of them moves in front of it.
__device__ __forceinline__ void tmem_load_wait(float (&v)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                   "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])
                 :
                 : "memory");
}

// Four columns of this warp's 32 tensor-memory lanes; tmem_store_wait before another thread is told.
__device__ __forceinline__ void tmem_store4(uint32_t addr, const uint32_t (&v)[4])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
                 : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Adds 64 columns of an accumulator to the warp's registers (those of them below `columns`).
__device__ __forceinline__ void tmem_add(float (&acc)[64], uint32_t addr, int columns)
{
#pragma unroll
    for (int j = 0; j < 64; j += 16) {
        if (j < columns) {
            float v[16];
            tmem_load16(addr + j, v);
            tmem_load_wait(v);
#pragma unroll
            for (int x = 0; x < 16; x += 2) {
                const float2 sum = __fadd2_rn(make_float2(acc[j + x], acc[j + x + 1]), make_float2(v[x], v[x + 1]));
                acc[j + x] = sum.x;
                acc[j + x + 1] = sum.y;
            }
        }
    }
}

// Shared-memory operand descriptors.  Swizzled layouts repeat every 8 rows; byte offsets between repetitions:
// `lead` and `stride` as in the canonical layouts of the PTX manual.
constexpr uint64_t kSwizzle128 = 2;
__device__ __forceinline__ uint64_t mma_descriptor(uint32_t smem, unsigned lead, unsigned stride, uint64_t swizzle)
{
    return (uint64_t)((smem & 0x3ffffu) >> 4) | ((uint64_t)(lead >> 4) << 16) | ((uint64_t)(stride >> 4) << 32) | (1ull << 46) |
           (swizzle << 61);
}
// bf16 operands, fp32 accumulators, M x N tile; `a_mn`, `b_mn`: the operand's rows run along K (its M or N
// dimension is the contiguous one).
__host__ __device__ constexpr uint32_t mma_instruction(int M, int N, bool a_mn, bool b_mn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}
template <bool PAIR>
__device__ __forceinline__ void mma_bf16(uint32_t acc, uint64_t a, uint64_t b, uint32_t instruction, bool add)
{
    if constexpr (PAIR)
        asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc),
                     "l"(a), "l"(b), "r"(instruction), "r"(add ? 1u : 0u)
                     : "memory");
    else
        asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc),
                     "l"(a), "l"(b), "r"(instruction), "r"(add ? 1u : 0u)
                     : "memory");
}
// The first operand from tensor memory (a lane a row, two neighbouring elements of K a word), by a pair of blocks.
__device__ __forceinline__ void mma_bf16_tmem(uint32_t acc, uint32_t a, uint64_t b, uint32_t instruction, bool add)
{
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(acc),
                 "r"(a), "l"(b), "r"(instruction), "r"(add ? 1u : 0u)
                 : "memory");
}
// The barrier (of both blocks of the pair) receives one arrival when all multiplies issued so far are done.
template <bool PAIR>
__device__ __forceinline__ void mma_commit(unsigned long long *bar, unsigned pair_mask)
{
    if constexpr (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                     "h"((unsigned short)pair_mask)
                     : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace dlspm
