// tcgen05 building blocks of the tensor-core stages (sm_103a): operand
// descriptors, kind::f16 products, completion, fences, named barriers.
#pragma once
#include <cstdint>

#include "qg_bulk.cuh"

namespace qg {

// Shared-memory matrix descriptor: start address, leading-dimension byte
// offset (between core matrices along K; unused by swizzled K-major
// layouts), stride-dimension byte offset (between 8-row groups), descriptor
// version 1, layout type (0 = no swizzle, 2 = 128-byte swizzle).
__device__ __forceinline__ uint64_t smem_desc(unsigned saddr, unsigned lbo, unsigned sbo,
                                              unsigned layout = 0) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) |
           ((uint64_t)(sbo >> 4) << 32) | (1ull << 46) | ((uint64_t)layout << 61);
}

// Instruction descriptor of kind::f16 with an m x n accumulator: D = F32,
// A = B = F16, both K-major.
constexpr unsigned idesc_f16(unsigned m, unsigned n) {
    return (1u << 4) | (0u << 7) | (0u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(unsigned dtmem, uint64_t a, uint64_t b, unsigned acc,
                                        unsigned idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %4, p;\n\t}\n" ::"r"(dtmem),
        "l"(a), "l"(b), "r"(acc), "r"(idesc)
        : "memory");
}

// A wait of a tensor stage gave up: its status word, which later launches look at,
// and the host's, which calls that return results look at (its device address, set
// when the engine starts).
struct StageStatus {
    unsigned bits;
    unsigned *host;
};
__device__ __forceinline__ void report_stage(StageStatus *s, unsigned bits, unsigned host_bits) {
    atomicOr(&s->bits, bits);
    unsigned *h = *(unsigned *volatile *)&s->host;
    if (h) atomicOr_system(h, host_bits);
}

// One lane of a converged warp (the same one at every call): code that the
// whole warp walks keeps descriptors in uniform registers, where tcgen05.mma
// takes them; issued from a single thread's branch the same products cost 100
// to 200 cycles each in operand moves (48 to 80 are the products' own).
__device__ __forceinline__ unsigned elect_lane() {
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(r));
    return r;
}

// mma_f16 by the lane whose `lane` is set (acc: 0 overwrites).
__device__ __forceinline__ void mma_f16_lane(unsigned dtmem, uint64_t a, uint64_t b, unsigned acc,
                                             unsigned idesc, unsigned lane) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %3, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %4, p;\n\t}\n" ::"r"(dtmem),
        "l"(a), "l"(b), "r"(acc), "r"(idesc), "r"(lane)
        : "memory");
}

__device__ __forceinline__ void mma_commit(unsigned bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}

__device__ __forceinline__ void tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// Barrier `id` over the `threads` threads of a tile group.
__device__ __forceinline__ void group_sync(unsigned id, unsigned threads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// Bit in which the Gray codes of i - 1 and i differ (ctz(i)), at compile
// time once the loops are unrolled.
__host__ __device__ constexpr int gray_bit(int i) {
    return (i & 1) ? 0 : (i & 2) ? 1 : (i & 4) ? 2 : (i & 8) ? 3 : 4;
}
// Inverse Gray code of j (5 bits).
__host__ __device__ constexpr int gray_index(int j) {
    return j ^ (j >> 1) ^ (j >> 2) ^ (j >> 3) ^ (j >> 4);
}

}  // namespace qg
