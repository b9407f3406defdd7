// tcgen05 (5th-generation tensor core) building blocks for sm_100a: shared-memory
// matrix descriptors, the instruction descriptors (f16 x f16 -> f32, int8 x int8 -> int32),
// TMEM allocation, MMA issue, commit, and TMEM loads. One thread issues an MMA
// for the whole CTA; accumulators live in tensor memory (128 lanes x 512
// 32-bit columns per SM) and come back to registers with tcgen05.ld.
//
// Operand tiles sit in shared memory in the K-major "no swizzle" canonical
// layout: 8-row x 16-byte core matrices, each 128 contiguous bytes, those of 16 bytes of K
// (8 f16 or 16 int8) one after another, R / 8 of them for R rows. So SBO (stride between
// 8-row groups) = 128 bytes and LBO (stride between 16-byte pieces of K) = R * 16 bytes.
// Global memory holds the tiles in exactly this order (f16_tile_offset), so one bulk copy
// brings a tile in ready for the MMA.
#pragma once

#include <stdint.h>

namespace tc {
namespace umma {

// 64-bit shared-memory matrix descriptor (K-major, no swizzle).
__device__ __forceinline__ uint64_t smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= uint64_t((smem_addr >> 4) & 0x3FFFu);         // start address, 16-byte units
    d |= uint64_t((lbo_bytes >> 4) & 0x3FFFu) << 16;   // leading (K) byte offset
    d |= uint64_t((sbo_bytes >> 4) & 0x3FFFu) << 32;   // stride (row-group) byte offset
    d |= uint64_t(1) << 46;                            // descriptor version for sm_100
    return d;                                          // base offset 0, layout type 0 = no swizzle
}

// Instruction descriptor: D s32, A and B signed 8-bit, both K-major, dense.
__host__ __device__ constexpr uint32_t idesc_s8(int m, int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

// The same for f16 operands and an f32 accumulator.
__host__ __device__ constexpr uint32_t idesc_f16(int m, int n) {
    return (1u << 4) | (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     uint32_t(__cvta_generic_to_shared(dst_smem))),
                 "r"(columns)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T, one K = 32 step; issued by ONE thread.
__device__ __forceinline__ void mma_s8(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t yes;
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}" : "=r"(yes));
    return yes != 0;
}

// The same with f16 operands, one K = 16 step. Of the descriptors only the low words (address, leading offset) are given;
// the high one is that of every operand tile here: SBO 128 bytes, version, no swizzle.
__device__ __forceinline__ uint32_t smem_desc_low(uint32_t smem_addr, uint32_t lbo_bytes) {
    return ((smem_addr >> 4) & 0x3FFFu) | ((lbo_bytes >> 4) & 0x3FFFu) << 16;
}
__device__ __forceinline__ void mma_f16_low(uint32_t tmem_d, uint32_t a_low, uint32_t b_low, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %6};\n\tmov.b64 db, {%2, %6};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(a_low), "r"(b_low), "r"(idesc), "r"(accumulate), "r"(0u), "n"((128 >> 4) | 1 << 14)
        : "memory");
}

// Arrives on an mbarrier once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     uint32_t(__cvta_generic_to_shared(bar)))
                 : "memory");
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 lanes (the lower or upper half of this warp's quadrant, by taddr's lane) x 32 or 16 consecutive columns of
// f32 values, in the order of an m16n8 accumulator: v[4 j], v[4 j + 1] are row lane / 4, columns 8 j + 2 (lane % 4)
// and the next; v[4 j + 2], v[4 j + 3] the same of row lane / 4 + 8.
__device__ __forceinline__ void ld_half_f32(uint32_t taddr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void ld_half_f32(uint32_t taddr, float (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x2.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "r"(taddr)
        : "memory");
}

// Waits for this thread's TMEM loads. The values pass through the statement so
// that no use of them can be scheduled above the wait.
__device__ __forceinline__ void wait_ld(float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                   "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void wait_ld(float (&v)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7])
                 :
                 : "memory");
}

// Byte offset of (row, k) in a block's operand tile of `rows` rows x 32 f16.
__host__ __device__ constexpr uint32_t f16_tile_offset(uint32_t rows, uint32_t row, uint32_t k) {
    return (k / 8) * (rows * 16) + (row / 8) * 128 + (row % 8) * 16 + (k % 8) * 2;
}

}  // namespace umma
}  // namespace tc
