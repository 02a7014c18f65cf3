// The fifth-generation tensor core of sm_100a (tcgen05) as inline PTX: tensor
// memory allocation, the instruction descriptor of the integer MMA, the MMA
// itself, its commit to an mbarrier, and loads and stores of tensor memory. The
// descriptor's bits follow the PTX ISA (tcgen05 "Instruction descriptor" table),
// as CUTLASS's cute/arch/mma_sm100_desc.hpp also lays them out.
#pragma once

#include "fb_tma.cuh"

namespace fb {
namespace umma {

// Instruction descriptor of kind::i8 with signed 8-bit A and B, both
// K-major, a signed 32-bit accumulator, shape M x N (bits: c_format [4,6) = 2,
// a_format [7,10) = 1, b_format [10,13) = 1, N >> 3 at [17,23), M >> 4 at
// [24,29)).
__host__ __device__ constexpr uint32_t idesc_s8s8_s32(int M, int N) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[tmem] B[smem]^T, issued by one thread: A is M x K in tensor memory, row i in lane
// i, K packed four 8-bit values to a 32-bit column.
__device__ __forceinline__ void mma_s8_tmem_a(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                              bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

// Arrives once on bar when every MMA this thread issued before has finished.
__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Makes this thread's generic-proxy shared-memory writes visible to the
// tensor core (async proxy) reads that are ordered after it.
__device__ __forceinline__ void fence_smem_to_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Tensor memory allocation, by one whole warp. The address lands in *slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(slot)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 16 consecutive columns of 32-bit words: thread t of the warp
// gets lane (taddr lane + t), columns [col, col + 16). A warp may only touch
// the 32 lanes of its own quarter (warp id % 4).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// 16 lanes (from the address's lane on) x 8 consecutive 32-bit columns:
// thread t writes lanes t / 4 (a0, a1) and t / 4 + 8 (b0, b1), columns t % 4
// (a0, b0) and 4 + t % 4 (a1, b1).
__device__ __forceinline__ void tmem_st_16x128b_x2(uint32_t taddr, uint32_t a0, uint32_t b0, uint32_t a1,
                                                   uint32_t b1) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1, %2, %3, %4};"
                 ::"r"(taddr), "r"(a0), "r"(b0), "r"(a1), "r"(b1) : "memory");
}

__device__ __forceinline__ void tmem_wait_st() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace umma
}  // namespace fb
