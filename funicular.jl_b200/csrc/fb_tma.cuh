// TMA tile loads, mbarriers with bounded waits, and the FP64 tensor-core MMA,
// as inline PTX for sm_100a. Every wait here gives up after a time limit and
// reports it, so a kernel can never spin forever on a shared GPU.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include "fb_common.cuh"

namespace fb {

// A wait gives up after this long; a healthy wait takes microseconds.
constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull;
constexpr long long WAIT_LIMIT_CYCLES = 4000000000ll;   // the same at 2 GHz

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Makes barrier initialisation visible to the TMA unit before first use.
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for the phase with the given parity to complete; false after
// WAIT_LIMIT_CYCLES without it. The limit is counted in SM cycles: reading the
// global timer in the polling loop goes through the same queue as the other
// warps' shared-memory and barrier operations and holds them up for hundreds
// of cycles each.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > WAIT_LIMIT_CYCLES) return false;
    }
    return true;
}

// Values read from shared memory, marked as arrived. A load and what gives its
// buffer back (an mbarrier arrival, the next copy into it) take different
// paths, and the later one can overtake the load. So what gives the buffer back
// takes an address that depends on every value read: bar + (seen & zero), with
// `zero` a kernel argument that is always 0, which the compiler cannot see.
__device__ __forceinline__ void mark_loaded(uint32_t& seen, double v) { seen |= (uint32_t)__double2hiint(v); }

// mbar_wait by a whole converged warp, every lane polling and the warp
// deciding together. The branch is then uniform: lanes that left a polling
// loop of their own at different turns would stay apart until the code joins
// again, which where a failed wait leaves the loop is past its end, and every
// instruction between would issue once per group of lanes.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    const long long t0 = clock64();
    while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
        if (__any_sync(0xffffffffu, clock64() - t0 > WAIT_LIMIT_CYCLES)) return false;
    }
    return true;
}

// One 2-D tile of a tensor map into shared memory, completion counted on bar.
// No multicast: the tile is read from this GPU's memory by this CTA alone.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// The same from a 4-D map.
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int w, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// D(8x8) += A(8x4) B(4x8) in FP64 on the tensor cores. Fragments: a is
// A[lane/4][lane%4], b is B[lane%4][lane/4], d0/d1 are D[lane/4][2*(lane%4)+0/1].
__device__ __forceinline__ void dmma_884(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// Host: a 2-D tensor map over a column-major ComplexF64 matrix (rows x cols,
// leading dimension ld elements), seen as FP64 pairs. A box is 8 complex rows
// (128 bytes, the 128-byte swizzle span) by box_cols columns; rows and
// columns past the matrix read as zero.
int encode_panel_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_cols);

// Host: a 4-D tensor map over `cols` columns of ComplexF64 grid functions on
// nx x ny x nz points (column c at base + c ld, x fastest), seen as FP64
// pairs. A box is box_x by box_y points of one plane; points outside the grid
// read as zero.
int encode_grid_map(CUtensorMap* map, const void* base, int64_t nx, int64_t ny, int64_t nz, int64_t cols, int64_t ld,
                    int box_x, int box_y);

}  // namespace fb
