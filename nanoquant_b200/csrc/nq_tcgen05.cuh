// PTX of the 5th-generation tensor cores, tensor memory and thread-block clusters, as the GEMM kernels use it.
#pragma once

#include <cuda.h>

#include "nq_common.cuh"

namespace nq {

constexpr unsigned kMbarWaitLimit = 1u << 21;   // attempts of up to ~2 us each

// Bounded wait on an mbarrier phase.  Returns false when the limit expired or another
// thread of the CTA already gave up; the caller then leaves its loop.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned* status) {
    if (mbar_try(bar, parity)) return true;   // the common case: already complete
    for (unsigned i = 0; i < kMbarWaitLimit; ++i) {
        if (mbar_try(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    atomicExch(status, (unsigned)(-NQ_ERR_TIMEOUT));
    return false;
}

// The same for a whole warp: every lane returns the same.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, unsigned* status) {
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
    for (unsigned i = 0; i < kMbarWaitLimit; ++i) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
        if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
    }
    *abort_flag = 1;
    if ((threadIdx.x & 31) == 0) atomicExch(status, (unsigned)(-NQ_ERR_TIMEOUT));
    return false;
}
// One lane of the (converged) warp.  The compiler knows that the branch has one thread, which the uniform-register operands of
// tcgen05 and bulk copy instructions profit from.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred != 0;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    const uint32_t lo = ((smem_addr >> 4) & 0x3FFFu) | (1u << 16);          // start address, LBO = 1 (unused)
    const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);             // SBO, version 1, SWIZZLE_128B
    return ((uint64_t)hi << 32) | lo;
}

// Address of this CTA's shared-memory location `local` in the CTA of rank `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_map(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_store4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// The same, counted by an mbarrier of the receiving CTA.
__device__ __forceinline__ void cluster_store4_tx(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];"
                 ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar) : "memory");
}
// mbar_try for a barrier that other CTAs of the cluster signal.
__device__ __forceinline__ bool mbar_try_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(2000u) : "memory");
    return ok != 0;
}

}  // namespace nq
