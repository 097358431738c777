// PTX of the 5th-generation tensor cores, tensor memory and thread-block clusters, as the GEMM kernels use it.
#pragma once

#include <cuda.h>

#include "nq_common.cuh"
#include "nq_stage.h"

namespace nq {

// mbar_try for a barrier that other CTAs of the cluster signal.
__device__ __forceinline__ bool mbar_try_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait of a whole warp on an mbarrier phase; every lane returns the same.  False when `limit` more attempts (of some 4 us each)
// after the first were in vain, which sets the status word, or when another warp of the CTA has already given up; the caller then leaves
// its loop.  `status` and `limit` are taken from the kernel's parameters (__grid_constant__): as constants they occupy no registers.  Read from
// the descriptors' copy in shared memory both GEMMs spilled 8 to 16 bytes (128 tokens module by module 135 -> 133 us without, 517 tokens 186 -> 183).
// CLUSTER: a barrier that other CTAs of the cluster signal.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, unsigned* status, unsigned limit) {
    auto done = [&]() { return __all_sync(0xffffffffu, CLUSTER ? mbar_try_cluster(bar, parity) : mbar_try(bar, parity)); };
    if (done()) return true;   // the common case: already complete
    for (unsigned i = 0; i < limit; ++i) {
        if (done()) return true;
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
// Store to the shared memory of a CTA of the cluster, counted by an mbarrier of that CTA.
__device__ __forceinline__ void cluster_store4_tx(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];"
                 ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar) : "memory");
}

// ---------------------------------------------------------------------------
// sign bits -> the A operand in tensor memory
// ---------------------------------------------------------------------------
// tcgen05.st 16x256b: of a 16-column block of 16 rows, lane 4g + q has the columns 4q..4q+3 (two words) of the rows g and g + 8: what the
// same lane holds in the tile layout.
__device__ __forceinline__ void tmem_st_frag4(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                 "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
// 64 columns of 16 rows: `w` with the bits of column class j at 8 b + j + 4 - (j & 4), half `hf` of the 128 columns -> the words of
// tcgen05.st 16x256b.x4, +-pn.  Two ALU operations per two weights, and a PRMT per two words for all eight classes.  (A PRMT that spreads sign bits
// per two weights beside half a shift before: two layers of 64 / 128 / 256 / 517 tokens, Qwen3-8B 133.6 / 164.2 / 223.0 / 335.8 -> 130.2 /
// 160.3 / 217.4 / 329.4 us, Llama-2-7B 145.3 / 204.0 / 260.2 / 390.8 -> 143.6 / 197.2 / 253.0 / 387.9.  Shifts as products, beside the ALU pipe: level.)
__device__ __forceinline__ void expand_columns(const uint4& w, int hf, const uint2 (&pn)[4], uint32_t (&v)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int sh = 3 - (2 * hf + (i >> 1));
        const uint32_t w0 = (i & 1) ? w.z : w.x, w1 = (i & 1) ? w.w : w.y;
        v[4 * i + 0] = and_xor(spread_bytes(w0, 0) << sh, 0x80008000u, pn[i].x);
        v[4 * i + 1] = and_xor(spread_bytes(w0, 1) << sh, 0x80008000u, pn[i].y);
        v[4 * i + 2] = and_xor(spread_bytes(w1, 0) << sh, 0x80008000u, pn[i].x);
        v[4 * i + 3] = and_xor(spread_bytes(w1, 1) << sh, 0x80008000u, pn[i].y);
    }
}
// The same for +-1 and columns whose middle two of every four are swapped (kOrderIn): the bits of a pair are 16 apart, one ALU
// operation per two weights.
__device__ __forceinline__ void expand_swapped(const uint4& w, int hf, uint32_t one2, uint32_t (&v)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int sh = 3 - (2 * hf + (i >> 1));
        const uint32_t w0 = (i & 1) ? w.z : w.x, w1 = (i & 1) ? w.w : w.y;
        v[4 * i + 0] = and_xor(w0 << (sh + 8), 0x80008000u, one2);
        v[4 * i + 1] = and_xor(w0 << sh, 0x80008000u, one2);
        v[4 * i + 2] = and_xor(w1 << (sh + 8), 0x80008000u, one2);
        v[4 * i + 3] = and_xor(w1 << sh, 0x80008000u, one2);
    }
}
// 0 2 1 3 4 6 5 7
__device__ __forceinline__ int swap_middle(int g) { return (g & 4) | ((g & 1) << 1) | ((g >> 1) & 1); }

// ---------------------------------------------------------------------------
// outputs
// ---------------------------------------------------------------------------
enum : int { kOutFp16, kOutBf16, kOutBf16Saturated };      // kinds of a stage's output, a template argument of the kernels
inline int out_kind(const StageTypes& ty, int saturate) { return !ty.out_bf16 ? kOutFp16 : saturate ? kOutBf16Saturated : kOutBf16; }

__device__ __forceinline__ float io_float(uint16_t h, int is_bf16) {
    return is_bf16 ? __uint_as_float((uint32_t)h << 16) : __half2float(__ushort_as_half(h));
}
// Two outputs, the first in the lower half.
template <int OUT>
__device__ __forceinline__ uint32_t pack_outputs(float o0, float o1, int saturate) {
    uint32_t r;
    if (OUT == kOutBf16Saturated) asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(o1), "f"(o0));
    else if (OUT == kOutBf16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(o1), "f"(o0));
    else {
        if (saturate) { o0 = clamp_or_nan(o0, 64504.0f); o1 = clamp_or_nan(o1, 64504.0f); }
        const __half2 h2 = __floats2half2_rn(o0, o1);
        r = *reinterpret_cast<const uint32_t*>(&h2);
    }
    return r;
}
// Four 8 x 8 matrices, transposed: accumulator fragments (rows across the lanes) -> rows of one token side by side.
__device__ __forceinline__ void stmatrix_trans(uint32_t addr, const uint32_t (&v)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// Eight rows of a token, of which `left` exist; `whole`: all do, at a 16-byte boundary.
__device__ __forceinline__ void store_rows(uint16_t* dst, const uint4& v, int left, bool whole) {
    if (whole) {
        *reinterpret_cast<uint4*>(dst) = v;
    } else {
        const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (e < left) dst[e] = (uint16_t)(vw[e >> 1] >> (16 * (e & 1)));
    }
}

}  // namespace nq
