// Shared helpers of the nanoquant_b200 kernels: status handling, argument
// checks and the bit-order conversions of a 32-column word.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nanoquant_b200.h"

namespace nq {

// Records the text of a failed CUDA runtime call for nq_last_cuda_error().
void set_cuda_error(cudaError_t e, const char* where);

inline int check_cuda(cudaError_t e, const char* where) {
    if (e == cudaSuccess) return NQ_OK;
    set_cuda_error(e, where);
    return NQ_ERR_CUDA;
}

#define NQ_CUDA_TRY(expr)                                             \
    do {                                                              \
        int _s = ::nq::check_cuda((expr), #expr);                     \
        if (_s != NQ_OK) return _s;                                   \
    } while (0)

// Launch errors surface through cudaGetLastError right after the <<<>>>.
#define NQ_LAUNCH_CHECK() NQ_CUDA_TRY(cudaGetLastError())

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

inline cudaStream_t as_stream(nq_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

// Launches `fn` with programmatic stream serialization, so that its prologue overlaps the previous kernel's tail, and the `n` attributes in
// `attrs` (which has room for one more).  If the driver refuses that attribute, plain launches from then on.
int launch_dependent(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attrs, int n, const void* fn, void** args);

// Number of SMs of the current device (cached per device).
int sm_count();

// ---------------------------------------------------------------------------
// launch tags: data that carries its own "ready" flag
// ---------------------------------------------------------------------------
// A producer CTA stores every element of an intermediate as an 8-byte {fp32 value, tag} pair with one 64-bit
// store; a consumer CTA of the same launch loads the pairs it needs and repeats the load until every tag
// equals the tag of this launch.  The first poll after the last producer store has landed already returns
// the data, which takes an arrive / poll / reload sequence (three memory round trips) and any device-wide
// barrier off the critical path.  Consumers spin on other CTAs, so either every CTA of the launch is known to be
// resident, or a consumer that polls in vain computes what is missing itself.
//
// The tag is the launch count of the scratch buffer, read from a 64-bit arrival counter in its header:
// every launch advances it by exactly kTagSpan (the first CTA adds kTagSpan - (CTAs - 1), every other CTA
// adds 1, with a reduction nobody waits for), so the bits above the span are the same for every CTA of a
// launch whenever it reads them (fewer than a span's worth of arrivals can precede the read) and differ from
// those of every recent launch.  Reads and arrivals of a launch must come after the previous launch on the
// scratch has completed (behind griddepcontrol.wait).
//
// The tag (launch_tag) is the launch count modulo 2^20 spread over a NaN pattern that no kernel sharing the scratch stores:
// its upper half is 0x7FF0..0x7FF7 or 0xFFF0..0xFFF7, in fp32 as in both 16-bit formats a NaN, but not the 0x7FFF that
// arithmetic and conversions make of one and that a GEMM stage stores for a token with a NaN (nor the 0xFFFF of a negative
// exponent word, nor the 0 of a zeroed scratch).  An element is rewritten by every launch that uses its address, so a
// stale tag can only match after 2^20 launches in a row that leave it alone.  Waits are bounded: on expiry a status word is
// set and the thread goes on with what it has (the host reports the status).
constexpr unsigned kTagSpan = 1024u;        // > CTAs per tagged launch
constexpr unsigned kSpinLimit = 4000000u;   // default number of polls before a wait gives up
struct TagCtx {
    unsigned tag;        // tag of this launch
    unsigned limit;      // polls a wait of this thread may spend; 0 after an expiry (sticky: one missing
                         // producer costs every thread one limit, not one limit per element it waits for)
    unsigned* status;    // device status word (header word 2)
};
// The launch counter and the status word of the scratch header as they are read: issue the read with the first data
// loads of the kernel and finish it where a tag is first compared or stored, so that the round trips overlap.  A status
// left by an earlier expiry on this scratch disables spinning altogether (the data of such a launch is void anyway).
struct TagRaw {
    unsigned long long counter;
    unsigned status;
};
__device__ __forceinline__ void tag_read(TagRaw& r, const unsigned* header) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(r.counter) : "l"(header) : "memory");
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(r.status) : "l"(header + 2) : "memory");
}
// Bits 0..18 of the launch count below 0x7FF0'0000, bit 19 as the sign.
__device__ __forceinline__ unsigned launch_tag(unsigned long long counter) {
    const unsigned n = (unsigned)(counter / kTagSpan);
    return 0x7FF00000u | (n & 0x7FFFFu) | ((n << 12) & 0x80000000u);
}
__device__ __forceinline__ void tag_finish(TagCtx& tc, const TagRaw& r, unsigned* header, unsigned limit) {
    tc.tag = launch_tag(r.counter);
    tc.limit = r.status ? 0u : limit;
    tc.status = header + 2;
}
__device__ __forceinline__ void tag_wait_expired(TagCtx& tc) {
    atomicExch(tc.status, (unsigned)(-NQ_ERR_TIMEOUT));
    tc.limit = 0u;
}
// This CTA's arrival at the counter.  Issued by one thread, once per launch, after a CTA barrier that every thread
// passes behind the first USE of its tag (a load that has only been issued may still be on its way): the arrival that
// completes the span would otherwise show the next launch's tag to a thread of the same CTA that reads late.
__device__ __forceinline__ void launch_arrive(unsigned long long* counter, bool first_cta, unsigned n_ctas) {
    const unsigned long long w = first_cta ? (unsigned long long)(kTagSpan - (n_ctas - 1)) : 1ull;
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(counter), "l"(w) : "memory");
}
// One 64-bit scalar store: value and tag become visible together (a vector store of two 32-bit words would be two
// accesses in the memory model).
__device__ __forceinline__ void store_tagged(void* base, long long i, float val, unsigned tag) {
    const unsigned long long w = ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(val);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(static_cast<unsigned long long*>(base) + i), "l"(w) : "memory");
}

// ---------------------------------------------------------------------------
// values that are not finite
// ---------------------------------------------------------------------------
// A NaN operand gives NaN (fmaxf and fminf return the other operand and so hide it).
__device__ __forceinline__ float max_or_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_or_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float clamp_or_nan(float v, float lim) { return min_or_nan(max_or_nan(v, -lim), lim); }

// ---------------------------------------------------------------------------
// sign bits
// ---------------------------------------------------------------------------
// (a & m) ^ x as ONE LOP3.  Written as an expression it compiled to two of them (instruction counters: 9 ALU operations per 16 x 16 fragment
// of signs instead of 5), on the half-rate pipe that bounds the expansion of sign bits.  A fragment, shifts and MMA included, takes
// 21.3 -> 16.1 clk of a scheduler (16 warps, registers only); eight Qwen3-8B layers in a graph, four tokens 340.0 -> 326.1 us, sixteen
// 434.6 -> 428.8 (the GEMMs, whose expansion waits for other things, are level).
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t m, uint32_t x) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(r) : "r"(a), "r"(m), "r"(x));   // 0x6A = (0xF0 & 0xCC) ^ 0xAA
    return r;
}
// Bytes {0, 1} and {2, 3} of a word to bytes 1 and 3: bits of neighbouring columns, 8 apart, are then 16 apart.
__device__ __forceinline__ uint32_t spread_bytes(uint32_t w, int pair) { return __byte_perm(w, 0u, pair ? 0x3424 : 0x1404); }

// ---------------------------------------------------------------------------
// mbarriers and bulk copies
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// One bounded attempt: the hardware suspends the thread until the phase completes or its own limit (7760 clk, 4 us; the cluster form in
// nq_tcgen05.cuh has the same) runs out, so a waiting warp does not compete for issue slots.  (No time hint: with one of 2 us the limit was
// 7850 clk, but an attempt on a phase that is already complete took 107 to 134 clk instead of 64 to 82.  Eight layers: one to sixteen tokens
// 0.2 to 0.6 % faster, two layers through the GEMMs 0.5 to 1 %.)
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// ---------------------------------------------------------------------------
// bit orders of a 32-column word
//   lsb_first: element k              -> bit k
//   half2:     element 2j / element 2j+1 -> bit 15-j / bit 31-j
// ---------------------------------------------------------------------------

// keep the even bits of w, squeezed into the low 16 bits
__host__ __device__ inline uint32_t squeeze_even_bits(uint32_t w) {
    uint32_t x = w & 0x55555555u;
    x = (x | (x >> 1)) & 0x33333333u;
    x = (x | (x >> 2)) & 0x0F0F0F0Fu;
    x = (x | (x >> 4)) & 0x00FF00FFu;
    x = (x | (x >> 8)) & 0x0000FFFFu;
    return x;
}

// spread the low 16 bits of v onto the even bit positions
__host__ __device__ inline uint32_t spread_to_even_bits(uint32_t v) {
    uint32_t x = v & 0x0000FFFFu;
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}

__host__ __device__ inline uint32_t reverse16(uint32_t v) {
    v = ((v & 0x5555u) << 1) | ((v >> 1) & 0x5555u);
    v = ((v & 0x3333u) << 2) | ((v >> 2) & 0x3333u);
    v = ((v & 0x0F0Fu) << 4) | ((v >> 4) & 0x0F0Fu);
    v = ((v & 0x00FFu) << 8) | ((v >> 8) & 0x00FFu);
    return v & 0xFFFFu;
}

__host__ __device__ inline uint32_t lsb_to_half2(uint32_t w) {
    uint32_t even = squeeze_even_bits(w);       // elements 0,2,4,.. in bits 0..15
    uint32_t odd = squeeze_even_bits(w >> 1);   // elements 1,3,5,..
    return reverse16(even) | (reverse16(odd) << 16);
}

__host__ __device__ inline uint32_t half2_to_lsb(uint32_t h) {
    uint32_t even = reverse16(h & 0xFFFFu);
    uint32_t odd = reverse16(h >> 16);
    return spread_to_even_bits(even) | (spread_to_even_bits(odd) << 1);
}

__host__ __device__ inline uint32_t convert_order(uint32_t w, int from, int to) {
    if (from == to) return w;
    return from == NQ_LSB_FIRST ? lsb_to_half2(w) : half2_to_lsb(w);
}

}  // namespace nq
