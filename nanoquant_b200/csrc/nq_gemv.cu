// Decode kernel for the binary low-rank linear, one launch per group of linears.
//
//   y = s_out * (U . (s_mid * (V . (s_in * x))))          T <= 4 tokens per launch
//
// For 8B-class layers the launch is a chain of dependent latencies (dependency on the previous kernel, input load,
// main loop, hand-over of the rank-R intermediate between CTAs, main loop, output), not a bandwidth problem: the
// packed factors of a launch are a few MB.  The design keeps every step of that chain short.
//
//  * The packed sign bits are the A operand of an integer tensor-core MMA
//    (mma.sync m16n8k32 s8*s8->s32) WITHOUT unpacking: in the tile layout (see
//    nq_rows_to_tiles) `word & (0x01010101 << j)` is an int8x4 register with values
//    {0, 2^j} ({0, -128} for j = 7), so one LOP3 prepares four weights and the eight
//    masks j = 0..7 consume a whole 32-bit word.  Columns [32j, 32j+32) of a
//    256-column chunk form the "class" j.
//  * The input of a phase (s_in*x, or the rank-R intermediate t) becomes fixed point with one scale per token and
//    CHUNK: a warp takes a (token, chunk) unit, its maximum is one warp reduction, and no CTA-wide maximum (a barrier
//    and a second pass) stands between the load and the conversion.  A column of class j is stored as
//    Z = round(p * inv * 2^(7-j)) (negated for j = 7), at most 23 bits, split into three signed bytes.  2^j * Z is
//    128 * p * inv for every class, so all eight masks accumulate into ONE accumulator per output row and byte
//    term.  The three byte terms of a token are three of the N = 8 MMA columns.
//  * sum(+-p) = sum(p) - 2 * sum_{bit=1}(p): exact int32 per (row, chunk).  These sums go through shared memory and
//    are added in fp32 in an order that depends on nothing but the number of chunks: a linear's result is the same
//    bits alone, in a launch group and however its rows are dealt to CTAs and warps.
//  * The 16 warps of a CTA split its rows x chunks into `wk` chunk slices x `wr` row slices; a warp keeps the B
//    fragments of a chunk in registers for all its rows.
//  * Two CTA barriers per phase: quantised input complete, partial sums complete.
//
// Phases: phase 1 computes t[T,R] (fp32, in scratch), phase 2 computes y.  Several
// linears that share the two phases (q/k/v, gate/up) are processed in one launch.
// There is no device-wide barrier between the phases: every element of t is stored
// together with a tag of the launch and phase 2 polls the elements it needs until
// they carry this launch's tag (nq_common.cuh).  A CTA that polls in vain computes the missing rows itself, once, so no wait
// depends on CTAs that are not running (help_phase1).  From then on only the poll limit ends a wait (two launches that share
// a scratch by mistake overwrite each other's tags): a status word is set and the thread goes on.  The launch has
// programmatic stream serialization: the weight loads of both phases are started before griddepcontrol.wait.
//
// Measured against the first versions of this kernel (cooperative launch, one scale per token, partial sums added with
// shared-memory atomics, weights by cp.async per warp): Qwen3-8B decode, eight layers in a graph, one token 291 -> 250 us, and 217
// with the token count a constant, whole sectors polled, the tag read once per CTA and the scales prefetched.
//
// A SIMT sign-flip-add inner loop issues ~1.5 instructions per weight and tops out
// near one third of the HBM rate on this part, which is why the integer MMA is
// used as a wide dot-product unit here.
//
// replaces: src/nanoquant/kernel/cuda/gemv_kernel.cu:43-301 of the reference
// (two kernels per linear, fp16/bf16 accumulation, sign-flip adds).
#include <cstddef>
#include <cstring>

#include "nq_common.cuh"
#include "nq_plan.h"
#include "nq_stage.h"

namespace nq {

constexpr int kGemvThreads = 512;
constexpr int kGemvWarps = kGemvThreads / 32;
constexpr int kMaxJobs = 4;         // linears per launch
constexpr int kMaxTok = 4;          // tokens per launch (3 byte terms each in two column groups of 8)
constexpr int kMaxCtas = 256;
constexpr float kQMax = 32500.f;    // |p * inv| bound: Z <= kQMax * 2^7 stays inside the magic-number conversion
constexpr int kMaxK = 32768;
constexpr int kMaxChunks = kMaxK / 256;
constexpr size_t kHeaderBytes = 256;
constexpr int kMaxSlots = 8;        // weight blocks in flight
// shared memory: mbarriers; the launch's descriptors; {unit value, sum} per chunk and token; weight slots
constexpr size_t kOffTag = 8 * kMaxSlots, kOffParams = 128, kOffMeta = 1280;
constexpr size_t kFixedBytes = kOffMeta + (size_t)kMaxTok * kMaxChunks * 8;
static_assert(8 * kMaxSlots <= kOffParams && kFixedBytes % 128 == 0, "shared memory map");
constexpr size_t kPartBytes = 32 << 10;    // partial sums of a row block
constexpr size_t kSlotBytes = 64 << 10;    // weights of a row block
constexpr unsigned kWeightWaitLimit = 1u << 20;   // attempts of some 4 us each
constexpr unsigned kPollBackoffNs = 20;    // pause between two polls of the tagged intermediate (100: 0.4 to 0.9 % slower, 300: more)
constexpr unsigned kHelpAfter = 256;       // polls (about 0.1 ms) before a CTA helps; 1/16 of the limit where that is less,
                                           // never with a limit below 16

enum : int { KIND_F16 = 0, KIND_BF16 = 1 };

// One linear's share of a phase, 128 bytes.
struct alignas(16) Job {
    const uint4* tiles;   // [row_groups][chunks][32]
    const void* in;       // [T, ld_in]  fp16/bf16 (phase 1) or tagged fp32 (phase 2)
    const void* pre;      // [K] scale in the I/O dtype (phase 1)
    const void* post;     // [rows] scale in the I/O dtype, or nullptr
    void* out;            // [T, ld_out] tagged fp32 (phase 1) or fp16/bf16 (phase 2)
    const void* bias;     // [rows] in the I/O dtype or nullptr (phase 2)
    const void* resid;    // [T, ld_res] in the I/O dtype or nullptr (phase 2)
    long long ld_in, ld_out, ld_res;
    int rows, K;
    int cta0, ncta;       // CTAs [cta0, cta0 + ncta) work on this job
    int g_q, g_r;         // row groups (16 rows) per CTA of the range: g_q, one more for its first g_r CTAs
    int chunks;           // ceil(K / 256)
    int gb;               // row groups per block (a block's weights and partial sums are in shared memory together)
    uint16_t wk, wr;      // chunk slices x row slices of a CTA's work, one warp each
    int vec;              // phase 1: rows of `in` and `pre` are 16-byte aligned, K a multiple of 8
    int wk_magic, wr_magic;   // ceil(2^16 / wk), ceil(2^16 / wr): exact quotients of what the slices divide
};
static_assert(sizeof(Job) == 128 && offsetof(Job, cta0) == 88, "cta0..g_r are read as two 8-byte words");

struct alignas(16) GemvParams {
    Job job[2 * kMaxJobs];  // phase 1, phase 2
    unsigned* header;       // [0..1] 64-bit arrival counter (launch tags), [2] status, [3] CTAs that have helped
    unsigned spin_limit;    // polls before a wait for the tagged intermediate gives up
    unsigned help_after;    // polls before a CTA computes missing rows of the intermediate itself
    int slots, slot_bytes;  // weight blocks in shared memory
    int xq_off, part_off;   // shared-memory offsets behind the weight slots
    uint8_t cta_job[kMaxCtas];   // per CTA: job of phase 1 + 16 * job of phase 2 (kMaxJobs: none)
};
constexpr int kParamWords = (int)(offsetof(GemvParams, cta_job) + 15) / 16;   // all but the table, rounded up
static_assert(kOffParams + 16 * kParamWords <= kOffMeta, "shared memory map");

template <int KIND>
__device__ __forceinline__ float to_float(uint16_t h) {
    return KIND == KIND_F16 ? __half2float(__ushort_as_half(h)) : __uint_as_float((uint32_t)h << 16);
}

__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---------------------------------------------------------------------------
// input -> fixed point
// ---------------------------------------------------------------------------
// Quantised input in shared memory: per chunk 3*T rows of 256 bytes, row 3*tok + term (term 0 = least significant byte).
// Inside a row the byte of column 32j + 16h + 4q + b sits at unit u = 4*(j/2) + q (16 bytes each, u ^= 4 in odd
// rows), offset 8*(j%2) + 4h + b: lane (g, q) fetches the B registers {k = 4q.., k = 16+4q..} of masks 2i, 2i+1 with
// ONE 128-bit load, and the eight lanes of a load phase (two rows) touch all 32 banks.
__device__ __forceinline__ uint32_t xq_unit(int row, int u) { return (uint32_t)(u ^ ((row & 1) << 2)) * 16u; }

// One unit, token `tok` of a chunk: lane l holds the products of columns 8l..8l+7 of the chunk (zeros beyond K).
// `xq_chunk`: the chunk's rows; `meta`: {unit value, sum} of the unit.
__device__ __forceinline__ void quantise_unit(float (&p)[8], unsigned char* xq_chunk, int tok, int2* meta) {
    const int lane = threadIdx.x & 31, j = lane >> 2;
    float m = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) m = max_or_nan(m, fabsf(p[e]));
    m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));   // as bits: a NaN is above infinity
    float unit = m * (1.0f / (128.f * kQMax));
    if (!(m > 1e-31f && m < 1e37f)) {
        // Below 1e-31 the scale of the integers overflows; above 2^126 (8.5e37) the reciprocal is subnormal, which the approximate one flushes to zero
        // (1e37 keeps a distance from it).  There the same integers come from p * 2^64 or p * 2^-64.
        const float f = m > 0.f && m <= 1e-31f ? 1.8446744e19f : m >= 1e37f && m <= 3.4028235e38f ? 5.4210109e-20f : 0.f;
        // All zero, or not finite.  A value that is not finite makes the unit a NaN, and with it every sum over this
        // chunk and every output of this token, as the same sums in floating point would be (an infinity meets another of
        // the opposite sign); left in, its bits would spill into the bytes of neighbouring columns.
        if (f == 0.f && m != 0.f) unit = __uint_as_float(0x7FFFFFFFu);
        m = f != 0.f ? m * f : 1.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) p[e] = f != 0.f ? p[e] * f : 0.f;
    }
    // The approximate reciprocal is some (1 + d) / m with |d| <= 2^-23.  The integers may be of any unit, as long as it is the one that they
    // are multiplied by again: the unit takes the factor 1 - d = 2 - m * inv.  (The rounded reciprocal is a sequence of dependent
    // instructions and a branch: eight layers, one / two / three tokens, Qwen3-8B 208 / 246 / 322 -> 206 / 240 / 319 us,
    // Llama-3.2-1B 159 / 182 / 231 -> 156 / 179 / 229.)
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(m));
    unit *= fmaf(-m, inv, 2.f);
    // times 2^(7-j), negative for j = 7 (the A operand of class 7 is -128)
    const float inv_j = kQMax * inv * __uint_as_float(j == 7 ? 0xBF800000u : (uint32_t)(127 + 7 - j) << 23);
    // 1.5 * 2^23 + v rounds v to an integer Z in the low mantissa bits (|v| < 2^22).  With 0x8080 added, bytes 0 and 1
    // of the sum are the two low signed bytes of Z with their top bits flipped, and bits 16..22 are the high byte + 64.
    uint32_t z[8], zsum = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        z[e] = __float_as_uint(fmaf(p[e], inv_j, 12582912.f + 32896.f));
        zsum += z[e];
    }
    unsigned char* r0 = xq_chunk + tok * (3 * 256) + 8 * (j & 1) + 2 * (lane & 2);
    const int row0 = 3 * tok, u0 = 4 * (j >> 1) + 2 * (lane & 1);
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const uint32_t* y = z + 4 * w;
        const uint32_t lo01 = __byte_perm(y[0], y[1], 0x5140), lo23 = __byte_perm(y[2], y[3], 0x5140);   // {b0, b0', b1, b1'}
        const uint32_t hi01 = __byte_perm(y[0], y[1], 0x0062), hi23 = __byte_perm(y[2], y[3], 0x0062);   // {b2, b2'}
        const uint32_t b0 = __byte_perm(lo01, lo23, 0x5410) ^ 0x80808080u;
        const uint32_t b1 = __byte_perm(lo01, lo23, 0x7632) ^ 0x80808080u;
        const uint32_t b2 = (__byte_perm(hi01, hi23, 0x5410) + 0x40404040u) ^ 0x80808080u;   // - 64
        *reinterpret_cast<uint32_t*>(r0 + xq_unit(row0, u0 + w)) = b0;
        *reinterpret_cast<uint32_t*>(r0 + 256 + xq_unit(row0 + 1, u0 + w)) = b1;
        *reinterpret_cast<uint32_t*>(r0 + 512 + xq_unit(row0, u0 + w)) = b2;
    }
    int sum = (int)(zsum - 8u * (0x4B400000u + 0x8080u));    // |sum| * 2^j <= 2^25
    sum = __reduce_add_sync(0xffffffffu, j == 7 ? sum * -128 : sum * (1 << j));
    if (lane == 0) *meta = make_int2(__float_as_int(unit), sum);
}

template <int KIND>
__device__ __forceinline__ void to_float8(const uint4& r, float (&v)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (KIND == KIND_F16) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
            v[2 * e] = f.x; v[2 * e + 1] = f.y;
        } else {  // bf16 -> fp32 is a 16-bit shift
            v[2 * e] = __uint_as_float(w[e] << 16);
            v[2 * e + 1] = __uint_as_float(w[e] & 0xFFFF0000u);
        }
    }
}

// Chunks a warp quantises: c, c + step, ... of `chunks`, of each the tokens [t0, t1).  One warp per chunk; with more
// than one token and no more than half as many chunks as warps, two warps share a chunk's tokens.
struct Share {
    int c, step, t0, t1;
};
__device__ __forceinline__ Share share_of(int chunks, int T) {
    const int warp = threadIdx.x >> 5;
    if (T == 1 || 2 * chunks > kGemvWarps) return Share{warp, kGemvWarps, 0, T};
    const int half = (T + 1) >> 1;
    return (warp & 1) ? Share{warp >> 1, kGemvWarps / 2, half, T} : Share{warp >> 1, kGemvWarps / 2, 0, half};
}

// Phase 1: s_in * x.  MT: most tokens of a share.  `also` issues other loads beside the first ones.  The loads of a chunk's tokens, and those of the next chunk, are in
// flight together; the conversion is one body that the tokens are shifted through.
template <int KIND, int MT, typename Also>
__device__ __forceinline__ void quantise_x(const Job& jb, int T, unsigned char* xq, int2* meta, Also also) {
    const int lane8 = (threadIdx.x & 31) * 8, K = jb.K, chunks = jb.chunks;
    const Share sh = share_of(chunks, T);
    const uint16_t* in = static_cast<const uint16_t*>(jb.in) + sh.t0 * jb.ld_in + lane8;
    const uint16_t* pre = static_cast<const uint16_t*>(jb.pre) + lane8;
    const long long ld = jb.ld_in;
    uint4 x[MT], s, xn[MT], sn;
    auto load = [&](int c, uint4 (&xr)[MT], uint4& sr) {
        sr = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int t = 0; t < MT; ++t) xr[t] = make_uint4(0u, 0u, 0u, 0u);
        if (c * 256 + lane8 < K) {
            sr = *reinterpret_cast<const uint4*>(pre + c * 256);
#pragma unroll
            for (int t = 0; t < MT; ++t)
                if (t < sh.t1 - sh.t0) xr[t] = *reinterpret_cast<const uint4*>(in + t * ld + c * 256);
        }
    };
    load(sh.c, x, s);
    also();
#pragma unroll 1
    for (int c = sh.c; c < chunks; c += sh.step) {
        load(c + sh.step, xn, sn);
#pragma unroll 1
        for (int t = sh.t0; t < sh.t1; ++t) {
            float p[8], q[8];
            to_float8<KIND>(x[0], p);
            to_float8<KIND>(s, q);
#pragma unroll
            for (int e = 0; e < 8; ++e) p[e] *= q[e];
            quantise_unit(p, xq + c * T * (3 * 256), t, meta + c * T + t);
#pragma unroll
            for (int k = 0; k + 1 < MT; ++k) x[k] = x[k + 1];
        }
#pragma unroll
        for (int k = 0; k < MT; ++k) x[k] = xn[k];
        s = sn;
    }
}
// The same for inputs of any alignment and size: element loads, lane by lane.
template <int KIND>
__device__ __noinline__ void quantise_x_any(const Job& jb, int T, unsigned char* xq, int2* meta) {
    const int lane8 = (threadIdx.x & 31) * 8, K = jb.K, chunks = jb.chunks;
    const uint16_t* pre = static_cast<const uint16_t*>(jb.pre);
    const Share sh = share_of(chunks, T);
#pragma unroll 1
    for (int c = sh.c; c < chunks; c += sh.step) {
#pragma unroll 1
        for (int t = sh.t0; t < sh.t1; ++t) {
            const uint16_t* in = static_cast<const uint16_t*>(jb.in) + t * jb.ld_in;
            uint16_t x[8], s[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int k = c * 256 + lane8 + e;
                x[e] = k < K ? in[k] : (uint16_t)0;
                s[e] = k < K ? pre[k] : (uint16_t)0;
            }
            float p[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) p[e] = to_float<KIND>(x[e]) * to_float<KIND>(s[e]);
            quantise_unit(p, xq + c * T * (3 * 256), t, meta + c * T + t);
        }
    }
}
// Phase 2: the tagged intermediate, polled until every element of a share's chunk (MT tokens at most) carries this
// launch's tag.  Every element is one 64-bit word {value, tag}: a 64-bit access is single-copy atomic, so a matching
// tag implies its value.  Returns false (for the whole warp) after `help_after` polls in vain for one element, and goes
// on without the data when the limit is spent.
template <int MT>
__device__ __forceinline__ bool quantise_t(const Job& jb, int T, unsigned char* xq, int2* meta, TagCtx& tc, unsigned help_after) {
    constexpr int B = MT > 2 ? 2 : MT;       // tokens whose loads are in flight together
    const int lane8 = (threadIdx.x & 31) * 8, K = jb.K, chunks = jb.chunks;
    const Share sh = share_of(chunks, T);
    const unsigned long long* in = static_cast<const unsigned long long*>(jb.in) + lane8;
    const int ld = (int)jb.ld_in;
#pragma unroll 1
    for (int c = sh.c; c < chunks; c += sh.step) {
        const int left = K - (c * 256 + lane8);      // elements of the row from here on; rows are padded to eight
#pragma unroll 1
        for (int t0 = sh.t0; t0 < sh.t1; t0 += B) {
            float v[B][8];
#pragma unroll 1
            for (unsigned spins = 0;; ++spins) {
                unsigned wrong = 0;
                unsigned long long e[B][8];
#pragma unroll
                for (int i = 0; i < B; ++i)
                    if (left > 0 && t0 + i < sh.t1) {
#pragma unroll
                        for (int u = 0; u < 2; ++u)      // whole sectors: in 16-byte loads every sector was asked for twice (231 -> 217 us)
                            asm volatile("ld.relaxed.gpu.global.v4.b64 {%0,%1,%2,%3}, [%4];"
                                         : "=l"(e[i][4 * u]), "=l"(e[i][4 * u + 1]), "=l"(e[i][4 * u + 2]), "=l"(e[i][4 * u + 3])
                                         : "l"(in + (t0 + i) * ld + c * 256 + 4 * u) : "memory");
                    } else {
#pragma unroll
                        for (int u = 0; u < 8; ++u) e[i][u] = (unsigned long long)tc.tag << 32;
                    }
#pragma unroll
                for (int i = 0; i < B; ++i)
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        wrong |= (unsigned)(e[i][u] >> 32) ^ tc.tag;
                        v[i][u] = __uint_as_float((unsigned)e[i][u]);
                    }
                if (left > 0 && left < 8) {          // the padding of a row is not written
                    wrong = 0;
#pragma unroll
                    for (int i = 0; i < B; ++i)
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            if (u < left) wrong |= (unsigned)(e[i][u] >> 32) ^ tc.tag;
                            else v[i][u] = 0.f;
                        }
                }
                if (__all_sync(0xffffffffu, wrong == 0u)) break;
                if (spins >= tc.limit) { tag_wait_expired(tc); break; }   // the same in every lane
                if (spins >= help_after) return false;
                __nanosleep(kPollBackoffNs);   // failed polls of 148 CTAs load the L2 lines the producers are storing to
            }
#pragma unroll 1
            for (int t = t0; t < t0 + B && t < sh.t1; ++t) {
                quantise_unit(v[0], xq + c * T * (3 * 256), t, meta + c * T + t);
                if (B > 1) {
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[0][u] = v[B - 1][u];
                }
            }
        }
    }
    return true;
}

// ---------------------------------------------------------------------------
// main loop and output of a row block
// ---------------------------------------------------------------------------
// What a warp does in a phase: chunk slice [c0, c1) of row slice rw of wr.
struct Slice {
    int c0, c1, rw;
};
__device__ __forceinline__ Slice slice_of(const Job& jb) {
    const int warp = threadIdx.x >> 5;
    Slice s;
    s.rw = (warp * jb.wk_magic) >> 16;
    const int kc = (warp - s.rw * jb.wk) * jb.chunks;
    s.c0 = (kc * jb.wk_magic) >> 16;
    s.c1 = ((kc + jb.chunks) * jb.wk_magic) >> 16;
    return s;
}
// Floats of a (chunk, token) in the partial sums: 8 mod 32 spreads the tokens over the banks.
__device__ __forceinline__ int part_stride(const Job& jb) { return jb.gb * 16 + 8; }

// Partial sums of `nb` row groups whose weights lie at `weights` (shared memory, or global for kShared = false):
// part[chunk][token][row of the block].
template <int CG, bool kShared>
__device__ __forceinline__ void mma_block(const Job& jb, const Slice& sl, int nb, int T, const unsigned char* weights,
                                          const unsigned char* xq, const int2* meta, float* part) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int chunks = jb.chunks, tok_stride = part_stride(jb), slice = T * tok_stride;
    // rows [r0, r1) of the block (a warp beyond the row slices has none)
    const int r0 = (sl.rw * nb * jb.wr_magic) >> 16, r1 = sl.rw < jb.wr ? ((sl.rw + 1) * nb * jb.wr_magic) >> 16 : 0;
    if (r0 >= r1) return;
    // MMA columns (see above for the rows of xq): CG = 1: column g = term min(g%4, 2) of token g/4; CG = 2: column g
    // of group 0 = term g%2 of token g/2, of group 1 = term 2 of token g/2.  Columns of tokens that do not exist re-read
    // the last one.
    int row_b[CG];
    if (CG == 1) {
        row_b[0] = 3 * min(g >> 2, T - 1) + min(g & 3, 2);
    } else {
        row_b[0] = 3 * min(g >> 1, T - 1) + (g & 1);
        row_b[CG - 1] = 3 * min(g >> 1, T - 1) + 2;
    }
    const int my_tok = CG == 1 ? q >> 1 : q;
    float* my_part = part + my_tok * tok_stride + g + (CG == 1 ? 8 * (q & 1) : 0) + r0 * 16;
#pragma unroll 1
    for (int c = sl.c0; c < sl.c1; ++c) {
        uint32_t b[CG][16];
#pragma unroll
        for (int cg = 0; cg < CG; ++cg) {
            const unsigned char* src = xq + c * T * (3 * 256) + row_b[cg] * 256 + xq_unit(row_b[cg], q);
#pragma unroll
            for (int i = 0; i < 4; ++i) {   // unit 4 * i + q: the flipped bit (4) is bit 0 of i
                const uint4 v = *reinterpret_cast<const uint4*>(src + ((row_b[cg] & 1) ? ((i ^ 1) - 1) * 64 : i * 64));
                b[cg][4 * i] = v.x; b[cg][4 * i + 1] = v.y; b[cg][4 * i + 2] = v.z; b[cg][4 * i + 3] = v.w;
            }
        }
        const int2 mt = meta[c * T + min(my_tok, T - 1)];
        const float d = __int_as_float(mt.x);
        const unsigned char* w = weights + (r0 * chunks + c) * 512 + lane * 16;
        float* dst = my_part + c * slice;
#pragma unroll 1
        for (int r = r0; r < r1; ++r, w += chunks * 512, dst += 16) {
            uint4 t;
            if (kShared) t = *reinterpret_cast<const uint4*>(w);
            else t = __ldg(reinterpret_cast<const uint4*>(w));
            // two accumulator sets: the MMAs of a set depend on each other, and a warp of a small layer has one or
            // two of these steps
            int acc[2][CG][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int cg = 0; cg < CG; ++cg)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[h][cg][i] = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t m = 0x01010101u << j;
#pragma unroll
                for (int cg = 0; cg < CG; ++cg)
                    mma_s8(acc[j & 1][cg], t.x & m, t.y & m, t.z & m, t.w & m, b[cg][2 * j], b[cg][2 * j + 1]);
            }
#pragma unroll
            for (int cg = 0; cg < CG; ++cg)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[0][cg][i] += acc[1][cg][i];
            // sum(+-p) of the chunk = unit * (sum - 2 * S), S the sum over the set bits from its three byte
            // terms: exact modulo 2^32, and the result is below 2^30
            auto bits_sum = [](int t0, int t1, int t2) { return (uint32_t)t0 + ((uint32_t)t1 << 8) + ((uint32_t)t2 << 16); };
            auto value = [&](uint32_t S) { return d * (float)(int)((uint32_t)mt.y - 2u * S); };
            const int* a = acc[0][0];
            if (CG == 1) {
                // lanes 2t (terms 0, 1) and 2t+1 (term 2) of token t trade halves: each keeps one row
                const uint32_t va = (q & 1) ? bits_sum(0, 0, a[0]) : bits_sum(a[0], a[1], 0);   // row g
                const uint32_t vb = (q & 1) ? bits_sum(0, 0, a[2]) : bits_sum(a[2], a[3], 0);   // row g + 8
                const uint32_t other = __shfl_xor_sync(0xffffffffu, (q & 1) ? va : vb, 1);
                if (my_tok < T) dst[0] = value(((q & 1) ? vb : va) + other);
            } else if (my_tok < T) {
                const int* a2 = acc[0][CG - 1];
                dst[0] = value(bits_sum(a[0], a[1], a2[0]));
                dst[8] = value(bits_sum(a[2], a[3], a2[2]));
            }
        }
    }
}

// Outputs of a block: adds the chunks, scales, stores.  Four neighbouring threads share an output (token-major, rows of
// the block): thread i of them adds the chunks c = i mod 4 in order, then the four sums are added pairwise.
struct RawOut {          // scale, bias, residual as loaded: conversions wait for the data, so they come where it is used
    uint32_t post, bias, resid;
};
__device__ __forceinline__ uint32_t load_raw(const void* p, long long i) {   // (a plain 16-bit load is widened, that is waited for, at once)
    uint16_t h;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(h) : "l"(static_cast<const uint16_t*>(p) + i));
    return h;
}
__device__ __forceinline__ uint32_t load_raw_rw(const void* p, long long i) {   // (the residual may be the output buffer)
    uint16_t h;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(h) : "l"(static_cast<const uint16_t*>(p) + i) : "memory");
    return h;
}
__device__ __forceinline__ void output_of(int o, int nb16, int T, int& tok, int& idx) {
    tok = 0; idx = o;
#pragma unroll
    for (int t = 1; t < kMaxTok; ++t)
        if (t < T && idx >= nb16) { idx -= nb16; ++tok; }
}
__device__ __forceinline__ void load_raw_out(RawOut& r, const Job& jb, int row0, int nb16, int T, int o) {
    int tok, idx;
    output_of(o, nb16, T, tok, idx);
    const int row = row0 + idx;
    if (o < T * nb16 && row < jb.rows) {
        if (jb.post) r.post = load_raw(jb.post, row);
        if (jb.bias) r.bias = load_raw(jb.bias, row);
        if (jb.resid) r.resid = load_raw_rw(jb.resid, tok * jb.ld_res + row);
    }
}
// kTagged: the intermediate (fp32 with the launch's tag), else the result.  `raw`: the operands of the first output.
template <int KIND, bool kTagged>
__device__ __forceinline__ void emit_block(const Job& jb, int row0, int nb, int T, const float* part, unsigned tag, RawOut raw) {
    const int i = threadIdx.x & 3, nb16 = nb * 16;
    const int chunks = jb.chunks, tok_stride = part_stride(jb), slice = T * tok_stride;
#pragma unroll 1
    for (int o = (int)threadIdx.x >> 2; (o & ~7) < T * nb16; o += kGemvThreads / 4) {   // whole warps: eight outputs each
        int tok, idx;
        output_of(o, nb16, T, tok, idx);
        const int row = row0 + idx;
        const bool live = o < T * nb16 && row < jb.rows;
        if (o >= kGemvThreads / 4) load_raw_out(raw, jb, row0, nb16, T, o);
        float v = 0.f;
        if (live) {
            const float* src = part + tok * tok_stride + idx + i * slice;
#pragma unroll 4
            for (int c = i; c < chunks; c += 4, src += 4 * slice) v += *src;
        }
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if (live && i == 0) {
            if (jb.post) v *= to_float<KIND>((uint16_t)raw.post);
            if (kTagged) {
                store_tagged(jb.out, tok * jb.ld_out + row, v, tag);
            } else {
                // bias and residual in fp32 behind the output scale; same saturation bounds as the reference epilogue
                if (jb.bias) v += to_float<KIND>((uint16_t)raw.bias);
                if (jb.resid) v += to_float<KIND>((uint16_t)raw.resid);
                constexpr float lim = KIND == KIND_F16 ? 64504.0f : 3.3895313892515355e+38f;
                v = clamp_or_nan(v, lim);
                if (KIND == KIND_F16) static_cast<__half*>(jb.out)[tok * jb.ld_out + row] = __float2half(v);
                else static_cast<__nv_bfloat16*>(jb.out)[tok * jb.ld_out + row] = __float2bfloat16(v);
            }
        }
    }
}

// Phase 1 of a job for every CTA whose rows are not there yet: called by a CTA that has polled in vain for a while.  The
// missing CTAs may not be running (other work holds their SMs), so a wait must not depend on them: this makes the
// launch finish however few of its CTAs run at a time, without the cooperative attribute (which cost 0.5 us per launch in
// a graph and 3 us in a stream).  A row computed twice is written with the same bits.  The header counts the helpers.
template <int KIND, int CG>
__device__ __noinline__ void help_phase1(const Job& jb, int T, unsigned char* xq, int2* meta, float* part, unsigned tag,
                                         unsigned* helpers) {
    const int tid = threadIdx.x;
    if (tid == 0) atomicAdd(helpers, 1u);
    const Slice sl = slice_of(jb);
    bool have_input = false;
    for (int k = 0; k < jb.ncta; ++k) {
        const int b = (int)((blockIdx.x + k) % (unsigned)jb.ncta);       // every helper starts at another share
        const int first = b * jb.g_q + min(b, jb.g_r), groups = jb.g_q + (b < jb.g_r ? 1 : 0);
        bool there = true;
        for (int e = tid; e < T * groups * 16; e += kGemvThreads) {
            const int tok = e / (groups * 16), row = first * 16 + e - tok * groups * 16;
            unsigned long long w = (unsigned long long)tag << 32;
            if (row < jb.rows)
                asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];"
                             : "=l"(w) : "l"(static_cast<unsigned long long*>(jb.out) + tok * jb.ld_out + row) : "memory");
            there = there && (unsigned)(w >> 32) == tag;
        }
        if (__syncthreads_and(there)) continue;
        if (!have_input) {
            quantise_x_any<KIND>(jb, T, xq, meta);
            have_input = true;
            __syncthreads();
        }
        for (int blk = 0; blk < groups; blk += jb.gb) {
            const int nb = min(jb.gb, groups - blk), row0 = (first + blk) * 16;
            mma_block<CG, false>(jb, sl, nb, T, reinterpret_cast<const unsigned char*>(jb.tiles + (size_t)(first + blk) * jb.chunks * 32),
                                 xq, meta, part);
            __syncthreads();
            RawOut raw = {};
            load_raw_out(raw, jb, row0, nb * 16, T, tid >> 2);
            emit_block<KIND, true>(jb, row0, nb, T, part, tag, raw);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
// TOK: tokens of the launch; one column group of 8 MMA columns up to two of them, two from three on.  The count as a constant takes
// loops and divisions out of a chain of dependent instructions: eight layers in a graph, one token, Qwen3-8B 248 -> 238 us, Llama-3.2-1B
// 195 -> 188; with a copy of the code per phase 237 and 183; three tokens 340 -> 332 and 238 -> 234.
//
// The launch takes about 7 us; its 16 warps need 4 issue cycles of every scheduler, 2 ns, for each instruction of the
// common path, and most of them wait for something short.  So the descriptors come into shared memory in one round trip,
// quotients are precomputed, batches go through one copy of the code, nothing lives in local memory (a spilled
// register is a cold line: 40 bytes of stack made the launch 10 % slower), and ONE thread moves the weights: a CTA's row
// groups are contiguous in the tile layout, so a block of them is one bulk copy, and the blocks of both phases that fit
// in shared memory (all of them, for 8B-class layers) are on their way before the dependency wait.
template <int KIND, int TOK>
__global__ void __launch_bounds__(kGemvThreads, 1) gemv_group_kernel(const __grid_constant__ GemvParams Pc) {
    constexpr int CG = TOK <= 2 ? 1 : 2;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t bars = smem_u32(smem);                                  // weight slot s is full: bars + 8 s
    // Nothing is read from the parameter bank but here, in one round trip for all of it: a first touch of a line there
    // costs some 700 cycles, and scalars read where they were needed cost that several times over in every launch.
    // Every warp reads its share with addresses that are the same in all lanes (different ones are served one by one).
    const unsigned my_jobs = Pc.cta_job[blockIdx.x];
    {
        const int warp = tid >> 5;
        uint4 w[(kParamWords + kGemvWarps - 1) / kGemvWarps];
#pragma unroll
        for (int i = 0; i * kGemvWarps < kParamWords; ++i)
            w[i] = reinterpret_cast<const uint4*>(&Pc)[min(warp + i * kGemvWarps, kParamWords - 1)];
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i * kGemvWarps < kParamWords; ++i)
                reinterpret_cast<uint4*>(smem + kOffParams)[min(warp + i * kGemvWarps, kParamWords - 1)] = w[i];
        }
    }
    if (tid >= kGemvThreads - kMaxSlots) {
        mbar_init(bars + 8 * (tid - (kGemvThreads - kMaxSlots)), 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // initialised barriers -> the bulk copies
    }
    __syncthreads();
    const GemvParams& P = *reinterpret_cast<const GemvParams*>(smem + kOffParams);
    const Job* jobs = P.job;
    int2* meta = reinterpret_cast<int2*>(smem + kOffMeta);                 // [chunk][token] {unit value, sum}
    unsigned char* weights = smem + kFixedBytes;
    constexpr int T = TOK;
    const int slots = P.slots, slot_bytes = P.slot_bytes;
    unsigned char* xq = smem + P.xq_off;
    float* part = reinterpret_cast<float*>(smem + P.part_off);
    unsigned* const header = P.header;
    unsigned help_after = P.help_after;
    // This CTA's job in each phase and its row groups of it: every job has a contiguous range of CTAs of its own, so a
    // CTA prepares the input of one job per phase.
    int first[2], groups[2], ji[2];
#pragma unroll
    for (int ph = 0; ph < 2; ++ph) {
        const int i = (int)(my_jobs >> (4 * ph)) & 15;
        ji[ph] = ph * kMaxJobs + min(i, kMaxJobs - 1);
        const Job& jb = jobs[ji[ph]];
        const int2 range = *reinterpret_cast<const int2*>(&jb.cta0), share = *reinterpret_cast<const int2*>(&jb.g_q);
        const int c = (int)blockIdx.x - range.x;
        first[ph] = c * share.x + min(c, share.y);
        groups[ph] = i == kMaxJobs ? 0 : share.x + (c < share.y ? 1 : 0);   // 0: no work in that phase
    }
    // weight blocks in the order they are used: phase, then row groups; block i goes to slot i % slots
    int l_ph = 0, l_g = 0, l_slot = 0;       // next block to load (one thread's)
    auto load_block = [&]() {
        if (l_ph == 0 && l_g >= groups[0]) { l_ph = 1; l_g = 0; }
        if (l_ph == 1 && l_g >= groups[1]) return;
        const Job& jb = jobs[l_ph ? ji[1] : ji[0]];
        const int nb = min(jb.gb, (l_ph ? groups[1] : groups[0]) - l_g);
        const uint32_t bytes = (uint32_t)(nb * jb.chunks) * 512u, bar = bars + 8 * l_slot;
        mbar_expect_tx(bar, bytes);
        bulk_load(smem_u32(weights) + (uint32_t)(l_slot * slot_bytes),
                  jb.tiles + (size_t)((l_ph ? first[1] : first[0]) + l_g) * jb.chunks * 32, bytes, bar);
        l_g += nb;
        l_slot = l_slot + 1 == slots ? 0 : l_slot + 1;
    };
    const bool loader = tid == kGemvThreads - kMaxSlots;
    if (loader) {
#pragma unroll 1
        for (int s = 0; s < slots; ++s) load_block();
    }
    // Scales on their way to L2: a model's are in memory when its turn comes, and the input's would be waited for beside the input
    // (eight Qwen3-8B layers at one token 223.5 -> 217.0 us; one bulk prefetch of the input's alone 221.9).
    if (tid < 64) {
#pragma unroll
        for (int ph = 0; ph < 2; ++ph) {
            if (groups[ph] == 0) continue;
            const Job& jb = jobs[ji[ph]];
            if (ph == 0)
                for (int k = 64 * tid; k < jb.K; k += 64 * 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint16_t*>(jb.pre) + k));
            if (jb.post && 64 * tid < 16 * groups[ph])
                asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint16_t*>(jb.post) + min(16 * first[ph] + 64 * tid, jb.rows - 1)));
        }
    }
    // Programmatic dependent launch: everything above may overlap with the tail of the previous kernel in the stream;
    // activations and scratch (shared with that kernel) are only touched after it has completed.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // let the next kernel begin its prologue wherever an SM frees up
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    TagCtx tc;

    int slot = 0;                            // of the next weight block, and its barrier's phase
    uint32_t parity = 0;
    // A copy of the code for each phase: the compiler then keeps the phase's descriptor in fewer registers.  (One copy for both, while the
    // token count was not a constant either: 250 us and 254; now 234 and 231.)
#pragma unroll 2
    for (int ph = 0; ph < 2; ++ph) {
        const int my_groups = ph ? groups[1] : groups[0], row0 = 16 * (ph ? first[1] : first[0]);
        const Job& jb = jobs[ph ? ji[1] : ji[0]];
        const Slice sl = slice_of(jb);
        // Operands of this thread's first output: needed behind the loop, on their way from here.  (They and the tag are
        // not carried around a loop: that would copy the registers, and the copy would wait for the loads.)
        RawOut raw0 = {};
        if (ph == 0) {
            // Tag of this launch: one thread's read, used behind the barrier; the round trip overlaps the input loads.  (Read by every
            // warp it was 16 requests of each CTA for one line of L2, and the launch 1 to 5 % slower.)
            TagRaw tag_raw = {};
            if (tid == kGemvThreads - 1) tag_read(tag_raw, header);
            if (my_groups > 0) {
                // (The operands of the output beside the first loads of the input; behind its conversion they were waited for: eight layers, one / two / three
                // tokens, Qwen3-8B 215 / 251 / 329 -> 209 / 247 / 325 us, Llama-3.2-1B 164 / 186 / 234 -> 159 / 182 / 232.)
                auto operands = [&]() { load_raw_out(raw0, jb, row0, min(jb.gb, my_groups) * 16, T, tid >> 2); };
                if (jb.vec) quantise_x<KIND, TOK>(jb, T, xq, meta, operands);
                else {
                    quantise_x_any<KIND>(jb, T, xq, meta);
                    operands();
                }
            }
            if (tid == kGemvThreads - 1) *reinterpret_cast<TagRaw*>(smem + kOffTag) = tag_raw;
            __syncthreads();   // quantised input complete
            tag_finish(tc, *reinterpret_cast<const TagRaw*>(smem + kOffTag), header, P.spin_limit);
        } else if (my_groups > 0) {
            load_raw_out(raw0, jb, row0, min(jb.gb, my_groups) * 16, T, tid >> 2);
            while (!__syncthreads_and(quantise_t<TOK>(jb, T, xq, meta, tc, help_after))) {
                help_phase1<KIND, CG>(jobs[ji[1] - kMaxJobs], T, xq, meta, part, tc.tag, header + 3);
                help_after = ~0u;     // every row has carried the tag now: what is missing again, another launch overwrites
            }
        }
#pragma unroll 1
        for (int blk = 0; blk < my_groups; blk += jb.gb) {
            const int nb = min(jb.gb, my_groups - blk);
#pragma unroll 1
            for (unsigned spins = 0; !mbar_try(bars + 8 * slot, parity); ++spins)
                if (spins >= kWeightWaitLimit) { tag_wait_expired(tc); break; }
            mma_block<CG, true>(jb, sl, nb, T, weights + slot * slot_bytes, xq, meta, part);
            __syncthreads();   // partial sums complete, this block's weights have been read
            if (++slot == slots) { slot = 0; parity ^= 1u; }
            if (loader) load_block();
            // every thread has compared or stored the tag, or never will
            if (ph == 1 && blk == 0 && tid == kGemvThreads - 1) launch_arrive(reinterpret_cast<unsigned long long*>(header), blockIdx.x == 0, gridDim.x);
            RawOut raw = raw0;
            if (blk > 0) load_raw_out(raw, jb, row0 + blk * 16, nb * 16, T, tid >> 2);
            if (ph == 0) emit_block<KIND, true>(jb, row0 + blk * 16, nb, T, part, tc.tag, raw);
            else emit_block<KIND, false>(jb, row0 + blk * 16, nb, T, part, tc.tag, raw);
            if (blk + jb.gb < my_groups) __syncthreads();   // the partial sums have been read
        }
    }
    if (groups[1] == 0) {
        __syncthreads();
        if (tid == 0) launch_arrive(reinterpret_cast<unsigned long long*>(header), blockIdx.x == 0, gridDim.x);
    }
}

static size_t round_up(size_t v, size_t m) { return (v + m - 1) / m * m; }

template <int KIND>
static const void* gemv_kernel_of(int tokens) {
    return tokens == 1 ? (const void*)gemv_group_kernel<KIND, 1> : tokens == 2 ? (const void*)gemv_group_kernel<KIND, 2>
           : tokens == 3 ? (const void*)gemv_group_kernel<KIND, 3> : (const void*)gemv_group_kernel<KIND, kMaxTok>;
}
static const void* gemv_kernel(int kind, int tokens) { return kind == KIND_F16 ? gemv_kernel_of<KIND_F16>(tokens) : gemv_kernel_of<KIND_BF16>(tokens); }

// Opt-in shared memory limit of every instantiation, set once per device.
static int dynamic_smem_limit(int dev, int* out) {
    static int cached[64];
    if (cached[dev & 63] == 0) {
        int optin = 0, lim = 1 << 30;
        NQ_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        for (int i = 0; i < 2 * kMaxTok; ++i) {
            const void* fn = gemv_kernel(i & 1 ? KIND_BF16 : KIND_F16, 1 + i / 2);
            cudaFuncAttributes fa;
            NQ_CUDA_TRY(cudaFuncGetAttributes(&fa, fn));
            const int v = optin - (int)fa.sharedSizeBytes;  // the opt-in limit covers static + dynamic
            NQ_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, v));
            lim = v < lim ? v : lim;
        }
        cached[dev & 63] = lim;
    }
    *out = cached[dev & 63];
    return NQ_OK;
}

// Chunk slices x row slices of the 16 warps for `groups` row groups of `chunks` chunks.  A step (512 bytes of weights)
// costs about twice as much as fetching the B fragments of a chunk once.
static void split_warps(int groups, int chunks, Job& j) {
    int best = 1 << 30;
    for (int k = 1; k <= kGemvWarps && k <= chunks; ++k) {
        int r = kGemvWarps / k;
        if (r > groups) r = groups;
        const int cost = ((chunks + k - 1) / k) * (2 * ((groups + r - 1) / r) + 1);
        if (cost < best) { best = cost; j.wk = (uint16_t)k; j.wr = (uint16_t)r; }
    }
    j.wk_magic = (65536 + j.wk - 1) / j.wk;
    j.wr_magic = (65536 + j.wr - 1) / j.wr;
}

// ---------------------------------------------------------------------------
// GEMV without caller-provided scratch
// ---------------------------------------------------------------------------
// Scratch of nq_gemv_fwd_static: lives in the library image on every GPU that loads it, until
// the process exits.  256-byte header + tagged fp32 intermediate (8 bytes per element) for up to 4 tokens x rank 8192.
constexpr int kStaticMaxRank = 8192;
constexpr size_t kStaticScratchBytes = kHeaderBytes + (size_t)kMaxTok * kStaticMaxRank * sizeof(uint2);
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// Device address of g_static_scratch on the current device.  In host code the symbol name is
// only a handle: the address a kernel can use comes from cudaGetSymbolAddress, looked up once
// per device with that device current.  The cached address stays valid as long as the device's
// primary context is not reset.
static int static_scratch_ptr(void** out) {
    static void* cached[64];
    int dev = 0;
    NQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return NQ_ERR_UNSUPPORTED;
    if (!cached[dev]) {
        void* p = nullptr;
        NQ_CUDA_TRY(cudaGetSymbolAddress(&p, g_static_scratch));
        if (!p) return NQ_ERR_CUDA;
        cached[dev] = p;
    }
    *out = cached[dev];
    return NQ_OK;
}

// {fp32, tag} words of a linear's intermediate, rows padded to eight elements
static size_t intermediate_bytes(int R) { return round_up((size_t)kMaxTok * (size_t)((R + 7) / 8 * 8) * sizeof(uint2), 256); }

// Four tokens of a linear by the batch kernel's two launches instead of one of the decode kernel.  Every CTA of the
// decode kernel converts the whole input and the whole intermediate of its linear to fixed point, and at four tokens that
// is the largest part of a launch; the batch kernel takes 16-bit floats as they come, with the intermediate as value and
// remainder, at eight columns of which it computes all anyway.  (Three tokens measured level and stay.)
//
// The rule looks at the linear alone, so that a module and a launch group give it the same bits, and at the size that the
// linears of a group share, so that a group is not torn apart.  The line: input of 14 chunks and more (above 3328
// columns).  us at four tokens, 0.8 bits per weight, one launch -> two:
//                                    2048 columns       3072              3584              4096              8192
//   q/k/v, in a graph                6.2 -> 4.8        7.8 -> 5.2        8.8 -> 6.2        8.8 -> 6.5       14.9 -> 12.1
//   gate/up, in a graph              7.9 -> 6.0       10.1 -> 8.0       12.4 -> 9.3       13.8 -> 11.1      40.5 -> 36.5
//   square linear alone, in a graph  6.0 -> 4.7        7.2 -> 5.1        8.0 -> 5.4        8.3 -> 5.7       13.8 -> 9.6
//   square linear called eagerly     5.8 -> 7.7        7.0 -> 7.9        7.9 -> 7.8        8.1 -> 7.9       13.7 -> 9.7
//   its quarter (k) called eagerly   5.3 -> 7.5        6.1 -> 7.7        6.5 -> 7.6        6.6 -> 7.7        9.6 -> 7.7
// A graph gains from 2048 columns on, but a call in a stream is bound by the host there, which pays 2 us for the second
// launch; from 3584 on the seven linears of a layer gain called one by one as well, though not the smallest of them.
constexpr int kTwoStageChunks = 14;
static bool takes_two_stages(const nq_linear_desc& L) {
    return (L.N + 255) / 256 >= kTwoStageChunks && L.N % 8 == 0 && L.R % 8 == 0 && L.ldx % 8 == 0 && aligned16(L.x) &&
           aligned16(L.s_in) && batch_fragment_bytes(2 * kSplitTokens, L.R) <= intermediate_bytes(L.R);   // (ranks from 128)
}
static int launch_two_stages(const nq_linear_desc* d, int n, int t0, int dtype, void* scratch, cudaStream_t stream) {
    StageJob s1[kMaxJobs], s2[kMaxJobs];
    size_t off = kHeaderBytes;
    for (int i = 0; i < n; ++i) {
        const nq_linear_desc& L = d[i];
        void* t = static_cast<char*>(scratch) + off;
        off += intermediate_bytes(L.R);
        s1[i] = {static_cast<const uint16_t*>(L.x) + (size_t)t0 * L.ldx, L.ldx, L.v_tiles, L.s_in, L.s_mid, t, L.R, L.N, L.R, nullptr, nullptr, 0, nullptr};
        s2[i] = {t, L.R, L.u_tiles, nullptr, L.s_out, static_cast<uint16_t*>(L.y) + (size_t)t0 * L.ldy, L.ldy, L.R, L.M, L.bias,
                 L.residual ? static_cast<const uint16_t*>(L.residual) + (size_t)t0 * L.ldr : nullptr, L.ldr, nullptr};
    }
    const int b16 = dtype == NQ_BF16;
    unsigned* status = static_cast<unsigned*>(scratch) + 2;
    const int st = launch_batch_stage(s1, n, kSplitTokens, StageTypes{b16, b16, 1, 0}, 0, false, true, true, status, stream);
    return st != NQ_OK ? st : launch_batch_stage(s2, n, kSplitTokens, StageTypes{b16, 1, b16, 0}, 1, true, false, true, status, stream);
}

static unsigned g_spin_limit = kSpinLimit;   // polls before a wait for the tagged intermediate gives up

}  // namespace nq

using namespace nq;

extern "C" {

size_t nq_gemv_scratch_bytes(int T, int N, int R, int M) {
    if (T <= 0 || N <= 0 || R <= 0 || M <= 0) return 0;
    return kHeaderBytes + intermediate_bytes(R);
}

size_t nq_gemv_group_scratch_bytes(const nq_linear_desc* d, int n_linears, int T) {
    if (!d || n_linears <= 0 || n_linears > kMaxJobs || T <= 0) return 0;
    size_t b = kHeaderBytes;
    for (int i = 0; i < n_linears; ++i) {
        if (d[i].R <= 0) return 0;
        b += intermediate_bytes(d[i].R);
    }
    return b;
}

static int check_group(const nq_linear_desc* d, int n_linears, int T, int dtype, const void* scratch, size_t scratch_bytes) {
    if (!d || !scratch) return NQ_ERR_NULL;
    if (n_linears <= 0 || n_linears > kMaxJobs) return NQ_ERR_UNSUPPORTED;
    if (T <= 0) return NQ_ERR_SHAPE;
    if (dtype != NQ_F16 && dtype != NQ_BF16) return NQ_ERR_DTYPE;
    if (!aligned16(scratch)) return NQ_ERR_ALIGN;
    if (scratch_bytes < nq_gemv_group_scratch_bytes(d, n_linears, T)) return NQ_ERR_SCRATCH;
    for (int i = 0; i < n_linears; ++i) {
        const nq_linear_desc& L = d[i];
        if (!L.x || !L.s_in || !L.v_tiles || !L.u_tiles || !L.s_out || !L.y) return NQ_ERR_NULL;
        if (L.N <= 0 || L.R <= 0 || L.M <= 0) return NQ_ERR_SHAPE;
        if (L.ldx < L.N || L.ldy < L.M) return NQ_ERR_SHAPE;
        if (L.residual && L.ldr < L.M) return NQ_ERR_SHAPE;
        if (L.N > kMaxK || L.R > kMaxK) return NQ_ERR_UNSUPPORTED;
        if (!aligned16(L.v_tiles) || !aligned16(L.u_tiles)) return NQ_ERR_ALIGN;
    }
    return NQ_OK;
}

// Tokens [t_first, T) of a group that check_group has passed, by the decode kernel.
static int launch_decode(const nq_linear_desc* d, int n_linears, int t_first, int T, int dtype, void* scratch, nq_stream_t stream) {
    int max_chunks = 0;
    int rg[2][kMaxJobs], ck[2][kMaxJobs];      // row groups and chunks of the two phases
    size_t packed = 0;
    for (int i = 0; i < n_linears; ++i) {
        const nq_linear_desc& L = d[i];
        rg[0][i] = (L.R + 15) / 16; ck[0][i] = (L.N + 255) / 256;
        rg[1][i] = (L.M + 15) / 16; ck[1][i] = (L.R + 255) / 256;
        for (int ph = 0; ph < 2; ++ph) max_chunks = ck[ph][i] > max_chunks ? ck[ph][i] : max_chunks;
        packed += (size_t)L.R * ((size_t)L.N + L.M) / 8;
    }
    int dev = 0, smem_limit = 0;
    NQ_CUDA_TRY(cudaGetDevice(&dev));
    {
        const int st = dynamic_smem_limit(dev, &smem_limit);
        if (st != NQ_OK) return st;
    }
    GemvParams P;
    memset(&P, 0, sizeof(P));
    P.header = static_cast<unsigned*>(scratch);
    P.spin_limit = g_spin_limit;
    P.help_after = g_spin_limit < 16 ? ~0u : g_spin_limit / 16 < kHelpAfter ? g_spin_limit / 16 : kHelpAfter;

    // One CTA per SM, fewer for launches with less than 2.25 MB of packed factors: their row groups do not divide any finer by
    // 148, every CTA fetches the whole input and polls the whole intermediate, and the SMs left free let CTAs of the next launch in.  One
    // token, us per launch in a graph by CTAs (52 / 74 / 103 / 148):
    //   0.4 MB (4096 -> 1024)  4.5 / 4.5 / 4.5 / 4.5      2.1 MB (8192 -> 2048)           6.0 / 5.8 / 5.7 / 5.7
    //   0.7 MB (q/k/v of 2048) 4.5 / 4.4 / 4.5 / 4.5      2.4 MB (q/k/v of 4096)          6.1 / 5.7 / 5.2 / 5.2
    //   1.7 MB (4096 -> 4096)  5.4 / 5.2 / 5.2 / 5.2      4.1 MB (gate/up of 2048)        8.6 / 6.5 / 6.3 / 5.7
    //   1.8 MB (3072 -> 3072)  5.5 / 5.2 / 5.1 / 5.2      5.0 MB (12288 -> 4096)          9.3 / 8.9 / 7.2 / 7.0
    // (While the intermediate was polled in 16-byte loads the line was at 3 MB.  Eight layers, 3 MB and now, one / two / three tokens: 4096
    // columns 216.0 / 253.8 / 331.4 -> 215.3 / 252.2 / 328.9, 3072 columns 188.8 / 217.5 / 276.9 -> 187.4 / 215.2 / 273.0.)
    int grid = sm_count() < kMaxCtas ? sm_count() : kMaxCtas;
    if (packed < ((size_t)9 << 18)) grid = grid * 7 / 10;
    {   // no more CTAs than the larger phase has row groups
        int g[2] = {0, 0};
        for (int i = 0; i < n_linears; ++i) { g[0] += rg[0][i]; g[1] += rg[1][i]; }
        const int most = g[0] > g[1] ? g[0] : g[1];
        if (grid > most) grid = most;
        if (grid < n_linears) grid = n_linears;
    }
    // tokens are processed in groups that fit the MMA columns (3 per token) and shared memory: the quantised input,
    // one row group's weights and its partial sums at least
    int tg = T - t_first < kMaxTok ? T - t_first : kMaxTok;
    auto fixed_bytes = [&](int t) { return kFixedBytes + (size_t)3 * t * max_chunks * 256; };
    const size_t least = (size_t)max_chunks * 512, least_part = (size_t)max_chunks * (16 + 8) * 4;   // part: per token
    while (tg > 1 && fixed_bytes(tg) + least + tg * least_part > (size_t)smem_limit) --tg;
    if (fixed_bytes(tg) + least + tg * least_part > (size_t)smem_limit) return NQ_ERR_UNSUPPORTED;

    int cta_n[2][kMaxJobs];
    for (int ph = 0; ph < 2; ++ph) deal_ctas(grid, n_linears, rg[ph], ck[ph], cta_n[ph]);

    const size_t esz = 2;
    for (int t0 = t_first; t0 < T; t0 += tg) {
        const int tn = (T - t0) < tg ? (T - t0) : tg;
        memset(P.cta_job, kMaxJobs * 17, sizeof(P.cta_job));
        // room for a block's partial sums and weights; a single row group is always allowed (see above)
        const size_t room = smem_limit - fixed_bytes(tn);
        const size_t slot_room = room / 2 < kSlotBytes ? room / 2 : kSlotBytes;
        const size_t slot_most = slot_room > least ? slot_room : least;
        const size_t part_room = room - slot_most < kPartBytes ? room - slot_most : kPartBytes;
        size_t part_used = 0, slot_used = 0;
        int most_blocks = 0;
        // the intermediate is loaded in 32 bytes: 16 back into the unused end of the header for a scratch between two multiples of 32
        size_t off = kHeaderBytes - (reinterpret_cast<uintptr_t>(scratch) & 16);
        int cta[2] = {0, 0};            // first CTA of the next job's range in the two phases
        for (int i = 0; i < n_linears; ++i) {
            const nq_linear_desc& L = d[i];
            void* tbuf = static_cast<char*>(scratch) + off;   // {fp32, tag} pairs, 8 bytes per element
            const int ld_t = (L.R + 7) / 8 * 8;               // rows of the intermediate start on 64-byte boundaries
            off += intermediate_bytes(L.R);
            Job& a = P.job[i];
            a.tiles = static_cast<const uint4*>(L.v_tiles);
            a.in = static_cast<const char*>(L.x) + (size_t)t0 * L.ldx * esz;
            a.pre = L.s_in;
            a.post = L.s_mid;
            a.out = tbuf;
            a.ld_in = L.ldx;
            a.ld_out = ld_t;
            a.rows = L.R;
            a.K = L.N;
            a.vec = (L.N % 8 == 0) && (L.ldx % 8 == 0) && aligned16(a.in) && aligned16(L.s_in);
            Job& b = P.job[kMaxJobs + i];
            b.tiles = static_cast<const uint4*>(L.u_tiles);
            b.in = tbuf;
            b.post = L.s_out;
            b.out = static_cast<char*>(L.y) + (size_t)t0 * L.ldy * esz;
            b.bias = L.bias;
            b.resid = L.residual ? static_cast<const char*>(L.residual) + (size_t)t0 * L.ldr * esz : nullptr;
            b.ld_res = L.ldr;
            b.ld_in = ld_t;
            b.ld_out = L.ldy;
            b.rows = L.M;
            b.K = L.R;
            for (int ph = 0; ph < 2; ++ph) {
                Job& j = P.job[ph * kMaxJobs + i];
                j.chunks = ck[ph][i];
                j.cta0 = cta[ph];
                j.ncta = cta_n[ph][i];
                j.g_q = rg[ph][i] / j.ncta;
                j.g_r = rg[ph][i] % j.ncta;
                for (int c = 0; c < j.ncta; ++c) {
                    uint8_t& m = P.cta_job[cta[ph] + c];
                    m = (uint8_t)(ph ? (m & 0x0F) | (i << 4) : (m & 0xF0) | i);
                }
                cta[ph] += j.ncta;
                // blocks of row groups whose weights and partial sums fit their space, as equal as possible
                const int most = j.g_q + (j.g_r ? 1 : 0);
                auto part_bytes = [&](int gb) { return (size_t)j.chunks * tn * (gb * 16 + 8) * 4; };
                for (int blocks = 1;; ++blocks) {
                    j.gb = (most + blocks - 1) / blocks;
                    if (j.gb == 1 || (part_bytes(j.gb) <= part_room && (size_t)j.gb * j.chunks * 512 <= slot_room && j.gb <= 128)) break;
                }
                split_warps(j.gb, j.chunks, j);
                const size_t part = part_bytes(j.gb), slot = (size_t)j.gb * j.chunks * 512;
                part_used = part > part_used ? part : part_used;
                slot_used = slot > slot_used ? slot : slot_used;
                const int blocks = (most + j.gb - 1) / j.gb;
                most_blocks = blocks > most_blocks ? blocks : most_blocks;
            }
        }
        int slots = 2 * most_blocks;      // no CTA has more blocks than that in its two phases
        if (slots > kMaxSlots) slots = kMaxSlots;
        while (slots > 1 && fixed_bytes(tn) + part_used + slots * slot_used > (size_t)smem_limit) --slots;
        P.slots = slots;
        P.slot_bytes = (int)slot_used;
        P.xq_off = (int)(kFixedBytes + slots * slot_used);
        P.part_off = P.xq_off + 3 * tn * max_chunks * 256;
        const size_t smem_bytes = P.part_off + part_used;
        if (smem_bytes > (size_t)smem_limit) return NQ_ERR_UNSUPPORTED;
        void* args[] = {&P};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(kGemvThreads);
        cfg.dynamicSmemBytes = smem_bytes;
        cfg.stream = as_stream(stream);
        cudaLaunchAttribute attr[1];
        const int st = launch_dependent(cfg, attr, 0, gemv_kernel(dtype, tn), args);
        if (st != NQ_OK) return st;
    }
    return NQ_OK;
}

int nq_gemv_group_fwd(const nq_linear_desc* d, int n_linears, int T, int dtype, void* scratch, size_t scratch_bytes,
                      nq_stream_t stream) {
    const int st = check_group(d, n_linears, T, dtype, scratch, scratch_bytes);
    return st != NQ_OK ? st : launch_decode(d, n_linears, 0, T, dtype, scratch, stream);
}

int nq_decode_group_fwd(const nq_linear_desc* d, int n_linears, int T, int dtype, void* scratch, size_t scratch_bytes,
                        nq_stream_t stream) {
    int st = check_group(d, n_linears, T, dtype, scratch, scratch_bytes);
    const int whole = T - T % kSplitTokens;
    if (st != NQ_OK || whole == 0) return st != NQ_OK ? st : launch_decode(d, n_linears, 0, T, dtype, scratch, stream);
    // Each linear by its own rule (the linears of a layer that share their input share it, too), one set of launches for
    // those of a kind; the launches follow one another, so they use the same scratch.
    nq_linear_desc two[kMaxJobs], one[kMaxJobs];
    int n_two = 0, n_one = 0;
    for (int i = 0; i < n_linears; ++i) {
        if (takes_two_stages(d[i])) two[n_two++] = d[i];
        else one[n_one++] = d[i];
    }
    for (int t0 = 0; n_two > 0 && st == NQ_OK && t0 < whole; t0 += kSplitTokens)
        st = launch_two_stages(two, n_two, t0, dtype, scratch, as_stream(stream));
    if (n_two > 0 && st == NQ_OK && whole < T) st = launch_decode(two, n_two, whole, T, dtype, scratch, stream);
    if (n_one > 0 && st == NQ_OK) st = launch_decode(one, n_one, 0, T, dtype, scratch, stream);
    return st;
}

int nq_gemv_fwd(const void* x, const void* s_in, const void* v_tiles, const void* s_mid,
                const void* u_tiles, const void* s_out, void* y, void* scratch, size_t scratch_bytes,
                int T, int N, int R, int M, int dtype, nq_stream_t stream) {
    nq_linear_desc d;
    memset(&d, 0, sizeof(d));
    d.x = x; d.s_in = s_in; d.v_tiles = v_tiles; d.s_mid = s_mid; d.u_tiles = u_tiles; d.s_out = s_out;
    d.y = y; d.N = N; d.R = R; d.M = M; d.ldx = N; d.ldy = M;
    return nq_gemv_group_fwd(&d, 1, T, dtype, scratch, scratch_bytes, stream);
}

int nq_gemv_fwd_static(const void* x, const void* s_in, const void* v_tiles, const void* s_mid,
                       const void* u_tiles, const void* s_out, void* y,
                       int T, int N, int R, int M, int dtype, nq_stream_t stream) {
    if (T <= 0 || N <= 0 || R <= 0 || M <= 0) return NQ_ERR_SHAPE;
    if (R > kStaticMaxRank || nq_gemv_scratch_bytes(T, N, R, M) > kStaticScratchBytes) return NQ_ERR_TOO_LARGE;
    void* scratch = nullptr;
    const int st = static_scratch_ptr(&scratch);   // first call on a device: symbol lookup
    if (st != NQ_OK) return st;
    // Nothing has to be cleared between calls: the array is zero when the library is loaded, the arrival
    // counter in its header runs freely (every launch derives a fresh tag from it) and stale intermediate
    // elements carry older tags.
    return nq_gemv_fwd(x, s_in, v_tiles, s_mid, u_tiles, s_out, y, scratch, kStaticScratchBytes, T, N, R, M, dtype,
                       stream);
}

size_t nq_gemv_static_max_rank(void) { return (size_t)kStaticMaxRank; }

unsigned nq_gemv_set_wait_limit(unsigned polls) {
    const unsigned old = g_spin_limit;
    g_spin_limit = polls ? polls : kSpinLimit;
    return old;
}

int nq_scratch_status(const void* scratch, nq_stream_t stream) {
    if (!scratch) {   // the array of nq_gemv_fwd_static
        void* p = nullptr;
        const int st = static_scratch_ptr(&p);
        if (st != NQ_OK) return st;
        scratch = p;
    }
    unsigned h[4] = {0, 0, 0, 0};
    NQ_CUDA_TRY(cudaMemcpyAsync(h, scratch, sizeof(h), cudaMemcpyDeviceToHost, as_stream(stream)));
    NQ_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    return h[2] == 0 ? NQ_OK : -(int)h[2];
}

}  // extern "C"
