// One stage of a decode batch (5 to 16 tokens, and split four): Out[T, rows] = (A[T, K] . W[rows, K]^T) * post.
//
// At these sizes a stage is a few microseconds of fixed chain around very little arithmetic.  The tcgen05 GEMM spends 12 to
// 13 us on it: 128-row tiles leave most SMs idle unless K is split, and the split costs slabs or a cluster exchange.
// Here the unit of work is a row group of 16 weight rows, as in the decode kernel (nq_gemv.cu): every linear of the
// launch has a contiguous range of CTAs, a CTA owns a few row groups and all of K, its 16 warps split chunks (256
// columns) x row groups, and the partial sums of the chunk slices meet in shared memory.
//
//  * Weights: a CTA's row groups are contiguous in the tile layout; ONE thread fetches them as bulk copies before the
//    dependency wait, all of them where they fit.
//  * mma.sync m16n8k16 (16 rows x 8 tokens).  The bits of columns {4q, 4q+2} and {4q+1, 4q+3} of a 16-column block are
//    16 apart in the lane's word, so a shift and ONE LOP3 ((word & 0x80008000) ^ {s, s'}) make an A register +-s: the
//    product x * (+-s_in) is exact.  The columns of a block may be permuted as long as A and B agree, so the B fragment
//    of a token is its four consecutive columns 4q..4q+3.
//  * B fragments.  The intermediate is stored in fragment order (see fragment_index): a warp's load of one is 256
//    contiguous bytes.  Activations come in rows: every warp stages its own columns through shared memory with 16-byte
//    copies, 192 of them in flight.  (Fragments loaded from rows touch eight lines each.)
//  * Two barriers; no K split over CTAs, no counters, no slabs.
//
// Splitting K over the CTAs of a cluster (partial sums exchanged through distributed shared memory) and staging the whole
// input by bulk copies before the loop both measured slower than this at every size.
// It ends at 16 tokens (8 for large launches, see batch_max_tokens): 17 tokens took three column groups, eight Qwen3-8B layers 625 us, 473 through nq_wgemm.cu.
//
// What bounds it (counters of single launches at 16 tokens, cold): no throughput limit is near.  DRAM 3 to 6 % of its peak,
// L2 4 to 16, tensor pipe 12 to 19.  The two stages of a group with little work take 8.8 us together, two launches of a fixed
// chain (dependency, weights' arrival, a loop of a few steps, two barriers, output).  In first stages the 16 warps issue in
// 56 to 60 % of the active cycles: copies, shifts and LOP3 around the MMAs; down's reads 56 MB through L2, since every CTA
// stages the whole input.  Gate/up's second stage waits for the fragments of t (long scoreboard, 3.1 warps per issue, is its
// largest stall) with four warps per scheduler to hide that.
#include <cstddef>
#include <cstring>
#include <type_traits>

#include "nq_common.cuh"
#include "nq_plan.h"
#include "nq_stage.h"

namespace nq {

constexpr int kBatchThreads = 512;
constexpr int kBatchWarps = kBatchThreads / 32;
// 16-column blocks of the intermediate whose B fragments a warp loads together
constexpr int blocks_in_flight(int nt, int rows) { return nt == 1 || rows < 4 ? 8 : 4; }
constexpr int tokens_groups(int T) { return T <= 8 ? 1 : 2; }
constexpr int kMostRows = 4;             // row groups of a pass
constexpr int kPieces = 3;               // pieces of 64 columns a warp has in flight
constexpr int kPieceStride = 128 + 32;   // bytes of a staged row: 32 mod 128, so the eight tokens of a fragment fall on
                                         // different banks
constexpr int kBatchSlots = 8;           // weight blocks in flight
constexpr int kBatchMaxCtas = 256;
constexpr size_t kOffParams = 64, kFixedBytes = 1024;
constexpr unsigned kWeightWaitLimit = 1u << 20;   // attempts of up to ~2 us each

struct alignas(16) BatchJob {
    const uint4* tiles;
    const void* a;
    const void* pre;
    const void* post;
    void* out;
    const void* bias;
    const void* resid;
    const int* row_exp;
    long long lda, ld_out, ld_res;
    int rows, K, chunks;
    int cta0, g_q, g_r;      // first CTA of the range; row groups per CTA, one more for its first g_r CTAs
    int gb;                  // row groups per block
    uint16_t wk, wr;         // chunk slices x row slices of a CTA's work, one warp each
    int wk_magic, wr_magic;  // ceil(2^16 / .)
};
static_assert(sizeof(BatchJob) == 128, "128 bytes");
struct alignas(16) BatchParams {
    BatchJob job[kMaxGemmJobs];
    unsigned* status;
    int T, io_bf16, out_bf16, saturate, exp_sign;   // T: columns of partial sums (tokens, or 8 for a split input)
    int slots, slot_bytes, part_off;
    int stage_off, frag_out;      // activation staging buffers; output in fragment order
    uint8_t cta_job[kBatchMaxCtas];
};
constexpr int kBatchWords = (int)offsetof(BatchParams, cta_job) / 16;
static_assert(offsetof(BatchParams, cta_job) % 16 == 0 && kOffParams + kBatchWords * 16 <= kFixedBytes, "shared memory map");

template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (BF16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float float_of(uint16_t h, int bf16) {
    return bf16 ? __uint_as_float((uint32_t)h << 16) : __half2float(__ushort_as_half(h));
}
// {a.lo, b.lo} and {a.hi, b.hi} of four consecutive 16-bit values: columns {0, 2} and {1, 3}
__device__ __forceinline__ uint32_t even_columns(uint2 v) { return __byte_perm(v.x, v.y, 0x5410); }
__device__ __forceinline__ uint32_t odd_columns(uint2 v) { return __byte_perm(v.x, v.y, 0x7632); }

// Fragment order of an intermediate [T, K]: per chunk, 16-column block (32 j + 16 h) and group of eight tokens, the 8
// bytes {columns 4q, 4q+2, 4q+1, 4q+3} of lane 4g + q (token g of the group).  Element index; the layout has
// chunks * 16 * NT * 128 elements, those of columns and tokens that do not exist are never used.
template <int NT>
__device__ __forceinline__ long long fragment_index(int tok, int k) {
    const int b = k & 3;
    return (((long long)(k >> 4) * NT + (tok >> 3)) * 32 + 4 * (tok & 7) + ((k >> 2) & 3)) * 4 + ((b >> 1) | ((b & 1) << 1));
}
__device__ __forceinline__ void copy16_or_zero(uint32_t dst, const void* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// NT: column groups of eight tokens.  ROWS: row groups a warp takes in a pass.  FRAG: the input is in fragment order
// and has no scale (the second stage); otherwise it is [T, lda].  SPLIT: the intermediate is value and remainder (see
// kSplitTokens).
template <bool BF16, int NT, int ROWS, bool FRAG, bool SPLIT>
__global__ void __launch_bounds__(kBatchThreads, 1) batch_stage_kernel(const __grid_constant__ BatchParams Pc) {
    constexpr int kRows = ROWS, kB = blocks_in_flight(NT, ROWS);
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const uint32_t bars = smem_u32(smem);
    // the parameter bank is read here and nowhere else, in one round trip (see nq_gemv.cu)
    const unsigned my_job = Pc.cta_job[blockIdx.x];
    {
        constexpr int kRounds = (kBatchWords + kBatchWarps - 1) / kBatchWarps;
        uint4 w[kRounds];
#pragma unroll
        for (int i = 0; i < kRounds; ++i) w[i] = reinterpret_cast<const uint4*>(&Pc)[min(warp + i * kBatchWarps, kBatchWords - 1)];
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < kRounds; ++i)
                reinterpret_cast<uint4*>(smem + kOffParams)[min(warp + i * kBatchWarps, kBatchWords - 1)] = w[i];
        }
    }
    if (tid >= kBatchThreads - kBatchSlots) {
        mbar_init(bars + 8 * (tid - (kBatchThreads - kBatchSlots)), 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    const BatchParams& P = *reinterpret_cast<const BatchParams*>(smem + kOffParams);
    const BatchJob& jb = P.job[my_job];
    unsigned char* weights = smem + kFixedBytes;
    float* part = reinterpret_cast<float*>(smem + P.part_off);        // [chunk slice][token][row of the block]
    // (a constant where it is one: eight Qwen3-8B layers of four tokens 347.4 -> 338.9 us, two of 8192 columns 273 -> 267.5)
    const int T = SPLIT ? (FRAG ? 2 * kSplitTokens : kSplitTokens) : P.T, slots = P.slots, slot_bytes = P.slot_bytes, chunks = jb.chunks, gb = jb.gb, rows = jb.rows;
    int first, groups;
    {
        const int c = (int)blockIdx.x - jb.cta0;
        first = c * jb.g_q + min(c, jb.g_r);
        groups = jb.g_q + (c < jb.g_r ? 1 : 0);
    }
    int l_g = 0, l_slot = 0;
    auto load_block = [&]() {
        if (l_g >= groups) return;
        const int nb = min(gb, groups - l_g);
        const uint32_t bytes = (uint32_t)(nb * chunks) * 512u, bar = bars + 8 * l_slot;
        mbar_expect_tx(bar, bytes);
        bulk_load(smem_u32(weights) + (uint32_t)(l_slot * slot_bytes), jb.tiles + (size_t)(first + l_g) * chunks * 32, bytes, bar);
        l_g += nb;
        l_slot = l_slot + 1 == slots ? 0 : l_slot + 1;
    };
    const bool loader = tid == kBatchThreads - kBatchSlots;
    if (loader) {
#pragma unroll 1
        for (int s = 0; s < slots; ++s) load_block();
    }
    // this warp: chunks [c0, c1), row slice rw
    const int wk = jb.wk, wr = jb.wr;
    const int rw = (warp * jb.wk_magic) >> 16, kw = warp - rw * wk;
    const int c0 = (kw * chunks * jb.wk_magic) >> 16, c1 = ((kw + 1) * chunks * jb.wk_magic) >> 16;
    const int wr_magic = jb.wr_magic, K = jb.K, tok_stride = gb * 16 + 4;   // 4 mod 16: an accumulator's 32 stores fall on 32 banks
    const uint16_t* const pre = static_cast<const uint16_t*>(jb.pre);
    const uint16_t* const a_in = static_cast<const uint16_t*>(jb.a);
    const long long lda = jb.lda;
    // staging: buffers of T + 1 rows (the scales last) of 64 columns, one piece each
    const int piece_bytes = (T + 1) * kPieceStride;
    unsigned char* const stage = smem + P.stage_off + warp * kPieces * piece_bytes;
    int a_row[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) a_row[nt] = min(8 * nt + g, T - 1) * kPieceStride + 8 * q;   // tokens beyond T: not stored
    int s_in = 0, s_out = 0;             // next buffer to fill, to read
    // piece `pc` (columns 64 pc ..): eight lanes per row
    auto stage_piece = [&](int pc) {
        if (pc < 4 * c1) {
            const int col = pc * 64 + (lane & 7) * 8, t0 = lane >> 3;
            const bool there = col < K;          // K is a multiple of 8
            const uint32_t dst = smem_u32(stage + s_in * piece_bytes) + (uint32_t)(t0 * kPieceStride + (lane & 7) * 16);
            const uint16_t* src = a_in + (there ? col : 0);
#pragma unroll
            for (int t = 0; t < 8 * NT; t += 4)
                if (t + t0 < T) copy16_or_zero(dst + (uint32_t)(t * kPieceStride), src + (t + t0) * lda, there);
            if (pre && lane < 8) copy16_or_zero(dst + (uint32_t)(T * kPieceStride), pre + (there ? col : 0), there);
            s_in = s_in + 1 == kPieces ? 0 : s_in + 1;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    int slot = 0;
    uint32_t parity = 0;
#pragma unroll 1
    for (int blk = 0; blk < groups; blk += gb) {
        const int nb = min(gb, groups - blk);
        const int r0 = (rw * nb * wr_magic) >> 16, r1 = rw < wr ? ((rw + 1) * nb * wr_magic) >> 16 : r0;
        // quotient by the rows of a block: exact below 2^22 / rows, and there are at most 16 times as many outputs as rows, 512 of them
        const unsigned nb16_magic = ((1u << 22) + nb * 16 - 1) / (nb * 16);
        // output scale and bias of row `tid` of the block (asm: a plain 16-bit load is widened, that is waited for, at once)
        const int row0 = (first + blk) * 16;
        uint16_t post_raw = 0, bias_raw = 0;
        if (tid < nb * 16 && row0 + tid < rows) {
            if (jb.post) asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(post_raw) : "l"(static_cast<const uint16_t*>(jb.post) + row0 + tid));
            if (jb.bias) asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(bias_raw) : "l"(static_cast<const uint16_t*>(jb.bias) + row0 + tid));
        }
#pragma unroll 1
        for (int rb = r0; rb < r1; rb += kRows) {
            const int nr = min(kRows, r1 - rb);
            float acc[kRows][NT][4];
#pragma unroll
            for (int r = 0; r < kRows; ++r)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[r][nt][i] = 0.f;
            if (!FRAG && c0 < c1) {
#pragma unroll 1
                for (int i = 0; i < kPieces; ++i) stage_piece(4 * c0 + i);
            }
            if (rb == r0) {
#pragma unroll 1
                for (unsigned spins = 0; !mbar_try(bars + 8 * slot, parity); ++spins)
                    if (spins >= kWeightWaitLimit) { atomicExch(P.status, (unsigned)(-NQ_ERR_TIMEOUT)); break; }
            }
            const uint32_t one2 = BF16 ? 0x3F803F80u : 0x3C003C00u;
            // Shifts as products with powers of two the compiler cannot see: multiplications do not wait for the half-rate pipe of the LOP3s
            // (16 tokens, eight layers: Llama-3.2-1B 315 -> 293 us, Qwen3-8B 438 -> 432, two of 8192 columns 393 -> 399; four and eight: level).
            uint32_t pw[8], p256;
            asm volatile("mov.u32 %0, %1;" : "=r"(p256) : "r"(256u));
#pragma unroll
            for (int i = 0; i < 8; ++i) asm volatile("mov.u32 %0, %1;" : "=r"(pw[i]) : "r"(1u << i));
            // block b of a chunk (columns 32 j + 16 h + ..) against all row groups
            auto block = [&](const uint4 (&w)[kRows], int b, uint32_t se, uint32_t so, const uint32_t (&be)[NT], const uint32_t (&bo)[NT]) {
                const int j = b >> 1, h = b & 1;
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                    if (r < nr) {
                        const uint32_t w0 = h ? w[r].z : w[r].x, w1 = h ? w[r].w : w[r].y;   // rows g, g + 8
                        const uint32_t u0 = w0 * pw[7 - j], u1 = w1 * pw[7 - j];
                        const uint32_t a0 = and_xor(u0 * p256, 0x80008000u, se), a2 = and_xor(u0, 0x80008000u, so);
                        const uint32_t a1 = and_xor(u1 * p256, 0x80008000u, se), a3 = and_xor(u1, 0x80008000u, so);
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) mma_16816<BF16>(acc[r][nt], a0, a1, a2, a3, be[nt], bo[nt]);
                    }
            };
#pragma unroll 1
            for (int c = c0; c < c1; ++c) {
                uint4 w[kRows];
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                    w[r] = *reinterpret_cast<const uint4*>(weights + slot * slot_bytes + ((rb + min(r, nr - 1)) * chunks + c) * 512 + lane * 16);
                if (FRAG) {
                    const uint2* src = reinterpret_cast<const uint2*>(a_in) + (size_t)c * (16 * NT * 32) + lane;
#pragma unroll
                    for (int b0 = 0; b0 < 16; b0 += kB) {
                        uint2 x[kB][NT];
#pragma unroll
                        for (int b = 0; b < kB; ++b) {
                            const bool in = c * 256 + (b0 + b) * 16 + 4 * q < K;
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt) x[b][nt] = in ? src[((b0 + b) * NT + nt) * 32] : make_uint2(0u, 0u);
                        }
#pragma unroll
                        for (int b = 0; b < kB; ++b) {
                            uint32_t be[NT], bo[NT];
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt) { be[nt] = x[b][nt].x; bo[nt] = x[b][nt].y; }
                            block(w, b0 + b, one2, one2, be, bo);
                        }
                    }
                } else {
#pragma unroll
                    for (int pc = 0; pc < 4; ++pc) {
                        asm volatile("cp.async.wait_group %0;" ::"n"(kPieces - 1) : "memory");
                        __syncwarp();
                        const unsigned char* buf = stage + s_out * piece_bytes;
                        s_out = s_out + 1 == kPieces ? 0 : s_out + 1;
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            uint32_t se = one2, so = one2, be[NT], bo[NT];
                            if (pre) {
                                const uint2 sv = *reinterpret_cast<const uint2*>(buf + T * kPieceStride + 8 * q + b * 32);
                                se = even_columns(sv); so = odd_columns(sv);
                            }
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt) {
                                const uint2 xv = *reinterpret_cast<const uint2*>(buf + a_row[nt] + b * 32);
                                be[nt] = even_columns(xv); bo[nt] = odd_columns(xv);
                            }
                            block(w, 4 * pc + b, se, so, be, bo);
                        }
                        __syncwarp();            // the buffer has been read
                        stage_piece(4 * c + pc + kPieces);
                    }
                }
            }
            if (!FRAG) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncwarp();
            }
            // lane (g, q): rows g, g + 8 of each row group, tokens 8 nt + 2q, + 1
            float* dst = part + (size_t)kw * T * tok_stride + (2 * q) * tok_stride + rb * 16 + g;
#pragma unroll
            for (int r = 0; r < kRows; ++r)
                if (r < nr) {
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (8 * nt + 2 * q + (i & 1) < T) dst[(8 * nt + (i & 1)) * tok_stride + r * 16 + 8 * (i >> 1)] = acc[r][nt][i];
                }
        }
        const int io_bf16 = P.io_bf16, out_bf16 = P.out_bf16;
        float2* const scale = reinterpret_cast<float2*>(part + (size_t)wk * T * tok_stride);   // {output scale, bias} of a row
        if (tid < nb * 16) scale[tid] = make_float2(jb.post ? float_of(post_raw, io_bf16) : 1.f, jb.bias ? float_of(bias_raw, io_bf16) : 0.f);
        __syncthreads();   // partial sums complete, this block's weights have been read
        if (++slot == slots) { slot = 0; parity ^= 1u; }
        if (loader) load_block();
        // Outputs, [token][row of the block] dealt to all threads, three at a time where there are more: the sums over the chunk slices are
        // chains of shared-memory loads.  Of a split intermediate two neighbouring lanes sum value and remainder.  (A warp per token left
        // 12 of 16 warps idle at four tokens: eight Qwen3-8B layers 356 -> 346 us, Llama-3.2-1B 264 -> 244, two of 8192 columns 289 -> 269.)
        // An intermediate that is not a pair becomes infinite beyond its type's range, as in the GEMM; the value of a pair
        // stays finite, and it is the remainder that an infinity goes to.  NaN passes every clamp.
        constexpr bool kPair = SPLIT && FRAG;
        const float lim = P.saturate || (SPLIT && !FRAG) ? (out_bf16 ? 3.3895313892515355e+38f : 64504.0f) : 3.4e38f;
        const uint16_t* const resid = static_cast<const uint16_t*>(jb.resid);
        const int* const row_exp = jb.row_exp;
        const int kslice = T * tok_stride, frag_out = P.frag_out, nb16 = nb * 16;
        const int sums = (SPLIT ? kSplitTokens : T) * nb16 * (kPair ? 2 : 1);
        auto emit = [&](auto many, int e0) {
            constexpr int U = decltype(many)::value;
            float v[U];
            const float* src[U];
            int tok[U], idx[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = min(e0 + u * kBatchThreads, sums - 1), o = kPair ? e >> 1 : e;
                tok[u] = (int)((unsigned)o * nb16_magic >> 22);
                idx[u] = o - tok[u] * nb16;
                src[u] = part + (tok[u] + (kPair && (e & 1) ? kSplitTokens : 0)) * tok_stride + idx[u];
                v[u] = 0.f;
            }
#pragma unroll 4
            for (int k = 0; k < wk; ++k)
#pragma unroll
                for (int u = 0; u < U; ++u) { v[u] += *src[u]; src[u] += kslice; }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (kPair) v[u] += __shfl_xor_sync(0xffffffffu, v[u], 1);
                const float2 sc = scale[idx[u]];
                const int row = row0 + idx[u];
                if (e0 + u * kBatchThreads >= sums || row >= rows || (kPair && (lane & 1))) continue;
                const float rs = row_exp ? exp2f((float)(P.exp_sign * row_exp[tok[u]])) : 1.f;
                float extra = sc.y;
                if (resid) extra += float_of(resid[tok[u] * jb.ld_res + row], io_bf16);
                const float exact = v[u] * (sc.x * rs) + extra, w = clamp_or_nan(exact, lim);
                uint16_t* const out = static_cast<uint16_t*>(jb.out);
                if (SPLIT && !FRAG) {
                    const __nv_bfloat16 value = __float2bfloat16(w);
                    out[fragment_index<1>(tok[u], row)] = __bfloat16_as_ushort(value);
                    out[fragment_index<1>(kSplitTokens + tok[u], row)] = __bfloat16_as_ushort(__float2bfloat16(exact - __bfloat162float(value)));
                } else {
                    out[frag_out ? fragment_index<NT>(tok[u], row) : tok[u] * jb.ld_out + row] = out_bf16 ? __bfloat16_as_ushort(__float2bfloat16(w)) : __half_as_ushort(__float2half(w));
                }
            }
        };
        if (sums <= kBatchThreads) {
            if ((tid & ~31) < sums) emit(std::integral_constant<int, 1>{}, tid);
        } else {
#pragma unroll 1
            for (int e0 = tid; (e0 & ~31) < sums; e0 += 3 * kBatchThreads) emit(std::integral_constant<int, 3>{}, e0);
        }
        if (blk + gb < groups) __syncthreads();   // the partial sums have been read
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

template <bool BF16, int NT, bool FRAG>
static const void* batch_kernel_rows(int rows) {
    if (rows == 1) return (const void*)batch_stage_kernel<BF16, NT, 1, FRAG, false>;
    if (rows == 2) return (const void*)batch_stage_kernel<BF16, NT, 2, FRAG, false>;
    return (const void*)batch_stage_kernel<BF16, NT, kMostRows, FRAG, false>;
}
template <bool BF16, bool FRAG>
static const void* batch_kernel_tokens(int nt, int rows) {
    return nt == 1 ? batch_kernel_rows<BF16, 1, FRAG>(rows) : batch_kernel_rows<BF16, 2, FRAG>(rows);
}
template <bool BF16, bool FRAG>
static const void* split_kernel_rows(int rows) {
    return rows == 1 ? (const void*)batch_stage_kernel<BF16, 1, 1, FRAG, true>
           : rows == 2 ? (const void*)batch_stage_kernel<BF16, 1, 2, FRAG, true> : (const void*)batch_stage_kernel<BF16, 1, 4, FRAG, true>;
}
static const void* split_kernel(int bf16, int rows, bool frag) {     // (a split intermediate is bf16)
    return frag ? split_kernel_rows<true, true>(rows) : bf16 ? split_kernel_rows<true, false>(rows) : split_kernel_rows<false, false>(rows);
}
static const void* batch_kernel(int bf16, int nt, int rows, bool frag) {
    if (frag) return bf16 ? batch_kernel_tokens<true, true>(nt, rows) : batch_kernel_tokens<false, true>(nt, rows);
    return bf16 ? batch_kernel_tokens<true, false>(nt, rows) : batch_kernel_tokens<false, false>(nt, rows);
}
static int batch_smem_limit(int* out) {
    static int cached[64];
    int dev = 0;
    NQ_CUDA_TRY(cudaGetDevice(&dev));
    if (cached[dev & 63] == 0) {
        int optin = 0;
        NQ_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        for (int i = 0; i < 24; ++i)
            NQ_CUDA_TRY(cudaFuncSetAttribute(batch_kernel(i & 1, 1 + (i / 4) % 2, 1 << (i / 8), (i & 2) != 0), cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
        for (int i = 0; i < 12; ++i)
            NQ_CUDA_TRY(cudaFuncSetAttribute(split_kernel(i & 1, 1 << (i / 4), (i & 2) != 0), cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
        cached[dev & 63] = optin;
    }
    *out = cached[dev & 63];
    return NQ_OK;
}

// From nine tokens on the second column group doubles the matrix instructions, and every CTA stages the whole input of a first stage:
// launches with much of both are faster through nq_wgemm.cu and nq_pgemm.cu.  The rule looks at each stage's packed factors, and either stage
// decides for both.  Groups in a graph, bf16, 16 tokens: MB of the two stages, here / there in us; * marks what the rule sends there.
//               q/k/v                        o                          gate/up                       down
//   2048 cols   0.4 + 0.2   7.2 /  8.0      0.2 + 0.2   7.1 /  7.7      0.6 +  1.8   9.0 /  9.6       0.9 + 0.3   9.7 /  9.5
//   4096        1.4 + 1.0  10.0 / 10.6      0.8 + 0.8   8.4 /  9.7      2.5 +  7.5  19.2 / 17.6       3.7 + 1.2  16.2 / 16.0
//   5120        2.3 + 1.5  14.0 / 13.3      1.3 + 1.3  10.8 / 11.3      3.9 + 11.7  31.0 / 22.3 *     5.8 + 1.9  21.8 / 20.4 *
//   6144        3.3 + 2.2  17.0 / 15.0      1.9 + 1.9  14.8 / 12.6      5.6 + 16.8  37.7 / 27.2 *     8.4 + 2.8  34.3 / 21.9 *
//   8192        5.9 + 4.0  25.8 / 21.3 *    3.3 + 3.3  17.0 / 16.5     10.4 + 36.2  73.0 / 55.8 *    18.1 + 5.2  66.0 / 36.7 *
// (0.8 bits per weight, inner width 3 times the columns, 28672 at 8192.)  A layer of all four, us, all here / all there / by the rule:
//   9 tokens    2048  31.3 / 34.3 / 31.3    4096  51.5 / 52.9 / 51.5    5120  75.6 / 65.3 / 67.3    6144   90.4 / 75.4 / 79.8
//               8192 157.7 / 126.8 / 129.1  4096 at 1.5 bits  63.7 / 66.5 / 65.4    5120 at 1.2 bits  95.8 / 80.8 / 89.6
//   16 tokens   2048  31.9 / 34.4 / 31.9    4096  53.4 / 52.9 / 53.5    5120  76.3 / 65.4 / 67.4    6144  102.8 / 75.3 / 81.1
//               8192 180.3 / 126.8 / 129.6  4096 at 1.5 bits  70.4 / 66.5 / 67.3    5120 at 1.2 bits  96.6 / 80.9 / 89.2
// Changing kernels inside a layer costs what a group of 4096 columns gains, so the lines (8 MB; 4.5 MB with 8192 columns) leave such layers in
// one kernel: they are within 3 % of the better one.  From 5120 columns on they are on the safe side: all of a layer through the GEMMs would be
// 1 to 11 % faster still.  (A line at 4.5 MB for any K changes no layer from 5120 columns on, and loses 2 to 4 % at 4096.)
int batch_max_tokens(const StageJob* jobs, int n) {
    double bytes = 0;                       // of this stage
    int most_k = 0;
    for (int i = 0; i < n; ++i) {
        if (jobs[i].K > 32768) return 0;    // one row group's weights have to fit beside staging and partial sums
        bytes += (double)jobs[i].K * jobs[i].Nout / 8;
        most_k = jobs[i].K > most_k ? jobs[i].K : most_k;
    }
    if (bytes >= 8e6 || (bytes >= 4.5e6 && most_k >= 8192)) return 8;
    return kBatchMostTokens;
}

size_t batch_fragment_bytes(int T, int K) { return (size_t)((K + 255) / 256) * 16 * tokens_groups(T) * 256; }

// Chunk slices x row slices of the warps for a block of `gb` row groups: a step (a row group's chunk) against a chunk's B
// fragments, once per pass.
static void split_warps(int gb, int chunks, int nt, int& wk, int& wr) {
    int best = 1 << 30;
    for (int k = 1; k <= kBatchWarps && k <= chunks; ++k) {
        int r = kBatchWarps / k;
        if (r > gb) r = gb;
        const int per = (gb + r - 1) / r;
        const int cost = ((chunks + k - 1) / k) * (per * (8 + 2 * nt) + ((per + kMostRows - 1) / kMostRows) * (3 + 3 * nt));
        if (cost < best) { best = cost; wk = k; wr = r; }
    }
}

int launch_batch_stage(const StageJob* jobs, int n, int tokens, StageTypes ty, int saturate, bool frag_in, bool frag_out, bool split,
                       unsigned* status, cudaStream_t stream) {
    const int T = split && frag_in ? 2 * kSplitTokens : tokens;
    for (int i = 0; i < n; ++i) {      // 16-byte copies of rows and scales
        if (jobs[i].K % 8 != 0 || (!frag_in && (!aligned16(jobs[i].a) || jobs[i].lda % 8 != 0))) return NQ_ERR_ALIGN;
        if (jobs[i].pre && !aligned16(jobs[i].pre)) return NQ_ERR_ALIGN;
    }
    int limit = 0;
    { const int st = batch_smem_limit(&limit); if (st != NQ_OK) return st; }
    BatchParams P;
    memset(&P, 0, sizeof(P));
    P.status = status;
    P.T = T;
    P.io_bf16 = ty.io_bf16; P.out_bf16 = ty.out_bf16; P.saturate = saturate; P.exp_sign = ty.exp_sign;
    const int nt = tokens_groups(T);
    int groups[kMaxGemmJobs], chunks[kMaxGemmJobs], ncta[kMaxGemmJobs], total = 0;
    for (int i = 0; i < n; ++i) {
        groups[i] = (jobs[i].Nout + 15) / 16;
        chunks[i] = (jobs[i].K + 255) / 256;
        total += groups[i];
    }
    int grid = sm_count() < kBatchMaxCtas ? sm_count() : kBatchMaxCtas;
    if (grid > total) grid = total;
    if (grid < n) grid = n;
    deal_ctas(grid, n, groups, chunks, ncta);
    const size_t stage_bytes = frag_in ? 0 : (size_t)kBatchWarps * kPieces * (T + 1) * kPieceStride;
    const size_t room = limit - kFixedBytes - stage_bytes;      // weights and partial sums of a block
    size_t slot_used = 0, part_used = 0;
    int cta = 0, most_blocks = 1, most_rows = 1;
    for (int i = 0; i < n; ++i) {
        const StageJob& S = jobs[i];
        BatchJob& j = P.job[i];
        j.tiles = static_cast<const uint4*>(S.tiles);
        j.a = S.a; j.pre = S.pre; j.post = S.post; j.out = S.out; j.bias = S.bias; j.resid = S.resid;
        j.row_exp = ty.exp_sign ? S.row_exp : nullptr;
        j.lda = S.lda; j.ld_out = S.ld_out; j.ld_res = S.ld_res;
        j.rows = S.Nout; j.K = S.K; j.chunks = chunks[i];
        j.cta0 = cta;
        j.g_q = groups[i] / ncta[i];
        j.g_r = groups[i] % ncta[i];
        memset(P.cta_job + cta, i, (size_t)ncta[i]);
        cta += ncta[i];
    }
    // Row blocks, as equal as possible: each job's weights and partial sums fit the room together; where the largest of
    // both over the jobs do not, each of them gets half; and where one row group does not fit half, one row group per
    // block (64 KB of weights at the largest K, 21 KB of partial sums).
    for (int attempt = 0; attempt < 3; ++attempt) {
        slot_used = part_used = 0;
        most_blocks = most_rows = 1;
        for (int i = 0; i < n; ++i) {
            BatchJob& j = P.job[i];
            const int most = j.g_q + (j.g_r ? 1 : 0);
            size_t part = 0, slot = 0;
            for (int blocks = 1;; ++blocks) {
                j.gb = attempt == 2 ? 1 : (most + blocks - 1) / blocks;
                int wk = 1, wr = 1;
                // the sums of a split linear have to be the same alone and in a group: slices as for the linear alone
                split_warps(split ? (groups[i] + sm_count() - 1) / sm_count() : j.gb, chunks[i], nt, wk, wr);
                if (split) wr = kBatchWarps / wk < j.gb ? kBatchWarps / wk : j.gb;
                j.wk = (uint16_t)wk; j.wr = (uint16_t)wr;
                part = (size_t)j.wk * T * (j.gb * 16 + 4) * 4 + (size_t)j.gb * 16 * 8;
                slot = (size_t)j.gb * chunks[i] * 512;
                const bool fits = attempt == 0 ? part + slot <= room : part <= room / 2 && slot <= room / 2;
                if (j.gb == 1 || (fits && j.gb <= kBatchThreads / 16)) break;
            }
            part_used = part > part_used ? part : part_used;
            slot_used = slot > slot_used ? slot : slot_used;
            j.wk_magic = (65536 + j.wk - 1) / j.wk;
            j.wr_magic = (65536 + j.wr - 1) / j.wr;
            const int blocks = (most + j.gb - 1) / j.gb, per_warp = (j.gb + j.wr - 1) / j.wr;
            most_blocks = blocks > most_blocks ? blocks : most_blocks;
            most_rows = per_warp > most_rows ? per_warp : most_rows;
        }
        if (part_used + slot_used <= room) break;
    }
    int slots = most_blocks < kBatchSlots ? most_blocks : kBatchSlots;
    while (slots > 1 && part_used + slots * slot_used > room) --slots;
    P.slots = slots;
    P.slot_bytes = (int)slot_used;
    P.frag_out = frag_out;
    P.part_off = (int)(kFixedBytes + slots * slot_used);
    P.stage_off = (P.part_off + (int)part_used + 15) / 16 * 16;
    const size_t smem = P.stage_off + stage_bytes;
    if (smem > (size_t)limit) return NQ_ERR_UNSUPPORTED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cta);
    cfg.blockDim = dim3(kBatchThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    void* args[] = {&P};
    const int rows = most_rows == 1 ? 1 : most_rows == 2 ? 2 : 4;
    const void* fn = split ? split_kernel(ty.a_bf16, rows, frag_in) : batch_kernel(ty.a_bf16, nt, rows, frag_in);
    return launch_dependent(cfg, attr, 0, fn, args);
}

}  // namespace nq
