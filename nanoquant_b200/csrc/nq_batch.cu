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
//  * mma.sync m16n8k16 (16 rows x 8 tokens).  A shift and ONE LOP3 ((word & 0x80008000) ^ {s, s'}) make an A register +-s: the
//    product x * (+-s_in) is exact.  The columns of a block may be permuted as long as A and B agree, so the B fragment
//    of a token is its four consecutive columns 4q..4q+3, as they lie in memory: a PRMT per word and chunk brings the bits of neighbouring
//    columns, 8 apart in the tile layout, to 16 apart (two PRMTs per fragment of activations and of scales did before).
//  * B fragments.  The intermediate is stored in fragment order (see fragment_index): a warp's load of one is 256
//    contiguous bytes, and what a warp needs of a chunk is loaded at once.  Activations come in rows: every warp stages its own columns through
//    shared memory with 16-byte copies, a chunk (half of one for two column groups) at a time: the 16 blocks of it are then ONE
//    piece of code without a wait in between.  (Fragments loaded from rows touch eight lines each.)
//  * A launch is a chain, and the warps of an SM are few: what counts is the length of a warp's path.  Pieces of 64 columns with a wait,
//    a copy and 4 dependent MMAs each took 300 ns, whatever was in flight; a chunk with two accumulators in turn 700 to 900 ns for its 16 blocks.
//    A second stage's output scales and bias come by bulk copy beside the weights, the input scales are prefetched to L2.  Eight Qwen3-8B layers in
//    a graph, 4 / 8 / 12 / 16 tokens: 326 / 336 / 423 / 430 us -> 305 / 311 / 390 / 400; Llama-3.2-1B 238 / 233 / 279 / 289 -> 226 / 207 / 249 / 258.
//    With the steps beside the code below: 264 / 273 / 362 / 369; Llama-3.2-1B 222 / 191 / 239 / 242.
//  * Two barriers; no K split over CTAs, no counters, no slabs.
//
// Splitting K over the CTAs of a cluster (partial sums exchanged through distributed shared memory) and staging the whole
// input by bulk copies before the loop both measured slower than this at every size.
// It ends at 16 tokens (8 for large launches, see batch_max_tokens): 17 tokens took three column groups, eight Qwen3-8B layers 625 us, 473 through nq_wgemm.cu.
//
// What bounds it: the two stages of a group with little work are two launches of a fixed chain.  Stamps of o (4096 columns, 4 tokens; us after the last CTA
// of the launch before): dependency 0.7, activations on their way 1.2, weights there 1.3, activations 1.55, products 2.4, outputs 3.0.  In launches
// with much work the half-rate ALU pipe (a shift and a LOP3 per two weights, 16 clk of a scheduler per 16 x 16 weights, 12 with no shift)
// beside 9 clk per MMA; gate/up's second stage 4.1 us of 7.4.  Two CTAs per SM (64 registers, or 256 threads), so that the next launch has its
// weights before this one ends, lost 10 to 50 %: every phase is then longer.  The next stage's weights brought to L2 by this one: 1 to 4 % slower.
#include <cstddef>
#include <cstring>
#include <type_traits>

#include "nq_common.cuh"
#include "nq_plan.h"
#include "nq_stage.h"

namespace nq {

constexpr int kBatchThreads = 512;
constexpr int kBatchWarps = kBatchThreads / 32;
constexpr int tokens_groups(int T) { return T <= 8 ? 1 : 2; }
constexpr int kMostRows = 4;             // row groups of a pass
// 16-column blocks that a warp stages together, and fragments of the intermediate it loads together
constexpr int step_blocks(int nt) { return nt == 1 ? 16 : 8; }
constexpr int blocks_in_flight(int nt, int rows) { return nt == 1 && rows < 4 ? 16 : nt == 1 || rows < 4 ? 8 : 4; }
// staged fragments a warp holds for its row groups in turn
constexpr int fragments_held(int nt, int rows) { return nt * rows >= 8 ? 2 : 4; }
constexpr int kMostSteps = 2;            // steps in flight
constexpr int kBatchSlots = 8;           // weight blocks in flight
constexpr int kBatchMaxCtas = 256;
constexpr size_t kOffParams = 128, kFixedBytes = 1024;
constexpr int kMostBlock = 32;           // row groups of a block
constexpr size_t kMostRowBytes = 8192;   // output scales of a CTA in shared memory
constexpr unsigned kWeightWaitLimit = 1u << 20;   // attempts of some 4 us each

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
    uint8_t wk, wr;          // chunk slices x row slices of a CTA's work, one warp each
    uint8_t bulk, whole;     // output scales and bias come by bulk copy beside the weights (second stages); two neighbouring outputs are one 4-byte store
    int wk_magic, wr_magic;  // ceil(2^16 / .)
};
static_assert(sizeof(BatchJob) == 128, "128 bytes");
struct alignas(16) BatchParams {
    BatchJob job[kMaxGemmJobs];
    unsigned* status;
    int T, io_bf16, out_bf16, saturate, exp_sign;   // T: columns of partial sums (tokens, or 8 for a split input)
    int slots, slot_bytes, part_off;
    int stage_off, steps, frag_out;      // activation staging buffers, their number per warp; output in fragment order
    int post_off, bias_off;       // output scales and bias of the CTA's rows
    int t_magic;                  // ceil(2^16 / tokens of the output)
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
__device__ __forceinline__ uint2 lds8(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}

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
    constexpr int kRows = ROWS, kB = blocks_in_flight(NT, ROWS), kStep = step_blocks(NT), kStepRow = kStep * 32, kQ = fragments_held(NT, ROWS);
    constexpr uint32_t one2 = BF16 ? 0x3F803F80u : 0x3C003C00u;
    // Accumulators of a fragment's blocks in turn: MMAs on one of them wait for each other.  (Of a split intermediate it must not depend on
    // ROWS, which may differ between a linear alone and in a group.)
    constexpr int kChains = SPLIT || NT * ROWS < 4 ? 2 : 1;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const uint32_t bars = smem_u32(smem);       // weight slots, then the constants
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
    constexpr int kLoader = kBatchThreads - 32;
    if (tid >= kLoader && tid <= kLoader + kBatchSlots) {
        mbar_init(bars + 8 * (tid - kLoader), 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    const BatchParams& P = *reinterpret_cast<const BatchParams*>(smem + kOffParams);
    const BatchJob& jb = P.job[my_job];
    unsigned char* weights = smem + kFixedBytes;
    // (a constant where it is one: eight Qwen3-8B layers of four tokens 347.4 -> 338.9 us, two of 8192 columns 273 -> 267.5)
    const int T = SPLIT ? (FRAG ? 2 * kSplitTokens : kSplitTokens) : P.T, slots = P.slots, slot_bytes = P.slot_bytes, chunks = jb.chunks, gb = jb.gb, rows = jb.rows, K = jb.K;
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
    const bool loader = tid == kLoader;
    const uint32_t const_bar = bars + 8 * kBatchSlots;
    const bool bulk = FRAG && jb.bulk;
    if (loader) {
#pragma unroll 1
        for (int s = 0; s < slots; ++s) load_block();
        if (!FRAG && jb.pre) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(jb.pre), "r"(2 * K) : "memory");
        if (bulk) {
            const uint32_t row_bytes = 2u * min(groups * 16, rows - first * 16);
            mbar_expect_tx(const_bar, row_bytes * ((jb.post ? 1u : 0u) + (jb.bias ? 1u : 0u)));
            if (jb.post) bulk_load(smem_u32(smem + P.post_off), static_cast<const uint16_t*>(jb.post) + first * 16, row_bytes, const_bar);
            if (jb.bias) bulk_load(smem_u32(smem + P.bias_off), static_cast<const uint16_t*>(jb.bias) + first * 16, row_bytes, const_bar);
        }
    }
    // this warp: chunks [c0, c1), row slice rw
    const int wk = jb.wk, wr = jb.wr;
    const int rw = (warp * jb.wk_magic) >> 16, kw = warp - rw * wk;
    const int c0 = (kw * chunks * jb.wk_magic) >> 16, c1 = ((kw + 1) * chunks * jb.wk_magic) >> 16;
    const int wr_magic = jb.wr_magic, tok_stride = gb * 16 + 4;   // 4 mod 16: an accumulator's 32 stores fall on 32 banks
    float* part = reinterpret_cast<float*>(smem + P.part_off);        // [chunk slice][token][row of the block]
    // Staging: steps of kStep * 16 columns, T rows and the input scales.  The 32-byte blocks of four are swapped by the token (t & 3), so
    // that the tokens of a fragment fall on different banks.  A lane copies column 8 (lane % kLanes) of the rows lane / kLanes + i * kPer.
    constexpr int kLanes = kStep * 2, kPer = 32 / kLanes;      // lanes of a row, rows of a copy
    const int step_bytes = (T + 1) * kStepRow, n_steps = P.steps;
    const uint32_t stage = smem_u32(smem) + P.stage_off + warp * n_steps * step_bytes;
    const int x_lane = (lane % kLanes) * 8;
    const uint16_t* const x_src = static_cast<const uint16_t*>(jb.a) + x_lane;
    const uint16_t* const pre_src = static_cast<const uint16_t*>(jb.pre) + x_lane;
    const long long lda = jb.lda;
    const bool scaled = !FRAG && jb.pre;
    int s_in = 0, s_out = 0;             // next buffer to fill, to read (bytes)
    // the step from column `col` on
    auto stage_step = [&](int col) {
        if (col < c1 * 256) {
            const bool there = col + x_lane < K;          // K is a multiple of 8
            const int off = there ? col : -x_lane;
            const uint32_t row0 = stage + s_in + (lane / kLanes) * kStepRow;
            const uint16_t* src = x_src + off + (lane / kLanes) * lda;
#pragma unroll
            for (int t = 0; t < (SPLIT ? kSplitTokens : 8 * NT); t += kPer) {
                const int tok = t + lane / kLanes;
                if (SPLIT || tok < T) copy16_or_zero(row0 + t * kStepRow + ((x_lane * 2) ^ ((tok & 3) * 32)), src, there);
                src += kPer * lda;
            }
            if (scaled && lane < kLanes) copy16_or_zero(stage + s_in + T * kStepRow + x_lane * 2, pre_src + off, there);
            s_in = s_in + step_bytes == n_steps * step_bytes ? 0 : s_in + step_bytes;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // of a fragment: token g (+ 8), columns 4 q.. ; tokens beyond T: not stored
    const uint32_t t_row[2] = {(uint32_t)(min(g, T - 1) * kStepRow + 8 * q), (uint32_t)((NT == 2 ? min(8 + g, T - 1) : 0) * kStepRow + 8 * q)};
    const uint32_t t_swap[2] = {(uint32_t)(min(g, T - 1) & 3) * 32, (uint32_t)(NT == 2 ? min(8 + g, T - 1) & 3 : 0) * 32};
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    int slot = 0;
    uint32_t parity = 0;
#pragma unroll 1
    for (int blk = 0; blk < groups; blk += gb) {
        const int nb = min(gb, groups - blk);
        const int r0 = (rw * nb * wr_magic) >> 16, r1 = rw < wr ? ((rw + 1) * nb * wr_magic) >> 16 : r0;
        const int row0 = (first + blk) * 16;
        // Output scale and bias of row `tid` of the block, where they do not come by bulk copy: into registers before the main loop (asm: a plain
        // 16-bit load is widened, that is waited for, at once).  Those of a first stage are not copied ahead of the dependency wait: a kernel
        // before it may have let it in early and still be writing them.  (The predecessor of a second stage is the first stage of the same call, which lets it
        // in behind its own wait.)  Two stages in a graph, 8 copies of 4096 -> 1024 -> 4096, 5 / 16 tokens: 5.30 / 6.95 us with that copy, 5.16 / 6.94 so; with
        // 4099 outputs and a bias 5.55 / 7.26 when a second stage read them behind its last barrier, 5.25 / 6.95 so; 700000 outputs, 8 tokens, 39.1 -> 36.0.
        uint16_t post_raw = 0, bias_raw = 0;
        if (!bulk && tid < nb * 16 && row0 + tid < rows) {
            if (jb.post) asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(post_raw) : "l"(static_cast<const uint16_t*>(jb.post) + row0 + tid));
            if (jb.bias) asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(bias_raw) : "l"(static_cast<const uint16_t*>(jb.bias) + row0 + tid));
        }
#pragma unroll 1
        for (int rb = r0; rb < r1; rb += kRows) {
            const int nr = min(kRows, r1 - rb);
            float acc[kChains][kRows][NT][4];
#pragma unroll
            for (int k = 0; k < kChains; ++k)
#pragma unroll
                for (int r = 0; r < kRows; ++r)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[k][r][nt][i] = 0.f;
            if (!FRAG) {
#pragma unroll 1
                for (int i = 0; i < n_steps; ++i) stage_step(c0 * 256 + i * (kStep * 16));
            }
            auto wait_weights = [&]() {
#pragma unroll 1
                for (unsigned spins = 0; !(mbar_try(bars + 8 * slot, parity) && (!bulk || mbar_try(const_bar, 0))); ++spins)
                    if (spins >= kWeightWaitLimit) { atomicExch(P.status, (unsigned)(-NQ_ERR_TIMEOUT)); break; }
            };
            if (!FRAG && rb == r0) wait_weights();
            const unsigned char* wp = weights + slot * slot_bytes + (rb * chunks + c0) * 512 + lane * 16;
            const int w_row = chunks * 512;
#pragma unroll 1
            for (int c = c0; c < c1; ++c, wp += 512) {
                if (FRAG) {
                    // neighbouring columns of a fragment are {0, 2} and {1, 3}: a word's bits are 16 apart as they are
                    const uint2* src = static_cast<const uint2*>(jb.a) + (size_t)c * (16 * NT * 32) + lane;
                    const bool full = c * 256 + 256 <= K;
                    // (Several fragments per row group in both kinds of stages: with the row groups inside, whether one exists was a branch around
                    // every MMA.  Eight Qwen3-8B layers, 4 / 8 / 12 / 16 tokens: 296 / 306 / 376 / 387 -> 267 / 278 / 364 / 373 us; two of 8192
                    // columns, 4 and 8 tokens, 189 / 209 -> 162 / 179.)
                    uint4 w[kRows];
#pragma unroll
                    for (int b0 = 0; b0 < 16; b0 += kB) {
                        uint2 x[kB][NT];
                        if (full) {
#pragma unroll
                            for (int b = 0; b < kB; ++b)
#pragma unroll
                                for (int nt = 0; nt < NT; ++nt) x[b][nt] = src[((b0 + b) * NT + nt) * 32];
                        } else {
#pragma unroll
                            for (int b = 0; b < kB; ++b) {
                                const bool in = c * 256 + (b0 + b) * 16 + 4 * q < K;
#pragma unroll
                                for (int nt = 0; nt < NT; ++nt) x[b][nt] = in ? src[((b0 + b) * NT + nt) * 32] : make_uint2(0u, 0u);
                            }
                        }
                        if (b0 == 0) {
                            if (c == c0 && rb == r0) wait_weights();
#pragma unroll
                            for (int r = 0; r < kRows; ++r) w[r] = *reinterpret_cast<const uint4*>(wp + min(r, nr - 1) * w_row);
                        }
#pragma unroll
                        for (int r = 0; r < kRows; ++r)
                            if (r < nr)
#pragma unroll
                                for (int b = 0; b < kB; ++b) {
                                    const int j = (b0 + b) >> 1;
                                    const uint32_t u0 = ((b & 1) ? w[r].z : w[r].x) << (7 - j), u1 = ((b & 1) ? w[r].w : w[r].y) << (7 - j);
                                    const uint32_t a0 = and_xor(u0 << 8, 0x80008000u, one2), a2 = and_xor(u0, 0x80008000u, one2);
                                    const uint32_t a1 = and_xor(u1 << 8, 0x80008000u, one2), a3 = and_xor(u1, 0x80008000u, one2);
#pragma unroll
                                    for (int nt = 0; nt < NT; ++nt) mma_16816<BF16>(acc[b % kChains][r][nt], a0, a1, a2, a3, x[b][nt].x, x[b][nt].y);
                                }
                    }
                } else {
                    // words with the bits of neighbouring columns 16 apart, rows g and g + 8, halves of 16 columns
                    uint32_t p[kRows][8];
#pragma unroll
                    for (int r = 0; r < kRows; ++r) {
                        const uint4 w = *reinterpret_cast<const uint4*>(wp + min(r, nr - 1) * w_row);
                        p[r][0] = spread_bytes(w.x, 0); p[r][1] = spread_bytes(w.x, 1); p[r][2] = spread_bytes(w.y, 0); p[r][3] = spread_bytes(w.y, 1);
                        p[r][4] = spread_bytes(w.z, 0); p[r][5] = spread_bytes(w.z, 1); p[r][6] = spread_bytes(w.w, 0); p[r][7] = spread_bytes(w.w, 1);
                    }
#pragma unroll
                    for (int s0 = 0; s0 < 16; s0 += kStep) {
                        if (n_steps > 1) asm volatile("cp.async.wait_group %0;" ::"n"(kMostSteps - 1) : "memory");
                        else asm volatile("cp.async.wait_group 0;" ::: "memory");
                        __syncwarp();
                        const uint32_t buf = stage + s_out, s_addr = buf + T * kStepRow + 8 * q;
                        uint32_t x_addr[NT][4];
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                            for (int k = 0; k < 4; ++k) x_addr[nt][k] = buf + t_row[nt] + ((32 * k) ^ t_swap[nt]);
                        s_out = s_out + step_bytes == n_steps * step_bytes ? 0 : s_out + step_bytes;
#pragma unroll
                        for (int q0 = 0; q0 < kStep; q0 += kQ) {
                            uint2 sv[kQ], xv[kQ][NT];
#pragma unroll
                            for (int b = 0; b < kQ; ++b) {
                                sv[b] = scaled ? lds8(s_addr + (q0 + b) * 32) : make_uint2(one2, one2);
#pragma unroll
                                for (int nt = 0; nt < NT; ++nt) xv[b][nt] = lds8(x_addr[nt][(q0 + b) & 3] + ((q0 + b) >> 2) * 128);
                            }
#pragma unroll
                            for (int r = 0; r < kRows; ++r)
                                if (r < nr)
#pragma unroll
                                    for (int b = 0; b < kQ; ++b) {
                                        const int j = (s0 + q0 + b) >> 1;
                                        const uint32_t* v = p[r] + 4 * ((q0 + b) & 1);
                                        const uint32_t a0 = and_xor(v[0] << (7 - j), 0x80008000u, sv[b].x), a2 = and_xor(v[1] << (7 - j), 0x80008000u, sv[b].y);
                                        const uint32_t a1 = and_xor(v[2] << (7 - j), 0x80008000u, sv[b].x), a3 = and_xor(v[3] << (7 - j), 0x80008000u, sv[b].y);
#pragma unroll
                                        for (int nt = 0; nt < NT; ++nt) mma_16816<BF16>(acc[(q0 + b) % kChains][r][nt], a0, a1, a2, a3, xv[b][nt].x, xv[b][nt].y);
                                    }
                        }
                        __syncwarp();            // the buffer has been read
                        stage_step(c * 256 + s0 * 16 + n_steps * (kStep * 16));
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
                            if (8 * nt + 2 * q + (i & 1) < T) dst[(8 * nt + (i & 1)) * tok_stride + r * 16 + 8 * (i >> 1)] = kChains == 2 ? acc[0][r][nt][i] + acc[kChains - 1][r][nt][i] : acc[0][r][nt][i];
                }
        }
        const int io_bf16 = P.io_bf16, out_bf16 = P.out_bf16;
        if (!bulk && tid < nb * 16) {
            reinterpret_cast<uint16_t*>(smem + P.post_off)[tid] = post_raw;
            reinterpret_cast<uint16_t*>(smem + P.bias_off)[tid] = bias_raw;
        }
        __syncthreads();   // partial sums complete, this block's weights have been read
        if (++slot == slots) { slot = 0; parity ^= 1u; }
        if (loader) load_block();
        // Outputs.  Up to 512 of them are dealt to the threads one by one; of a split intermediate two neighbouring lanes sum value and
        // remainder.  Larger blocks by two rows (two apart where they are neighbours in the next stage's fragments) of every tok_step-th
        // token, with their scales converted once: the outputs of gate/up's second stage took 1.8 us of 9, now 1.1.  Eight Qwen3-8B layers, 4 / 8 / 12 /
        // 16 tokens: 305 / 311 / 390 / 400 us -> 296 / 307 / 377 / 388; two of 8192 columns, 4 tokens, 192.8 -> 188.8.  (All blocks that way: one more
        // dependent step where there are few outputs, Llama-3.2-1B 226 -> 229 and, eight tokens, 207 -> 213.)
        // An intermediate that is not a pair becomes infinite beyond its type's range, as in the GEMM; the value of a pair
        // stays finite, and it is the remainder that an infinity goes to.  NaN passes every clamp.
        constexpr bool kPair = SPLIT && FRAG;
        const float lim = P.saturate || (SPLIT && !FRAG) ? (out_bf16 ? 3.3895313892515355e+38f : 64504.0f) : 3.4e38f;
        const uint16_t* const resid = static_cast<const uint16_t*>(jb.resid);
        const int* const row_exp = jb.row_exp;
        // output scale and bias of a row of the block
        auto row_value = [&](int copy, int idx) { return float_of(reinterpret_cast<const uint16_t*>(smem + copy)[(bulk ? blk * 16 : 0) + idx], io_bf16); };
        const int kslice = T * tok_stride, frag_out = P.frag_out, t_magic = P.t_magic, tokens = SPLIT ? kSplitTokens : T;
        const int sums = tokens * nb * 16 * (kPair ? 2 : 1);
        if (sums <= kBatchThreads) {
            if ((tid & ~31) < sums) {
                const int e = min(tid, sums - 1), o = kPair ? e >> 1 : e;
                const int gt = o >> 4, gi = SPLIT ? gt / kSplitTokens : (gt * t_magic) >> 16;      // [row group][token][row]
                const int tok = gt - gi * tokens, idx = gi * 16 + (o & 15), row = row0 + idx;
                const float* src = part + (tok + (kPair && (e & 1) ? kSplitTokens : 0)) * tok_stride + idx;
                float v = 0.f;
#pragma unroll 4
                for (int k = 0; k < wk; ++k, src += kslice) v += *src;
                if (kPair) v += __shfl_xor_sync(0xffffffffu, v, 1);
                if (tid < sums && row < rows && !(kPair && (lane & 1))) {
                    const float rs = row_exp ? exp2f((float)(P.exp_sign * row_exp[tok])) : 1.f;
                    const float sc = jb.post ? row_value(P.post_off, idx) : 1.f;
                    float extra = jb.bias ? row_value(P.bias_off, idx) : 0.f;
                    if (resid) extra += float_of(resid[tok * jb.ld_res + row], io_bf16);
                    const float exact = v * (sc * rs) + extra, w = clamp_or_nan(exact, lim);
                    uint16_t* const out = static_cast<uint16_t*>(jb.out);
                    if (SPLIT && !FRAG) {
                        const __nv_bfloat16 value = __float2bfloat16(w);
                        out[fragment_index<1>(tok, row)] = __bfloat16_as_ushort(value);
                        out[fragment_index<1>(kSplitTokens + tok, row)] = __bfloat16_as_ushort(__float2bfloat16(exact - __bfloat162float(value)));
                    } else {
                        out[frag_out ? fragment_index<NT>(tok, row) : tok * jb.ld_out + row] = out_bf16 ? __bfloat16_as_ushort(__float2bfloat16(w)) : __half_as_ushort(__float2half(w));
                    }
                }
            }
        } else {
            const int pair_bits = 3 + (nb > 1) + (nb > 2) + (nb > 4) + (nb > 8) + (nb > 16);
            const int pair = tid & ((1 << pair_bits) - 1), tok_step = kBatchThreads >> pair_bits;
            const bool frag = !FRAG && frag_out;
            const int apart = frag ? 2 : 1, idx = frag ? 4 * (pair >> 1) + (pair & 1) : 2 * pair, row = row0 + idx;
            if (idx < nb * 16 && row < rows) {
                const bool both = row + apart < rows;
                float sc0 = 1.f, sc1 = 1.f, bi0 = 0.f, bi1 = 0.f;
                if (jb.post) { sc0 = row_value(P.post_off, idx); if (both) sc1 = row_value(P.post_off, idx + apart); }
                if (jb.bias) { bi0 = row_value(P.bias_off, idx); if (both) bi1 = row_value(P.bias_off, idx + apart); }
                uint16_t* const out = static_cast<uint16_t*>(jb.out) + (frag ? 0 : row);
                const long long ld_out = jb.ld_out, ld_res = jb.ld_res;
                const bool pairs = both && jb.whole;
                const int exp_sign = P.exp_sign;
                // Two tokens at a time where a thread has more than one: the sums are chains of shared-memory loads (sixteen tokens 373 -> 368 us, six
                // layers of 3072 columns 258 -> 253).
                auto take = [&](auto many, int tok0) {
                    constexpr int U = decltype(many)::value;
                    float v0[U], v1[U], r0[U], r1[U];
                    const float* from = part + tok0 * tok_stride + idx;
                    const int next = tok0 + tok_step < tokens ? tok_step * tok_stride : 0;      // (a second token that does not exist: the first again)
#pragma unroll
                    for (int u = 0; u < U; ++u) v0[u] = v1[u] = r0[u] = r1[u] = 0.f;
#pragma unroll 4
                    for (int k = 0; k < wk; ++k, from += kslice) {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const float* f = from + (u ? next : 0);
                            if (FRAG) {       // (neighbouring rows)
                                const float2 a = *reinterpret_cast<const float2*>(f);
                                v0[u] += a.x; v1[u] += a.y;
                                if (kPair) {
                                    const float2 r = *reinterpret_cast<const float2*>(f + kSplitTokens * tok_stride);
                                    r0[u] += r.x; r1[u] += r.y;
                                }
                            } else {
                                v0[u] += f[0]; v1[u] += f[apart];
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int tok = tok0 + u * tok_step;
                        if (u && next == 0) break;
                        if (kPair) { v0[u] += r0[u]; v1[u] += r1[u]; }      // (the same order of sums as above: a linear's bits do not depend on the block)
                        float x0 = bi0, x1 = bi1, s0 = sc0, s1 = sc1;
                        if (resid) {
                            const uint16_t* const r = resid + tok * ld_res + row;
                            x0 += float_of(r[0], io_bf16);
                            if (both) x1 += float_of(r[1], io_bf16);
                        }
                        if (row_exp) { const float rs = exp2f((float)(exp_sign * row_exp[tok])); s0 *= rs; s1 *= rs; }
                        const float e0 = v0[u] * s0 + x0, e1 = v1[u] * s1 + x1, w0 = clamp_or_nan(e0, lim), w1 = clamp_or_nan(e1, lim);
                        if (SPLIT && !FRAG) {
                            const __nv_bfloat162 value = __floats2bfloat162_rn(w0, w1);
                            *reinterpret_cast<__nv_bfloat162*>(out + fragment_index<1>(tok, row)) = value;
                            *reinterpret_cast<__nv_bfloat162*>(out + fragment_index<1>(kSplitTokens + tok, row)) = __floats2bfloat162_rn(e0 - __low2float(value), e1 - __high2float(value));
                            continue;
                        }
                        uint32_t o;
                        if (out_bf16) { const __nv_bfloat162 h = __floats2bfloat162_rn(w0, w1); o = *reinterpret_cast<const uint32_t*>(&h); }
                        else { const __half2 h = __floats2half2_rn(w0, w1); o = *reinterpret_cast<const uint32_t*>(&h); }
                        uint16_t* const dst = out + (frag ? fragment_index<NT>(tok, row) : tok * ld_out);
                        if (pairs) *reinterpret_cast<uint32_t*>(dst) = o;
                        else {
                            dst[0] = (uint16_t)o;
                            if (both) dst[1] = (uint16_t)(o >> 16);
                        }
                    }
                };
                if (tokens <= tok_step) {
                    if ((tid >> pair_bits) < tokens) take(std::integral_constant<int, 1>{}, tid >> pair_bits);
                } else {
#pragma unroll 1
                    for (int tok = tid >> pair_bits; tok < tokens; tok += 2 * tok_step) take(std::integral_constant<int, 2>{}, tok);
                }
            }
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
//   2048 cols   0.4 + 0.2   6.2 /  8.0      0.2 + 0.2   6.0 /  7.9      0.6 +  1.8   7.7 /  9.4       0.9 + 0.3   7.8 /  9.4
//   4096        1.4 + 1.0   8.8 / 10.3      0.8 + 0.8   7.3 /  9.6      2.5 +  7.5  16.4 / 16.9       3.7 + 1.2  14.4 / 15.1
//   5120        2.3 + 1.5  11.5 / 12.2      1.3 + 1.3   8.8 / 10.9      3.9 + 11.7  22.8 / 21.5 *     5.8 + 1.9  18.0 / 19.1 *
//   6144        3.3 + 2.2  12.4 / 13.3      1.9 + 1.9  11.9 / 12.2      5.6 + 16.8  28.5 / 26.1 *     8.4 + 2.8  21.0 / 20.6 *
//   8192        5.9 + 4.0  14.2 / 17.7 *    3.3 + 3.3  13.9 / 15.6     10.4 + 36.2  58.2 / 52.8 *    18.1 + 5.2  45.7 / 33.3 *
// (0.8 bits per weight, inner width 3 times the columns, 28672 at 8192.)  A layer of all four, us, all here / all there / by the rule:
//   9 tokens    2048  26.3 / 34.5 / 26.2    4096  44.2 / 51.2 / 44.2    5120  59.1 / 62.8 / 60.8    6144   72.3 / 73.0 / 70.9
//               8192 126.5 / 117.9 / 117.5  4096 at 1.5 bits  55.7 / 65.2 / 61.7    5120 at 1.2 bits  74.1 / 76.9 / 77.7
//   16 tokens   2048  26.6 / 34.4 / 26.8    4096  46.1 / 51.3 / 46.2    5120  61.4 / 62.8 / 61.7    6144   74.9 / 72.9 / 71.9
//               8192 132.1 / 118.1 / 117.9  4096 at 1.5 bits  60.1 / 65.4 / 62.8    5120 at 1.2 bits  77.9 / 77.1 / 78.7
// The lines (8 MB; 4.5 MB with 8192 columns) were drawn for an earlier main loop, 15 % slower.  They leave layers in one kernel or send there what
// still belongs there, within 3 % of the better one, except nine tokens of 4096 columns at 1.5 bits (11 %) and of 5120 at 1.2 (5 %): lines at 16 MB, and
// 8 MB with 8192 columns, would be better for those, but every line in MB is wrong somewhere in this table (down of 5120 columns, q/k/v of 8192): what
// should decide is a predicted time, as between the two GEMMs.
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
    const size_t step_bytes = frag_in ? 0 : (size_t)kBatchWarps * (T + 1) * step_blocks(nt) * 32;
    size_t row_bytes = 0, slot_used = 0, part_used = 0;      // row_bytes: output scales of a CTA, and as much for the bias
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
        const size_t bytes = (size_t)(j.g_q + (j.g_r ? 1 : 0)) * 32;
        j.bulk = frag_in && (!S.post || aligned16(S.post)) && (!S.bias || aligned16(S.bias)) && S.Nout % 8 == 0 && bytes <= kMostRowBytes;
        const size_t kept = j.bulk || bytes < 32 * kMostBlock ? bytes : 32 * kMostBlock;      // of all rows of a CTA, or of a block
        if (kept > row_bytes) row_bytes = kept;
        j.whole = frag_out || (reinterpret_cast<uintptr_t>(S.out) % 4 == 0 && S.ld_out % 2 == 0);
        memset(P.cta_job + cta, i, (size_t)ncta[i]);
        cta += ncta[i];
    }
    // Row blocks, as equal as possible: each job's weights and partial sums fit the room together; where the largest of
    // both over the jobs do not, each of them gets half; and where one row group does not fit half, one row group per
    // block (64 KB of weights at the largest K, 21 KB of partial sums).
    // Two staged steps per warp where that leaves each job in one block.
    int steps = kMostSteps;
    for (int attempt = -1; attempt < 3; ++attempt) {
        steps = attempt < 0 ? kMostSteps : 1;
        const size_t taken = kFixedBytes + steps * step_bytes + 2 * row_bytes + 256;
        const size_t room = limit > (int)taken ? limit - taken : 0;      // weights and partial sums of a block
        slot_used = part_used = 0;
        int most_block = 1;
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
                j.wk = (uint8_t)wk; j.wr = (uint8_t)wr;
                part = (size_t)j.wk * T * (j.gb * 16 + 4) * 4;
                slot = (size_t)j.gb * chunks[i] * 512;
                const bool fits = attempt <= 0 ? part + slot <= room : part <= room / 2 && slot <= room / 2;
                if (j.gb == 1 || attempt < 0 || (fits && j.gb <= kMostBlock)) break;
            }
            part_used = part > part_used ? part : part_used;
            slot_used = slot > slot_used ? slot : slot_used;
            j.wk_magic = (65536 + j.wk - 1) / j.wk;
            j.wr_magic = (65536 + j.wr - 1) / j.wr;
            const int blocks = (most + j.gb - 1) / j.gb, per_warp = (j.gb + j.wr - 1) / j.wr;
            most_blocks = blocks > most_blocks ? blocks : most_blocks;
            most_block = j.gb > most_block ? j.gb : most_block;
            most_rows = per_warp > most_rows ? per_warp : most_rows;
        }
        if (part_used + slot_used <= room && (attempt >= 0 || most_block <= kMostBlock)) break;
    }
    const size_t rest = kFixedBytes + steps * step_bytes + 2 * row_bytes + 256;
    int slots = most_blocks < kBatchSlots ? most_blocks : kBatchSlots;
    while (slots > 1 && part_used + slots * slot_used + rest > (size_t)limit) --slots;
    P.slots = slots;
    P.slot_bytes = (int)slot_used;
    P.frag_out = frag_out;
    P.steps = steps;
    P.part_off = (int)(kFixedBytes + slots * slot_used);
    P.post_off = (P.part_off + (int)part_used + 15) / 16 * 16;
    P.bias_off = P.post_off + (int)row_bytes;
    P.stage_off = (P.bias_off + (int)row_bytes + 127) / 128 * 128;
    const int tokens_out = split ? kSplitTokens : T;
    P.t_magic = (65536 + tokens_out - 1) / tokens_out;
    const size_t smem = P.stage_off + steps * step_bytes;
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
