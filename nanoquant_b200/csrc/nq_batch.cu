// One stage of a decode batch (a handful to a few dozen tokens): Out[T, rows] = (A[T, K] . W[rows, K]^T) * post.
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
//    of a token is its four consecutive columns 4q..4q+3: one 64-bit load from global memory, no staging.
//  * Two barriers; no K split over CTAs, no counters, no slabs.
//
// Qwen3-8B decode, eight layers in a graph, GEMM against this kernel: 8 tokens 804 -> 433 us, 16 tokens 825 -> 544 us; 32
// tokens 842 -> 1141 us, where it stops.
#include <cstddef>
#include <cstring>

#include "nq_common.cuh"
#include "nq_plan.h"
#include "nq_stage.h"

namespace nq {

constexpr int kBatchThreads = 512;
constexpr int kBatchWarps = kBatchThreads / 32;
constexpr int rows_per_pass(int nt) { return nt == 4 ? 2 : 4; }     // row groups a warp keeps accumulators for
constexpr int blocks_in_flight(int nt) { return nt == 1 ? 8 : 4; }  // 16-column blocks whose B fragments are loaded together
constexpr int kBatchSlots = 8;           // weight blocks in flight
constexpr int kBatchMaxCtas = 256;
constexpr size_t kOffParams = 64, kFixedBytes = 1024;
constexpr size_t kSlotBytes = 64 << 10;  // weights of a row block
constexpr size_t kPartBytes = 64 << 10;  // partial sums of a row block
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
    int T, io_bf16, out_bf16, saturate, exp_sign;
    int slots, slot_bytes, part_off, pad[2];
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

// NT: column groups of eight tokens.
template <bool BF16, int NT>
__global__ void __launch_bounds__(kBatchThreads, 1) batch_stage_kernel(const __grid_constant__ BatchParams Pc) {
    constexpr int kRows = rows_per_pass(NT), kB = blocks_in_flight(NT);
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
    const int T = P.T, slots = P.slots, slot_bytes = P.slot_bytes, chunks = jb.chunks, gb = jb.gb, rows = jb.rows;
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
    const uint16_t* a_row[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
        a_row[nt] = static_cast<const uint16_t*>(jb.a) + (long long)min(8 * nt + g, T - 1) * jb.lda + 4 * q;   // tokens beyond T: not stored
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    int slot = 0;
    uint32_t parity = 0;
#pragma unroll 1
    for (int blk = 0; blk < groups; blk += gb) {
        const int nb = min(gb, groups - blk);
        const int r0 = (rw * nb * wr_magic) >> 16, r1 = rw < wr ? ((rw + 1) * nb * wr_magic) >> 16 : r0;
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
#pragma unroll 1
            for (int c = c0; c < c1; ++c) {
#pragma unroll
                for (int b0 = 0; b0 < 16; b0 += kB) {
                    uint2 x[NT][kB], s[kB];
#pragma unroll
                    for (int b = 0; b < kB; ++b) {
                        const int k = c * 256 + (b0 + b) * 16;        // + 4q in a_row: K is a multiple of 8
                        const bool in = k + 4 * q < K;
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt)
                            x[nt][b] = in ? *reinterpret_cast<const uint2*>(a_row[nt] + k) : make_uint2(0u, 0u);
                        s[b] = pre && in ? __ldg(reinterpret_cast<const uint2*>(pre + k + 4 * q))
                                         : (BF16 ? make_uint2(0x3F803F80u, 0x3F803F80u) : make_uint2(0x3C003C00u, 0x3C003C00u));
                    }
                    if (b0 == 0 && c == c0 && rb == r0) {
#pragma unroll 1
                        for (unsigned spins = 0; !mbar_try(bars + 8 * slot, parity); ++spins)
                            if (spins >= kWeightWaitLimit) { atomicExch(P.status, (unsigned)(-NQ_ERR_TIMEOUT)); break; }
                    }
                    uint4 w[kRows];
#pragma unroll
                    for (int r = 0; r < kRows; ++r)
                        w[r] = *reinterpret_cast<const uint4*>(weights + slot * slot_bytes +
                                                               ((size_t)(rb + min(r, nr - 1)) * chunks + c) * 512 + lane * 16);
#pragma unroll
                    for (int b = 0; b < kB; ++b) {
                        const int j = (b0 + b) >> 1, h = b & 1;       // block = columns 32 j + 16 h + ..
                        const uint32_t se = even_columns(s[b]), so = odd_columns(s[b]);
                        uint32_t be[NT], bo[NT];
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) { be[nt] = even_columns(x[nt][b]); bo[nt] = odd_columns(x[nt][b]); }
#pragma unroll
                        for (int r = 0; r < kRows; ++r)
                            if (r < nr) {
                                const uint32_t w0 = h ? w[r].z : w[r].x, w1 = h ? w[r].w : w[r].y;   // rows g, g + 8
                                const uint32_t a0 = ((w0 << (15 - j)) & 0x80008000u) ^ se, a2 = ((w0 << (7 - j)) & 0x80008000u) ^ so;
                                const uint32_t a1 = ((w1 << (15 - j)) & 0x80008000u) ^ se, a3 = ((w1 << (7 - j)) & 0x80008000u) ^ so;
#pragma unroll
                                for (int nt = 0; nt < NT; ++nt) mma_16816<BF16>(acc[r][nt], a0, a1, a2, a3, be[nt], bo[nt]);
                            }
                    }
                }
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
        __syncthreads();   // partial sums complete, this block's weights have been read
        if (++slot == slots) { slot = 0; parity ^= 1u; }
        if (loader) load_block();
        // outputs: lanes take rows, warps take tokens
        const int io_bf16 = P.io_bf16, out_bf16 = P.out_bf16, kslice = T * tok_stride;
        const float lim = P.saturate ? (out_bf16 ? 3.3895313892515355e+38f : 64504.0f) : 3.4e38f;
        const uint16_t* const resid = static_cast<const uint16_t*>(jb.resid);
        const int row0 = (first + blk) * 16;
#pragma unroll 1
        for (int idx = lane; idx < nb * 16 && row0 + idx < rows; idx += 32) {
            const int row = row0 + idx;
            const float post = jb.post ? float_of(static_cast<const uint16_t*>(jb.post)[row], io_bf16) : 1.f;
            const float bias = jb.bias ? float_of(static_cast<const uint16_t*>(jb.bias)[row], io_bf16) : 0.f;
#pragma unroll 1
            for (int tok = warp; tok < T; tok += kBatchWarps) {
                const float* src = part + tok * tok_stride + idx;
                float v = 0.f;
#pragma unroll 4
                for (int k = 0; k < wk; ++k, src += kslice) v += *src;
                const float rs = jb.row_exp ? exp2f((float)(P.exp_sign * jb.row_exp[tok])) : 1.f;
                float extra = bias;
                if (resid) extra += float_of(resid[tok * jb.ld_res + row], io_bf16);
                v = fminf(fmaxf(v * (post * rs) + extra, -lim), lim);
                const long long at = tok * jb.ld_out + row;
                if (out_bf16) static_cast<__nv_bfloat16*>(jb.out)[at] = __float2bfloat16(v);
                else static_cast<__half*>(jb.out)[at] = __float2half(v);
            }
        }
        if (blk + gb < groups) __syncthreads();   // the partial sums have been read
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
constexpr int kMostTokens = 16;    // above, every CTA's fetch of the whole input outweighs the GEMM's fixed costs (see the figures above)

static const void* batch_kernel(int bf16, int T) {
    const int nt = T <= 8 ? 1 : T <= 16 ? 2 : 4;
    if (bf16) return nt == 1 ? (const void*)batch_stage_kernel<true, 1> : nt == 2 ? (const void*)batch_stage_kernel<true, 2> : (const void*)batch_stage_kernel<true, 4>;
    return nt == 1 ? (const void*)batch_stage_kernel<false, 1> : nt == 2 ? (const void*)batch_stage_kernel<false, 2> : (const void*)batch_stage_kernel<false, 4>;
}
static int batch_smem_limit(int* out) {
    static int cached[64];
    int dev = 0;
    NQ_CUDA_TRY(cudaGetDevice(&dev));
    if (cached[dev & 63] == 0) {
        int optin = 0;
        NQ_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        for (int i = 0; i < 6; ++i)
            NQ_CUDA_TRY(cudaFuncSetAttribute(batch_kernel(i & 1, 8 << (i >> 1)), cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
        cached[dev & 63] = optin;
    }
    *out = cached[dev & 63];
    return NQ_OK;
}

int batch_max_tokens(const StageJob* jobs, int n) {
    for (int i = 0; i < n; ++i)
        if (jobs[i].K > 65536) return 0;    // one row group's weights have to fit beside its partial sums
    return kMostTokens;
}

int launch_batch_stage(const StageJob* jobs, int n, int T, StageTypes ty, int saturate, unsigned* status, cudaStream_t stream) {
    int limit = 0;
    { const int st = batch_smem_limit(&limit); if (st != NQ_OK) return st; }
    BatchParams P;
    memset(&P, 0, sizeof(P));
    P.status = status;
    P.T = T;
    P.io_bf16 = ty.io_bf16; P.out_bf16 = ty.out_bf16; P.saturate = saturate; P.exp_sign = ty.exp_sign;
    const int nt = T <= 8 ? 1 : T <= 16 ? 2 : 4;
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
    size_t slot_used = 0, part_used = 0;
    int cta = 0, most_blocks = 1;
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
        const int most = j.g_q + (j.g_r ? 1 : 0);
        for (int blocks = 1;; ++blocks) {   // row blocks whose weights and partial sums fit, as equal as possible
            j.gb = (most + blocks - 1) / blocks;
            // Chunk slices x row slices: a step (a row group's chunk) against fetching a chunk's B fragments, which a
            // warp does once per pass over its row groups.
            int best = 1 << 30;
            for (int k = 1; k <= kBatchWarps && k <= chunks[i]; ++k) {
                int r = kBatchWarps / k;
                if (r > j.gb) r = j.gb;
                const int per = (j.gb + r - 1) / r;
                const int cost = ((chunks[i] + k - 1) / k) * (per * (2 + T / 8) + ((per + rows_per_pass(nt) - 1) / rows_per_pass(nt)) * (2 + T / 4));
                if (cost < best) { best = cost; j.wk = (uint16_t)k; j.wr = (uint16_t)r; }
            }
            const size_t part = (size_t)j.wk * T * (j.gb * 16 + 4) * 4, slot = (size_t)j.gb * chunks[i] * 512;
            if (j.gb == 1 || (part <= kPartBytes && slot <= kSlotBytes && j.gb <= 128)) {
                part_used = part > part_used ? part : part_used;
                slot_used = slot > slot_used ? slot : slot_used;
                break;
            }
        }
        j.wk_magic = (65536 + j.wk - 1) / j.wk;
        j.wr_magic = (65536 + j.wr - 1) / j.wr;
        const int blocks = (most + j.gb - 1) / j.gb;
        most_blocks = blocks > most_blocks ? blocks : most_blocks;
    }
    int slots = most_blocks < kBatchSlots ? most_blocks : kBatchSlots;
    while (slots > 1 && kFixedBytes + part_used + slots * slot_used > (size_t)limit) --slots;
    P.slots = slots;
    P.slot_bytes = (int)slot_used;
    P.part_off = (int)(kFixedBytes + slots * slot_used);
    const size_t smem = P.part_off + part_used;
    if (smem > (size_t)limit) return NQ_ERR_UNSUPPORTED;
    static bool pdl_ok = true;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cta);
    cfg.blockDim = dim3(kBatchThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = pdl_ok ? 1 : 0;
    void* args[] = {&P};
    const void* fn = batch_kernel(ty.a_bf16, T);
    cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    if (e != cudaSuccess && pdl_ok) {
        (void)cudaGetLastError();
        pdl_ok = false;
        cfg.numAttrs = 0;
        e = cudaLaunchKernelExC(&cfg, fn, args);
    }
    NQ_CUDA_TRY(e);
    return NQ_OK;
}

}  // namespace nq
