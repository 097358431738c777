// GEMM of a stage with the weights on the row side of the MMA, for prompts: pairs of CTAs, each pair with several tiles in turn.
//
// Two CTAs (a cluster) share a tile of 256 weight rows x 32..256 tokens: tcgen05.mma cta_group::2, M = 256, each CTA expands its 128
// rows into its own tensor memory and loads half of the tokens; one thread of the first CTA issues for both.
//
//   warp 0       activations by TMA, two boxes of 64 columns per step, counted by the first CTA's barrier
//   warp 1       MMAs (first CTA), eight per step of 128 columns
//   warp 2       the input scales of all jobs, once (beyond shared memory's room they are read from global memory)
//   warp 3       the first tile's weights to L2
//   warps 4-19   expansion, two groups of eight warps on alternate steps; weights two chunks ahead, across the tiles
//   warps 20-27  epilogue, two sets of four warps, 32 tokens in turn, through a transposing staging buffer
//
//  * As in nq_wgemm.cu no expanded weight passes through shared memory, and the token side has any multiple of 32: 517 tokens pay
//    for 544 to 576, not for 640 or 768.  A pair fetches every activation once (48 to 64 bytes per cycle and SM with 128-row tiles alone).
//  * The grid is one pair per two SMs; a pair takes tiles p, p + pairs, ...  With two accumulators (up to 160 tokens: 3 and more stages
//    of 64 columns remain for the A operand) the epilogue of a tile runs beside the main loop of the next.
//  * Every arrival on the other CTA's barriers has the default (CTA) scope: tensor memory and TMA writes are ordered by their own
//    waits and fences, and a cluster-scope release waited for the weight loads in flight (0.24 us per 64 columns, 0.14 without).
//  * An expand group takes every second step of the CTA's whole sequence, whatever tile it belongs to.
//
// Per step of 128 columns, on few SMs, us: 0.35 at 160 tokens and 0.555 at 256 are the MMAs; the expansion takes 0.26 for +-1 in the
// swapped order (kOrderIn) and 0.345 with input scales.  On all SMs at 2048 tokens the clocks fall under the power cap.
//
// Stages through 256-token tiles whose weights were expanded into shared memory (the GEMM that this and nq_wgemm.cu replaced) and as the
// planners choose now, one launch after another in a graph, us:
//   K -> rows            517 tokens      1024            2048
//   4096 -> 2 x 2432     31.2 -> 21.8    50.3 -> 32.7    92.3 -> 57.2
//   2432 -> 2 x 12288    69 -> 46.8      104 -> 79.7     221 -> 154
//   12288 -> 2432        44.7 -> 37.6    66.7 -> 48.0    139 -> 93.7
//   1600 -> 4096         15.8 -> 11.2    17.2 -> 14.5    26.5 -> 21.7
// Layers: Qwen3-8B 517 tokens 244 -> 175, Llama-2-7B 2048 tokens 720 -> 580 (1.41 PFLOP/s).
//
#include <cuda.h>

#include <cstring>

#include "nq_common.cuh"
#include "nq_stage.h"
#include "nq_tcgen05.cuh"

namespace nq {

constexpr int kPExpandWarps = 16, kPEpilogueWarps = 8;
constexpr int kPThreads = 32 * (4 + kPExpandWarps + kPEpilogueWarps);
constexpr int kPGroups = 2;                      // expand groups of eight warps, on alternate steps of 128 columns
constexpr int kPRows = 256;                      // weight rows of a pair's tile
constexpr int kPMaxStages = 8;
constexpr int kPTmemCols = 512;

struct alignas(16) PJob {
    const uint4* tiles;
    const void* pre;
    const void* post;
    void* out;
    const int* row_exp;
    const void* bias;
    const void* resid;
    long long ld_out, ld_res;
    int K, Nout;
    int chunks, row_groups;
    int row_tiles, tile0;
    int pre0, unused[3];
};
static_assert(sizeof(PJob) == 112, "seven 16-byte words");
struct alignas(16) PHead {
    unsigned* status;      // (this and the wait limit are read from the parameters, not from the copy)
    int njobs, tiles;
    int T;
    int ntok, stages, accs;   // tokens of a tile (a multiple of 16), pipeline stages of 64 columns, accumulators (1 or 2)
    int is_bf16, a_bf16, saturate, exp_sign;
    int order;                // kOrderOut, kOrderIn
    int off_out, off_pre;     // output staging; input scales of job j from off_pre + pre0 (pre0 < 0: read from global memory)
    unsigned wait_limit;
};
struct alignas(64) PParams {
    CUtensorMap map_a[kMaxGemmJobs];     // activations [T, K], box 64 x half of a tile's tokens, 128-byte swizzle
    PJob job[kMaxGemmJobs];
    PHead head;            // (the jobs and the head are copied to shared memory together)
};
constexpr int kPParamWords = (int)(sizeof(PJob) * kMaxGemmJobs + sizeof(PHead)) / 16;
// shared memory (from a 1024-byte boundary): descriptors, barriers, B stages, output staging, input scales
constexpr int kPBarOff = 640, kPBOff = 1024, kPOutBytes = 4 * 32 * 256;
static_assert(kPParamWords * 16 <= kPBarOff && kPBOff % 1024 == 0, "shared memory map");

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {   // `bar`: an address of cluster_map
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Load into this CTA's shared memory, counted by a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {      // the barrier at this offset in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// 32 columns of 16 rows.
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, float (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
                   "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;"      // (the registers are operands, so that no use moves above it)
                 : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]),
                   "+f"(r[8]), "+f"(r[9]), "+f"(r[10]), "+f"(r[11]), "+f"(r[12]), "+f"(r[13]), "+f"(r[14]), "+f"(r[15]) :: "memory");
}
template <int OUT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPThreads, 1) pgemm_kernel(const __grid_constant__ PParams Pc) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < kPParamWords)
        reinterpret_cast<uint4*>(smem)[threadIdx.x] = reinterpret_cast<const uint4*>(&Pc.job[0])[threadIdx.x];
    const uint32_t bars = sbase + kPBarOff;
    auto bar_ready = [&](int s) { return bars + 8 * s; };                                   // used in the leader
    auto bar_free = [&](int s) { return bars + 8 * (kPMaxStages + s); };
    const uint32_t bar_pre = bars + 8 * (2 * kPMaxStages);
    auto bar_acc_full = [&](int a) { return bars + 8 * (2 * kPMaxStages + 1 + a); };
    auto bar_acc_empty = [&](int a) { return bars + 8 * (2 * kPMaxStages + 3 + a); };   // used in the leader
    constexpr int kMisc = kPBarOff + 8 * (2 * kPMaxStages + 6);
    static_assert(kMisc + 8 <= kPBOff, "shared memory map");
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kMisc);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kMisc + 4);
    const int rank = (int)(blockIdx.x & 1);          // in the pair; 0 issues the MMAs
    if (warp == 2) {
        if (lane < kPMaxStages) {
            mbar_init(bar_ready(lane), 1 + 16);      // the leader's producer, eight expand warps of each CTA
            mbar_init(bar_free(lane), 1);
        }
        if (lane < 2) {
            mbar_init(bar_acc_full(lane), 1);
            mbar_init(bar_acc_empty(lane), 2 * kPEpilogueWarps);
        }
        if (lane == 0) {
            mbar_init(bar_pre, 1);
            *abort_flag = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(const_cast<uint32_t*>(tmem_slot))), "r"((uint32_t)kPTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // both CTAs' barriers and tensor memory are there
    tc_fence_after();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const PHead& P = *reinterpret_cast<const PHead*>(smem + sizeof(PJob) * kMaxGemmJobs);
    const PJob* jobs = reinterpret_cast<const PJob*>(smem);
    const int pairs = (int)(gridDim.x >> 1), tiles = P.tiles, first = (int)(blockIdx.x >> 1);
    const int ntok = P.ntok, stages = P.stages, accs = P.accs;
    const uint32_t tmem_base = *tmem_slot;                    // accumulators, then the A stages of 64 columns
    const uint32_t tmem_a = tmem_base + (uint32_t)(accs * ntok);
    const uint32_t b_base = sbase + kPBOff, stage_bytes = (uint32_t)ntok * 128u;     // this CTA's half of the tokens
    auto job_of = [&](int t) { int j = 0; while (j + 1 < P.njobs && t >= jobs[j + 1].tile0) ++j; return j; };

    if (warp == 0) {
        // ---------------------------------------------------------------- activations
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int t = first; t < tiles && ok; t += pairs) {
            const int j = job_of(t), local = t - jobs[j].tile0, mt = local / jobs[j].row_tiles;
            const CUtensorMap* map = &Pc.map_a[j];
            const int m0 = mt * ntok + rank * (ntok >> 1), nst = (jobs[j].K + 127) >> 7;
            for (int st = 0; st < nst; ++st) {
                ok = mbar_wait_warp(bar_free(s), ph ^ 1, abort_flag, Pc.head.status, Pc.head.wait_limit);
                if (!ok) break;
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(bar_ready(s), 2u * stage_bytes);
                    const uint32_t dst = b_base + (uint32_t)s * stage_bytes, bar = cluster_map(bar_ready(s), 0);
                    tma_load_2d_pair(dst, map, 128 * st, m0, bar);
                    tma_load_2d_pair(dst + (stage_bytes >> 1), map, 128 * st + 64, m0, bar);
                }
                if (++s == stages) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issue
        if (rank == 0) {
            const uint32_t fmt = P.a_bf16 ? 1u : 0u;
            const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(ntok >> 3) << 17) | ((uint32_t)(kPRows >> 4) << 24);
            int s = 0, a = 0;
            uint32_t ph = 0, aph = 0;
            bool ok = true;
            for (int t = first; t < tiles && ok; t += pairs) {
                const int nst = (jobs[job_of(t)].K + 127) >> 7;
                const uint32_t d = tmem_base + (uint32_t)(a * ntok);
                ok = mbar_wait_warp<true>(bar_acc_empty(a), aph ^ 1, abort_flag, Pc.head.status, Pc.head.wait_limit);
                for (int st = 0; st < nst && ok; ++st) {
                    ok = mbar_wait_warp<true>(bar_ready(s), ph, abort_flag, Pc.head.status, Pc.head.wait_limit);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t b_desc = umma_desc(b_base + (uint32_t)s * stage_bytes);
                        const uint32_t wa = tmem_a + (uint32_t)(64 * s);
                        const uint64_t half = (uint64_t)(stage_bytes >> 5);
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            umma_pair(d, wa + 8 * k, b_desc + (k >> 2) * half + (uint64_t)(2 * (k & 3)), idesc, (st | k) ? 1u : 0u);
                        umma_commit_pair(bar_free(s));
                    }
                    if (++s == stages) { s = 0; ph ^= 1; }
                }
                if (ok && elect_one()) umma_commit_pair(bar_acc_full(a));
                if (++a == accs) { a = 0; aph ^= 1; }
            }
        }
    } else if (warp == 2) {
        // ---------------------------------------------------------------- input scales of all jobs
        if (elect_one()) {
            uint32_t bytes = 0;
            for (int j = 0; j < P.njobs; ++j)
                if (jobs[j].pre && jobs[j].pre0 >= 0) bytes += (uint32_t)jobs[j].K * 2u;
            mbar_expect_tx(bar_pre, bytes);
            for (int j = 0; j < P.njobs; ++j)
                if (jobs[j].pre && jobs[j].pre0 >= 0)
                    bulk_load(sbase + (uint32_t)(P.off_pre + jobs[j].pre0), jobs[j].pre, (uint32_t)jobs[j].K * 2u, bar_pre);
        }
    } else if (warp == 3) {
        // ---------------------------------------------------------------- the first tile's weights on their way to L2
        if (first < tiles) {
            const PJob& J = jobs[job_of(first)];
            const int rg = (first - J.tile0) % J.row_tiles * 16 + 8 * rank + lane;
            if (lane < 8 && rg < J.row_groups)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(J.tiles + (size_t)rg * J.chunks * 32), "r"((uint32_t)J.chunks * 512u) : "memory");
        }
    } else if (warp < 4 + kPExpandWarps) {
        // ---------------------------------------------------------------- expansion
        const int grp = (warp - 4) >> 3, q = lane & 3;
        const int rgl = 2 * (warp & 3) + ((warp >> 2) & 1 ^ 1);     // row group of the CTA's eight
        const uint32_t one2 = P.a_bf16 ? 0x3F803F80u : 0x3C003C00u;
        const bool in_order = P.order != kOrderIn;
        const int src_lane = P.order == kOrderOut ? 4 * swap_middle(lane >> 2) + q : lane;
        const uint32_t a_lane = tmem_a + ((uint32_t)(16 * rgl) << 16);
        const uint32_t ready0 = cluster_map(bar_ready(0), 0);
        // weights two chunks ahead, across the tiles of this CTA
        int nt = first, left = 0;
        const uint4* wp = nullptr;
        bool there = false;
        auto seek = [&]() {
            if (nt < tiles) {
                const PJob& J = jobs[job_of(nt)];
                const int rg = (nt - J.tile0) % J.row_tiles * 16 + 8 * rank + rgl;
                left = J.chunks;
                there = rg < J.row_groups;
                wp = J.tiles + (size_t)(there ? rg : 0) * J.chunks * 32 + src_lane;
            }
        };
        auto fetch = [&]() {
            uint4 w = make_uint4(0u, 0u, 0u, 0u);
            if (nt < tiles) {
                if (there) w = __ldg(wp);
                wp += 32;
                if (--left == 0) { nt += pairs; seek(); }
            }
            return w;
        };
        seek();
        uint4 w1 = fetch(), w2 = fetch();
        unsigned base = 0;                 // steps before this tile
        bool ok = mbar_wait_warp(bar_pre, 0, abort_flag, Pc.head.status, Pc.head.wait_limit);
        for (int t = first; t < tiles && ok; t += pairs) {
            const PJob& J = jobs[job_of(t)];
            const int K = J.K, nst = (K + 127) >> 7, chunks = J.chunks;
            const bool pre = J.pre != nullptr;
            // (a generic pointer: shared memory unless the scales of the launch do not fit)
            const uint2* sp = (J.pre0 >= 0 ? reinterpret_cast<const uint2*>(smem + P.off_pre + J.pre0) : static_cast<const uint2*>(J.pre)) + q;
            // A group takes every other step of all this CTA has, not of every tile: it then never skips a turn, and a turn is at
            // most one round of the stages, so that a stage's phase cannot be mistaken for the one before the last.
            const int sub = (int)((grp - base) & 1), pre_shift = sub ? 0 : 4;
            int s = (int)((base + sub) % (unsigned)stages);
            uint32_t ph = (base + sub) / (unsigned)stages & 1u;
            base += (unsigned)nst;
            for (int c = 0; c < chunks && ok; ++c) {
                uint4 w = w1;
                w1 = w2;
                w2 = fetch();
                const int st = 2 * c + sub;
                if (st < nst) {
                    w.x <<= pre_shift; w.y <<= pre_shift; w.z <<= pre_shift; w.w <<= pre_shift;
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {       // 64 columns
                        uint32_t v[16];
                        if (in_order) {
                            uint2 pn[4];
                            const int k0 = 128 * st + 64 * hf;
                            if (!pre) {
#pragma unroll
                                for (int i = 0; i < 4; ++i) pn[i] = make_uint2(one2, one2);
                            } else if (k0 + 64 <= K) {
#pragma unroll
                                for (int i = 0; i < 4; ++i) pn[i] = sp[(k0 >> 2) + 4 * i];
                            } else {                       // some of the columns are beyond K
#pragma unroll
                                for (int i = 0; i < 4; ++i) pn[i] = k0 + 16 * i + 4 * q < K ? sp[(k0 >> 2) + 4 * i] : make_uint2(0u, 0u);
                            }
                            expand_columns(w, hf, pn, v);
                        } else {
                            expand_swapped(w, hf, one2, v);
                        }
                        if (hf == 0) {
                            ok = mbar_wait_warp(bar_free(s), ph ^ 1, abort_flag, Pc.head.status, Pc.head.wait_limit);
                            tc_fence_after();
                        }
                        tmem_st_frag4(a_lane + (uint32_t)(64 * s + 32 * hf), v);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0 && ok) mbar_arrive_cluster(ready0 + 8 * s);
                    s += kPGroups;
                    if (s >= stages) { s -= stages; ph ^= 1; }
                }
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue: two sets of four warps, 32 tokens in turn
        const int ew = warp & 3, g = lane >> 2, q = lane & 3, set = (warp - 4 - kPExpandWarps) >> 2;
        const int tu = (int)(threadIdx.x & 127);
        const int row_g = P.order == kOrderOut ? swap_middle(g) : g;
        const uint32_t out_stage = sbase + (uint32_t)P.off_out + (uint32_t)set * (2 * 32 * 256);
        // matrix i of the transposing store: tokens 8 (i >> 1) .., rows 8 (i & 1) ..; 16-byte units of a row swizzled by the token
        const int st_tok = 8 * (lane >> 4) + (lane & 7), st_unit = 4 * ew + ((lane >> 3) & 1);
        const int unit = tu & 15, ld_tok = tu >> 4;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int a = 0, buf = 0;
        uint32_t aph = 0;
        bool ok = true;
        for (int t = first; t < tiles; t += pairs) {
            const PJob& J = jobs[job_of(t)];
            const int local = t - J.tile0, mt = local / J.row_tiles;
            const int n0 = (local - mt * J.row_tiles) * kPRows + 128 * rank, m0 = mt * ntok, Nout = J.Nout;
            float sc[4], bi[4];                       // rows g, g + 8 of both row groups of this warp
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = n0 + 32 * ew + 8 * i + row_g;
                sc[i] = J.post && row < Nout ? io_float(__ldg(static_cast<const unsigned short*>(J.post) + row), P.is_bf16) : 1.f;
                bi[i] = J.bias && row < Nout ? io_float(__ldg(static_cast<const unsigned short*>(J.bias) + row), P.is_bf16) : 0.f;
            }
            const uint16_t* resid = static_cast<const uint16_t*>(J.resid);
            const int* row_exp = J.row_exp;
            const int row_s = n0 + 8 * unit, live = min(ntok, P.T - m0);
            const long long ld_out = J.ld_out;
            uint16_t* out = static_cast<uint16_t*>(J.out) + (size_t)(m0 + 32 * set + ld_tok) * ld_out + row_s;
            const bool whole = row_s + 8 <= Nout && ((reinterpret_cast<uintptr_t>(out) | (uintptr_t)(2 * ld_out)) & 15u) == 0;
            ok = ok && mbar_wait_warp(bar_acc_full(a), aph, abort_flag, Pc.head.status, Pc.head.wait_limit);
            tc_fence_after();                         // (not ok: on all the same, the four warps pass the same barriers)
            const uint32_t d_lane = tmem_base + (uint32_t)(a * ntok) + ((uint32_t)(32 * ew) << 16);
            bool held = true;                         // the accumulator
#pragma unroll 1
            for (int tb = 32 * set; tb < live; tb += 64) {
                const uint32_t stage = out_stage + (uint32_t)buf * (32 * 256);
#pragma unroll
                for (int rr = 0; rr < 2; ++rr) {
                    float r[16] = {};
                    if (ok) tmem_ld_frag(d_lane + ((uint32_t)(16 * rr) << 16) + (uint32_t)tb, r);
                    if (rr == 1 && tb + 64 >= live) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(cluster_map(bar_acc_empty(a), 0));
                        held = false;
                    }
                    // r[8 h + 2 i + e]: token 16 h + 8 (i >> 1) + 2 q + e, row 16 rr + 8 (i & 1) + g
                    if (row_exp) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const int tok = m0 + tb + 16 * (k >> 2) + 8 * ((k >> 1) & 1) + 2 * q + (k & 1);
                            const float ts = tok < P.T ? exp2f((float)(P.exp_sign * row_exp[tok])) : 1.f;
                            r[8 * (k >> 2) + 4 * ((k >> 1) & 1) + (k & 1)] *= ts;
                            r[8 * (k >> 2) + 4 * ((k >> 1) & 1) + 2 + (k & 1)] *= ts;
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 16; ++k) r[k] = fmaf(r[k], sc[2 * rr + ((k >> 1) & 1)], bi[2 * rr + ((k >> 1) & 1)]);
                    if (resid) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) {
                            const int tok = m0 + tb + 16 * (k >> 3) + 8 * ((k >> 2) & 1) + 2 * q + (k & 1);
                            const int row = n0 + 32 * ew + 16 * rr + 8 * ((k >> 1) & 1) + g;
                            if (tok < P.T && row < Nout) {
                                r[k] += io_float(resid[(size_t)tok * J.ld_res + row], P.is_bf16);
                            }
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t pk[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) pk[i] = pack_outputs<OUT>(r[8 * h + 2 * i], r[8 * h + 2 * i + 1], P.saturate);
                        const int tl = 16 * h + st_tok;
                        const uint32_t addr = stage + (uint32_t)(tl * 256 + (((st_unit + 2 * rr) ^ (tl & 7)) << 4));
                        stmatrix_trans(addr, pk);
                    }
                }
                asm volatile("bar.sync %0, 128;" ::"r"(3 + set) : "memory");     // (buffers alternate: one barrier per 32 tokens)
                if (ok && row_s < Nout) {
                    uint4 v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int tl = 8 * i + ld_tok;
                        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[i].x), "=r"(v[i].y), "=r"(v[i].z), "=r"(v[i].w)
                                     : "r"(stage + (uint32_t)(tl * 256 + ((unit ^ (tl & 7)) << 4))) : "memory");
                    }
                    uint16_t* dst = out;
#pragma unroll
                    for (int i = 0; i < 4; ++i, dst += 8 * ld_out) {
                        if (tb + 8 * i + ld_tok < live) {
                            store_rows(dst, v[i], Nout - row_s, whole);
                        }
                    }
                }
                out += 64 * ld_out;
                buf ^= 1;
            }
            if (held) {                               // (fewer tokens than the sets take)
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(cluster_map(bar_acc_empty(a), 0));
            }
            if (++a == accs) { a = 0; aph ^= 1; }
        }
    }
    // On an expired wait, give the copies in flight a bounded time to land before shared memory is released.
    if (*abort_flag && threadIdx.x == 0) {
        for (unsigned i = 0; i < (1u << 20); ++i) __nanosleep(64);
    }
    __syncwarp();
    tc_fence_before();
    // the other CTA may still signal barriers here, and its MMAs and epilogue use the pair's tensor memory
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kPTmemCols) : "memory");
    }
}

static const void* p_kernel(int out) {
    return out == kOutFp16 ? (const void*)pgemm_kernel<kOutFp16> : out == kOutBf16 ? (const void*)pgemm_kernel<kOutBf16>
                                                                                     : (const void*)pgemm_kernel<kOutBf16Saturated>;
}

constexpr int kPSmemMost = 226 * 1024;

// Tile width and accumulators by a cost in microseconds, fitted to 1300 measured launches (20 shapes of 512..24576 rows and 512..12288
// columns, 128 to 2048 tokens, the eight widths); together with nq_wgemm.cu's plan the choice is 1.3 % above the best of both on average.  A
// step of 128 columns takes what its expansion or its MMAs take, whichever is longer.
PgemmPlan plan_pgemm(const StageJob* jobs, int n, int T, int order) {
    static const int sizes[] = {32, 64, 96, 128, 160, 192, 224, 256};
    PgemmPlan best = {0.f, 0, 0};
    const int most_pairs = sm_count() / 2;
    const float expand = order == kOrderIn ? 0.256f : 0.345f;
    for (int ntok : sizes) {
        if (ntok >= T + 32 && ntok > 32) continue;
        const int mt = (T + ntok - 1) / ntok, accs = ntok <= 160 ? 2 : 1;
        int ends[kMaxGemmJobs], tiles = 0;
        for (int j = 0; j < n; ++j) ends[j] = tiles += (jobs[j].Nout + kPRows - 1) / kPRows * mt;
        const int pairs = tiles < most_pairs ? tiles : most_pairs;
        const float mma = 0.0021f * ntok, step = (expand > mma ? expand : mma) + 0.037f * pairs / most_pairs;
        float t = 3.4f + 0.0086f * ntok + 0.00079f * T;
        for (int first = 0, j = 0; first < tiles; first += pairs) {      // rounds of one tile per pair, the longest tile of each
            while (ends[j] <= first) ++j;
            int steps = 0;
            for (int i = j; i < n && (i == j || ends[i - 1] < first + pairs); ++i) {
                const int st = (jobs[i].K + 127) / 128;
                steps = st > steps ? st : steps;
            }
            t += steps * step + 0.28f + (first > 0 && accs == 1 ? 0.0104f * ntok : 0.f);
        }
        if (best.ntok == 0 || t < best.us) best = {t, ntok, accs};
    }
    return best;
}

int launch_pgemm_stage(const StageJob* jobs_in, int n, int T, StageTypes ty, int saturate, const PgemmPlan& pl, unsigned* status,
                       cudaStream_t stream) {
    static bool attr_set[64];
    int dev = 0;
    NQ_CUDA_TRY(cudaGetDevice(&dev));
    if (!attr_set[dev & 63]) {
        for (int o = 0; o < 3; ++o) NQ_CUDA_TRY(cudaFuncSetAttribute(p_kernel(o), cudaFuncAttributeMaxDynamicSharedMemorySize, kPSmemMost));
        attr_set[dev & 63] = true;
    }
    StageJob jobs[kMaxGemmJobs];           // the longest tiles first
    for (int j = 0; j < n; ++j) {
        int i = j;
        for (; i > 0 && jobs[i - 1].K < jobs_in[j].K; --i) jobs[i] = jobs[i - 1];
        jobs[i] = jobs_in[j];
    }
    const int ntok = pl.ntok, accs = pl.accs;
    PParams P;
    memset(&P, 0, sizeof(P));
    PHead& H = P.head;
    int stages = (kPTmemCols - accs * ntok) / 64;
    if (stages > kPMaxStages) stages = kPMaxStages;
    H.njobs = n; H.status = status; H.wait_limit = gemm_wait_limit(); H.T = T; H.ntok = ntok; H.stages = stages; H.accs = accs;
    H.is_bf16 = ty.io_bf16; H.a_bf16 = ty.a_bf16; H.saturate = saturate; H.exp_sign = ty.exp_sign; H.order = ty.order;
    H.off_out = kPBOff + stages * ntok * 128;
    H.off_pre = H.off_out + kPOutBytes;
    int smem = 1024 + H.off_pre;
    const int mt = (T + ntok - 1) / ntok;
    int tiles = 0;
    for (int j = 0; j < n; ++j) {
        const StageJob& S = jobs[j];
        PJob& J = P.job[j];
        const int st = encode_activations(&P.map_a[j], S, ty.a_bf16, T, ntok / 2);
        if (st != NQ_OK) return st;
        J.tiles = static_cast<const uint4*>(S.tiles);
        J.pre = S.pre; J.post = S.post; J.out = S.out; J.ld_out = S.ld_out;
        J.row_exp = ty.exp_sign ? S.row_exp : nullptr;
        J.bias = S.bias; J.resid = S.resid; J.ld_res = S.ld_res;
        J.K = S.K; J.Nout = S.Nout;
        J.chunks = (S.K + 255) / 256;
        J.row_groups = (S.Nout + 15) / 16;
        J.row_tiles = (S.Nout + kPRows - 1) / kPRows;
        J.tile0 = tiles;
        J.pre0 = -1;
        if (S.pre && smem + S.K * 2 <= kPSmemMost) {
            J.pre0 = smem - 1024 - H.off_pre;
            smem += (S.K * 2 + 15) / 16 * 16;
        }
        tiles += J.row_tiles * mt;
    }
    H.tiles = tiles;
    const int pairs = sm_count() / 2 < tiles ? sm_count() / 2 : tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(kPThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    void* args[] = {&P};
    return launch_dependent(cfg, attr, 0, p_kernel(out_kind(ty, saturate)), args);
}

}  // namespace nq
