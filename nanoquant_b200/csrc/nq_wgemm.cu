// GEMM of a stage with the weights on the row side of the MMA, for a few dozen to a few hundred tokens:
// Out[T, rows] = (A[T, K] . W[rows, K]^T) * post.
//
// A CTA takes 128 weight rows (MMA M) x 16..128 tokens (MMA N, any multiple of 16) x a share of K:
//
//   warp 0      activations by TMA (128-byte swizzle), two boxes of 64 columns per step
//   warp 1      tcgen05.mma, eight per step, A from tensor memory, B from shared memory
//   warp 2      the input scales of the CTA's columns, one bulk copy
//   warps 4-11  expansion: sign bits (global memory, two chunks ahead) -> +-s_in[k] straight into tensor memory; then the
//               exchange and the epilogue
//
//  * No expanded weight passes through shared memory.  tcgen05.st 16x256b gives lane 4g + q the columns 4q..4q+3 of rows g and
//    g + 8 of a 16-column block, which are the bits that this lane holds in the tile layout: a PRMT that spreads
//    sign bits and one LOP3 per two weights.  Written to shared memory and read back by the MMA, as the operand of a 128 x 128
//    tile of the first GEMM here was, they made it shared-memory bound (485 cycles per 64 columns for 256 of MMA).
//  * Tokens are columns, so 33 tokens pay for 48 and not for 128.
//  * K is split over the CTAs of a cluster where tiles are few.  Blocks of 16 tokens x 128 rows are dealt to the CTAs; every
//    CTA sends the blocks it does not own by st.async, counted by an mbarrier of the owner, which adds them in rank order (the
//    result does not depend on timing).  Receive buffers of their own: nobody has to be done with its main loop before.
//    (A cluster barrier behind plain stores took 1.4 us, this 0.5.)
//  * Half of the SM's shared memory, tensor memory and registers: the CTAs of the next launch set up, fetch their weights and
//    expand the first steps while this one drains, and up to two CTAs of a launch share an SM.
//
// What a launch costs (globaltimer stamps, 4096 -> 2016, 64 tokens, 64 CTAs = 16 tiles x 4, us): dependency 1.0, activations
// 0.6, eight steps 2.4, last MMAs 0.3, exchange 0.5, output 0.9, exit 0.3.  A step of 128 columns takes 0.27 us alone on its SM, most
// of it the expansion (64 half-rate ALU operations of every warp per step, plus wait, store and signal), and 64 tokens of MMA are half
// of that.  k blocks of 64 cost 0.24 each: the signalling.  An issuing branch by lane number instead of elect.sync costs 0.05 more.
//
// Stages through tiles of 128 tokens whose weights were expanded into shared memory, and through this kernel, one launch after another in a
// graph, us, before the second stage's swapped column order (kOrderIn), which takes 5 to 10 % off it:
//   K -> rows            33 tokens       64              128             256             384
//   4096 -> 2016         9.8 -> 5.8      9.8 -> 7.0      10.9 -> 7.7     12.3 -> 9.7     15.1 -> 13
//   2944 -> 11008        15.9 -> 8.6     16.1 -> 9.3     18.2 -> 13.6    23.5 -> 19.6    31.4 -> 21.1
//   1024 -> 512          5.6 -> 3.5      5.6 -> 3.6      6.6 -> 3.7      6.6 -> 3.9      6.6 -> 4.0
//
#include <cuda.h>

#include <cstring>

#include "nq_common.cuh"
#include "nq_stage.h"
#include "nq_tcgen05.cuh"

namespace nq {

constexpr int kWThreads = 384;
constexpr int kWRows = 128;         // weight rows of a tile: MMA M, tensor-memory lanes
constexpr int kWMaxStages = 8, kWMaxSplit = 8;
constexpr int kWTmemCols = 256;
constexpr int kWExpandWarps = 8;

struct alignas(16) WJob {
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
    int chunks_per, tile0;
};
static_assert(sizeof(WJob) == 96, "six 16-byte words");
struct alignas(16) WHead {
    unsigned* status;      // (this and the wait limit are read from the parameters, not from the copy)
    int njobs;
    int T;
    int ntok, stages;      // tokens of a tile (a multiple of 16), pipeline stages of 128 columns
    int is_bf16, a_bf16, saturate, exp_sign;
    int order;             // kOrderOut, kOrderIn
    int csplit, owned;
    int off_recv, off_pre;
    unsigned wait_limit;
};
struct alignas(64) WParams {
    CUtensorMap map_a[kMaxGemmJobs];     // activations [T, K], box 64 x tokens of a tile, 128-byte swizzle
    WJob job[kMaxGemmJobs];
    WHead head;            // (the jobs and the head are copied to shared memory together)
};
constexpr int kWParamWords = (int)(sizeof(WJob) * kMaxGemmJobs + sizeof(WHead)) / 16;
// shared memory (from a 1024-byte boundary): descriptors, barriers, output scales and bias, B stages, received sums, input scales
constexpr int kWBarOff = 512, kWScaleOff = 1024, kWBOff = 2048;
static_assert(kWParamWords * 16 <= kWBarOff, "shared memory map");

__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_w(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld_frag2(uint32_t taddr, float (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld_frag8(uint32_t taddr, float (&r)[4][8]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=f"(r[0][0]), "=f"(r[0][1]), "=f"(r[0][2]), "=f"(r[0][3]), "=f"(r[0][4]), "=f"(r[0][5]), "=f"(r[0][6]), "=f"(r[0][7]),
                   "=f"(r[1][0]), "=f"(r[1][1]), "=f"(r[1][2]), "=f"(r[1][3]), "=f"(r[1][4]), "=f"(r[1][5]), "=f"(r[1][6]), "=f"(r[1][7]),
                   "=f"(r[2][0]), "=f"(r[2][1]), "=f"(r[2][2]), "=f"(r[2][3]), "=f"(r[2][4]), "=f"(r[2][5]), "=f"(r[2][6]), "=f"(r[2][7]),
                   "=f"(r[3][0]), "=f"(r[3][1]), "=f"(r[3][2]), "=f"(r[3][3]), "=f"(r[3][4]), "=f"(r[3][5]), "=f"(r[3][6]), "=f"(r[3][7])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
template <int OUT>
__global__ void __launch_bounds__(kWThreads, 2) wgemm_kernel(const __grid_constant__ WParams Pc) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // The launch's descriptors, copied to shared memory in one round trip (a first touch of a parameter line costs ~700 cycles)
    if (threadIdx.x < kWParamWords)
        reinterpret_cast<uint4*>(smem)[threadIdx.x] = reinterpret_cast<const uint4*>(&Pc.job[0])[threadIdx.x];
    const uint32_t bars = sbase + kWBarOff;
    auto bar_ready = [&](int s) { return bars + 8 * s; };
    auto bar_free = [&](int s) { return bars + 8 * (kWMaxStages + s); };
    const uint32_t bar_accum = bars + 8 * (2 * kWMaxStages), bar_pre = bar_accum + 8, bar_recv = bar_accum + 16;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kWBarOff + 8 * (2 * kWMaxStages) + 24);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kWBarOff + 8 * (2 * kWMaxStages) + 28);
    if (warp == 2) {
        if (lane < kWMaxStages) {
            mbar_init(bar_ready(lane), 1 + kWExpandWarps / 2);
            mbar_init(bar_free(lane), 1);
        }
        if (lane == 0) {
            mbar_init(bar_accum, 1);
            mbar_init(bar_pre, 1);
            mbar_init(bar_recv, 1);
            *abort_flag = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(const_cast<uint32_t*>(tmem_slot))), "r"((uint32_t)kWTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // only now: a CTA of the next kernel may take the SM's other half, and must not take tensor memory this one waits for
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const WHead& P = *reinterpret_cast<const WHead*>(smem + sizeof(WJob) * kMaxGemmJobs);
    const WJob* jobs = reinterpret_cast<const WJob*>(smem);
    int ji = 0;
    while (ji + 1 < P.njobs && (int)blockIdx.x >= jobs[ji + 1].tile0) ++ji;
    const WJob& J = jobs[ji];
    const int n0 = ((int)blockIdx.x - J.tile0) * kWRows;
    const int ntok = P.ntok, stages = P.stages, csplit = P.csplit;
    const int m0 = (int)blockIdx.y * ntok;
    const int c_begin = (int)blockIdx.z * J.chunks_per;
    const int c_end = min(J.chunks, c_begin + J.chunks_per);
    const int nks = min((J.K + 127) / 128, 2 * c_end) - 2 * c_begin;    // steps of 128 columns
    float* s_post = reinterpret_cast<float*>(smem + kWScaleOff);
    float* s_bias = s_post + kWRows;
    const uint32_t tmem_base = *tmem_slot;                    // the accumulator, then the A stages of 64 columns
    const uint32_t tmem_a = tmem_base + (uint32_t)((ntok + 31) & ~31);
    const uint32_t b_base = sbase + kWBOff, stage_bytes = (uint32_t)ntok * 256u;
    const int nblk = ntok >> 4, crank = csplit > 1 ? (int)blockIdx.z : 0;
    const int live = min(nblk, (P.T - m0 + 15) >> 4);         // blocks of 16 tokens that exist
    const int owned = P.owned;                                // blocks a CTA finishes, at most
    if (csplit > 1) {
        if (threadIdx.x == 96) {
            int mine = 0;
            for (int b = crank; b < live; b += csplit) ++mine;
            mbar_expect_tx(bar_recv, (uint32_t)(mine * (csplit - 1)) * 8192u);
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }

    bool ok = true;
    const int ew = warp - 4;
    const int rgl = 2 * (warp & 3) + (ew >> 2);               // row group of the tile this warp expands and finishes
    if (warp == 0) {
        const CUtensorMap* map = &Pc.map_a[ji];
        if (elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
        __syncwarp();
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int s = 0;
        uint32_t ph = 0;
        for (int ks = 0; ks < nks; ++ks) {
            if (!mbar_wait_warp(bar_free(s), ph ^ 1, abort_flag, Pc.head.status, Pc.head.wait_limit)) break;
            if (elect_one()) {
                const uint32_t dst = b_base + (uint32_t)s * stage_bytes;
                mbar_expect_tx(bar_ready(s), stage_bytes);
                tma_load_2d(dst, map, 256 * c_begin + 128 * ks, m0, bar_ready(s));
                tma_load_2d(dst + (stage_bytes >> 1), map, 256 * c_begin + 128 * ks + 64, m0, bar_ready(s));
            }
            if (++s == stages) { s = 0; ph ^= 1; }
        }
    } else if (warp == 1) {
        const uint32_t fmt = P.a_bf16 ? 1u : 0u;
        const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(ntok >> 3) << 17) | ((uint32_t)(kWRows >> 4) << 24);
        int s = 0;
        uint32_t ph = 0;
        bool good = true;
        for (int ks = 0; ks < nks; ++ks) {
            good = mbar_wait_warp(bar_ready(s), ph, abort_flag, Pc.head.status, Pc.head.wait_limit);
            if (!good) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t b_desc = umma_desc(b_base + (uint32_t)s * stage_bytes);
                const uint64_t half = (uint64_t)(stage_bytes >> 5);
                const uint32_t a = tmem_a + (uint32_t)(64 * s);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    umma_ts(tmem_base, a + 8 * k, b_desc + (k >> 2) * half + (uint64_t)(2 * (k & 3)), idesc, (ks | k) ? 1u : 0u);
                umma_commit_w(bar_free(s));
            }
            if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (good && elect_one()) umma_commit_w(bar_accum);
    } else if (warp == 2) {
        if (J.pre && nks > 0) {      // the input scales of this CTA's columns
            const int cols = min(J.K - 256 * c_begin, 128 * nks);
            if (elect_one()) {
                mbar_expect_tx(bar_pre, (uint32_t)cols * 2u);
                bulk_load(sbase + (uint32_t)P.off_pre, static_cast<const uint16_t*>(J.pre) + 256 * c_begin, (uint32_t)cols * 2u, bar_pre);
            }
        }
    } else if (warp >= 4) {
        const int q = lane & 3;
        // four warps per step (32 rows each), two groups of them on alternate steps: the group is the half of a chunk
        const int grp = ew >> 2, rg0 = (n0 >> 4) + 2 * (warp & 3);
        const bool there0 = rg0 < J.row_groups, there1 = rg0 + 1 < J.row_groups;
        const int chunks = J.chunks;
        const int src_lane = P.order == kOrderOut ? 4 * swap_middle(lane >> 2) + q : lane;
        const uint4* wt0 = J.tiles + ((size_t)(there0 ? rg0 : 0) * chunks + c_begin) * 32 + src_lane;
        const uint4* wt1 = J.tiles + ((size_t)(there1 ? rg0 + 1 : 0) * chunks + c_begin) * 32 + src_lane;
        uint4 w0n = make_uint4(0u, 0u, 0u, 0u), w1n = w0n, w0nn = w0n, w1nn = w0n;
        if (c_begin < c_end) {
            if (there0) w0n = __ldg(wt0);
            if (there1) w1n = __ldg(wt1);
        }
        if (c_begin + 1 < c_end) {
            if (there0) w0nn = __ldg(wt0 + 32);
            if (there1) w1nn = __ldg(wt1 + 32);
        }
        if (lane == 0 && c_begin + 2 < c_end && (grp ? there1 : there0))
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((grp ? wt1 : wt0) - src_lane + 64), "r"((uint32_t)(c_end - c_begin - 2) * 512u) : "memory");
        const int tu = (int)threadIdx.x - 128;
        uint16_t raw_post = 0, raw_bias = 0;
        if (tu < kWRows && n0 + tu < J.Nout) {
            if (J.post) asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(raw_post) : "l"(static_cast<const uint16_t*>(J.post) + n0 + tu));
            if (J.bias) asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(raw_bias) : "l"(static_cast<const uint16_t*>(J.bias) + n0 + tu));
        }
        const uint32_t one2 = P.a_bf16 ? 0x3F803F80u : 0x3C003C00u;
        const bool pre = J.pre != nullptr, in_order = P.order != kOrderIn;
        const uint2* s_pre = reinterpret_cast<const uint2*>(smem + P.off_pre) + q;
        const int K_left = J.K - 256 * c_begin;
        const uint32_t a_lane = tmem_a + ((uint32_t)(32 * (warp & 3)) << 16);
        if (pre && nks > 0) ok = mbar_wait_warp(bar_pre, 0, abort_flag, Pc.head.status, Pc.head.wait_limit);
        int s = grp;
        uint32_t ph = 0;
        const int pre_shift = grp ? 0 : 4;
        for (int ks = grp; ks < nks && ok; ks += 2) {
            uint4 w0 = w0n, w1 = w1n;
            w0n = w0nn; w1n = w1nn;
            wt0 += 32; wt1 += 32;
            if (ks - grp + 4 < nks) {
                if (there0) w0nn = __ldg(wt0 + 32);
                if (there1) w1nn = __ldg(wt1 + 32);
            }
            w0.x <<= pre_shift; w0.y <<= pre_shift; w0.z <<= pre_shift; w0.w <<= pre_shift;
            w1.x <<= pre_shift; w1.y <<= pre_shift; w1.z <<= pre_shift; w1.w <<= pre_shift;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {       // 64 columns
                uint2 pn[4];
                if (in_order) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) pn[i] = pre ? s_pre[(128 * ks + 64 * hf + 16 * i) >> 2] : make_uint2(one2, one2);
                    if (pre && 128 * ks + 64 * hf + 64 > K_left) {       // columns beyond K
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (128 * ks + 64 * hf + 16 * i + 4 * q >= K_left) pn[i] = make_uint2(0u, 0u);
                    }
                }
#pragma unroll
                for (int rr = 0; rr < 2; ++rr) {
                    const uint4& w = rr ? w1 : w0;
                    uint32_t v[16];
                    if (in_order) expand_columns(w, hf, pn, v);
                    else expand_swapped(w, hf, one2, v);
                    if (hf == 0 && rr == 0) {
                        ok = mbar_wait_warp(bar_free(s), ph ^ 1, abort_flag, Pc.head.status, Pc.head.wait_limit);
                        tc_fence_after();
                    }
                    tmem_st_frag4(a_lane + ((uint32_t)(16 * rr) << 16) + (uint32_t)(64 * s + 32 * hf), v);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive(bar_ready(s));
            s += 2;
            if (s >= stages) { s -= stages; ph ^= 1; }
        }
        if (tu < kWRows) {
            s_post[tu] = J.post ? io_float(raw_post, P.is_bf16) : 1.f;
            s_bias[tu] = J.bias ? io_float(raw_bias, P.is_bf16) : 0.f;
        }
        if (ok) ok = mbar_wait_warp(bar_accum, 0, abort_flag, Pc.head.status, Pc.head.wait_limit);
        tc_fence_after();
    }
    // ---------------------------------------------------------------- exchange of the partial sums
    const uint32_t d_lane = tmem_base + ((uint32_t)(16 * rgl) << 16);
    __syncwarp();
    if (csplit > 1) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every CTA of the cluster has started
        if (warp >= 4 && ok) {
            int owner = 0, idx = 0;
            for (int b0 = 0; b0 < live; b0 += 4) {
                float r[4][8];
                if (nks > 0) tmem_ld_frag8(d_lane + (uint32_t)(16 * b0), r);
                else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int e = 0; e < 8; ++e) r[i][e] = 0.f;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (b0 + i < live && owner != crank) {
                        const int src = crank < owner ? crank : crank - 1;
                        const uint32_t slot = sbase + (uint32_t)(P.off_recv + (src * owned + idx) * 8192 + rgl * 1024 + lane * 16);
                        const uint32_t dst = cluster_map(slot, (uint32_t)owner);
                        const uint32_t bar = cluster_map(bar_recv, (uint32_t)owner);
                        cluster_store4_tx(dst, bar, __float_as_uint(r[i][0]), __float_as_uint(r[i][1]), __float_as_uint(r[i][2]), __float_as_uint(r[i][3]));
                        cluster_store4_tx(dst + 512, bar, __float_as_uint(r[i][4]), __float_as_uint(r[i][5]), __float_as_uint(r[i][6]), __float_as_uint(r[i][7]));
                    }
                    if (++owner == csplit) { owner = 0; ++idx; }
                }
            }
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    }
    if (warp >= 4) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("bar.sync 2, 256;" ::: "memory");        // scales visible
        const int g = lane >> 2, q = lane & 3;
        if (ok) {
            const int r0 = 16 * rgl + g, rs = 16 * rgl + (P.order == kOrderOut ? swap_middle(g) : g);
            const float sc0 = s_post[rs], sc1 = s_post[rs + 8], bi0 = s_bias[rs], bi1 = s_bias[rs + 8];
            const uint16_t* resid = static_cast<const uint16_t*>(J.resid);
            int idx = 0;
            for (int b = crank; b < live; b += csplit, ++idx) {
                const int t0 = m0 + 16 * b;
                float r[8];
                if (nks > 0) tmem_ld_frag2(d_lane + (uint32_t)(16 * b), r);
                else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) r[e] = 0.f;
                }
                if (csplit > 1 && b == crank) {
                    ok = mbar_wait_warp<true>(bar_recv, 0, abort_flag, Pc.head.status, Pc.head.wait_limit);
                    if (!ok) break;      // (all 256 threads still pass the barrier below)
                }
                for (int rk = 0; rk < csplit - 1; ++rk) {
                    const unsigned char* src = smem + P.off_recv + (rk * owned + idx) * 8192 + rgl * 1024 + lane * 16;
                    const float4 a = *reinterpret_cast<const float4*>(src), c = *reinterpret_cast<const float4*>(src + 512);
                    r[0] += a.x; r[1] += a.y; r[2] += a.z; r[3] += a.w;
                    r[4] += c.x; r[5] += c.y; r[6] += c.z; r[7] += c.w;
                }
                float ts[4] = {1.f, 1.f, 1.f, 1.f};
                if (J.row_exp) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int tok = t0 + 8 * (e >> 1) + 2 * q + (e & 1);
                        if (tok < P.T) ts[e] = exp2f((float)(P.exp_sign * J.row_exp[tok]));
                    }
                }
                // r[4 h + 2 hi + e]: token 8 h + 2 q + e, row g + 8 hi
                float o[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int e = 2 * (i >> 2) + (i & 1);
                    float add = (i & 2) ? bi1 : bi0;
                    if (resid) {
                        const int tok = t0 + 8 * (i >> 2) + 2 * q + (i & 1), row = n0 + r0 + ((i & 2) ? 8 : 0);
                        if (tok < P.T && row < J.Nout) {
                            add += io_float(resid[(size_t)tok * J.ld_res + row], P.is_bf16);
                        }
                    }
                    o[i] = r[i] * (((i & 2) ? sc1 : sc0) * ts[e]) + add;
                }
                uint32_t pk[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) pk[i] = pack_outputs<OUT>(o[2 * i], o[2 * i + 1], P.saturate);
                // matrix i of the transposing store: tokens 8 (i >> 1) .., rows 8 (i & 1) ..
                const int mi = lane >> 3, tl = 16 * idx + 8 * (mi >> 1) + (lane & 7), unit = 2 * rgl + (mi & 1);
                const uint32_t addr = b_base + (uint32_t)(tl * 256 + ((unit ^ (tl & 7)) << 4));
                stmatrix_trans(addr, pk);
            }
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        if (ok) {
            const int tu = (int)threadIdx.x - 128, unit = tu & 15, tr = tu >> 4;
            const int row = n0 + 8 * unit;
            if (row < J.Nout) {
                uint16_t* out = static_cast<uint16_t*>(J.out) + row;
                int tl = tr;
                for (int b = crank; b < live; b += csplit, tl += 16) {
                    const int tok = m0 + 16 * b + tr;
                    if (tok >= P.T) break;
                    const uint4 v = *reinterpret_cast<const uint4*>(smem + kWBOff + tl * 256 + ((unit ^ (tl & 7)) << 4));
                    uint16_t* dst = out + (size_t)tok * J.ld_out;
                    store_rows(dst, v, J.Nout - row, row + 8 <= J.Nout && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0);
                }
            }
        }
    }
    if (*abort_flag && threadIdx.x == 0) {
        for (unsigned i = 0; i < (1u << 20); ++i) __nanosleep(64);
    }
    tc_fence_before();
    __syncthreads();
    if (csplit > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kWTmemCols) : "memory");
    }
}

static const void* w_kernel(int out) {
    return out == kOutFp16 ? (const void*)wgemm_kernel<kOutFp16> : out == kOutBf16 ? (const void*)wgemm_kernel<kOutBf16>
                                                                                     : (const void*)wgemm_kernel<kOutBf16Saturated>;
}

constexpr int kWSmemMost = 112 * 1024;   // two CTAs per SM

// Shared memory of a plan; false if it does not fit half an SM.
static bool w_layout(int ntok, int csplit, int pre_bytes, WgemmPlan& p) {
    const int owned = (ntok / 16 + csplit - 1) / csplit;
    const int recv = (csplit - 1) * owned * 8192;
    p.ntok = ntok; p.csplit = csplit; p.owned = owned;
    int st = (kWTmemCols - (ntok + 31) / 32 * 32) / 64;
    if (st > kWMaxStages) st = kWMaxStages;
    while (st > 0 && 1024 + kWBOff + st * ntok * 256 + recv + pre_bytes > kWSmemMost) --st;
    if (st < 2 || owned * 4096 > st * ntok * 256) return false;
    p.stages = st;
    p.off_recv = kWBOff + st * ntok * 256;
    p.off_pre = p.off_recv + recv;
    p.smem = 1024 + p.off_pre + pre_bytes;
    if (p.smem < 78 * 1024) p.smem = 78 * 1024;   // never a third CTA: its tensor memory would not fit
    return true;
}

static int w_attributes() {
    static bool done[64];
    int dev = 0;
    NQ_CUDA_TRY(cudaGetDevice(&dev));
    if (!done[dev & 63]) {
        for (int o = 0; o < 3; ++o) {
            NQ_CUDA_TRY(cudaFuncSetAttribute(w_kernel(o), cudaFuncAttributeMaxDynamicSharedMemorySize, kWSmemMost));
            // (by default the driver makes room for one CTA's shared memory)
            NQ_CUDA_TRY(cudaFuncSetAttribute(w_kernel(o), cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        }
        done[dev & 63] = true;
    }
    return NQ_OK;
}

// CTAs that can be resident at once when they are launched as clusters of `s` (clusters are placed inside one GPC, so this
// is less than two per SM for most sizes); 0: this size cannot be launched.
static int w_capacity(int s) {
    static int cached[kWMaxSplit + 1];
    int& c = cached[s];
    if (c == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, 1, s);
        cfg.blockDim = dim3(kWThreads);
        cfg.dynamicSmemBytes = kWSmemMost;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 1; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = (unsigned)s;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (w_attributes() != NQ_OK || cudaOccupancyMaxActiveClusters(&clusters, w_kernel(kOutFp16), &cfg) != cudaSuccess || clusters <= 0) {
            (void)cudaGetLastError();
            clusters = 0;
        }
        c = clusters > 0 ? 2 * clusters * s : -1;     // (the query counts one CTA per SM)
    }
    return c > 0 ? c : 0;
}

// Tokens of a tile and k split by a cost in microseconds, fitted to 3200 measured launches (14 shapes of 512..28672 rows and
// 608..11008 columns, 33 to 384 tokens, 1 to 8 CTAs per cluster, all tile widths): the plan it picks is 1.3 % above the best on
// average.  A CTA's steps cost less while it has its SM for itself (`one`) than when two share it (`two`); up to 56 tokens the
// expansion hides the MMA; every CTA more is contention; clusters above four exchange more and fit less well.
bool plan_wgemm(const StageJob* jobs, int n, int T, int order, WgemmPlan& best) {
    int most_chunks = 0, most_pre = 0;
    for (int j = 0; j < n; ++j) {
        const int c = (jobs[j].K + 255) / 256;
        most_chunks = c > most_chunks ? c : most_chunks;
        if (jobs[j].pre && c > most_pre) most_pre = c;
    }
    int rows = 0;
    for (int j = 0; j < n; ++j) rows += (jobs[j].Nout + kWRows - 1) / kWRows;
    const int all = (T + 15) / 16 * 16;
    static const int sizes[] = {16, 32, 48, 64, 80, 96, 112, 128};
    bool found = false;
    const int sms = sm_count();
    for (int ntok : sizes) {
        if (ntok > all || (ntok < 32 && ntok < all)) continue;
        const int tiles = rows * ((T + ntok - 1) / ntok);
        for (int s = 1; s <= kWMaxSplit && s <= most_chunks; ++s) {
            WgemmPlan p;
            if (!w_layout(ntok, s, (most_pre + s - 1) / s * 512, p)) continue;
            const int resident = w_capacity(s);
            if (resident <= 0) continue;
            const int steps = 2 * ((most_chunks + s - 1) / s), ctas = tiles * s;
            const float over = ntok > 56 ? ntok - 56.f : 0.f;
            const float one = 0.38f + 0.002f * over, two = 0.46f + 0.0024f * over;
            const int full = ctas / resident, rest = ctas % resident;
            float t = 0.5f + 0.03f * ntok + 2.2f * ctas / sms + (ctas > sms ? -0.7f : 0.f) + (s > 1 ? -0.18f + 0.01f * s + (s > 4 ? 0.22f * (s - 4) : 0.f) : 0.f);
            t += (order == kOrderIn ? 0.82f : most_pre ? 1.14f : 1.f) * steps * (full * (resident > sms ? two : one) + (rest == 0 ? 0.f : rest > sms ? two : one));
            if (!found || t < best.us) { best = p; best.us = t; found = true; }
        }
    }
    return found;
}

int launch_wgemm_stage(const StageJob* jobs, int n, int T, StageTypes ty, int saturate, const WgemmPlan& pl, unsigned* status,
                       cudaStream_t stream) {
    { const int st = w_attributes(); if (st != NQ_OK) return st; }
    WParams P;
    memset(&P, 0, sizeof(P));
    WHead& H = P.head;
    H.njobs = n; H.status = status; H.wait_limit = gemm_wait_limit(); H.T = T; H.ntok = pl.ntok; H.stages = pl.stages; H.csplit = pl.csplit;
    H.owned = pl.owned; H.off_recv = pl.off_recv; H.off_pre = pl.off_pre;
    H.is_bf16 = ty.io_bf16; H.a_bf16 = ty.a_bf16; H.saturate = saturate; H.exp_sign = ty.exp_sign; H.order = ty.order;
    int tiles = 0;
    for (int j = 0; j < n; ++j) {
        const StageJob& S = jobs[j];
        WJob& J = P.job[j];
        const int st = encode_activations(&P.map_a[j], S, ty.a_bf16, T, pl.ntok);
        if (st != NQ_OK) return st;
        J.tiles = static_cast<const uint4*>(S.tiles);
        J.pre = S.pre; J.post = S.post; J.out = S.out; J.ld_out = S.ld_out;
        J.row_exp = ty.exp_sign ? S.row_exp : nullptr;
        J.bias = S.bias; J.resid = S.resid; J.ld_res = S.ld_res;
        J.K = S.K; J.Nout = S.Nout;
        J.chunks = (S.K + 255) / 256;
        J.row_groups = (S.Nout + 15) / 16;
        J.chunks_per = (J.chunks + pl.csplit - 1) / pl.csplit;
        J.tile0 = tiles;
        tiles += (S.Nout + kWRows - 1) / kWRows;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles, (T + pl.ntok - 1) / pl.ntok, pl.csplit);
    cfg.blockDim = dim3(kWThreads);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    int na = 0;
    if (pl.csplit > 1) {
        attrs[na].id = cudaLaunchAttributeClusterDimension;
        attrs[na].val.clusterDim.x = 1; attrs[na].val.clusterDim.y = 1; attrs[na].val.clusterDim.z = (unsigned)pl.csplit;
        ++na;
    }
    void* args[] = {&P};
    return launch_dependent(cfg, attrs, na, w_kernel(out_kind(ty, saturate)), args);
}

}  // namespace nq
