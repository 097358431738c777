// Prefill GEMM of the binary low-rank linear, host side:
//
//   stage 1:  t[T, R] = ((x * s_in) . V^T) * s_mid        (t kept in the I/O dtype by default)
//   stage 2:  y[T, M] = (t . U^T) * s_out
//
// Each stage is one launch, Out[T, Nout] = (A[T, K] . W[Nout, K]^T) * post for up to four linears, of the kernel that costs
// least: 5 to 16 tokens nq_batch.cu, then nq_wgemm.cu (K split over clusters, two CTAs per SM) or nq_pgemm.cu (pairs of CTAs with
// several tiles each), whose planners predict a launch's time.  The packed operand is the same tile layout the decode GEMV
// streams (nq_rows_to_tiles), so a layer keeps one copy of its weights for all of them.
//
// bf16 linears may keep their intermediate as fp16 times a per-token power of two (row_bound_kernel,
// nq_gemm_set_precise_intermediate).
//
// replaces: src/nanoquant/kernel/cuda/gemm_kernel.cu:278-791 (Marlin-derived mma.sync
// kernel with register-level dequantisation) and src/nanoquant/kernel/cuda/gemm.cpp:59-122
// of the reference.
#include <cuda.h>

#include <cstring>

#include "nq_common.cuh"
#include "nq_stage.h"

namespace nq {

// ---------------------------------------------------------------------------
// Per-token exponents of a bf16 linear's intermediate.  |t[tok, r]| <= max|s_mid| * sum_k |s_in[k] * x[tok, k]| =: B,
// so t * 2^e with B * 2^e <= 2^14 fits fp16 for every r, whatever the signs in V are; typical elements sit
// sqrt(K) below the bound, far above fp16's subnormal range.  One CTA per eight tokens, up to four linears (grid.y).
// ---------------------------------------------------------------------------
struct BoundJob {
    const uint16_t* x;      // [T, ldx] bf16
    long long ldx;
    const uint16_t* s_in;   // [K] bf16
    const uint16_t* s_mid;  // [R] bf16 or nullptr (ones)
    int* row_exp;           // [T]
    int K, R;
};
struct BoundParams {
    BoundJob job[kMaxGemmJobs];
    int T;
};

__global__ void __launch_bounds__(256) row_bound_kernel(const __grid_constant__ BoundParams P) {
    const BoundJob& J = P.job[blockIdx.y];
    __shared__ float s_red[8][9];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    auto bf = [](uint16_t h) { return __uint_as_float((uint32_t)h << 16); };
    // the layer's constants first (they do not depend on the previous kernel)
    float m = J.s_mid ? 0.f : 1.f;
    if (J.s_mid)
        for (int r = threadIdx.x; r < J.R; r += 256) m = fmaxf(m, fabsf(bf(J.s_mid[r])));
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the activations come from the previous kernel
    // every thread takes 8-column pieces of all eight tokens of the CTA: the loads of a round are independent,
    // so a row costs one memory round trip, not one per piece
    const int tok0 = blockIdx.x * 8;
    float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const bool vec = (reinterpret_cast<uintptr_t>(J.x) & 15u) == 0 && (J.ldx % 8) == 0 &&
                     (reinterpret_cast<uintptr_t>(J.s_in) & 15u) == 0;
    const int kvec = vec ? (J.K & ~7) : 0;
    for (int k = threadIdx.x * 8; k < kvec; k += 2048) {
        const uint4 b = *reinterpret_cast<const uint4*>(J.s_in + k);
        uint4 a[8];
#pragma unroll
        for (int t = 0; t < 8; ++t)
            a[t] = tok0 + t < P.T ? *reinterpret_cast<const uint4*>(J.x + (size_t)(tok0 + t) * J.ldx + k) : make_uint4(0, 0, 0, 0);
        const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const uint32_t aw[4] = {a[t].x, a[t].y, a[t].z, a[t].w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                sum[t] += fabsf(__uint_as_float(aw[i] << 16) * __uint_as_float(bw[i] << 16)) +
                          fabsf(__uint_as_float(aw[i] & 0xFFFF0000u) * __uint_as_float(bw[i] & 0xFFFF0000u));
        }
    }
    for (int k = kvec + threadIdx.x; k < J.K; k += 256) {
        const float sk = bf(J.s_in[k]);
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (tok0 + t < P.T) sum[t] += fabsf(bf(J.x[(size_t)(tok0 + t) * J.ldx + k]) * sk);
    }
#pragma unroll
    for (int t = 0; t < 8; ++t)
        for (int o = 16; o; o >>= 1) sum[t] += __shfl_xor_sync(0xffffffffu, sum[t], o);
    if (lane == 0) {
#pragma unroll
        for (int t = 0; t < 8; ++t) s_red[warp][t] = sum[t];
        s_red[warp][8] = m;
    }
    __syncthreads();
    if (threadIdx.x < 8 && tok0 + (int)threadIdx.x < P.T) {
        float total = 0.f, mm = 0.f;
        for (int w = 0; w < 8; ++w) { total += s_red[w][threadIdx.x]; mm = fmaxf(mm, s_red[w][8]); }
        const float bound = total * mm * 1.0001f;   // (rounding of the sum itself)
        int e = 0;
        if (bound > 0.f && bound < 3.0e38f) {
            int q;
            (void)frexpf(bound, &q);                // bound = f * 2^q, 0.5 <= f < 1
            e = 14 - q;
            e = e > 100 ? 100 : (e < -100 ? -100 : e);
        }
        J.row_exp[tok0 + threadIdx.x] = e;
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup: no link against libcuda.
static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

int encode_activations(CUtensorMap* map, const StageJob& S, int bf16, int T, int box_rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return NQ_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)S.K, (cuuint64_t)T};
    const cuuint64_t strides[1] = {(cuuint64_t)S.lda * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                           2, const_cast<void*>(S.a), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? NQ_OK : NQ_ERR_UNSUPPORTED;
}

// The kernel of a stage, with its plan.  (An intermediate in the GEMMs' column order is theirs.)
static int pick_kernel(const StageJob* jobs, int n, int T, int order, WgemmPlan& w, PgemmPlan& p) {
    if (order == 0 && T <= batch_max_tokens(jobs, n)) return NQ_KERNEL_BATCH;
    p = plan_pgemm(jobs, n, T, order);
    return plan_wgemm(jobs, n, T, order, w) && w.us <= p.us ? NQ_KERNEL_WGEMM : NQ_KERNEL_PGEMM;
}
// Both stages of a group by the batch kernel, which keeps the intermediate in its own order.
static bool both_batch(const StageJob* s1, const StageJob* s2, int n, int T) {
    return T <= batch_max_tokens(s1, n) && T <= batch_max_tokens(s2, n);
}

// One stage of up to four linears: out_j[T, Nout_j] = (a_j[T, K_j] . W_j^T) * post_j.
static int launch_stage(const StageJob* jobs, int n, int T, StageTypes ty, int saturate, unsigned* status, cudaStream_t stream) {
    if (n < 1 || n > kMaxGemmJobs) return NQ_ERR_UNSUPPORTED;
    for (int j = 0; j < n; ++j) {
        const StageJob& S = jobs[j];
        if (!aligned16(S.a) || (S.lda % 8) != 0 || (S.K % 8) != 0) return NQ_ERR_ALIGN;   // TMA: 16-byte base and stride
        if (S.pre && !aligned16(S.pre)) return NQ_ERR_ALIGN;
    }
    WgemmPlan w;
    PgemmPlan p;
    switch (pick_kernel(jobs, n, T, ty.order, w, p)) {
        case NQ_KERNEL_BATCH: return launch_batch_stage(jobs, n, T, ty, saturate, false, false, false, status, stream);
        case NQ_KERNEL_WGEMM: return launch_wgemm_stage(jobs, n, T, ty, saturate, w, status, stream);
        default: return launch_pgemm_stage(jobs, n, T, ty, saturate, p, status, stream);
    }
}

constexpr unsigned kGemmWaitLimit = 1u << 21;      // seconds
static unsigned g_gemm_wait_limit = kGemmWaitLimit;
unsigned gemm_wait_limit() { return g_gemm_wait_limit; }

static int g_precise_intermediate = 0;   // see nq_gemm_set_precise_intermediate

}  // namespace nq

using namespace nq;

extern "C" {

// Scratch of a GEMM group: header (status word), the intermediates t_j[T, R_j] (16-bit, 256-byte aligned each; in the
// batch kernel's order for few tokens), the per-token exponents of each intermediate (T words each; used by bf16 linears).
static size_t gemm_group_layout(const nq_linear_desc* d, int n, int T, size_t* t_off, size_t* exp_off) {
    size_t off = 256;
    for (int j = 0; j < n; ++j) {
        if (t_off) t_off[j] = off;
        size_t t_bytes = (size_t)T * (size_t)d[j].R * 2;
        if (T <= kBatchMostTokens && batch_fragment_bytes(T, d[j].R) > t_bytes) t_bytes = batch_fragment_bytes(T, d[j].R);
        off += (t_bytes + 255) / 256 * 256;
    }
    for (int j = 0; j < n; ++j) {
        if (exp_off) exp_off[j] = off;
        off += ((size_t)T * sizeof(int) + 255) / 256 * 256;
    }
    return off;
}

size_t nq_gemm_group_scratch_bytes(const nq_linear_desc* d, int n_linears, int T) {
    if (!d || n_linears <= 0 || n_linears > kMaxGemmJobs || T <= 0) return 0;
    for (int j = 0; j < n_linears; ++j)
        if (d[j].N <= 0 || d[j].R <= 0 || d[j].M <= 0) return 0;
    return gemm_group_layout(d, n_linears, T, nullptr, nullptr);
}

size_t nq_gemm_scratch_bytes(int T, int N, int R, int M) {
    if (T <= 0 || N <= 0 || R <= 0 || M <= 0) return 0;
    nq_linear_desc d;
    memset(&d, 0, sizeof(d));
    d.N = N; d.R = R; d.M = M;
    return gemm_group_layout(&d, 1, T, nullptr, nullptr);
}

int nq_onebit_gemm_fwd(const void* x, const void* tiles, const void* s_in, const void* s_out, void* y,
                       void* status_word, int T, int K, int Nout, int dtype, nq_stream_t stream) {
    if (!x || !tiles || !y || !status_word) return NQ_ERR_NULL;
    if (T <= 0 || K <= 0 || Nout <= 0) return NQ_ERR_SHAPE;
    if (dtype != NQ_F16 && dtype != NQ_BF16) return NQ_ERR_DTYPE;
    if (!aligned16(tiles)) return NQ_ERR_ALIGN;
    const StageJob job = {x, K, tiles, s_in, s_out, y, Nout, K, Nout, nullptr, nullptr, 0, nullptr};
    const int b16 = dtype == NQ_BF16;
    return launch_stage(&job, 1, T, StageTypes{b16, b16, b16, 0}, 1, static_cast<unsigned*>(status_word) + 2, as_stream(stream));
}

int nq_gemm_group_fwd(const nq_linear_desc* d, int n_linears, int T, int dtype, void* scratch,
                      size_t scratch_bytes, nq_stream_t stream) {
    if (!d || !scratch) return NQ_ERR_NULL;
    if (n_linears <= 0 || n_linears > kMaxGemmJobs) return NQ_ERR_UNSUPPORTED;
    if (T <= 0) return NQ_ERR_SHAPE;
    if (dtype != NQ_F16 && dtype != NQ_BF16) return NQ_ERR_DTYPE;
    if (!aligned16(scratch)) return NQ_ERR_ALIGN;
    for (int j = 0; j < n_linears; ++j) {
        const nq_linear_desc& L = d[j];
        if (!L.x || !L.s_in || !L.v_tiles || !L.u_tiles || !L.s_out || !L.y) return NQ_ERR_NULL;
        if (L.N <= 0 || L.R <= 0 || L.M <= 0 || L.ldx < L.N || L.ldy < L.M) return NQ_ERR_SHAPE;
        if (L.residual && L.ldr < L.M) return NQ_ERR_SHAPE;
        if (L.N % 8 || L.R % 8) return NQ_ERR_SHAPE;
        if (!aligned16(L.v_tiles) || !aligned16(L.u_tiles)) return NQ_ERR_ALIGN;
    }
    size_t t_off[kMaxGemmJobs], exp_off[kMaxGemmJobs];
    if (scratch_bytes < gemm_group_layout(d, n_linears, T, t_off, exp_off)) return NQ_ERR_SCRATCH;
    unsigned* status = static_cast<unsigned*>(scratch) + 2;   // same word as the GEMV header's status
    StageJob s1[kMaxGemmJobs], s2[kMaxGemmJobs];
    for (int j = 0; j < n_linears; ++j) {
        const nq_linear_desc& L = d[j];
        void* t = static_cast<char*>(scratch) + t_off[j];
        int* row_exp = reinterpret_cast<int*>(static_cast<char*>(scratch) + exp_off[j]);
        s1[j] = {L.x, L.ldx, L.v_tiles, L.s_in, L.s_mid, t, L.R, L.N, L.R, nullptr, nullptr, 0, row_exp};
        s2[j] = {t, L.R, L.u_tiles, nullptr, L.s_out, L.y, L.ldy, L.R, L.M, L.bias, L.residual, L.ldr, row_exp};
    }
    const bool batch = both_batch(s1, s2, n_linears, T);
    auto stages = [&](StageTypes ty1, StageTypes ty2) -> int {
        if (batch) {
            const int st = launch_batch_stage(s1, n_linears, T, ty1, 0, false, true, false, status, as_stream(stream));
            return st != NQ_OK ? st : launch_batch_stage(s2, n_linears, T, ty2, 1, true, false, false, status, as_stream(stream));
        }
        ty1.order = kOrderOut;
        ty2.order = kOrderIn;
        const int st = launch_stage(s1, n_linears, T, ty1, 0, status, as_stream(stream));
        return st != NQ_OK ? st : launch_stage(s2, n_linears, T, ty2, 1, status, as_stream(stream));
    };
    if (dtype == NQ_F16 || !g_precise_intermediate) {   // the intermediate in the I/O type, as it comes
        const int b16 = dtype == NQ_BF16;
        const StageTypes ty = {b16, b16, b16, 0};
        return stages(ty, ty);
    }
    // bf16 with the precise intermediate switched on: a bf16 intermediate carries 8 significant bits into stage 2
    // (its rounding alone is up to 1.6e-3 of the output's maximum); here it is kept as fp16 times a per-token
    // power of two instead.  row_bound_kernel finds the exponents from a bound on |t| that holds for any signs;
    // stage 2 then runs as an fp16 MMA on +-1 weights.  One more small kernel per launch group.
    {
        BoundParams B;
        memset(&B, 0, sizeof(B));
        B.T = T;
        for (int j = 0; j < n_linears; ++j) {
            const nq_linear_desc& L = d[j];
            B.job[j] = {static_cast<const uint16_t*>(L.x), L.ldx, static_cast<const uint16_t*>(L.s_in),
                        static_cast<const uint16_t*>(L.s_mid), const_cast<int*>(s1[j].row_exp), L.N, L.R};
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)((T + 7) / 8), (unsigned)n_linears);
        cfg.blockDim = dim3(256);
        cfg.stream = as_stream(stream);
        cudaLaunchAttribute attr[1];
        void* args[] = {&B};
        const int st = launch_dependent(cfg, attr, 0, (const void*)row_bound_kernel, args);
        if (st != NQ_OK) return st;
    }
    return stages(StageTypes{1, 1, 0, +1}, StageTypes{1, 0, 1, -1});
}

int nq_gemm_group_kernels(const nq_linear_desc* d, int n_linears, int T, int* kernels) {
    if (!d || !kernels) return NQ_ERR_NULL;
    if (n_linears <= 0 || n_linears > kMaxGemmJobs) return NQ_ERR_UNSUPPORTED;
    if (T <= 0) return NQ_ERR_SHAPE;
    StageJob s1[kMaxGemmJobs] = {}, s2[kMaxGemmJobs] = {};
    for (int j = 0; j < n_linears; ++j) {
        if (d[j].N <= 0 || d[j].R <= 0 || d[j].M <= 0 || d[j].N % 8 || d[j].R % 8) return NQ_ERR_SHAPE;
        s1[j].K = d[j].N; s1[j].Nout = s2[j].K = d[j].R; s2[j].Nout = d[j].M;
        s1[j].pre = d;      // (not read: a first stage has input scales)
    }
    WgemmPlan w;
    PgemmPlan p;
    const bool batch = both_batch(s1, s2, n_linears, T);
    kernels[0] = batch ? (int)NQ_KERNEL_BATCH : pick_kernel(s1, n_linears, T, kOrderOut, w, p);
    kernels[1] = batch ? (int)NQ_KERNEL_BATCH : pick_kernel(s2, n_linears, T, kOrderIn, w, p);
    return NQ_OK;
}

int nq_gemm_fwd(const void* x, const void* s_in, const void* v_tiles, const void* s_mid, const void* u_tiles,
                const void* s_out, void* y, void* scratch, size_t scratch_bytes, int T, int N, int R, int M,
                int dtype, nq_stream_t stream) {
    if (!x || !s_in || !v_tiles || !u_tiles || !s_out || !y || !scratch) return NQ_ERR_NULL;
    if (T <= 0 || N <= 0 || R <= 0 || M <= 0) return NQ_ERR_SHAPE;
    nq_linear_desc d;
    memset(&d, 0, sizeof(d));
    d.x = x; d.s_in = s_in; d.v_tiles = v_tiles; d.s_mid = s_mid; d.u_tiles = u_tiles; d.s_out = s_out;
    d.y = y; d.N = N; d.R = R; d.M = M; d.ldx = N; d.ldy = M;
    return nq_gemm_group_fwd(&d, 1, T, dtype, scratch, scratch_bytes, stream);
}


int nq_gemm_set_precise_intermediate(int on) {
    const int old = g_precise_intermediate;
    g_precise_intermediate = on ? 1 : 0;
    return old;
}

unsigned nq_gemm_set_wait_limit(unsigned attempts) {
    const unsigned old = g_gemm_wait_limit;
    g_gemm_wait_limit = attempts ? attempts : kGemmWaitLimit;
    return old;
}

// The decode path takes up to four tokens (the largest groups of four by the batch kernel, see nq_decode_group_fwd); from five
// on the batch kernel's two stages are faster than two decode launches, and keep the intermediate in the I/O type.
int nq_gemv_max_tokens(void) { return 4; }

size_t nq_linear_scratch_bytes(int T, int N, int R, int M) {
    const size_t a = nq_gemv_scratch_bytes(T, N, R, M), b = nq_gemm_scratch_bytes(T, N, R, M);
    return a > b ? a : b;
}

int nq_linear_fwd(const void* x, const void* s_in, const void* v_tiles, const void* s_mid, const void* u_tiles,
                  const void* s_out, void* y, void* scratch, size_t scratch_bytes, int T, int N, int R, int M,
                  int dtype, nq_stream_t stream) {
    if (T <= nq_gemv_max_tokens() || (N % 8) || (R % 8)) {
        nq_linear_desc d;
        memset(&d, 0, sizeof(d));
        d.x = x; d.s_in = s_in; d.v_tiles = v_tiles; d.s_mid = s_mid; d.u_tiles = u_tiles; d.s_out = s_out; d.y = y;
        d.N = N; d.R = R; d.M = M; d.ldx = N; d.ldy = M;
        return nq_decode_group_fwd(&d, 1, T, dtype, scratch, scratch_bytes, stream);
    }
    return nq_gemm_fwd(x, s_in, v_tiles, s_mid, u_tiles, s_out, y, scratch, scratch_bytes, T, N, R, M, dtype, stream);
}

}  // extern "C"
