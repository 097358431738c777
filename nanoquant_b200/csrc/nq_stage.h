// One stage of a launch group as the host sees it: Out_j[T, Nout_j] = (A_j[T, K_j] . W_j^T) * post_j for up to four
// linears.  Implemented by the tensor-core GEMMs (nq_wgemm.cu, nq_pgemm.cu) and, for few tokens, by the batch kernel (nq_batch.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

namespace nq {

constexpr int kMaxGemmJobs = 4;

struct StageJob {
    const void* a;          // activations [T, K], row stride lda elements; 16-byte aligned rows, K a multiple of 8
    long long lda;
    const void* tiles;
    const void* pre;        // [K] input scales or nullptr (ones)
    const void* post;       // [Nout] output scales or nullptr
    void* out;
    long long ld_out;
    int K, Nout;
    const void* bias;       // [Nout] or nullptr
    const void* resid;      // [T, ld_res] or nullptr
    long long ld_res;
    const int* row_exp;     // [T] per-token exponents of the intermediate or nullptr
};
// Types of a stage: scales / bias / residual, MMA operands, output; sign of the row exponents (0: none).
struct StageTypes {
    int io_bf16, a_bf16, out_bf16, exp_sign;
    int order = 0;          // kOrderOut, kOrderIn
};
// The intermediate between two stages of nq_wgemm.cu or nq_pgemm.cu has the middle two of every four columns swapped, which costs the
// first stage nothing (its MMA rows may have any order) and halves the expansion of the second.
enum : int { kOrderOut = 1, kOrderIn = 2 };

constexpr int kBatchMostTokens = 16;    // of the batch kernel: its two column groups (beyond, nq_wgemm.cu is faster; figures in nq_batch.cu)
// The same, or 0 where it cannot take the jobs.
int batch_max_tokens(const StageJob* jobs, int n);
// `frag_in` / `frag_out`: the activations / the output are an intermediate in the batch kernel's fragment order, of
// batch_fragment_bytes each, without an input scale.
size_t batch_fragment_bytes(int T, int K);
// `split` (with a fragment-order side, kSplitTokens tokens): the intermediate is bf16 twice, value and remainder, as the
// columns t and 4 + t of eight; 16 significant bits at fp32's range.  A linear's results are then the same bits in any group.
constexpr int kSplitTokens = 4;
int launch_batch_stage(const StageJob* jobs, int n, int T, StageTypes ty, int saturate, bool frag_in, bool frag_out, bool split,
                       unsigned* status, cudaStream_t stream);

// Tensor map of a stage's activations: boxes of 64 columns x `box_rows` tokens, 128-byte swizzle.
int encode_activations(CUtensorMap* map, const StageJob& S, int bf16, int T, int box_rows);

// Attempts (of some 4 us each) that a wait inside the GEMMs may spend before it gives up (nq_gemm_set_wait_limit).
unsigned gemm_wait_limit();

// GEMMs with the weights on the row side of the MMA; `us` is the predicted time of the launch.
// nq_wgemm.cu: tiles of 128 rows, K split over a cluster, two CTAs per SM.  False: no plan (input scales of too many columns).
struct WgemmPlan {
    float us;
    int ntok, stages, csplit, owned, off_recv, off_pre, smem;
};
bool plan_wgemm(const StageJob* jobs, int n, int T, int order, WgemmPlan& plan);
int launch_wgemm_stage(const StageJob* jobs, int n, int T, StageTypes ty, int saturate, const WgemmPlan& plan, unsigned* status,
                       cudaStream_t stream);
// nq_pgemm.cu: tiles of 256 rows by pairs of CTAs, several tiles each.  Takes everything.
struct PgemmPlan {
    float us;
    int ntok, accs;
};
PgemmPlan plan_pgemm(const StageJob* jobs, int n, int T, int order);
int launch_pgemm_stage(const StageJob* jobs, int n, int T, StageTypes ty, int saturate, const PgemmPlan& plan, unsigned* status,
                       cudaStream_t stream);

}  // namespace nq
