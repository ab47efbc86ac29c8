// Launchers of the fp32 linear cross-entropy on the tensor cores (linear_ce_split.cu).
//
// Operands are planes: an fp32 matrix (rows, cols) as (3, rows, cols) bf16 whose sum it is.
#pragma once

#include "common.h"

namespace b200tp {

// When a launch does its work: while *run_if is set (null: always) and *unless is not (null: always).  Every CTA reads
// both first, so a kernel must not write either.
struct SplitGuard {
  const int* run_if = nullptr;
  const int* unless = nullptr;
  __host__ __device__ bool any() const { return run_if != nullptr || unless != nullptr; }
};

// x (count values, a multiple of 8) -> planes; sets *flag when a value has no such form (inf, NaN, or so near the
// largest fp32 that bf16 rounds it to infinity).
int ce_split_planes(const float* x, int64_t count, void* planes, int* flag, cudaStream_t stream,
                    const SplitGuard& guard = {});

// Vocab shares of a logits launch.
int ce_split_splits(int64_t n, int64_t width);

// Forward partials of one vocab chunk (`width` rows from `vocab_id0`): 2 * splits triples per row.
int ce_split_fwd(const void* h3, const void* w3, int64_t n, int d, int64_t width, int64_t vocab_id0,
                 const int64_t* targets, int64_t ignore_index, int splits, float* pm, float* ps, float* pt,
                 cudaStream_t stream, int* status);

// g3 (3, n, ldg) = (exp(z - lse) - onehot) * ct of one chunk, zero past its width up to the next multiple of 256;
// sets *flag when a value is not finite.
int ce_split_bwd_g(const void* h3, const void* w3, int64_t n, int d, int64_t width, int64_t vocab_id0,
                   const int64_t* targets, int64_t ignore_index, const float* lse, const float* ct, int splits,
                   void* g3, int ldg, int* flag, cudaStream_t stream, int* status, const SplitGuard& guard = {});

// The forward that also forms the gradient's sum (see linear_ce_grad.h): ref, then per chunk the partials and
// g3 = exp(z - ref), zero at the target and on ignored rows; *flag is set when g3 is void (a logit more than 69 above
// the reference of a row that is not ignored, or *bad), the partials are right unless *bad.
int ce_split_reference(const float* hidden, const float* w, int64_t n, int d, int64_t v, const int64_t* targets,
                       int64_t ignore_index, float* ref, cudaStream_t stream);
int ce_split_fwd_grad(const void* h3, const void* w3, int64_t n, int d, int64_t width, int64_t vocab_id0,
                      const int64_t* targets, int64_t ignore_index, const float* ref, int splits, float* pm, float* ps,
                      float* pt, void* g3, int ldg, const int* bad, int* flag, cudaStream_t stream, int* status);
// d_hidden from the shares' sums, nothing while flags[0] (they are void; set here when one overflowed) is set; flags[2] = flags[1] (an operand has no
// planes) in any case.
int ce_split_finish(const float* acc, int shares, const float* ref, int* flags, const float* w, int64_t n, int d,
                    int64_t v, const int64_t* targets, int64_t ignore_index, const float* lse, const float* tgt,
                    const float* ct, float* out, cudaStream_t stream);

// out (ksplit shares of (n, d) fp32, `keep`: added to) = g @ w over the chunk.
int ce_split_dh_shares(int64_t n, int d, int64_t width);
int ce_split_dh(const void* g3, int ldg, const void* w3, int64_t n, int d, int64_t width, int ksplit, float* out,
                int keep, cudaStream_t stream, int* status, const SplitGuard& guard = {});

// out = (keep ? out : 0) + sum of the shares in index order.
int ce_split_sum(const float* acc, int shares, int64_t count, float* out, int keep, const SplitGuard& guard,
                 cudaStream_t stream);

}  // namespace b200tp
