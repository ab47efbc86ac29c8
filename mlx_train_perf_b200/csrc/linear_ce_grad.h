// Row kernels of the forward that also forms the gradient (see linear_ce_grad.cu).
#pragma once

#include "linear_ce_tc.h"

namespace b200tp {

// ref2[n] = log2(e) * (logit of the row's target, or of vocab row 0 when it has none), 0 where that
// is not finite; *overflow = 0.
// `q` non-null: 4-bit head, else `w` (v, d) bf16.
int launch_ce_reference(const void* hidden, const void* w, const QuantHead* q, int64_t n, int d, int64_t v,
                        const int64_t* targets, int64_t ignore_index, float* ref2, int* overflow,
                        cudaStream_t stream);

// d_hidden[n][d] (bf16) = ct * (exp(ref - lse) * sum_s acc[s] + (p_target - 1) * W[target]), 0 on ignored rows;
// does nothing when *overflow is set, and sets it when a sum overflowed (d_hidden is void then).
int launch_ce_grad_finish(const float* acc, int shares, const float* ref2, int* overflow, const void* w,
                          const QuantHead* q, int64_t n, int d, int64_t v, const int64_t* targets,
                          int64_t ignore_index, const float* lse, const float* tgt, const float* ct, void* d_hidden,
                          cudaStream_t stream);

}  // namespace b200tp
