// Launchers of the tcgen05 linear-cross-entropy kernels (bf16 operands, fp32 accumulate).
#pragma once

#include "common.h"

namespace b200tp {

constexpr int kCeTileRows = 128;   // rows of hidden per tile
constexpr int kCeTileCols = 256;   // vocab columns (logits) / hidden columns (dH) per tile

// A 4-bit affine group-64 head (codes (V, D/8) uint32 low nibble first, scales / biases (V, D/64) bf16
// or fp32).  Passed to the launchers below, the weight operand is expanded inside the kernels and `w`
// is ignored; a null pointer (or a null `wq`) means a dense bf16 weight matrix `w`.
struct QuantHead {
  const uint32_t* wq;
  const void* scales;
  const void* biases;
  int qp_f32;
};

// A launch that is only needed when a flag in device memory is set (or is not): every CTA reads it first and
// leaves at once otherwise.  A null `flag` means "always".
struct LaunchGuard {
  const int* flag = nullptr;
  int run_if_set = 0;
};

// Vocab splits the forward uses for (n rows, v_rows vocab rows): one partial triple per
// (row, split) lands in the workspace.
int ce_tc_fwd_splits(int64_t n, int d, int64_t v_rows);
// The split count behind it, for `num_rb` row groups and `num_vt` vocab tiles on `ctas` CTAs (or pairs).
int ce_tc_choose_splits(int num_rb, int num_vt, int ctas);

// Forward partials over weight rows [vrow0, vrow1) of a (w_rows_total, d) bf16 matrix whose
// row 0 has global vocab id `vocab_id0`.  pm/ps/pt: [splits][n] f32.
int ce_tc_launch_fwd(const void* hidden, const void* w, int64_t w_rows_total, int64_t n, int d, int64_t vrow0,
                     int64_t vrow1, int64_t vocab_id0, const int64_t* targets, int64_t ignore_index, int splits,
                     float* pm, float* ps, float* pt, const QuantHead* q, cudaStream_t stream, int* status);

// The same partials for a 4-bit head expanded inside the kernel into tensor memory (linear_ce_int4.cu).
int ce_int4_fwd_splits(int64_t n, int64_t v_rows);
int ce_int4_launch_fwd(const void* hidden, const QuantHead& q, int64_t v_rows, int64_t n, int d, int64_t vocab_id0,
                       const int64_t* targets, int64_t ignore_index, int splits, float* pm, float* ps, float* pt,
                       cudaStream_t stream, int* status);

// g[n][ldg] (bf16) = (exp(z - lse) - onehot) * ct over weight rows [vrow0, vrow1); columns
// up to the next multiple of 256 are written (zeros past vrow1).
int ce_tc_launch_bwd_g(const void* hidden, const void* w, int64_t w_rows_total, int64_t n, int d, int64_t vrow0,
                       int64_t vrow1, int64_t vocab_id0, const int64_t* targets, int64_t ignore_index,
                       const float* lse, const float* ct, void* g, int ldg, const QuantHead* q,
                       const LaunchGuard& guard, cudaStream_t stream, int* status);

// Forward partials as ce_tc_launch_fwd and, from the same exponentials, g[n][ldg] (bf16) = exp(z - ref) with
// `ref2` = ref log2(e) per row, zero at the target's column and on ignored rows.  Any other row whose logits reach
// 69 above its reference sets *overflow (g is void then; the partials are right in any case).  Dense weights.
int ce_tc_launch_fwd_grad(const void* hidden, const void* w, int64_t w_rows_total, int64_t n, int d, int64_t vrow0,
                          int64_t vrow1, int64_t vocab_id0, const int64_t* targets, int64_t ignore_index,
                          const float* ref2, int* overflow, int splits, float* pm, float* ps, float* pt, void* g,
                          int ldg, cudaStream_t stream, int* status);

// dH = [acc_in +] G[:, :k_total] @ W[wrow0 : wrow0 + k_total, :]; written to out_bf16, else to acc_out (f32), which
// also holds the sums of the parts that a k_total above 16384 is accumulated in (without it, in one).  k_total is a multiple of 64; rows of W past w_rows_total read as zero.
// The 128 x 256 output tiles are numbered row-block-major; this launch computes tiles
// [tile0, tile1) (negative: from the first / through the last).  `ce_tc_dh_rows_done(n, d, t)` is
// the number of leading rows of d_hidden that are complete once tiles [0, t) have run.
// `ksplit` > 1 shares each tile's contraction between that many units, share s summing into acc + s * n * d
// (fp32, in place over chunks); `ce_tc_dh_ksplit` picks it for chunks of k_total columns.
int ce_tc_dh_tiles(int64_t n, int d);
int ce_tc_dh_ksplit(int64_t n, int d, int k_total);
int ce_tc_dh_rows_done(int64_t n, int d, int tiles_done);
int ce_tc_launch_dh(const void* g, int ldg, int k_total, int64_t n, const void* w, int64_t w_rows_total, int d,
                    int64_t wrow0, const float* acc_in, float* acc_out, void* out_bf16, int tile0, int tile1,
                    int ksplit, const QuantHead* q, const LaunchGuard& guard, cudaStream_t stream, int* status);

// d_weight block (v_rows, d) bf16 = G[:, :v_rows]^T @ hidden: g (n, ldg) bf16 as written by
// ce_tc_launch_bwd_g, hidden (n, d) bf16.  fp32 accumulation over the n rows, one rounding.
int ce_tc_launch_dw(const void* g, int ldg, int64_t v_rows, int64_t n, const void* hidden, int d, void* d_weight_block,
                    cudaStream_t stream, int* status);

}  // namespace b200tp
