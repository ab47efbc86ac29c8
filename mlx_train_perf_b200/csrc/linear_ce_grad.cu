// Row kernels around the forward that also forms the gradient of the hidden states (frozen heads, bf16).
//
// The gradient of row i's loss is  sum_v p_iv W_v - W_t  with p_iv = exp(z_iv - lse_i).  It needs the logits twice
// only because lse is known after all of them; with any reference r_i fixed beforehand,
//   exp(r_i - lse_i) * sum_{v != t} exp(z_iv - r_i) W_v  +  (p_it - 1) W_t
// is the same vector, and the sum can be formed chunk by chunk beside the forward's row sums: two contractions
// over N x V x D where forward + recomputing backward take three.  The reference is the target's own logit: it
// never exceeds the row maximum, so nothing that matters underflows, and logits may lie 69 above it before
// an exponential overflows (a loss of 69 nats; such calls set a flag and the backward recomputes, as it always did
// before: core/chunked.py:52-90 of the reference).  A sum over weights of 2^11 and more may overflow before that:
// the finish kernel then sets the flag.
#include "linear_ce_grad.h"

#include "dequant.cuh"
#include "ptx.cuh"

namespace b200tp {
namespace {

__device__ __forceinline__ float dot8(uint4 a, uint4 b, float acc) {
  const uint32_t x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[i]));
    const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&y[i]));
    acc = fmaf(u.x, v.x, acc);
    acc = fmaf(u.y, v.y, acc);
  }
  return acc;
}

// Eight consecutive weights of a vocab row: columns [8 i, 8 i + 8).
template <bool QUANT>
__device__ __forceinline__ uint4 weight8(const __nv_bfloat16* w, const QuantHead& q, long long row, int d, int i) {
  if constexpr (!QUANT) {
    return __ldg(reinterpret_cast<const uint4*>(w + row * d) + i);
  } else {
    const long long gi = row * (d / 64) + (i >> 3);
    const uint32_t sc = dq_load_param(q.scales, gi, q.qp_f32 != 0), bi = dq_load_param(q.biases, gi, q.qp_f32 != 0);
    const int sh = q.qp_f32 ? 0 : 16;
    return dq_word_f32(__ldg(q.wq + row * (d / 8) + i), __uint_as_float(sc << sh), __uint_as_float(bi << sh));
  }
}

__device__ __forceinline__ long long target_row(long long t, long long ignore_index, long long v) {
  return (t != ignore_index && t >= 0 && t < v) ? t : -1;
}

// One warp per row, four rows per block: two row reads of D bf16, HBM-bound (N = 8192, D = 4096: 134 MB).
template <bool QUANT>
__global__ void __launch_bounds__(128)
ce_reference_kernel(const __nv_bfloat16* __restrict__ hidden, const __nv_bfloat16* __restrict__ w, const QuantHead q,
                    int n, int d, long long v, const long long* __restrict__ targets, long long ignore_index,
                    float* __restrict__ ref2, int* __restrict__ overflow) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *overflow = 0;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n) return;
  const long long t = max(target_row(targets[row], ignore_index, v), 0ll);
  const uint4* h = reinterpret_cast<const uint4*>(hidden + static_cast<long long>(row) * d);
  float acc = 0.f;
#pragma unroll 4
  for (int i = lane; i < d / 8; i += 32) acc = dot8(__ldg(h + i), weight8<QUANT>(w, q, t, d, i), acc);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) ref2[row] = isfinite(acc) ? acc * kLog2e : 0.f;   // (any finite one serves)
}

// Eight columns of one row per thread.  HBM-bound: the fp32 sums, the target's weight row and the bf16 result
// (N = 8192, D = 4096: 268 MB).
constexpr int kFinishThreads = 128;
template <bool QUANT>
__global__ void __launch_bounds__(kFinishThreads)
ce_grad_finish_kernel(const float* __restrict__ acc, int shares, const float* __restrict__ ref2,
                      int* overflow, const __nv_bfloat16* __restrict__ w, const QuantHead q, int n,
                      int d, long long v, const long long* __restrict__ targets, long long ignore_index,
                      const float* __restrict__ lse, const float* __restrict__ tgt, const float* __restrict__ ct,
                      __nv_bfloat16* __restrict__ out) {
  if (*overflow != 0) return;
  const int row = blockIdx.x;
  const int i = blockIdx.y * kFinishThreads + threadIdx.x;
  if (i >= d / 8) return;
  const long long off = static_cast<long long>(row) * d + i * 8;
  const long long target = targets[row];
  if (target == ignore_index) {
    *reinterpret_cast<uint4*>(out + off) = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const long long stride = static_cast<long long>(n) * d;
#pragma unroll 4
  for (int k = 0; k < shares; ++k) {
    const float4 a = __ldcs(reinterpret_cast<const float4*>(acc + k * stride + off));
    const float4 b = __ldcs(reinterpret_cast<const float4*>(acc + k * stride + off) + 1);
    s[0] += a.x; s[1] += a.y; s[2] += a.z; s[3] += a.w;
    s[4] += b.x; s[5] += b.y; s[6] += b.z; s[7] += b.w;
  }
  bool finite = true;
#pragma unroll
  for (int k = 0; k < 8; ++k) finite = finite && isfinite(s[k]);
  if (!finite) {
    *overflow = 1;
    return;
  }
  // c last: exp(ref - lse) may be as small as 2^-117, and c too is often small
  const float c = ct[row], l = lse[row];
  const float f = exp2f(ref2[row] - l * kLog2e);
  const long long t = target_row(target, ignore_index, v);
  uint32_t o[4];
  if (t >= 0) {
    const float g = expm1f(tgt[row] - l);   // p_target - 1
    const uint4 w8 = weight8<QUANT>(w, q, t, d, i);
    const uint32_t wv[4] = {w8.x, w8.y, w8.z, w8.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&wv[k]));
      o[k] = pack_bf16x2(c * fmaf(f, s[2 * k], g * x.x), c * fmaf(f, s[2 * k + 1], g * x.y));
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = pack_bf16x2(c * (f * s[2 * k]), c * (f * s[2 * k + 1]));
  }
  *reinterpret_cast<uint4*>(out + off) = make_uint4(o[0], o[1], o[2], o[3]);
}

}  // namespace

int launch_ce_reference(const void* hidden, const void* w, const QuantHead* q, int64_t n, int d, int64_t v,
                        const int64_t* targets, int64_t ignore_index, float* ref2, int* overflow,
                        cudaStream_t stream) {
  const unsigned blocks = static_cast<unsigned>(ceil_div(n, 4));
  const auto* h = static_cast<const __nv_bfloat16*>(hidden);
  const auto* wd = static_cast<const __nv_bfloat16*>(w);
  const auto* t = reinterpret_cast<const long long*>(targets);
  if (q != nullptr)
    ce_reference_kernel<true><<<blocks, 128, 0, stream>>>(h, wd, *q, static_cast<int>(n), d, v, t, ignore_index, ref2,
                                                          overflow);
  else
    ce_reference_kernel<false><<<blocks, 128, 0, stream>>>(h, wd, QuantHead{}, static_cast<int>(n), d, v, t,
                                                           ignore_index, ref2, overflow);
  B200TP_CUDA_OK(cudaGetLastError());
  return B200TP_OK;
}

int launch_ce_grad_finish(const float* acc, int shares, const float* ref2, int* overflow, const void* w,
                          const QuantHead* q, int64_t n, int d, int64_t v, const int64_t* targets,
                          int64_t ignore_index, const float* lse, const float* tgt, const float* ct, void* d_hidden,
                          cudaStream_t stream) {
  const dim3 grid(static_cast<unsigned>(n), static_cast<unsigned>(ceil_div(d / 8, kFinishThreads)));
  const auto* wd = static_cast<const __nv_bfloat16*>(w);
  const auto* t = reinterpret_cast<const long long*>(targets);
  auto* out = static_cast<__nv_bfloat16*>(d_hidden);
  if (q != nullptr)
    ce_grad_finish_kernel<true><<<grid, kFinishThreads, 0, stream>>>(acc, shares, ref2, overflow, wd, *q,
                                                                     static_cast<int>(n), d, v, t, ignore_index, lse,
                                                                     tgt, ct, out);
  else
    ce_grad_finish_kernel<false><<<grid, kFinishThreads, 0, stream>>>(acc, shares, ref2, overflow, wd, QuantHead{},
                                                                      static_cast<int>(n), d, v, t, ignore_index,
                                                                      lse, tgt, ct, out);
  B200TP_CUDA_OK(cudaGetLastError());
  return B200TP_OK;
}

}  // namespace b200tp
