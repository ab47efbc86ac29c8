// fp32 linear cross-entropy on the tensor cores: each fp32 operand as three bf16 planes.
//
// x = hi + mid + lo with hi = bf16(x), mid = bf16(x - hi), lo = x - hi - mid is exact (three 8-bit significands
// cover fp32's 24 bits), so a product x y is the sum of nine bf16 products, each exact in fp32.  Six are formed:
// hi hi, hi mid, mid hi, mid mid, hi lo, lo hi; the other three are below 2^-25 of it and of random sign.  What is
// left is the summation.  The tensor core rounds its fp32 accumulator towards zero at every step, an error that
// grows with the number of steps and is biased, so a contraction is cut into segments of 128: each runs in a fresh
// tensor-memory accumulator, the five small products first (their steps round at 2^-8 of the size), and is added
// to a register sum with round-to-nearest.  Distance to float64 (2-norm, CUDA cores / here): 2048 x 1024 x 32768 losses
// 4.3e-7 / 1.3e-7, d_hidden 1.5e-6 / 5.1e-7; 60 x 4096 x 8192 losses 1.0e-6 / 1.5e-7, d_hidden 1.8e-6 / 4.7e-7.
//
// Tensor-bound: six bf16 products (6 x 2 N V D flops per contraction) against one product on the CUDA cores, whose
// fp32 rate is 1/25 of the bf16 tensor rate and whose kernels reach a third of it.  2048 x 1024 x 32768, forward +
// backward: 18.5 ms there, 2.57 with three contractions, 1.65 with the gradient's sum formed in the forward and CTA
// pairs: twelve bf16 products at 1.36 PFLOP/s inside the two kernels.
//
//   split_planes_kernel    fp32 rows -> three bf16 planes; raises a flag on values bf16 cannot hold (inf, NaN,
//                          within 2^-9 of the largest fp32), for which the CUDA-core kernels take over
//   split_logits_kernel    Z = H W^T per 128 x 256 tile, K = D; row sums (FWD), g as three planes (BWD_G), or row sums
//                          and exp(z - ref) as three planes (FWD_GRAD, as linear_ce_grad.cu does for bf16)
//   split_dh_kernel        dH (128 x 256) (+)= G W over the chunk's vocab rows
//   share_sum_kernel       adds the shares of a contraction that was spread over several CTAs
//
// Fallback launches, which nearly always have nothing to do, overlap their predecessors' tails (38 of them in a step of
// 2048 x 1024 x 32768: 1.70 -> 1.58 ms).
//
// Roles and CTA pairs as in linear_ce_tc.cu, with eight accumulating warps (two per lane quadrant, 128 columns each).
// Replaces core/chunked.py:35-90 of the reference for fp32 heads, beside linear_ce_simt.cu.
#include "linear_ce_split.h"

#include <algorithm>
#include <atomic>

#include "linear_ce_pipe.cuh"

namespace b200tp {
namespace {

constexpr int EPI_WARPS = 8;
constexpr int SPLIT_THREADS = 64 + 32 * EPI_WARPS;
constexpr int HALF = BN / 2;          // columns per accumulating warp
constexpr int SEG_KB = 2;             // k blocks (64) per accumulator segment
constexpr int PAIRS = 6;
// plane (0 hi, 1 mid, 2 lo) of A and of B for each pair, two bits each, smallest products first
constexpr uint32_t PLANE_A = 2u | 0u << 2 | 1u << 4 | 1u << 6 | 0u << 8 | 0u << 10;
constexpr uint32_t PLANE_B = 0u | 2u << 2 | 1u << 4 | 0u << 6 | 1u << 8 | 0u << 10;
__device__ __forceinline__ int plane_a(int pr) { return (PLANE_A >> (2 * pr)) & 3; }
__device__ __forceinline__ int plane_b(int pr) { return (PLANE_B >> (2 * pr)) & 3; }

enum { SPLIT_FWD = 0, SPLIT_BWD_G = 1, SPLIT_FWD_GRAD = 2 };
constexpr float kHeadroom = 69.f;   // FWD_GRAD: exponents above this raise the flag; 2^27 terms of e^69 fit fp32

// (A guarded launch may be scheduled under its predecessor's tail, as in linear_ce_simt.cu.)
__device__ __forceinline__ bool guard_skips(const SplitGuard& g) {
  if (g.any()) griddep_wait();
  return (g.run_if != nullptr && *g.run_if == 0) || (g.unless != nullptr && *g.unless != 0);
}

__device__ __forceinline__ void split3(float x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = __bfloat16_as_ushort(__float2bfloat16_rn(x));
  const float r = x - __uint_as_float(hi << 16);
  mid = __bfloat16_as_ushort(__float2bfloat16_rn(r));
  lo = __bfloat16_as_ushort(__float2bfloat16_rn(r - __uint_as_float(mid << 16)));
}

// N (8 or 16) consecutive values -> 2 N bytes of each plane, sixteen as whole sectors.
template <int N>
__device__ __forceinline__ bool split_store(const float (&x)[N], __nv_bfloat16* dst, long long plane) {
  uint32_t o[3][N / 2];
  bool bad = false;
#pragma unroll
  for (int e = 0; e < N; e += 2) {
    uint32_t h0, m0, l0, h1, m1, l1;
    split3(x[e], h0, m0, l0);
    split3(x[e + 1], h1, m1, l1);
    bad = bad || (h0 & 0x7F80u) == 0x7F80u || (h1 & 0x7F80u) == 0x7F80u;
    o[0][e >> 1] = h0 | h1 << 16;
    o[1][e >> 1] = m0 | m1 << 16;
    o[2][e >> 1] = l0 | l1 << 16;
  }
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    if constexpr (N == 16)
      st_global_32b(dst + p * plane, o[p]);
    else
      *reinterpret_cast<uint4*>(dst + p * plane) = make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
  }
  return bad;
}

// HBM-bound: 4 bytes read and 6 written per value.  `count` is a multiple of 8, `out` 16-byte aligned.
template <bool ALIGNED>
__global__ void __launch_bounds__(256)
split_planes_kernel(const float* __restrict__ x, long long count, __nv_bfloat16* __restrict__ out, int* flag,
                    const SplitGuard guard) {
  if (guard_skips(guard)) return;
  const long long i = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * 8;
  bool bad = false;
  if (i < count) {
    float v[8];
    if (ALIGNED) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(x + i)), b = __ldg(reinterpret_cast<const float4*>(x + i) + 1);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = __ldg(x + i + e);
    }
    bad = split_store(v, out + i, count);
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) *flag = 1;
}

// out = (keep ? out : 0) + sum of the shares, in index order (`out` may have any alignment).
__global__ void __launch_bounds__(256)
share_sum_kernel(const float* __restrict__ acc, int shares, long long count, float* __restrict__ out, int keep,
                 const SplitGuard guard) {
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (guard_skips(guard) || i >= count) return;
  float s = 0.f;
#pragma unroll 4
  for (int k = 0; k < shares; ++k) s += __ldcs(acc + k * count + i);
  out[i] = keep ? out[i] + s : s;
}

struct SplitLogitsParams {
  int n_rows, kblocks;
  int width;             // vocab rows of the chunk
  long long vocab_id0;   // global id of its first
  int num_rb, num_vt, splits;
  const long long* targets;
  long long ignore_index;
  float* pm;             // FWD: partial triples, [split][column half][N] each
  float* ps;
  float* pt;
  const float* lse;      // BWD_G
  const float* ct;
  __nv_bfloat16* g;      // (3, N, ldg)
  int ldg;
  const float* ref;      // FWD_GRAD: reference of the row's exponentials
  const int* bad;        // FWD_GRAD: an operand had no planes; raises the flag
  int* flag;             // BWD_G: set when a value of g is not finite; FWD_GRAD: when g is void
  SplitGuard guard;
  int* status;
};

struct SplitDhParams {
  int n_rows, d_cols;
  int kblocks;           // 64-row blocks of the chunk's vocab rows
  int num_rb, num_nt, ksplit;
  float* out;            // share s at out + s * n * d
  int keep;              // add to what `out` holds
  SplitGuard guard;
  int* status;
};

// One tile's stage sequence: segments of SEG_KB k blocks, in each the six plane pairs, in each its k blocks.
struct SplitWalk {
  int seg0, seg1, pr, kb, kb_end;
  __device__ __forceinline__ SplitWalk(int kb0, int kblocks_end) : seg0(kb0), pr(0), kb(kb0), kb_end(kblocks_end) {
    seg1 = min(seg0 + SEG_KB, kb_end);
  }
  __device__ __forceinline__ bool first() const { return pr == 0 && kb == seg0; }
  __device__ __forceinline__ bool last() const { return pr == PAIRS - 1 && kb + 1 == seg1; }
  __device__ __forceinline__ bool done() const { return seg0 >= kb_end; }
  __device__ __forceinline__ void next() {
    if (++kb < seg1) return;
    kb = seg0;
    if (++pr < PAIRS) return;
    pr = 0;
    seg0 = kb = seg1;
    seg1 = min(seg0 + SEG_KB, kb_end);
  }
};

// The MMA issuer's part of one tile.  B_MN: B is MN-major in 64 x 64 boxes (the weight rows of dH), else K-major.
template <bool B_MN, bool PAIR>
__device__ __forceinline__ bool issue_tile(const SmemView& sm, uint32_t tmem_base, int kb0, int kb1, uint32_t& it,
                                           uint32_t& seg, int lane, int* status) {
  constexpr uint32_t idesc = make_idesc_bf16(PAIR ? 2 * BM : BM, BN, 0, B_MN ? 1 : 0);
  constexpr uint32_t dhi = desc_hi_sw128(1024);
  constexpr uint32_t b_step = B_MN ? 128 : 2, kStages = PAIR ? PAIR_STAGES : STAGES;
  for (SplitWalk w(kb0, kb1); !w.done(); w.next(), ++it) {
    const uint32_t as = seg & 1;
    if (w.first()) {
      if (!mbar_wait_warp(&sm.tempty[as], ((seg >> 1) & 1) ^ 1, sm.abort_flag)) {
        if (lane == 0) raise_abort(sm, status, kDevTimeoutMma);
        return false;
      }
    }
    const int s = it % kStages;
    if (!mbar_wait_warp(&sm.full[s], (it / kStages) & 1, sm.abort_flag)) {
      if (lane == 0) raise_abort(sm, status, kDevTimeoutMma);
      return false;
    }
    tc_fence_after_sync();
    const uint32_t d_tmem = tmem_base + as * BN;
    const uint32_t a_lo = desc_lo(smem_u32(sm.a(s)), 16);
    const uint32_t b_lo = desc_lo(smem_u32(sm.b(s)), B_MN ? 64 * BK * 2 : 16);
    const bool fresh = w.first(), last = w.last();
    if (elect_one()) {
#pragma unroll
      for (int k = 0; k < BK / 16; ++k)
        umma<PAIR>(d_tmem, a_lo + k * 2, dhi, b_lo + k * b_step, dhi, idesc, (fresh && k == 0) ? 0u : 1u);
      commit<PAIR>(&sm.empty[s]);
      if (last) commit<PAIR>(&sm.tfull[as]);
    }
    __syncwarp();
    if (last) ++seg;
  }
  return true;
}

// A pair's CTA leaves only after the commits of its last stages have arrived.
__device__ __forceinline__ void pair_tail(const SmemView& sm, uint32_t it) {
  for (uint32_t j = it > PAIR_STAGES ? it - PAIR_STAGES : 0; j < it; ++j)
    mbar_wait(&sm.empty[j % PAIR_STAGES], (j / PAIR_STAGES) & 1, sm.abort_flag);
}

// An accumulating warp's part of one tile: acc = sum of the segments' accumulators over its 128 columns.
template <bool PAIR>
__device__ __forceinline__ bool gather_tile(const SmemView& sm, uint32_t taddr, int segs, uint32_t& seg, int lane,
                                            float (&acc)[HALF], int* status) {
#pragma unroll
  for (int e = 0; e < HALF; ++e) acc[e] = 0.f;
  for (int i = 0; i < segs; ++i, ++seg) {
    const uint32_t as = seg & 1;
    if (!mbar_wait_warp(&sm.tfull[as], (seg >> 1) & 1, sm.abort_flag)) {
      raise_abort(sm, status, kDevTimeoutEpilogue);
      return false;
    }
    tc_fence_after_sync();
#pragma unroll
    for (int c = 0; c < HALF / 32; ++c) {
      uint32_t r[32];
      tmem_ld_x32(taddr + as * BN + c * 32, r);
      tmem_wait_ld();
      tmem_regs_ready(r);
#pragma unroll
      for (int e = 0; e < 32; ++e) acc[c * 32 + e] += __uint_as_float(r[e]);
    }
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) release_acc<PAIR>(&sm.tempty[as]);
  }
  return true;
}

template <int MODE, bool PAIR>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
split_logits_kernel(const __grid_constant__ CUtensorMap tmap_h, const __grid_constant__ CUtensorMap tmap_w,
                    const SplitLogitsParams p) {
  if (guard_skips(p.guard)) return;
  extern __shared__ uint8_t smem_raw[];
  const SmemView sm = carve_smem(smem_raw, false, PAIR);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // provably warp-uniform
  const int lane = threadIdx.x & 31;
  const uint32_t tmem_base = cta_setup(sm, warp, 1, (PAIR ? 2 : 1) * EPI_WARPS, PAIR);
  constexpr uint32_t kStages = PAIR ? PAIR_STAGES : STAGES;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0;
  const int unit0 = PAIR ? blockIdx.x >> 1 : blockIdx.x, unit_step = PAIR ? gridDim.x >> 1 : gridDim.x;
  auto block_row = [&](int rb) { return (PAIR ? rb * 2 + static_cast<int>(rank) : rb) * BM; };
  const int total_units = p.num_rb * p.splits;
  auto vt_begin = [&](int split) { return static_cast<int>(static_cast<long long>(split) * p.num_vt / p.splits); };

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_h);
      tma_prefetch_desc(&tmap_w);
      uint32_t it = 0;
      bool ok = true;
      for (int u = unit0; u < total_units && ok; u += unit_step) {
        const int split = u / p.num_rb, rb = u - split * p.num_rb;
        for (int vt = vt_begin(split); vt < vt_begin(split + 1) && ok; ++vt) {
          for (SplitWalk w(0, p.kblocks); !w.done(); w.next(), ++it) {
            const int s = it % kStages;
            if (!mbar_wait(&sm.empty[s], ((it / kStages) & 1) ^ 1, sm.abort_flag)) {
              raise_abort(sm, p.status, kDevTimeoutProducer);
              ok = false;
              break;
            }
            if (PAIR) {   // both CTAs' copies complete on CTA 0's barrier
              if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2 * PAIR_STAGE_BYTES);
              const uint32_t bar = map_to_rank(&sm.full[s], 0);
              tma_load_4d_pair(sm.a(s), &tmap_h, bar, w.kb * BK, block_row(rb), 0, plane_a(w.pr));
              tma_load_4d_pair(sm.b(s), &tmap_w, bar, w.kb * BK, vt * BN + static_cast<int>(rank) * (BN / 2), 0,
                               plane_b(w.pr));
              continue;
            }
            mbar_arrive_expect_tx(&sm.full[s], STAGE_BYTES);
            tma_load_4d(sm.a(s), &tmap_h, &sm.full[s], w.kb * BK, rb * BM, 0, plane_a(w.pr));
            tma_load_4d(sm.b(s), &tmap_w, &sm.full[s], w.kb * BK, vt * BN, 0, plane_b(w.pr));
          }
        }
      }
      if (PAIR && ok) pair_tail(sm, it);
      if (!ok) producer_drain(sm, it);
    }
  } else if (warp == 1) {
    uint32_t it = 0, seg = 0;
    bool ok = rank == 0;   // CTA 0 issues for both
    for (int u = unit0; u < total_units && ok; u += unit_step) {
      const int split = u / p.num_rb;
      for (int vt = vt_begin(split); vt < vt_begin(split + 1) && ok; ++vt)
        ok = issue_tile<false, PAIR>(sm, tmem_base, 0, p.kblocks, it, seg, lane, p.status);
    }
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t taddr = tmem_base + half * HALF + (static_cast<uint32_t>(quad * 32) << 16);
    const int segs = (p.kblocks + SEG_KB - 1) / SEG_KB;
    uint32_t seg = 0;
    bool ok = true, bad = false;
    for (int u = unit0; u < total_units && ok; u += unit_step) {
      const int split = u / p.num_rb, rb = u - split * p.num_rb;
      const int row = block_row(rb) + quad * 32 + lane;
      const bool row_ok = row < p.n_rows;
      const long long target = row_ok ? p.targets[row] : p.ignore_index;
      const bool tvalid = row_ok && target != p.ignore_index;
      float run_m = -INFINITY, run_s = 0.f, run_t = 0.f;   // FWD
      float lse = 0.f, ct = 0.f;                           // BWD_G
      if (MODE == SPLIT_FWD_GRAD) run_m = row_ok ? p.ref[row] : 0.f;
      if (MODE == SPLIT_BWD_G && row_ok) {
        lse = p.lse[row];
        ct = tvalid ? p.ct[row] : 0.f;
      }
      for (int vt = vt_begin(split); vt < vt_begin(split + 1); ++vt) {
        float acc[HALF];
        ok = gather_tile<PAIR>(sm, taddr, segs, seg, lane, acc, p.status);
        if (!ok) break;
        const int col0 = vt * BN + half * HALF;          // chunk-relative column of acc[0]
        const int ncols = min(HALF, p.width - col0);     // columns that exist (may be <= 0)
        int tcol = -1;
        if (tvalid) {
          const long long rel = target - p.vocab_id0 - col0;
          if (rel >= 0 && rel < ncols) tcol = static_cast<int>(rel);
        }
        if (MODE == SPLIT_FWD) {
          if (ncols > 0) {
            float m4[4] = {run_m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < HALF; ++e) {
              if (e >= ncols) acc[e] = -INFINITY;
              if (e == tcol) run_t = acc[e];
              m4[e & 3] = fmaxf(m4[e & 3], acc[e]);
            }
            const float m = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
            float s4[4] = {run_s * expf(run_m - m), 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < HALF; ++e) s4[e & 3] += expf(acc[e] - m);
            run_s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
            run_m = m;
          }
        } else if (row_ok) {
          __nv_bfloat16* dst = p.g + static_cast<long long>(row) * p.ldg + col0;
          const long long plane = static_cast<long long>(p.n_rows) * p.ldg;
          if (MODE == SPLIT_FWD_GRAD) {
            float xm = -INFINITY;
#pragma unroll
            for (int e = 0; e < HALF; ++e) {
              if (e >= ncols) acc[e] = -INFINITY;
              if (e == tcol) run_t = acc[e];
              acc[e] -= run_m;
              xm = fmaxf(xm, acc[e]);
            }
            if (xm > kHeadroom) {   // rare: this thread's own sum moves to a larger reference; g is void then
              bad = bad || tvalid;  // (an ignored row's g is zero, and its reference an arbitrary logit)
              run_s *= expf(-xm);
              run_m += xm;
#pragma unroll
              for (int e = 0; e < HALF; ++e) acc[e] -= xm;
            }
          }
          float s4[4] = {run_s, 0.f, 0.f, 0.f};
#pragma unroll
          for (int e = 0; e < HALF; e += 16) {
            float g[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              if (MODE == SPLIT_FWD_GRAD) {
                // the target's own term p - 1 is added to d_hidden at the end
                const float v = expf(acc[e + k]);
                s4[k & 3] += v;
                g[k] = tvalid && e + k != tcol ? v : 0.f;
                continue;
              }
              float v = expf(acc[e + k] - lse);
              if (e + k == tcol) v -= 1.f;
              g[k] = e + k < ncols ? v * ct : 0.f;
            }
            bad = split_store(g, dst + e, plane) || bad;
          }
          if (MODE == SPLIT_FWD_GRAD) run_s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
        }
      }
      if (MODE != SPLIT_BWD_G && ok && row_ok) {
        const size_t o = static_cast<size_t>(split * 2 + half) * p.n_rows + row;
        p.pm[o] = run_m;
        p.ps[o] = run_s;
        p.pt[o] = run_t;
      }
    }
    if (MODE != SPLIT_FWD && bad) *p.flag = 1;
    if (MODE == SPLIT_FWD_GRAD && blockIdx.x == 0 && warp == 2 && lane == 0 && *p.bad != 0) *p.flag = 1;
  }
  cta_teardown(sm, warp, tmem_base, PAIR);
}

template <bool PAIR>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
split_dh_kernel(const __grid_constant__ CUtensorMap tmap_g, const __grid_constant__ CUtensorMap tmap_w,
                const SplitDhParams p) {
  if (guard_skips(p.guard)) return;
  extern __shared__ uint8_t smem_raw[];
  const SmemView sm = carve_smem(smem_raw, false, PAIR);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // provably warp-uniform
  const int lane = threadIdx.x & 31;
  const uint32_t tmem_base = cta_setup(sm, warp, 1, (PAIR ? 2 : 1) * EPI_WARPS, PAIR);
  constexpr uint32_t kStages = PAIR ? PAIR_STAGES : STAGES;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0;
  const int unit0 = PAIR ? blockIdx.x >> 1 : blockIdx.x, unit_step = PAIR ? gridDim.x >> 1 : gridDim.x;
  auto block_row = [&](int rb) { return (PAIR ? rb * 2 + static_cast<int>(rank) : rb) * BM; };
  const int tiles = p.num_rb * p.num_nt, total_units = tiles * p.ksplit;
  auto kb_begin = [&](int share) { return static_cast<int>(static_cast<long long>(share) * p.kblocks / p.ksplit); };

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_g);
      tma_prefetch_desc(&tmap_w);
      uint32_t it = 0;
      bool ok = true;
      for (int u = unit0; u < total_units && ok; u += unit_step) {
        const int share = u / tiles, t = u - share * tiles;
        const int rb = t / p.num_nt, nt = t - rb * p.num_nt;
        for (SplitWalk w(kb_begin(share), kb_begin(share + 1)); !w.done(); w.next(), ++it) {
          const int s = it % kStages;
          if (!mbar_wait(&sm.empty[s], ((it / kStages) & 1) ^ 1, sm.abort_flag)) {
            raise_abort(sm, p.status, kDevTimeoutProducer);
            ok = false;
            break;
          }
          if (PAIR) {
            if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2 * PAIR_STAGE_BYTES);
            const uint32_t bar = map_to_rank(&sm.full[s], 0);
            tma_load_4d_pair(sm.a(s), &tmap_g, bar, w.kb * BK, block_row(rb), 0, plane_a(w.pr));
#pragma unroll
            for (int j = 0; j < BN / 128; ++j)
              tma_load_4d_pair(sm.b(s) + j * (64 * BK * 2), &tmap_w, bar,
                               nt * BN + static_cast<int>(rank) * (BN / 2) + j * 64, w.kb * BK, 0, plane_b(w.pr));
            continue;
          }
          mbar_arrive_expect_tx(&sm.full[s], STAGE_BYTES);
          tma_load_4d(sm.a(s), &tmap_g, &sm.full[s], w.kb * BK, rb * BM, 0, plane_a(w.pr));
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)
            tma_load_4d(sm.b(s) + j * (64 * BK * 2), &tmap_w, &sm.full[s], nt * BN + j * 64, w.kb * BK, 0,
                        plane_b(w.pr));
        }
      }
      if (PAIR && ok) pair_tail(sm, it);
      if (!ok) producer_drain(sm, it);
    }
  } else if (warp == 1) {
    uint32_t it = 0, seg = 0;
    bool ok = rank == 0;   // CTA 0 issues for both
    for (int u = unit0; u < total_units && ok; u += unit_step) {
      const int share = u / tiles;
      ok = issue_tile<true, PAIR>(sm, tmem_base, kb_begin(share), kb_begin(share + 1), it, seg, lane, p.status);
    }
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t taddr = tmem_base + half * HALF + (static_cast<uint32_t>(quad * 32) << 16);
    uint32_t seg = 0;
    for (int u = unit0; u < total_units; u += unit_step) {
      const int share = u / tiles, t = u - share * tiles;
      const int rb = t / p.num_nt, nt = t - rb * p.num_nt;
      const int segs = (kb_begin(share + 1) - kb_begin(share) + SEG_KB - 1) / SEG_KB;
      float acc[HALF];
      if (!gather_tile<PAIR>(sm, taddr, segs, seg, lane, acc, p.status)) break;
      const int row = block_row(rb) + quad * 32 + lane, col0 = nt * BN + half * HALF;
      if (row < p.n_rows) {
        float* dst = p.out + (static_cast<long long>(share) * p.n_rows + row) * p.d_cols + col0;
#pragma unroll
        for (int e = 0; e < HALF; e += 4) {
          if (col0 + e < p.d_cols) {   // d_cols is a multiple of 8
            float4 v = make_float4(acc[e], acc[e + 1], acc[e + 2], acc[e + 3]);
            if (p.keep) {
              const float4 o = *reinterpret_cast<const float4*>(dst + e);
              v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
            }
            *reinterpret_cast<float4*>(dst + e) = v;
          }
        }
      }
    }
  }
  cta_teardown(sm, warp, tmem_base, PAIR);
}

// ref[row] = the target's logit (any vocab row's, where there is no target).  One warp per row; no alignment wanted.
__global__ void __launch_bounds__(128)
split_reference_kernel(const float* __restrict__ hidden, const float* __restrict__ w, int n, int d, long long v,
                       const long long* __restrict__ targets, long long ignore_index, float* __restrict__ ref) {
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n) return;
  const long long tg = targets[row], t = tg != ignore_index && tg >= 0 && tg < v ? tg : 0;
  const float *h = hidden + static_cast<long long>(row) * d, *wt = w + t * d;
  float acc = 0.f;
#pragma unroll 8
  for (int i = lane; i < d; i += 32) acc = fmaf(__ldg(h + i), __ldg(wt + i), acc);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) ref[row] = isfinite(acc) ? acc : 0.f;   // (any finite one serves)
}

// d_hidden = ct (exp(ref - lse) sum of shares + (p_t - 1) W_t); HBM-bound, one column per thread.
__global__ void __launch_bounds__(256)
split_finish_kernel(const float* __restrict__ acc, int shares, const float* __restrict__ ref, int* flags,
                    const float* __restrict__ w, int n, int d, long long v,
                    const long long* __restrict__ targets, long long ignore_index, const float* __restrict__ lse,
                    const float* __restrict__ tgt, const float* __restrict__ ct, float* __restrict__ out) {
  const int row = blockIdx.x, i = blockIdx.y * 256 + threadIdx.x;
  if (row == 0 && i == 0) flags[2] = flags[1];
  if (flags[0] != 0 || i >= d) return;
  const long long off = static_cast<long long>(row) * d + i, t = targets[row];
  if (t == ignore_index) {
    out[off] = 0.f;
    return;
  }
  float s = 0.f;
#pragma unroll 4
  for (int k = 0; k < shares; ++k) s += __ldcs(acc + static_cast<long long>(k) * n * d + off);
  if (!isfinite(s)) {   // large weights: the sum is void
    flags[0] = 1;
    return;
  }
  const float c = ct[row], l = lse[row];
  float g = expf(ref[row] - l) * s;
  if (t >= 0 && t < v) g = fmaf(expm1f(tgt[row] - l), __ldg(w + t * d + i), g);
  out[off] = c * g;
}

// CTA pairs over 256 rows, as in linear_ce_tc.cu, where an odd number of row blocks does not leave much of the last
// pair empty (2048 x 1024 x 32768, single CTAs against pairs and whole-sector stores of g: logits 176 / 124 us a chunk,
// d_hidden 138 / 119; the tensor pipe was 46 and 57 % active).  Forward / whole step in us, single CTAs, pairs, V = 32768:
//   D = 512:   200 rows 117 / 281, 115 / 274;  1024 rows 244 / 596, 211 / 563;  1100 rows (9 blocks) 246 / 621, 248 / 606
//   D = 1024:  200 rows 186 / 397, 176 / 375;  640 rows (5) 330 / 705, 291 / 666;  1100 rows 435 / 1020, 426 / 1147;
//              1300 rows (11) 531 / 1340, 509 / 1180;  2048 rows 756 / 1842, 631 / 1612
//   D = 2048:  200 rows 471 / 859, 408 / 774;  1024 rows 852 / 2003, 721 / 1798;  1100 rows 882 / 2112, 990 / 2092
//   D = 4096:  300 rows (3) 1311 / 2144, 1090 / 1989;  500 rows 1327 / 2339, 1101 / 2025
// Even counts gain throughout; of the odd ones 9 is about even and those below, left to single CTAs, would gain too.
bool split_pair(int64_t n) {
  const int64_t blocks = ceil_div(n, BM);
  return blocks % 2 == 0 || blocks >= 9;
}

std::atomic<int> g_configured[64];

int configure() {
  int dev = 0;
  B200TP_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && g_configured[dev].load(std::memory_order_acquire)) return B200TP_OK;
  const void* kernels[] = {
      reinterpret_cast<const void*>(split_logits_kernel<SPLIT_FWD, false>),
      reinterpret_cast<const void*>(split_logits_kernel<SPLIT_BWD_G, false>),
      reinterpret_cast<const void*>(split_logits_kernel<SPLIT_FWD_GRAD, false>),
      reinterpret_cast<const void*>(split_dh_kernel<false>),
      reinterpret_cast<const void*>(split_logits_kernel<SPLIT_FWD, true>),
      reinterpret_cast<const void*>(split_logits_kernel<SPLIT_BWD_G, true>),
      reinterpret_cast<const void*>(split_logits_kernel<SPLIT_FWD_GRAD, true>),
      reinterpret_cast<const void*>(split_dh_kernel<true>)};
  for (const void* k : kernels)
    B200TP_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  if (dev >= 0 && dev < 64) g_configured[dev].store(1, std::memory_order_release);
  return B200TP_OK;
}

// (3, rows, cols) planes as a 4-D map: coordinates (column, row, 0, plane).
int plane_map(CUtensorMap* out, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
  return make_tmap_bhsd_bf16(out, base, 3, 1, rows, cols, rows * ld, rows * ld, ld, box_rows, BK);
}

template <int MODE>
int launch_logits(const void* h3, const void* w3, int64_t n, int d, int64_t width, SplitLogitsParams& p,
                  cudaStream_t stream) {
  int rc = configure();
  if (rc) return rc;
  CUtensorMap tmap_h, tmap_w;
  rc = plane_map(&tmap_h, h3, n, d, d, BM);
  if (rc) return rc;
  const bool pair = split_pair(n);
  rc = plane_map(&tmap_w, w3, width, d, d, pair ? BN / 2 : BN);
  if (rc) return rc;
  p.n_rows = static_cast<int>(n);
  p.kblocks = static_cast<int>(ceil_div(d, BK));
  p.width = static_cast<int>(width);
  p.num_rb = static_cast<int>(ceil_div(n, pair ? 2 * BM : BM));
  p.num_vt = static_cast<int>(ceil_div(width, BN));
  return launch_units(pair ? split_logits_kernel<MODE, true> : split_logits_kernel<MODE, false>, SPLIT_THREADS, pair,
                      static_cast<long long>(p.num_rb) * p.splits, stream, tmap_h, tmap_w, p, p.guard.any());
}

}  // namespace

int ce_split_splits(int64_t n, int64_t width) {
  const bool pair = split_pair(n);
  return ce_tc_choose_splits(static_cast<int>(ceil_div(n, pair ? 2 * BM : BM)), static_cast<int>(ceil_div(width, BN)),
                             pair ? sm_count() / 2 : sm_count());
}

int ce_split_planes(const float* x, int64_t count, void* planes, int* flag, cudaStream_t stream,
                    const SplitGuard& guard) {
  const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  B200TP_CUDA_OK(launch_kernel(guard.any(), aligned ? split_planes_kernel<true> : split_planes_kernel<false>,
                               dim3(static_cast<unsigned>(ceil_div(count, 256 * 8))), dim3(256), 0, stream, x, count,
                               static_cast<__nv_bfloat16*>(planes), flag, guard));
  return B200TP_OK;
}

int ce_split_fwd(const void* h3, const void* w3, int64_t n, int d, int64_t width, int64_t vocab_id0,
                 const int64_t* targets, int64_t ignore_index, int splits, float* pm, float* ps, float* pt,
                 cudaStream_t stream, int* status) {
  SplitLogitsParams p{};
  p.vocab_id0 = vocab_id0;
  p.splits = splits;
  p.targets = reinterpret_cast<const long long*>(targets);
  p.ignore_index = ignore_index;
  p.pm = pm;
  p.ps = ps;
  p.pt = pt;
  p.status = status;
  return launch_logits<SPLIT_FWD>(h3, w3, n, d, width, p, stream);
}

int ce_split_bwd_g(const void* h3, const void* w3, int64_t n, int d, int64_t width, int64_t vocab_id0,
                   const int64_t* targets, int64_t ignore_index, const float* lse, const float* ct, int splits,
                   void* g3, int ldg, int* flag, cudaStream_t stream, int* status, const SplitGuard& guard) {
  SplitLogitsParams p{};
  p.flag = flag;
  p.guard = guard;
  p.vocab_id0 = vocab_id0;
  p.splits = splits;
  p.targets = reinterpret_cast<const long long*>(targets);
  p.ignore_index = ignore_index;
  p.lse = lse;
  p.ct = ct;
  p.g = static_cast<__nv_bfloat16*>(g3);
  p.ldg = ldg;
  p.status = status;
  return launch_logits<SPLIT_BWD_G>(h3, w3, n, d, width, p, stream);
}

int ce_split_reference(const float* hidden, const float* w, int64_t n, int d, int64_t v, const int64_t* targets,
                       int64_t ignore_index, float* ref, cudaStream_t stream) {
  split_reference_kernel<<<static_cast<unsigned>(ceil_div(n, 4)), 128, 0, stream>>>(
      hidden, w, static_cast<int>(n), d, v, reinterpret_cast<const long long*>(targets), ignore_index, ref);
  B200TP_CUDA_OK(cudaGetLastError());
  return B200TP_OK;
}

int ce_split_fwd_grad(const void* h3, const void* w3, int64_t n, int d, int64_t width, int64_t vocab_id0,
                      const int64_t* targets, int64_t ignore_index, const float* ref, int splits, float* pm, float* ps,
                      float* pt, void* g3, int ldg, const int* bad, int* flag, cudaStream_t stream, int* status) {
  SplitLogitsParams p{};
  p.vocab_id0 = vocab_id0;
  p.splits = splits;
  p.targets = reinterpret_cast<const long long*>(targets);
  p.ignore_index = ignore_index;
  p.pm = pm;
  p.ps = ps;
  p.pt = pt;
  p.g = static_cast<__nv_bfloat16*>(g3);
  p.ldg = ldg;
  p.ref = ref;
  p.bad = bad;
  p.flag = flag;
  p.status = status;
  return launch_logits<SPLIT_FWD_GRAD>(h3, w3, n, d, width, p, stream);
}

int ce_split_finish(const float* acc, int shares, const float* ref, int* flags, const float* w, int64_t n, int d,
                    int64_t v, const int64_t* targets, int64_t ignore_index, const float* lse, const float* tgt,
                    const float* ct, float* out, cudaStream_t stream) {
  const dim3 grid(static_cast<unsigned>(n), static_cast<unsigned>(ceil_div(d, 256)));
  split_finish_kernel<<<grid, 256, 0, stream>>>(acc, shares, ref, flags, w, static_cast<int>(n), d, v,
                                                reinterpret_cast<const long long*>(targets), ignore_index, lse, tgt,
                                                ct, out);
  B200TP_CUDA_OK(cudaGetLastError());
  return B200TP_OK;
}

// Shares of the d_hidden contraction: the fewest that keep the busiest CTA's work (k blocks, plus about two per unit
// for its prologue and epilogue) lowest, so that few tiles still fill the chip (2048 x 1024 has 64).
int ce_split_dh_shares(int64_t n, int d, int64_t width) {
  const bool pair = split_pair(n);
  const int64_t tiles = ceil_div(n, pair ? 2 * BM : BM) * ceil_div(d, BN), kblocks = ceil_div(width, BK),
                ctas = pair ? sm_count() / 2 : sm_count();
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int ks = 1; ks <= std::min<int64_t>(64, kblocks) && (ks == 1 || tiles * ks <= 4 * ctas); ++ks) {
    const int64_t cost = ceil_div(tiles * ks, ctas) * (ceil_div(kblocks, ks) + 2);
    if (cost < best_cost) {
      best_cost = cost;
      best = ks;
    }
  }
  return best;
}

int ce_split_dh(const void* g3, int ldg, const void* w3, int64_t n, int d, int64_t width, int ksplit, float* out,
                int keep, cudaStream_t stream, int* status, const SplitGuard& guard) {
  int rc = configure();
  if (rc) return rc;
  SplitDhParams p{};
  p.guard = guard;
  p.n_rows = static_cast<int>(n);
  p.d_cols = d;
  p.kblocks = static_cast<int>(ceil_div(width, BK));
  const bool pair = split_pair(n);
  p.num_rb = static_cast<int>(ceil_div(n, pair ? 2 * BM : BM));
  p.num_nt = static_cast<int>(ceil_div(d, BN));
  p.ksplit = ksplit;
  p.out = out;
  p.keep = keep;
  p.status = status;
  CUtensorMap tmap_g, tmap_w;
  rc = plane_map(&tmap_g, g3, n, ldg, ldg, BM);
  if (rc) return rc;
  rc = plane_map(&tmap_w, w3, width, d, d, BK);
  if (rc) return rc;
  return launch_units(pair ? split_dh_kernel<true> : split_dh_kernel<false>, SPLIT_THREADS, pair,
                      static_cast<long long>(p.num_rb) * p.num_nt * ksplit, stream, tmap_g, tmap_w, p, guard.any());
}

int ce_split_sum(const float* acc, int shares, int64_t count, float* out, int keep, const SplitGuard& guard,
                 cudaStream_t stream) {
  B200TP_CUDA_OK(launch_kernel(guard.any(), share_sum_kernel, dim3(static_cast<unsigned>(ceil_div(count, 256))),
                               dim3(256), 0, stream, acc, shares, count, out, keep, guard));
  return B200TP_OK;
}

}  // namespace b200tp
