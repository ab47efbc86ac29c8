// Fused linear cross-entropy on the Blackwell tensor cores (tcgen05 / TMEM / TMA).
//
// Four kernels:
//
//  ce_logits_kernel<FWD>    Z = H W^T tile by tile (128 rows x 256 vocab columns, K = D),
//                           accumulators double-buffered in tensor memory; the epilogue
//                           warps fold each tile into a per-row online (max, sum-exp,
//                           target-logit) and write ONE partial triple per (row, vocab
//                           split).  The logits never leave the SM.
//  ce_logits_kernel<BWD_G>  same main loop over one vocab chunk; the epilogue forms
//                           g = (exp(z - lse) - onehot) * cotangent, rounds it to bf16 and
//                           stores it to a (N, chunk) scratch matrix.
//  ce_dh_kernel             dH(128 x 256 tile) (+)= G(N, chunk) W[chunk, :] with the vocab
//                           axis as the contraction: A = G is K-major, B = W is read as an
//                           MN-major operand straight from its row-major storage.
//  ce_dw_kernel             trainable heads: dW_chunk(128 x 256 tile) = G^T hidden with the token
//                           axis as the contraction; both operands read MN-major from their
//                           row-major storage, written once (each vocab row has one chunk).
//
// Work split: persistent CTAs (one per SM), static round-robin over work units.  Roles in
// a CTA of 192 threads: warp 0 = TMA producer, warp 1 = MMA issuer (also owns the TMEM
// allocation), warps 2..5 = epilogue (one TMEM lane quadrant each).
//
// PAIR instantiations (dense heads): a cluster of two CTAs works on 256 rows.  Each holds its 128 rows of A, half of
// the weight tile and its rows' accumulators; CTA 0 issues one `cta_group::2` MMA for both, whose commits arrive in
// both.  Both CTAs' copies complete on CTA 0's full barriers; accumulators are handed back to it across the cluster.
// Training step of 8192 x 4096 x 151936: 18.2 -> 16.6 ms, 1000 rows 2.30 -> 2.05 ms, a trained head of 4096 x 1024 x
// 151936 4.94 -> 4.62 ms.
//
// 4-bit affine group-64 heads (QUANT instantiations of ce_logits_kernel and ce_dh_kernel): the
// weight operand is never materialised in global memory.  The TMA producer copies the packed codes
// of each stage's weight tile into a small shared-memory ring (8 KiB per stage) beside the other
// operand; eight more warps (256 threads, one (vocab row, 64-column group) each per stage) read
// their 32 bytes of codes from there and the group's scale / bias from global memory (prefetched in
// registers), expand them (dequant.cuh) and write the bf16 tile into the stage's swizzled slot,
// where the MMA reads it exactly as it reads a TMA-loaded dense tile.
// core/kernel/source.py:199-340 (K2) and core/kernel/launch.py:336-373.
//
// Replaces core/kernel/source.py:25-166 (forward MSL), :475-611 (dH MMA backward), :659-702 (dW)
// and the chunked backward of core/chunked.py:52-90 of the reference.
#include "linear_ce_tc.h"

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "dequant.cuh"
#include "linear_ce_pipe.cuh"

namespace b200tp {

namespace {

constexpr int THREADS = 192;
constexpr int THREADS_Q = THREADS + 32 * DQ_WARPS;
constexpr int DQ_FULL_ARRIVALS = DQ_WARPS;        // one arrival per dequantising warp on a stage's full barrier

enum { MODE_FWD = 0, MODE_BWD_G = 1, MODE_FWD_GRAD = 2 };

// MODE_FWD_GRAD: exponents (log2 units, relative to the row's reference) above this raise the overflow flag.
// Sums of 2^27 terms of 2^100 stay below the largest fp32, and 2^100 = e^69.
constexpr float kRefHeadroom = 100.f;

constexpr int kMostAccumulated = 16384;   // vocab rows per accumulation of d_hidden (see ce_dh_kernel)

__device__ __forceinline__ bool guard_skips(const LaunchGuard& g) {
  return g.flag != nullptr && (*g.flag != 0) != (g.run_if_set != 0);
}

// 32 columns of a row of g as whole sectors.  With 16-byte stores every sector was written in two halves, and at
// D = 1024 the L2 took them no faster than the tensor cores made them (15194 vocab rows x 4096 rows: 115 -> 90 us).
__device__ __forceinline__ void store_g(__nv_bfloat16* dst, const uint32_t (&v)[16]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    st_global_32b(dst + h * 16, {v[8 * h], v[8 * h + 1], v[8 * h + 2], v[8 * h + 3], v[8 * h + 4], v[8 * h + 5],
                                 v[8 * h + 6], v[8 * h + 7]});
}

struct LogitsParams {
  int n_rows;            // N
  int k_dim;             // D
  int vrow0, vrow1;      // rows of the weight matrix (tensor map coordinates) this launch covers
  long long vocab_id0;   // global vocab id of tensor-map row 0
  int num_rb, num_vt, splits;
  const long long* targets;
  long long ignore_index;
  // FWD: partial triples, [split][N] each
  float* pm;
  float* ps;
  float* pt;
  // BWD_G
  const float* lse;
  const float* ct;
  __nv_bfloat16* g;         // BWD_G, FWD_GRAD
  int ldg;
  // FWD_GRAD
  const float* ref2;        // per row: reference of the exponentials, log2 units
  int* overflow;            // set to 1 when some logit exceeds its (not ignored) row's reference by kRefHeadroom
  LaunchGuard guard;
  int* status;
  // QUANT: the packed head (rows indexed like the tensor map of a dense weight would be)
  const uint32_t* wq;
  const void* scales;
  const void* biases;
  int qp_f32;
  int qvec;              // bf16 scales / biases, D % 512 == 0, 16-byte aligned: eight groups per load
};

struct DhParams {
  int n_rows;     // N
  int d_cols;     // D
  int k_total;    // contraction length (multiple of 64; columns of G)
  int wrow0;      // first vocab row of this chunk in the weight tensor map
  int num_rb, num_nt;
  const float* acc_in;   // fp32 (N, D) partial sums to add, or nullptr
  float* acc_out;        // fp32 (N, D) destination, or nullptr
  __nv_bfloat16* out_bf16;  // bf16 (N, D) destination, or nullptr
  LaunchGuard guard;
  int* status;
  int tile0, tile1;         // units [tile0, tile1) are computed by this launch; unit = split * tiles + tile
  int ksplit;               // shares of the contraction: share s adds into acc + s * split_stride (ksplit 1: no shares)
  long long split_stride;
  int seg_kb;               // most k blocks of one accumulation; a unit's parts are added in acc_out
  int wide;                 // acc_in and acc_out are 32-byte aligned
  // QUANT: the packed head
  const uint32_t* wq;
  const void* scales;
  const void* biases;
  int qp_f32;
  int w_rows;               // vocab rows of the head (rows at or past it read as zero)
};

struct DwParams {
  int n_rows;     // N tokens = contraction length
  int d_cols;     // D
  int v_rows;     // vocab rows of this chunk (rows of the d_weight block written)
  int num_mt, num_nt;
  __nv_bfloat16* out;   // (v_rows, D) bf16 block of d_weight, row stride D
  int* status;
};

// A dequantising warp's part of "the stage's weight tile is written": every thread fences its own
// generic-proxy stores against the tensor core's async proxy, then one lane arrives for the warp.
__device__ __forceinline__ void dq_signal_written(uint64_t* full_bar, int lane) {
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) mbar_arrive(full_bar);
}

// -----------------------------------------------------------------------------------------
// Z = H W^T with fused epilogues
// -----------------------------------------------------------------------------------------
// Walk over the (work unit, vocab tile, k block) sequence of one persistent CTA, in the order the
// producer, the MMA issuer and the dequantising warps all follow.
struct LogitsWalk {
  int u, vt, vt1, kb;
  __device__ __forceinline__ void set_unit(const LogitsParams& p) {
    const int split = u / p.num_rb;
    vt = static_cast<int>(static_cast<long long>(split) * p.num_vt / p.splits);
    vt1 = static_cast<int>(static_cast<long long>(split + 1) * p.num_vt / p.splits);
    kb = 0;
  }
  __device__ __forceinline__ void init(const LogitsParams& p, int total_units) {
    u = blockIdx.x;
    if (u < total_units) set_unit(p);
  }
  __device__ __forceinline__ void next(const LogitsParams& p, int total_units, int kblocks) {
    if (++kb < kblocks) return;
    kb = 0;
    if (++vt < vt1) return;
    u += gridDim.x;
    if (u < total_units) set_unit(p);
  }
};

template <int MODE, bool QUANT, bool PAIR = false>
__global__ void __launch_bounds__(QUANT ? THREADS_Q : THREADS, 1)
ce_logits_kernel(const __grid_constant__ CUtensorMap tmap_h, const __grid_constant__ CUtensorMap tmap_w,
                 const LogitsParams p) {
  if (guard_skips(p.guard)) return;
  extern __shared__ uint8_t smem_raw[];
  const SmemView sm = carve_smem(smem_raw, QUANT, PAIR);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // provably warp-uniform
  const int lane = threadIdx.x & 31;
  const uint32_t tmem_base = cta_setup(sm, warp, QUANT ? 1 + DQ_FULL_ARRIVALS : 1, PAIR ? 8 : 4, PAIR);
  // a pair's units are 256 rows: CTA `rank` of it has rows [128 rank, +128) and that half of each weight tile
  constexpr uint32_t kStages = PAIR ? PAIR_STAGES : STAGES;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0;
  const int unit0 = PAIR ? blockIdx.x >> 1 : blockIdx.x, unit_step = PAIR ? gridDim.x >> 1 : gridDim.x;
  auto block_row = [&](int rb) { return (PAIR ? rb * 2 + static_cast<int>(rank) : rb) * BM; };

  const int total_units = p.num_rb * p.splits;
  const int kblocks = (p.k_dim + BK - 1) / BK;

  if (QUANT && warp >= THREADS / 32) {
    // ------------------------------ dequantising warps ------------------------------
    // Thread t owns row t of the stage's 256-row weight tile: one group of 64 codes per k block.  A code
    // tile (256 rows x 64 bytes, 64-byte swizzle) holds two k blocks.  Scales / biases: eight groups per
    // 16-byte load, one load ahead (`qvec`: bf16 parameters, D % 512 == 0), else one load per stage.
    const int trow = threadIdx.x - THREADS;
    const int groups = p.k_dim / 64;
    const bool qp_f32 = p.qp_f32 != 0, qvec = p.qvec != 0;
    const uint32_t swz = static_cast<uint32_t>((trow >> 1) & 3);
    LogitsWalk cur;
    cur.init(p, total_units);
    auto row_of = [&](const LogitsWalk& w) { return p.vrow0 + w.vt * BN + trow; };
    auto load8 = [&](const LogitsWalk& w, uint4& s8, uint4& b8) {
      const int row = row_of(w);
      if (row < p.vrow1) {
        const long long idx = static_cast<long long>(row) * groups + (w.kb & ~7);
        s8 = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p.scales) + idx));
        b8 = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p.biases) + idx));
      }
    };
    auto pick = [](const uint4& v, int k) -> uint32_t {   // k-th bf16 of eight
      const uint32_t lo = (k & 4) ? v.z : v.x, hi = (k & 4) ? v.w : v.y;
      return (((k & 2) ? hi : lo) >> ((k & 1) * 16)) & 0xFFFFu;
    };
    uint4 s_cur = make_uint4(0, 0, 0, 0), b_cur = s_cur, s_nxt = s_cur, b_nxt = s_cur;
    LogitsWalk pre = cur;      // start of the eight-block span after the current one
    if (qvec && cur.u < total_units) {
      load8(cur, s_nxt, b_nxt);
    }
    uint32_t it = 0, ci = 0;
    bool ok = true;
#pragma unroll 1
    for (; cur.u < total_units && ok; cur.next(p, total_units, kblocks), ++it) {
      const int row = row_of(cur);
      const bool valid = row < p.vrow1;
      uint32_t sc, bi;
      if (qvec) {
        if ((cur.kb & 7) == 0) {
          s_cur = s_nxt;
          b_cur = b_nxt;
          // the span after this one: eight k blocks on, or the next tile / unit (kblocks % 8 == 0 here)
          pre = cur;
          for (int k = 0; k < 8 && pre.u < total_units; ++k) pre.next(p, total_units, kblocks);
          if (pre.u < total_units) load8(pre, s_nxt, b_nxt);
        }
        sc = pick(s_cur, cur.kb & 7);
        bi = pick(b_cur, cur.kb & 7);
      } else {
        sc = bi = 0;
        if (valid) {
          sc = dq_load_param(p.scales, static_cast<long long>(row) * groups + cur.kb, qp_f32);
          bi = dq_load_param(p.biases, static_cast<long long>(row) * groups + cur.kb, qp_f32);
        }
      }
      // ---- this row's 32 bytes of codes from the TMA-filled tile (two k blocks per tile)
      const int half = cur.kb & 1;
      const uint32_t cs = ci % CODE_SLOTS_LOGITS;
      if (half == 0 && !mbar_wait_warp(&sm.cfull[cs], (ci / CODE_SLOTS_LOGITS) & 1, sm.abort_flag)) {
        if (lane == 0) raise_abort(sm, p.status, kDevTimeoutProducer);
        ok = false;
        break;
      }
      const uint32_t crow = smem_u32(sm.codes) + cs * (CODE_BYTES / CODE_SLOTS_LOGITS) + trow * 64;
      const uint4 lo = lds128(crow + (((2 * half) ^ swz) << 4));
      const uint4 hi = lds128(crow + (((2 * half + 1) ^ swz) << 4));
      const bool release_codes = half == 1 || cur.kb + 1 == kblocks;   // last k block served by this tile
      const int s = it % STAGES;
      if (!mbar_wait_warp(&sm.empty[s], ((it / STAGES) & 1) ^ 1, sm.abort_flag)) {
        if (lane == 0) raise_abort(sm, p.status, kDevTimeoutProducer);
        ok = false;
        break;
      }
      dq_store_row(smem_u32(sm.b(s)) + trow * 128, trow & 7, lo, hi, sc, bi, qp_f32, valid);
      dq_signal_written(&sm.full[s], lane);
      // The code slot goes back to the producer only now, after `lo` / `hi` have been consumed: an
      // mbarrier arrive issued right behind the shared-memory loads can be performed before those loads
      // have read their data when the load / store unit is backed up (observed: with the backward's
      // epilogue streaming G to global memory, the producer's refill overwrote rows a warp had not read yet).
      if (release_codes) {
        if (lane == 0) mbar_arrive(&sm.cempty[cs]);
        ++ci;
      }
    }
  } else if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      tma_prefetch_desc(&tmap_h);
      tma_prefetch_desc(&tmap_w);
      uint32_t it = 0, ci = 0;
      bool ok = true;
      for (int u = unit0; u < total_units && ok; u += unit_step) {
        const int split = u / p.num_rb;
        const int rb = u - split * p.num_rb;
        const int vt0 = static_cast<int>(static_cast<long long>(split) * p.num_vt / p.splits);
        const int vt1 = static_cast<int>(static_cast<long long>(split + 1) * p.num_vt / p.splits);
        for (int vt = vt0; vt < vt1 && ok; ++vt) {
          for (int kb = 0; kb < kblocks; ++kb, ++it) {
            const int s = it % kStages;
            if (!mbar_wait(&sm.empty[s], ((it / kStages) & 1) ^ 1, sm.abort_flag)) {
              raise_abort(sm, p.status, kDevTimeoutProducer);
              ok = false;
              break;
            }
            if (QUANT && (kb & 1) == 0) {
              // packed codes of k blocks kb, kb + 1 for the tile's 256 rows (tmap_w is the uint32 map here)
              const uint32_t cs = ci % CODE_SLOTS_LOGITS;
              if (!mbar_wait(&sm.cempty[cs], ((ci / CODE_SLOTS_LOGITS) & 1) ^ 1, sm.abort_flag)) {
                raise_abort(sm, p.status, kDevTimeoutProducer);
                ok = false;
                break;
              }
              mbar_arrive_expect_tx(&sm.cfull[cs], CODE_BYTES / CODE_SLOTS_LOGITS);
              tma_load_2d(sm.codes + cs * (CODE_BYTES / CODE_SLOTS_LOGITS), &tmap_w, &sm.cfull[cs], kb * 8,
                          p.vrow0 + vt * BN);
              ++ci;
            }
            if (PAIR) {   // both CTAs' copies complete on CTA 0's barrier
              if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2 * PAIR_STAGE_BYTES);
              const uint32_t bar = map_to_rank(&sm.full[s], 0);
              tma_load_2d_pair(sm.a(s), &tmap_h, bar, kb * BK, block_row(rb));
              tma_load_2d_pair(sm.b(s), &tmap_w, bar, kb * BK, p.vrow0 + vt * BN + static_cast<int>(rank) * (BN / 2));
              continue;
            }
            mbar_arrive_expect_tx(&sm.full[s], QUANT ? A_BYTES : STAGE_BYTES);
            tma_load_2d(sm.a(s), &tmap_h, &sm.full[s], kb * BK, rb * BM);
            if (!QUANT) tma_load_2d(sm.b(s), &tmap_w, &sm.full[s], kb * BK, p.vrow0 + vt * BN);
          }
        }
      }
      // the other CTA's commits land here: none may be on its way when this one leaves
      if (PAIR && ok)
        for (uint32_t j = it > kStages ? it - kStages : 0; j < it; ++j)
          mbar_wait(&sm.empty[j % kStages], (j / kStages) & 1, sm.abort_flag);
      if (!ok) {
        producer_drain(sm, it);
        if (QUANT)
          for (uint32_t c = ci > CODE_SLOTS_LOGITS ? ci - CODE_SLOTS_LOGITS : 0; c < ci; ++c)
            mbar_wait_drain(&sm.cfull[c % CODE_SLOTS_LOGITS], (c / CODE_SLOTS_LOGITS) & 1);
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
    // ------------------------------ MMA issuer ------------------------------
    // The whole warp runs the loop (its address arithmetic stays warp-uniform and cheap: this warp
    // shares an instruction scheduler with epilogue warps) and one elected lane issues.
    constexpr uint32_t idesc = make_idesc_bf16(PAIR ? 2 * BM : BM, BN, 0, 0);
    constexpr uint32_t dhi = desc_hi_sw128(1024);
    uint32_t it = 0, tile = 0;
    bool ok = true;
    for (int u = unit0; u < total_units && ok; u += unit_step) {
      const int split = u / p.num_rb;
      const int vt0 = static_cast<int>(static_cast<long long>(split) * p.num_vt / p.splits);
      const int vt1 = static_cast<int>(static_cast<long long>(split + 1) * p.num_vt / p.splits);
      for (int vt = vt0; vt < vt1 && ok; ++vt, ++tile) {
        const uint32_t as = tile & 1;
        if (!mbar_wait_warp(&sm.tempty[as], ((tile >> 1) & 1) ^ 1, sm.abort_flag)) {
          if (lane == 0) raise_abort(sm, p.status, kDevTimeoutMma);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + as * BN;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % kStages;
          if (!mbar_wait_warp(&sm.full[s], (it / kStages) & 1, sm.abort_flag)) {
            if (lane == 0) raise_abort(sm, p.status, kDevTimeoutMma);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t a_lo = desc_lo(smem_u32(sm.a(s)), 16);
          const uint32_t b_lo = desc_lo(smem_u32(sm.b(s)), 16);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma<PAIR>(d_tmem, a_lo + k * 2, dhi, b_lo + k * 2, dhi, idesc, (kb | k) != 0 ? 1u : 0u);
            commit<PAIR>(&sm.empty[s]);  // frees the stage once these MMAs have read it
          }
          __syncwarp();
        }
        if (ok && elect_one()) commit<PAIR>(&sm.tfull[as]);
        __syncwarp();
      }
    }
    }
  } else {
    // ------------------------------ epilogue warps ------------------------------
    const int quad = warp & 3;  // TMEM lane quadrant this warp may read
    const int row_in_tile = quad * 32 + lane;
    uint32_t tile = 0;
    bool ok = true;
    for (int u = unit0; u < total_units && ok; u += unit_step) {
      const int split = u / p.num_rb;
      const int rb = u - split * p.num_rb;
      const int vt0 = static_cast<int>(static_cast<long long>(split) * p.num_vt / p.splits);
      const int vt1 = static_cast<int>(static_cast<long long>(split + 1) * p.num_vt / p.splits);
      const int row = block_row(rb) + row_in_tile;
      const bool row_ok = row < p.n_rows;
      long long target = p.ignore_index;
      if (row_ok) target = p.targets[row];
      const bool tvalid = row_ok && target != p.ignore_index;

      float run_m = -INFINITY, run_s = 0.f, run_t = 0.f;  // FWD, FWD_GRAD state (log2 domain for m)
      bool over = false;                                  // FWD_GRAD: some exponent left the reference's range
      float lse2 = 0.f, ctv = 0.f;                        // BWD_G state
      if (MODE == MODE_BWD_G && row_ok) {
        lse2 = p.lse[row] * kLog2e;
        ctv = tvalid ? p.ct[row] : 0.f;
      }
      if (MODE == MODE_FWD_GRAD) run_m = row_ok ? p.ref2[row] : 0.f;

      for (int vt = vt0; vt < vt1 && ok; ++vt, ++tile) {
        const uint32_t as = tile & 1;
        if (!mbar_wait_warp(&sm.tfull[as], (tile >> 1) & 1, sm.abort_flag)) {
          raise_abort(sm, p.status, kDevTimeoutEpilogue);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const int tile_row0 = p.vrow0 + vt * BN;                      // tensor-map row of column 0
        const int ncols = min(BN, p.vrow1 - tile_row0);               // valid columns in this tile
        long long trel = -1;
        if (tvalid) trel = target - (p.vocab_id0 + tile_row0);
        const int tcol = (trel >= 0 && trel < ncols) ? static_cast<int>(trel) : -1;
        const uint32_t taddr0 = tmem_base + as * BN + (static_cast<uint32_t>(quad * 32) << 16);

#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          if (MODE == MODE_FWD && c * 32 >= ncols) break;
          uint32_t r[32];
          tmem_ld_x32(taddr0 + c * 32, r);
          tmem_wait_ld();
          tmem_regs_ready(r);
          const int cvalid = ncols - c * 32;  // columns of this chunk that exist (may exceed 32)
          if (MODE == MODE_FWD) {
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              x[j] = __uint_as_float(r[j]);
              if (j >= cvalid) x[j] = -INFINITY;
            }
            if (tcol >= 0 && (tcol >> 5) == c) {
              const int tj = tcol & 31;
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (j == tj) run_t = x[j];
            }
            float cm = x[0];
#pragma unroll
            for (int j = 1; j < 32; ++j) cm = fmaxf(cm, x[j]);
            // cm is finite: column c*32 exists (checked above) and logits are finite.
            const float new_m = fmaxf(run_m, cm * kLog2e);
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < 32; ++j) acc += fast_exp2(fmaf(x[j], kLog2e, -new_m));
            run_s = run_s * fast_exp2(run_m - new_m) + acc;
            run_m = new_m;
          } else if (MODE == MODE_FWD_GRAD) {
            // One exponential per logit serves both the row sum and the unnormalised gradient: relative to a
            // reference fixed before the launch, e = exp(z - ref) needs neither the row maximum nor the final
            // log-sum-exp, and the row's factor exp(ref - lse) is applied to d_hidden afterwards.
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              x[j] = __uint_as_float(r[j]);
              if (j >= cvalid) x[j] = -INFINITY;
            }
            const int tj = (tcol >= 0 && (tcol >> 5) == c) ? (tcol & 31) : -1;
            float xm = -INFINITY;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (j == tj) run_t = x[j];
              x[j] = fmaf(x[j], kLog2e, -run_m);
              xm = fmaxf(xm, x[j]);
            }
            if (xm > kRefHeadroom) {   // rare: move this thread's own sum to a larger reference; g is void then
              over = over || tvalid;   // (an ignored row's g is zero, and its reference an arbitrary logit)
              run_s *= fast_exp2(-xm);
              run_m += xm;
#pragma unroll
              for (int j = 0; j < 32; ++j) x[j] -= xm;
            }
            float acc4[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t packed[16];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              float e0 = fast_exp2(x[j]), e1 = fast_exp2(x[j + 1]);
              acc4[(j >> 1) & 3] += e0 + e1;
              // the target's own term p - 1 is added to d_hidden in fp32 later: rounding p to bf16 here would
              // lose it on rows whose target is nearly certain
              if (j == tj) e0 = 0.f;
              if (j + 1 == tj) e1 = 0.f;
              packed[j >> 1] = tvalid ? pack_bf16x2(e0, e1) : 0u;
            }
            run_s += (acc4[0] + acc4[1]) + (acc4[2] + acc4[3]);
            if (row_ok) {
              store_g(p.g + static_cast<size_t>(row) * p.ldg + (vt * BN + c * 32), packed);
            }
          } else {
            uint32_t packed[16];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              float g0 = fast_exp2(fmaf(__uint_as_float(r[j]), kLog2e, -lse2));
              float g1 = fast_exp2(fmaf(__uint_as_float(r[j + 1]), kLog2e, -lse2));
              if (c * 32 + j == tcol) g0 -= 1.f;
              if (c * 32 + j + 1 == tcol) g1 -= 1.f;
              g0 = (j < cvalid) ? g0 * ctv : 0.f;
              g1 = (j + 1 < cvalid) ? g1 * ctv : 0.f;
              packed[j >> 1] = pack_bf16x2(g0, g1);
            }
            if (row_ok) {
              store_g(p.g + static_cast<size_t>(row) * p.ldg + vt * BN + c * 32, packed);
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) release_acc<PAIR>(&sm.tempty[as]);
      }

      if (MODE == MODE_FWD_GRAD && over) *p.overflow = 1;
      if ((MODE == MODE_FWD || MODE == MODE_FWD_GRAD) && ok && row_ok) {
        const size_t o = static_cast<size_t>(split) * p.n_rows + row;
        p.pm[o] = run_m * kLn2;  // back to natural-log units
        p.ps[o] = run_s;
        p.pt[o] = run_t;
      }
    }
  }
  cta_teardown(sm, warp, tmem_base, PAIR);
}

// -----------------------------------------------------------------------------------------
// dH (+)= G W_chunk
// -----------------------------------------------------------------------------------------
// Tiles are numbered row-block-major (t = rb * num_nt + nt), so the row blocks of d_hidden complete
// in order as the persistent CTAs advance, and a launch can be given a sub-range [tile0, tile1) of
// them: vocab-sharded callers run the last chunk in a few such launches and start reducing the
// finished rows across ranks while the later ones are still being computed.
//
// The tensor core rounds its accumulator towards zero at every step of 16 terms, an error that is biased and grows with
// the steps.  A chunk wider than kMostAccumulated vocab rows is therefore accumulated in parts, which the epilogue adds in
// acc_out with round-to-nearest while the next part runs.  (One large row and 76000 small ones: the sum 1.6e-4 of itself
// too small in one part, 3.2e-5 in five; 1000 x 4096 x 151936, d_hidden of a chunk 444 -> 453 us with whole sectors read
// and written, 465 with halves: what the epilogue moves through L1 is taken from the operands.)
template <bool QUANT, bool PAIR = false>
__global__ void __launch_bounds__(QUANT ? THREADS_Q : THREADS, 1)
ce_dh_kernel(const __grid_constant__ CUtensorMap tmap_g, const __grid_constant__ CUtensorMap tmap_w,
             const DhParams p) {
  if (guard_skips(p.guard)) return;
  extern __shared__ uint8_t smem_raw[];
  const SmemView sm = carve_smem(smem_raw, QUANT, PAIR);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // provably warp-uniform
  const int lane = threadIdx.x & 31;
  const uint32_t tmem_base = cta_setup(sm, warp, QUANT ? 1 + DQ_FULL_ARRIVALS : 1, PAIR ? 8 : 4, PAIR);
  constexpr uint32_t kStages = PAIR ? PAIR_STAGES : STAGES;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0;
  const int unit_step = PAIR ? gridDim.x >> 1 : gridDim.x;
  auto block_row = [&](int rb) { return (PAIR ? rb * 2 + static_cast<int>(rank) : rb) * BM; };

  const int total_tiles = p.tile1;
  const int first_tile = p.tile0 + (PAIR ? blockIdx.x >> 1 : blockIdx.x);
  const int kblocks = p.k_total / BK;
  const int tiles = p.num_rb * p.num_nt;
  // k blocks [kb0, kb1) of a unit; a share can be empty when a later chunk is narrower than the first
  auto k_range = [&](int split, int& kb0, int& kb1) {
    kb0 = static_cast<int>(static_cast<long long>(split) * kblocks / p.ksplit);
    kb1 = static_cast<int>(static_cast<long long>(split + 1) * kblocks / p.ksplit);
  };
  auto num_segs = [&](int kb0, int kb1) { return (kb1 - kb0 + p.seg_kb - 1) / p.seg_kb; };

  if (QUANT && warp >= THREADS / 32) {
    // ------------------------------ dequantising warps ------------------------------
    // Stage tile: 64 vocab rows (k) x 256 hidden columns as four [64 k][64 n] boxes = four groups per
    // vocab row.  Warp w, lane l: vocab row 8 w + (l & 7), box l >> 3 -- eight consecutive rows per
    // quarter-warp, so the reads of the code tile (64 rows x 128 B, 128-byte swizzle), the writes of the
    // operand tile and the scale / bias loads (four consecutive values per row) are all conflict-free /
    // coalesced.  Scales and biases are prefetched three stages ahead in registers.
    const int dw = warp - THREADS / 32;
    const int krow = dw * 8 + (lane & 7), box = lane >> 3;
    const int groups = p.d_cols / 64;
    const bool qp_f32 = p.qp_f32 != 0;
    constexpr int PF = 3;
    int t_cur = first_tile, kb_cur = 0, t_pre = first_tile, kb_pre = 0;
    uint32_t sc_ring[PF], bi_ring[PF];
    auto coords = [&](int t, int kb, int& row, int& col) {
      const int nt = t % p.num_nt;
      row = p.wrow0 + kb * BK + krow;
      col = nt * BN + box * 64;
    };
    auto fetch = [&](uint32_t& sc, uint32_t& bi, int t, int kb) {
      int row, col;
      coords(t, kb, row, col);
      sc = bi = 0;
      if (row < p.w_rows && col < p.d_cols) {
        const long long idx = static_cast<long long>(row) * groups + col / 64;
        sc = dq_load_param(p.scales, idx, qp_f32);
        bi = dq_load_param(p.biases, idx, qp_f32);
      }
    };
    auto advance = [&](int& t, int& kb) {
      if (++kb == kblocks) {
        kb = 0;
        t += gridDim.x;
      }
    };
#pragma unroll
    for (int j = 0; j < PF; ++j) {
      if (t_pre < total_tiles) {
        fetch(sc_ring[j], bi_ring[j], t_pre, kb_pre);
        advance(t_pre, kb_pre);
      }
    }
    uint32_t it = 0;
    bool ok = true;
#pragma unroll 1
    while (t_cur < total_tiles && ok) {
#pragma unroll
      for (int j = 0; j < PF; ++j) {
        if (t_cur >= total_tiles || !ok) break;
        const uint32_t sc = sc_ring[j], bi = bi_ring[j];
        int row, col;
        coords(t_cur, kb_cur, row, col);
        const bool valid = row < p.w_rows && col < p.d_cols;
        if (t_pre < total_tiles) {
          fetch(sc_ring[j], bi_ring[j], t_pre, kb_pre);
          advance(t_pre, kb_pre);
        }
        const uint32_t cs = it % CODE_SLOTS_DH;
        if (!mbar_wait_warp(&sm.cfull[cs], (it / CODE_SLOTS_DH) & 1, sm.abort_flag)) {
          if (lane == 0) raise_abort(sm, p.status, kDevTimeoutProducer);
          ok = false;
          break;
        }
        const uint32_t crow = smem_u32(sm.codes) + cs * (CODE_BYTES / CODE_SLOTS_DH) + krow * 128;
        const uint4 lo = lds128(crow + (((2 * box) ^ (krow & 7)) << 4));
        const uint4 hi = lds128(crow + (((2 * box + 1) ^ (krow & 7)) << 4));
        const int s = it % STAGES;
        if (!mbar_wait_warp(&sm.empty[s], ((it / STAGES) & 1) ^ 1, sm.abort_flag)) {
          if (lane == 0) raise_abort(sm, p.status, kDevTimeoutProducer);
          ok = false;
          break;
        }
        dq_store_row(smem_u32(sm.b(s)) + box * (64 * BK * 2) + krow * 128, krow & 7, lo, hi, sc, bi, qp_f32, valid);
        dq_signal_written(&sm.full[s], lane);
        if (lane == 0) mbar_arrive(&sm.cempty[cs]);   // after the codes were consumed (see ce_logits_kernel)
        ++it;
        advance(t_cur, kb_cur);
      }
    }
  } else if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_g);
      tma_prefetch_desc(&tmap_w);
      uint32_t it = 0;
      bool ok = true;
      for (int u = first_tile; u < total_tiles && ok; u += unit_step) {
        const int split = u / tiles, t = u - split * tiles;
        const int rb = t / p.num_nt;
        const int nt = t - rb * p.num_nt;
        int kb0, kb1;
        k_range(split, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % kStages;
          if (!mbar_wait(&sm.empty[s], ((it / kStages) & 1) ^ 1, sm.abort_flag)) {
            raise_abort(sm, p.status, kDevTimeoutProducer);
            ok = false;
            break;
          }
          if (QUANT) {
            // packed codes of the stage's 64 vocab rows x 256 hidden columns (tmap_w is the uint32 map here)
            const uint32_t cs = it % CODE_SLOTS_DH;
            if (!mbar_wait(&sm.cempty[cs], ((it / CODE_SLOTS_DH) & 1) ^ 1, sm.abort_flag)) {
              raise_abort(sm, p.status, kDevTimeoutProducer);
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&sm.cfull[cs], CODE_BYTES / CODE_SLOTS_DH);
            tma_load_2d(sm.codes + cs * (CODE_BYTES / CODE_SLOTS_DH), &tmap_w, &sm.cfull[cs], nt * (BN / 8),
                        p.wrow0 + kb * BK);
          }
          if (PAIR) {
            if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2 * PAIR_STAGE_BYTES);
            const uint32_t bar = map_to_rank(&sm.full[s], 0);
            tma_load_2d_pair(sm.a(s), &tmap_g, bar, kb * BK, block_row(rb));
#pragma unroll
            for (int j = 0; j < BN / 128; ++j)
              tma_load_2d_pair(sm.b(s) + j * (64 * BK * 2), &tmap_w, bar,
                               nt * BN + static_cast<int>(rank) * (BN / 2) + j * 64, p.wrow0 + kb * BK);
            continue;
          }
          mbar_arrive_expect_tx(&sm.full[s], QUANT ? A_BYTES : STAGE_BYTES);
          tma_load_2d(sm.a(s), &tmap_g, &sm.full[s], kb * BK, rb * BM);
          // B tile: 64 vocab rows (K) x 256 hidden columns (N) as four [64 k][64 n] boxes.
          if (!QUANT) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_2d(sm.b(s) + j * (64 * BK * 2), &tmap_w, &sm.full[s], nt * BN + j * 64, p.wrow0 + kb * BK);
          }
        }
      }
      // the other CTA's commits land here: none may be on its way when this one leaves
      if (PAIR && ok)
        for (uint32_t j = it > kStages ? it - kStages : 0; j < it; ++j)
          mbar_wait(&sm.empty[j % kStages], (j / kStages) & 1, sm.abort_flag);
      if (!ok) {
        producer_drain(sm, it);
        if (QUANT)
          for (uint32_t c = it > CODE_SLOTS_DH ? it - CODE_SLOTS_DH : 0; c < it; ++c)
            mbar_wait_drain(&sm.cfull[c % CODE_SLOTS_DH], (c / CODE_SLOTS_DH) & 1);
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
    // whole-warp issue loop, one elected lane issues (see ce_logits_kernel)
    constexpr uint32_t idesc = make_idesc_bf16(PAIR ? 2 * BM : BM, BN, 0, 1);  // B is MN-major
    constexpr uint32_t dhi = desc_hi_sw128(1024);
    uint32_t it = 0, tile = 0;
    bool ok = true;
    for (int u = first_tile; u < total_tiles && ok; u += unit_step) {
      int kb0, kb1;
      k_range(u / tiles, kb0, kb1);
      const int segs = num_segs(kb0, kb1);
      for (int seg = 0; seg < segs && ok; ++seg, ++tile) {
        const int ks0 = kb0 + (kb1 - kb0) * seg / segs, ks1 = kb0 + (kb1 - kb0) * (seg + 1) / segs;
        const uint32_t as = tile & 1;
        if (!mbar_wait_warp(&sm.tempty[as], ((tile >> 1) & 1) ^ 1, sm.abort_flag)) {
          if (lane == 0) raise_abort(sm, p.status, kDevTimeoutMma);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + as * BN;
        for (int kb = ks0; kb < ks1; ++kb, ++it) {
          const int s = it % kStages;
          if (!mbar_wait_warp(&sm.full[s], (it / kStages) & 1, sm.abort_flag)) {
            if (lane == 0) raise_abort(sm, p.status, kDevTimeoutMma);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t a_lo = desc_lo(smem_u32(sm.a(s)), 16);
          // 16 k rows of 128 B each per step; 64-column chunks are 8 KiB apart.
          const uint32_t b_lo = desc_lo(smem_u32(sm.b(s)), 64 * BK * 2);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma<PAIR>(d_tmem, a_lo + k * 2, dhi, b_lo + k * 128, dhi, idesc, kb != ks0 || k != 0 ? 1u : 0u);
            commit<PAIR>(&sm.empty[s]);
          }
          __syncwarp();
        }
        if (ok && elect_one()) commit<PAIR>(&sm.tfull[as]);
        __syncwarp();
      }
    }
    }
  } else {
    const int quad = warp & 3;
    const int row_in_tile = quad * 32 + lane;
    uint32_t tile = 0;
    bool ok = true;
    for (int u = first_tile; u < total_tiles && ok; u += unit_step) {
      const int split = u / tiles, t = u - split * tiles;
      const int rb = t / p.num_nt;
      const int nt = t - rb * p.num_nt;
      int kb0, kb1;
      k_range(split, kb0, kb1);
      const int segs = num_segs(kb0, kb1);   // 0: the share keeps what earlier chunks left (see the host side)
      for (int seg = 0; seg < segs; ++seg, ++tile) {
        const float* acc_in = seg == 0 ? p.acc_in : p.acc_out;
        const bool last = seg == segs - 1;
        const uint32_t as = tile & 1;
        if (!mbar_wait_warp(&sm.tfull[as], (tile >> 1) & 1, sm.abort_flag)) {
          raise_abort(sm, p.status, kDevTimeoutEpilogue);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const int row = block_row(rb) + row_in_tile;
        const bool row_ok = row < p.n_rows;
        const uint32_t taddr0 = tmem_base + as * BN + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          const int col0 = nt * BN + c * 32;
          if (col0 >= p.d_cols) break;
          uint32_t r[32];
          tmem_ld_x32(taddr0 + c * 32, r);
          tmem_wait_ld();
          tmem_regs_ready(r);
          if (row_ok) {
            const size_t off = static_cast<size_t>(split) * p.split_stride + static_cast<size_t>(row) * p.d_cols + col0;
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              if (col0 + j < p.d_cols) {  // d_cols is a multiple of 8
                uint32_t v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = r[j + e];
                if (acc_in != nullptr) {
                  uint32_t o[8];
                  if (p.wide) ld_global_32b(acc_in + off + j, o);
                  else ld_global_2x16b(acc_in + off + j, o);
#pragma unroll
                  for (int e = 0; e < 8; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(o[e]));
                }
                if (last && p.out_bf16 != nullptr) {
#pragma unroll
                  for (int e = 0; e < 8; e += 4)
                    *reinterpret_cast<uint2*>(p.out_bf16 + off + j + e) =
                        make_uint2(pack_bf16x2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])),
                                   pack_bf16x2(__uint_as_float(v[e + 2]), __uint_as_float(v[e + 3])));
                } else if (p.wide) {
                  st_global_32b(p.acc_out + off + j, v);
                } else {
                  st_global_2x16b(p.acc_out + off + j, v);
                }
              }
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) release_acc<PAIR>(&sm.tempty[as]);
      }
    }
  }
  cta_teardown(sm, warp, tmem_base, PAIR);
}

// -----------------------------------------------------------------------------------------
// dW_chunk = G^T hidden   (trainable dense head; core/chunked.py:84-85, K5 of the reference)
// -----------------------------------------------------------------------------------------
// Tile = 128 vocab rows x 256 hidden columns per CTA of a pair, contraction over the N tokens in 64-row blocks.
// Both operands are read MN-major straight from their row-major homes: A = G (N, chunk) as two
// [64 tokens][64 vocab columns] boxes per stage, B = hidden (N, D) as four [64 tokens][64 hidden
// columns] boxes.  Token rows past N are zero-filled by TMA.  Each vocab row belongs to exactly one
// chunk, so the fp32 accumulator is complete after one pass and is rounded once to bf16.
__global__ void __launch_bounds__(THREADS, 1)
ce_dw_kernel(const __grid_constant__ CUtensorMap tmap_g, const __grid_constant__ CUtensorMap tmap_h,
             const DwParams p) {
  extern __shared__ uint8_t smem_raw[];
  const SmemView sm = carve_smem(smem_raw, false, true);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // provably warp-uniform
  const int lane = threadIdx.x & 31;
  const uint32_t tmem_base = cta_setup(sm, warp, 1, 8, true);
  constexpr uint32_t kStages = PAIR_STAGES;
  const uint32_t rank = cluster_ctarank();
  const int unit0 = blockIdx.x >> 1, unit_step = gridDim.x >> 1;
  auto block_row = [&](int mt) { return (mt * 2 + static_cast<int>(rank)) * BM; };

  const int total_tiles = p.num_mt * p.num_nt;
  const int kblocks = (p.n_rows + BK - 1) / BK;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_g);
      tma_prefetch_desc(&tmap_h);
      uint32_t it = 0;
      bool ok = true;
      for (int t = unit0; t < total_tiles && ok; t += unit_step) {
        const int nt = t / p.num_mt;
        const int mt = t - nt * p.num_mt;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % kStages;
          if (!mbar_wait(&sm.empty[s], ((it / kStages) & 1) ^ 1, sm.abort_flag)) {
            raise_abort(sm, p.status, kDevTimeoutProducer);
            ok = false;
            break;
          }
          if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2 * PAIR_STAGE_BYTES);
          const uint32_t bar = map_to_rank(&sm.full[s], 0);
#pragma unroll
          for (int j = 0; j < BM / 64; ++j)
            tma_load_2d_pair(sm.a(s) + j * (64 * BK * 2), &tmap_g, bar, block_row(mt) + j * 64, kb * BK);
#pragma unroll
          for (int j = 0; j < BN / 128; ++j)
            tma_load_2d_pair(sm.b(s) + j * (64 * BK * 2), &tmap_h, bar,
                             nt * BN + static_cast<int>(rank) * (BN / 2) + j * 64, kb * BK);
        }
      }
      // the other CTA's commits land here: none may be on its way when this one leaves
      if (ok)
        for (uint32_t j = it > kStages ? it - kStages : 0; j < it; ++j)
          mbar_wait(&sm.empty[j % kStages], (j / kStages) & 1, sm.abort_flag);
      if (!ok) producer_drain(sm, it);
    }
  } else if (warp == 1) {
    if (rank == 0) {
    // whole-warp issue loop, one elected lane issues (see ce_logits_kernel)
    constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, 1, 1);  // A and B are MN-major
    constexpr uint32_t dhi = desc_hi_sw128(1024);
    uint32_t it = 0, tile = 0;
    bool ok = true;
    for (int t = unit0; t < total_tiles && ok; t += unit_step, ++tile) {
      const uint32_t as = tile & 1;
      if (!mbar_wait_warp(&sm.tempty[as], ((tile >> 1) & 1) ^ 1, sm.abort_flag)) {
        if (lane == 0) raise_abort(sm, p.status, kDevTimeoutMma);
        break;
      }
      tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + as * BN;
      for (int kb = 0; kb < kblocks; ++kb, ++it) {
        const int s = it % kStages;
        if (!mbar_wait_warp(&sm.full[s], (it / kStages) & 1, sm.abort_flag)) {
          if (lane == 0) raise_abort(sm, p.status, kDevTimeoutMma);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        // 16 token rows of 128 B per step; 64-column chunks are 8 KiB apart (both operands).
        const uint32_t a_lo = desc_lo(smem_u32(sm.a(s)), 64 * BK * 2);
        const uint32_t b_lo = desc_lo(smem_u32(sm.b(s)), 64 * BK * 2);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma<true>(d_tmem, a_lo + k * 128, dhi, b_lo + k * 128, dhi, idesc, (kb | k) != 0 ? 1u : 0u);
          commit<true>(&sm.empty[s]);
        }
        __syncwarp();
      }
      if (ok && elect_one()) commit<true>(&sm.tfull[as]);
      __syncwarp();
    }
    }
  } else {
    const int quad = warp & 3;
    const int row_in_tile = quad * 32 + lane;
    uint32_t tile = 0;
    for (int t = unit0; t < total_tiles; t += unit_step, ++tile) {
      const int nt = t / p.num_mt;
      const int mt = t - nt * p.num_mt;
      const uint32_t as = tile & 1;
      if (!mbar_wait_warp(&sm.tfull[as], (tile >> 1) & 1, sm.abort_flag)) {
        raise_abort(sm, p.status, kDevTimeoutEpilogue);
        break;
      }
      tc_fence_after_sync();
      const int row = block_row(mt) + row_in_tile;   // vocab row inside the chunk
      const bool row_ok = row < p.v_rows;
      const uint32_t taddr0 = tmem_base + as * BN + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        const int col0 = nt * BN + c * 32;
        if (col0 >= p.d_cols) break;
        uint32_t r[32];
        tmem_ld_x32(taddr0 + c * 32, r);
        tmem_wait_ld();
        tmem_regs_ready(r);
        if (row_ok) {
          __nv_bfloat16* dst = p.out + static_cast<size_t>(row) * p.d_cols + col0;
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            if (col0 + j < p.d_cols) {  // d_cols is a multiple of 8
              *reinterpret_cast<uint4*>(dst + j) = make_uint4(
                  pack_bf16x2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])),
                  pack_bf16x2(__uint_as_float(r[j + 2]), __uint_as_float(r[j + 3])),
                  pack_bf16x2(__uint_as_float(r[j + 4]), __uint_as_float(r[j + 5])),
                  pack_bf16x2(__uint_as_float(r[j + 6]), __uint_as_float(r[j + 7])));
            }
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) release_acc<true>(&sm.tempty[as]);
    }
  }
  cta_teardown(sm, warp, tmem_base, true);
}

// -----------------------------------------------------------------------------------------
// Host-side scheduling
// -----------------------------------------------------------------------------------------
// Splits of the vocab-tile range: pick the count that minimises the busiest CTA's tile
// count under static round-robin, with a small per-unit cost for the partial writes.
// The search is O(splits * units) on the host, so results are memoised per shape.
int choose_splits(int num_rb, int num_vt, int ctas) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int>, int> memo;
  const auto key = std::make_tuple(num_rb, num_vt, ctas);
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = memo.find(key);
    if (it != memo.end()) return it->second;
  }
  int best = 1;
  double best_cost = 1e300;
  // More splits than ~8 waves of units buys nothing: cap the search.
  const int max_s = std::max(1, std::min(num_vt, std::max(1, 8 * ctas / std::max(1, num_rb) + 1)));
  std::vector<long long> load(ctas);
  for (int s = 1; s <= max_s; ++s) {
    std::fill(load.begin(), load.end(), 0);
    const long long units = static_cast<long long>(num_rb) * s;
    for (int split = 0; split < s; ++split) {
      const long long t0 = static_cast<long long>(split) * num_vt / s;
      const long long t1 = static_cast<long long>(split + 1) * num_vt / s;
      const long long u0 = static_cast<long long>(split) * num_rb;
      for (int rb = 0; rb < num_rb; ++rb) load[(u0 + rb) % ctas] += (t1 - t0);
    }
    const long long mx = *std::max_element(load.begin(), load.end());
    const double cost = static_cast<double>(mx) + 0.02 * static_cast<double>((units + ctas - 1) / ctas);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = s;
    }
  }
  std::lock_guard<std::mutex> lock(mu);
  memo[key] = best;
  return best;
}

}  // namespace

static std::atomic<int> g_smem_configured[64];

static int configure_kernels() {
  int dev = 0;
  B200TP_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && g_smem_configured[dev].load(std::memory_order_acquire)) return B200TP_OK;
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_logits_kernel<MODE_FWD, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      SMEM_BYTES));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_logits_kernel<MODE_BWD_G, false>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_logits_kernel<MODE_FWD_GRAD, false>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_logits_kernel<MODE_FWD, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      SMEM_BYTES_Q));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_logits_kernel<MODE_BWD_G, true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES_Q));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_dh_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_dh_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES_Q));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_dw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_logits_kernel<MODE_FWD, false, true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_logits_kernel<MODE_BWD_G, false, true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_logits_kernel<MODE_FWD_GRAD, false, true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  B200TP_CUDA_OK(cudaFuncSetAttribute(ce_dh_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      SMEM_BYTES));
  if (dev >= 0 && dev < 64) g_smem_configured[dev].store(1, std::memory_order_release);
  return B200TP_OK;
}

// Whether the dense kernels run as CTA pairs over 256 rows each.  A pair's MMA reads each weight tile once for two SMs
// and leaves room for two more stages; against that stand the padding of an odd number of row blocks and, in short
// kernels, the pair's start-up.  Forward / forward with gradient, us, single CTAs against pairs:
//   D = 4096, V = 151936:  200 rows 277 / 601, 252 / 528;  257 rows (3 blocks) 369 / 781, 412 / 859;  400 rows 467 / 999,
//   429 / 902;  850 rows (7) 818 / 1749, 965 / 1911;  1100 rows (9) 1041 / 2223, 1047 / 2280;  2100 rows (17)
//   1978 / 4386, 1769 / 4134;  8192 rows 7624 / 17976, 7234 / 16916
//   D = 1024, V = 50000:   200 rows 53 / 110, 59 / 125;  400 rows 60 / 129, 66 / 139;  2100 rows (17) 156 / 377, 153 / 368;
//   8192 rows 535 / 1530, 509 / 1378
// That head (102 MB) was in the L2.  Forward / whole step from a cold L2, V = 50000, where the line at D = 2048 leaves
// something to pairs below it:
//   D = 1024:  200 rows 46 / 101, 42 / 97;  1000 rows 87 / 210, 77 / 187;  1400 rows (11) 111 / 273, 108 / 265
//   D = 1536:  200 rows 64 / 144, 60 / 134;  1000 rows 140 / 337, 126 / 300;  1400 rows 161 / 394, 156 / 366
//   D = 2048:  200 rows 79 / 163, 71 / 150;  1000 rows 161 / 370, 140 / 331;  1400 rows 222 / 486, 208 / 478
static bool use_pair(int64_t n, int d) {
  const int64_t blocks = ceil_div(n, BM);
  return blocks >= 16 || (blocks % 2 == 0 && d >= 2048);
}

int ce_tc_choose_splits(int num_rb, int num_vt, int ctas) { return choose_splits(num_rb, num_vt, ctas); }

int ce_tc_fwd_splits(int64_t n, int d, int64_t v_rows) {
  const int num_vt = static_cast<int>(ceil_div(v_rows, BN));
  if (use_pair(n, d)) return choose_splits(static_cast<int>(ceil_div(n, 2 * BM)), num_vt, sm_count() / 2);
  return choose_splits(static_cast<int>(ceil_div(n, BM)), num_vt, sm_count());
}

// Tensor map of the weight operand: the dense bf16 matrix, or for a 4-bit head the map of its packed
// uint32 code words (box of `code_box_rows` rows x `code_box_words` words), which the producer copies
// into the code ring.
static int weight_map(CUtensorMap* out, const void* w, int64_t w_rows_total, int d, uint32_t box_rows,
                      uint32_t box_cols, const QuantHead* q, uint32_t code_box_rows, uint32_t code_box_words) {
  if (q != nullptr && q->wq != nullptr)
    return make_tmap_2d_u32(out, q->wq, w_rows_total, d / 8, d / 8, code_box_rows, code_box_words);
  return make_tmap_2d_bf16(out, w, w_rows_total, d, d, box_rows, box_cols);
}

static void fill_quant(LogitsParams& p, const QuantHead* q) {
  if (q == nullptr) return;
  p.wq = q->wq;
  p.scales = q->scales;
  p.biases = q->biases;
  p.qp_f32 = q->qp_f32;
  p.qvec = (!q->qp_f32 && p.k_dim % 512 == 0 && ((reinterpret_cast<uintptr_t>(q->scales) |
                                                  reinterpret_cast<uintptr_t>(q->biases)) & 15) == 0)
               ? 1
               : 0;
}

int ce_tc_launch_fwd(const void* hidden, const void* w, int64_t w_rows_total, int64_t n, int d, int64_t vrow0,
                     int64_t vrow1, int64_t vocab_id0, const int64_t* targets, int64_t ignore_index, int splits,
                     float* pm, float* ps, float* pt, const QuantHead* q, cudaStream_t stream, int* status) {
  int rc = configure_kernels();
  if (rc) return rc;
  CUtensorMap tmap_h, tmap_w;
  rc = make_tmap_2d_bf16(&tmap_h, hidden, n, d, d, BM, BK);
  if (rc) return rc;
  const bool quant = q != nullptr && q->wq != nullptr, pair = !quant && use_pair(n, d);
  rc = weight_map(&tmap_w, w, w_rows_total, d, pair ? BN / 2 : BN, BK, q, BN, 16);
  if (rc) return rc;
  LogitsParams p{};
  p.n_rows = static_cast<int>(n);
  p.k_dim = d;
  p.vrow0 = static_cast<int>(vrow0);
  p.vrow1 = static_cast<int>(vrow1);
  p.vocab_id0 = vocab_id0;
  p.num_rb = static_cast<int>(ceil_div(n, pair ? 2 * BM : BM));
  p.num_vt = static_cast<int>(ceil_div(vrow1 - vrow0, BN));
  p.splits = splits;
  p.targets = reinterpret_cast<const long long*>(targets);
  p.ignore_index = ignore_index;
  p.pm = pm;
  p.ps = ps;
  p.pt = pt;
  p.status = status;
  fill_quant(p, q);
  if (quant) {
    const int grid = std::min<long long>(sm_count(), static_cast<long long>(p.num_rb) * splits);
    ce_logits_kernel<MODE_FWD, true><<<grid, THREADS_Q, SMEM_BYTES_Q, stream>>>(tmap_h, tmap_w, p);
    B200TP_CUDA_OK(cudaGetLastError());
    return B200TP_OK;
  }
  return launch_units(pair ? ce_logits_kernel<MODE_FWD, false, true> : ce_logits_kernel<MODE_FWD, false>, THREADS, pair,
                      static_cast<long long>(p.num_rb) * splits, stream, tmap_h, tmap_w, p);
}

int ce_tc_launch_bwd_g(const void* hidden, const void* w, int64_t w_rows_total, int64_t n, int d, int64_t vrow0,
                       int64_t vrow1, int64_t vocab_id0, const int64_t* targets, int64_t ignore_index,
                       const float* lse, const float* ct, void* g, int ldg, const QuantHead* q,
                       const LaunchGuard& guard, cudaStream_t stream, int* status) {
  int rc = configure_kernels();
  if (rc) return rc;
  CUtensorMap tmap_h, tmap_w;
  rc = make_tmap_2d_bf16(&tmap_h, hidden, n, d, d, BM, BK);
  if (rc) return rc;
  const bool quant = q != nullptr && q->wq != nullptr, pair = !quant && use_pair(n, d);
  rc = weight_map(&tmap_w, w, w_rows_total, d, pair ? BN / 2 : BN, BK, q, BN, 16);
  if (rc) return rc;
  LogitsParams p{};
  p.n_rows = static_cast<int>(n);
  p.k_dim = d;
  p.vrow0 = static_cast<int>(vrow0);
  p.vrow1 = static_cast<int>(vrow1);
  p.vocab_id0 = vocab_id0;
  p.num_rb = static_cast<int>(ceil_div(n, pair ? 2 * BM : BM));
  p.num_vt = static_cast<int>(ceil_div(vrow1 - vrow0, BN));
  // One unit per (row block, vocab tile group): there is no cross-tile state in this
  // mode, so split as finely as balance asks for.
  p.splits = choose_splits(p.num_rb, p.num_vt, pair ? sm_count() / 2 : sm_count());
  p.targets = reinterpret_cast<const long long*>(targets);
  p.ignore_index = ignore_index;
  p.lse = lse;
  p.ct = ct;
  p.g = reinterpret_cast<__nv_bfloat16*>(g);
  p.ldg = ldg;
  p.guard = guard;
  p.status = status;
  fill_quant(p, q);
  if (quant) {
    const int grid = std::min<long long>(sm_count(), static_cast<long long>(p.num_rb) * p.splits);
    ce_logits_kernel<MODE_BWD_G, true><<<grid, THREADS_Q, SMEM_BYTES_Q, stream>>>(tmap_h, tmap_w, p);
    B200TP_CUDA_OK(cudaGetLastError());
    return B200TP_OK;
  }
  return launch_units(pair ? ce_logits_kernel<MODE_BWD_G, false, true> : ce_logits_kernel<MODE_BWD_G, false>, THREADS, pair,
                      static_cast<long long>(p.num_rb) * p.splits, stream, tmap_h, tmap_w, p);
}

int ce_tc_launch_fwd_grad(const void* hidden, const void* w, int64_t w_rows_total, int64_t n, int d, int64_t vrow0,
                          int64_t vrow1, int64_t vocab_id0, const int64_t* targets, int64_t ignore_index,
                          const float* ref2, int* overflow, int splits, float* pm, float* ps, float* pt, void* g,
                          int ldg, cudaStream_t stream, int* status) {
  int rc = configure_kernels();
  if (rc) return rc;
  CUtensorMap tmap_h, tmap_w;
  rc = make_tmap_2d_bf16(&tmap_h, hidden, n, d, d, BM, BK);
  if (rc) return rc;
  const bool pair = use_pair(n, d);
  rc = make_tmap_2d_bf16(&tmap_w, w, w_rows_total, d, d, pair ? BN / 2 : BN, BK);
  if (rc) return rc;
  LogitsParams p{};
  p.n_rows = static_cast<int>(n);
  p.k_dim = d;
  p.vrow0 = static_cast<int>(vrow0);
  p.vrow1 = static_cast<int>(vrow1);
  p.vocab_id0 = vocab_id0;
  p.num_rb = static_cast<int>(ceil_div(n, pair ? 2 * BM : BM));
  p.num_vt = static_cast<int>(ceil_div(vrow1 - vrow0, BN));
  p.splits = splits;
  p.targets = reinterpret_cast<const long long*>(targets);
  p.ignore_index = ignore_index;
  p.pm = pm;
  p.ps = ps;
  p.pt = pt;
  p.g = reinterpret_cast<__nv_bfloat16*>(g);
  p.ldg = ldg;
  p.ref2 = ref2;
  p.overflow = overflow;
  p.status = status;
  return launch_units(pair ? ce_logits_kernel<MODE_FWD_GRAD, false, true> : ce_logits_kernel<MODE_FWD_GRAD, false>, THREADS, pair,
                      static_cast<long long>(p.num_rb) * splits, stream, tmap_h, tmap_w, p);
}

int ce_tc_dh_tiles(int64_t n, int d) {
  return static_cast<int>(ceil_div(n, BM) * ceil_div(d, BN));
}

// Shares of the d_hidden contraction.  A call with few rows has few 128 x 256 tiles (four at 60 rows and
// D = 1024), and one CTA each would leave most of the chip idle; the shares' fp32 sums are added in a fixed order
// afterwards.  The cost of a choice is the busiest CTA's k blocks plus, per unit, what its prologue and
// epilogue take (about kUnitCost k blocks of 0.27 us).
int ce_tc_dh_ksplit(int64_t n, int d, int k_total) {
  constexpr int kUnitCost = 8, kMostShares = 64;
  const bool pair = use_pair(n, d);
  const int64_t tiles = ceil_div(n, pair ? 2 * BM : BM) * ceil_div(d, BN);
  const int kblocks = k_total / BK, ctas = pair ? sm_count() / 2 : sm_count();
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int ks = 1; ks <= std::min(kMostShares, kblocks); ++ks) {
    const int64_t cost = ceil_div(tiles * ks, ctas) * (ceil_div(kblocks, ks) + kUnitCost);
    if (cost < best_cost) {
      best_cost = cost;
      best = ks;
    }
    if (tiles * ks >= 4 * ctas) break;   // more shares than this only add partial sums
  }
  return best;
}

int ce_tc_dh_rows_done(int64_t n, int d, int tiles_done) {
  const int num_nt = static_cast<int>(ceil_div(d, BN));
  if (tiles_done >= ce_tc_dh_tiles(n, d)) return static_cast<int>(n);
  return static_cast<int>(std::min<int64_t>(n, static_cast<int64_t>(tiles_done / num_nt) * BM));
}

int ce_tc_launch_dh(const void* g, int ldg, int k_total, int64_t n, const void* w, int64_t w_rows_total, int d,
                    int64_t wrow0, const float* acc_in, float* acc_out, void* out_bf16, int tile0, int tile1,
                    int ksplit, const QuantHead* q, const LaunchGuard& guard, cudaStream_t stream, int* status) {
  if (ksplit > 1 && (out_bf16 != nullptr || (q != nullptr && q->wq != nullptr) ||
                     (acc_in == nullptr && ksplit > k_total / BK) || (acc_in != nullptr && acc_in != acc_out)))
    return fail(B200TP_ERR_CUDA, "d_hidden shares: fp32 sums of a dense weight, in place, no empty share at first");
  int rc = configure_kernels();
  if (rc) return rc;
  CUtensorMap tmap_g, tmap_w;
  rc = make_tmap_2d_bf16(&tmap_g, g, n, k_total, ldg, BM, BK);
  if (rc) return rc;
  rc = weight_map(&tmap_w, w, w_rows_total, d, /*box_rows=*/BK, /*box_cols=*/64, q, BK, BN / 8);
  if (rc) return rc;
  DhParams p{};
  p.n_rows = static_cast<int>(n);
  p.d_cols = d;
  p.k_total = k_total;
  p.wrow0 = static_cast<int>(wrow0);
  // a slab of the tiles (a staged backward) is counted in 128-row tiles and stays with them
  const bool quant = q != nullptr && q->wq != nullptr;
  const bool pair = !quant && use_pair(n, d) && tile0 <= 0 && (tile1 < 0 || tile1 >= ce_tc_dh_tiles(n, d) * ksplit);
  if (pair) tile0 = tile1 = -1;
  p.num_rb = static_cast<int>(ceil_div(n, pair ? 2 * BM : BM));
  p.num_nt = static_cast<int>(ceil_div(d, BN));
  p.acc_in = acc_in;
  p.acc_out = acc_out;
  p.out_bf16 = reinterpret_cast<__nv_bfloat16*>(out_bf16);
  p.status = status;
  p.guard = guard;
  p.ksplit = ksplit;
  p.split_stride = static_cast<long long>(n) * d;
  p.wide = ((reinterpret_cast<uintptr_t>(acc_in) | reinterpret_cast<uintptr_t>(acc_out)) & 31) == 0;
  p.seg_kb = acc_out != nullptr ? kMostAccumulated / BK : std::max(1, k_total / BK);
  const int total = p.num_rb * p.num_nt * ksplit;
  p.tile0 = tile0 < 0 ? 0 : tile0;
  p.tile1 = tile1 < 0 ? total : std::min(tile1, total);
  p.w_rows = static_cast<int>(w_rows_total);
  if (q != nullptr) {
    p.wq = q->wq;
    p.scales = q->scales;
    p.biases = q->biases;
    p.qp_f32 = q->qp_f32;
  }
  if (p.tile1 <= p.tile0) return B200TP_OK;
  if (quant) {
    const int grid = std::min<long long>(sm_count(), p.tile1 - p.tile0);
    ce_dh_kernel<true><<<grid, THREADS_Q, SMEM_BYTES_Q, stream>>>(tmap_g, tmap_w, p);
    B200TP_CUDA_OK(cudaGetLastError());
    return B200TP_OK;
  }
  return launch_units(pair ? ce_dh_kernel<false, true> : ce_dh_kernel<false>, THREADS, pair, p.tile1 - p.tile0, stream, tmap_g,
                      tmap_w, p);
}

int ce_tc_launch_dw(const void* g, int ldg, int64_t v_rows, int64_t n, const void* hidden, int d, void* d_weight_block,
                    cudaStream_t stream, int* status) {
  int rc = configure_kernels();
  if (rc) return rc;
  CUtensorMap tmap_g, tmap_h;
  // both maps: 64 token rows x 64 columns per box
  rc = make_tmap_2d_bf16(&tmap_g, g, n, ldg, ldg, /*box_rows=*/BK, /*box_cols=*/64);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tmap_h, hidden, n, d, d, /*box_rows=*/BK, /*box_cols=*/64);
  if (rc) return rc;
  DwParams p{};
  p.n_rows = static_cast<int>(n);
  p.d_cols = d;
  p.v_rows = static_cast<int>(v_rows);
  p.num_mt = static_cast<int>(ceil_div(v_rows, 2 * BM));   // pairs: chunks are whole multiples of 256 rows but the last
  p.num_nt = static_cast<int>(ceil_div(d, BN));
  p.out = reinterpret_cast<__nv_bfloat16*>(d_weight_block);
  p.status = status;
  return launch_units(ce_dw_kernel, THREADS, true, static_cast<long long>(p.num_mt) * p.num_nt, stream, tmap_g, tmap_h, p);
}

}  // namespace b200tp
