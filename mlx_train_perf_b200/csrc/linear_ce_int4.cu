// Forward of a 4-bit affine head, expanded inside the kernel: Z^T = W H^T on the tensor cores.
//
// The weight is the A operand and lives in TENSOR memory: a thread expands one vocab row's 64 codes of a k block and
// stores the 32 bf16 pairs into that row's lane.  The tokens are the N side: a CTA keeps up to kMostTokens of them
// against one 128-row weight tile, so a code is expanded once per kMostTokens tokens.  (With the tokens on the M side
// a weight tile was expanded again for every 128 of them, and padding went to multiples of 128: 257 rows x 4096 x
// 151936 took 773 us where this takes 304.)  An MMA reads only the tokens from shared memory, which
// leaves room for the TMA writes beside it; both operands there would need more than its bandwidth.
//
// The accumulator is transposed: a lane holds a vocab row, a column a token.  The epilogue warps turn 32 x 32 blocks
// around through shared memory and keep the running (max, sum-exp, target) of one token per lane; at the end of a
// vocab share the four lane quadrants' triples of a token are merged into one.
//
// Tensor-bound from about 200 tokens on, expansion-bound below (about 170 instructions per 64 weights; eight warps in
// two groups, each taking every other k block, keep it under the MMAs of 272 tokens; three groups make 60 tokens 260 ->
// 239 us, and 257 304 -> 313, 2048 2050 -> 2249).
//
// Roles (19 warps): two TMA producers, MMA issuer, eight epilogue warps, eight expanding warps.  Waits are bounded and end
// like those of linear_ce_tc.cu.  Replaces core/kernel/source.py:199-340 (K2) of the reference.
#include "linear_ce_tc.h"

#include <algorithm>
#include <atomic>

#include "dequant.cuh"
#include "ptx.cuh"

namespace b200tp {
namespace {

constexpr int VROWS = 128;                            // vocab rows per tile (M)
constexpr int KB = 64;
constexpr int kMostTokens = 320;                      // two MMAs of at most 160 columns
constexpr int STAGES = 4;
constexpr int STAGE_BYTES = kMostTokens * KB * 2;     // 40 KiB
constexpr int CODE_SLOTS = 4;
constexpr int CODE_BYTES = VROWS * 64;                // one row's codes of two k blocks: 64 bytes
constexpr int EPI_WARPS = 8, DQ_WARPS = 8;
constexpr int CTRL_WARPS = 3;                         // token producer, MMA issuer, code producer
constexpr int THREADS = 32 * (CTRL_WARPS + EPI_WARPS + DQ_WARPS);
constexpr int TURN_FLOATS = 32 * 33;                  // per epilogue warp: a 32 x 32 block, padded against conflicts
constexpr int BAR_BYTES = 256;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + CODE_SLOTS * CODE_BYTES + EPI_WARPS * TURN_FLOATS * 4 + BAR_BYTES + 1024;
constexpr uint32_t TMEM_COLS = 512, TMEM_A = 384;     // accumulators [0, 320), weight stages [384, 512)
constexpr int CHUNKS = kMostTokens / 32 / 2;          // 32-token chunks per epilogue warp
static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");

struct Int4Params {
  int n_rows, kblocks;
  int v_rows, num_vt, splits;
  int groups, gsz;       // token groups and their size (a multiple of 16)
  int n0, n1, boxes;     // columns of the two MMAs; the token box is n0 rows, loaded once or twice
  long long vocab_id0;
  const long long* targets;
  long long ignore_index;
  float* pm;             // [split][N]
  float* ps;
  float* pt;
  const void* scales;
  const void* biases;
  int qp_f32, qvec;
  int* status;
};

struct Smem {
  uint8_t* base;
  uint8_t* codes;
  float* turn;
  uint64_t *full, *empty, *cfull, *cempty, *tfull, *tempty;
  uint32_t* tmem_ptr;
  int* abort_flag;
};

__device__ __forceinline__ Smem carve(uint8_t* raw) {
  const uint32_t addr = smem_u32(raw);
  Smem s;
  s.base = raw + (((addr + 1023u) & ~1023u) - addr);
  s.codes = s.base + STAGES * STAGE_BYTES;
  s.turn = reinterpret_cast<float*>(s.codes + CODE_SLOTS * CODE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(s.turn + EPI_WARPS * TURN_FLOATS);
  s.full = bars;
  s.empty = bars + STAGES;
  s.cfull = bars + 2 * STAGES;
  s.cempty = s.cfull + CODE_SLOTS;
  s.tfull = s.cempty + CODE_SLOTS;
  s.tempty = s.tfull + 1;
  s.tmem_ptr = reinterpret_cast<uint32_t*>(s.tempty + 1);
  s.abort_flag = reinterpret_cast<int*>(s.tmem_ptr + 1);
  return s;
}

__device__ __forceinline__ void raise(const Smem& sm, int* status, int code) {
  atomicExch(sm.abort_flag, 1);
  if (status != nullptr) atomicCAS(status, 0, code);
}

// Whether any of the epilogue warps' threads says so; a barrier among them.
__device__ __forceinline__ bool epilogue_any(bool x) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "bar.red.or.pred q, 1, %2, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(r)
      : "r"(x ? 1u : 0u), "n"(EPI_WARPS * 32)
      : "memory");
  return r != 0;
}

// The (unit, vocab tile) sequence of one CTA; unit = share * groups + group, so neighbours read the same weights.
struct TileWalk {
  int u, vt, vt1;
  __device__ __forceinline__ void set(const Int4Params& p) {
    const int split = u / p.groups;
    vt = static_cast<int>(static_cast<long long>(split) * p.num_vt / p.splits);
    vt1 = static_cast<int>(static_cast<long long>(split + 1) * p.num_vt / p.splits);
  }
  __device__ __forceinline__ TileWalk(const Int4Params& p) : u(blockIdx.x) {
    if (!done(p)) set(p);
  }
  __device__ __forceinline__ bool done(const Int4Params& p) const { return u >= p.groups * p.splits; }
  __device__ __forceinline__ void next(const Int4Params& p) {
    if (++vt < vt1) return;
    u += gridDim.x;
    if (!done(p)) set(p);
  }
};

__global__ void __launch_bounds__(THREADS, 1)
int4_logits_kernel(const __grid_constant__ CUtensorMap tmap_h, const __grid_constant__ CUtensorMap tmap_c,
                   const Int4Params p) {
  extern __shared__ uint8_t smem_raw[];
  const Smem sm = carve(smem_raw);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // provably warp-uniform
  const int lane = threadIdx.x & 31;
  const int cblocks = (p.kblocks + 1) / 2;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sm.full[s], 1 + DQ_WARPS / 2);   // the token copy and the group that expands this k block
      mbar_init(&sm.empty[s], 1);
    }
    for (int s = 0; s < CODE_SLOTS; ++s) {
      mbar_init(&sm.cfull[s], 1);
      mbar_init(&sm.cempty[s], DQ_WARPS);
    }
    mbar_init(sm.tfull, 1);
    mbar_init(sm.tempty, EPI_WARPS);
    *sm.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(sm.tmem_ptr, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(sm.tmem_ptr);

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_h);
      const uint32_t box_bytes = static_cast<uint32_t>(p.n0) * KB * 2;
      uint32_t it = 0;
      bool ok = true;
      for (TileWalk w(p); !w.done(p) && ok; w.next(p)) {
        const int row0 = (w.u % p.groups) * p.gsz;
        for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(&sm.empty[s], ((it / STAGES) & 1) ^ 1, sm.abort_flag)) {
            raise(sm, p.status, kDevTimeoutProducer);
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&sm.full[s], p.boxes * box_bytes);
          for (int b = 0; b < p.boxes; ++b)
            tma_load_2d(sm.base + s * STAGE_BYTES + b * box_bytes, &tmap_h, &sm.full[s], kb * KB, row0 + b * p.n0);
        }
      }
      if (!ok)
        for (uint32_t j = it > STAGES ? it - STAGES : 0; j < it; ++j) mbar_wait_drain(&sm.full[j % STAGES], (j / STAGES) & 1);
    }
  } else if (warp == 2) {
    // The codes come from HBM and the tokens from L2, and codes must be asked for further ahead than the stages reach:
    // issued in step with the tokens, four k blocks ahead, stages waited for them (257 rows: 322 us, now 304).
    if (lane == 0) {
      tma_prefetch_desc(&tmap_c);
      uint32_t ci = 0;
      bool ok = true;
      for (TileWalk w(p); !w.done(p) && ok; w.next(p)) {
        for (int cb = 0; cb < cblocks; ++cb, ++ci) {
          const uint32_t cs = ci % CODE_SLOTS;
          if (!mbar_wait(&sm.cempty[cs], ((ci / CODE_SLOTS) & 1) ^ 1, sm.abort_flag)) {
            raise(sm, p.status, kDevTimeoutProducer);
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&sm.cfull[cs], CODE_BYTES);
          tma_load_2d(sm.codes + cs * CODE_BYTES, &tmap_c, &sm.cfull[cs], cb * 16, w.vt * VROWS);
        }
      }
      if (!ok)
        for (uint32_t c = ci > CODE_SLOTS ? ci - CODE_SLOTS : 0; c < ci; ++c)
          mbar_wait_drain(&sm.cfull[c % CODE_SLOTS], (c / CODE_SLOTS) & 1);
    }
  } else if (warp == 1) {
    // whole-warp issue loop, one elected lane issues (see ce_logits_kernel)
    const uint32_t idesc0 = make_idesc_bf16(VROWS, p.n0, 0, 0), idesc1 = make_idesc_bf16(VROWS, p.n1, 0, 0);
    constexpr uint32_t dhi = desc_hi_sw128(1024);
    const uint32_t second = static_cast<uint32_t>(p.n0) * KB * 2 / 16;
    uint32_t it = 0, tile = 0;
    bool ok = true;
    for (TileWalk w(p); !w.done(p) && ok; w.next(p), ++tile) {
      ok = mbar_wait_warp(sm.tempty, (tile & 1) ^ 1, sm.abort_flag);
      for (int kb = 0; kb < p.kblocks && ok; ++kb, ++it) {
        const int s = it % STAGES;
        ok = mbar_wait_warp(&sm.full[s], (it / STAGES) & 1, sm.abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t b_lo = desc_lo(smem_u32(sm.base + s * STAGE_BYTES), 16);
        const uint32_t a = tmem_base + TMEM_A + s * (KB / 2);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < KB / 16; ++k) {
            umma_ts_w(tmem_base, a + k * 8, b_lo + k * 2, dhi, idesc0, (kb | k) != 0 ? 1u : 0u);
            if (p.n1 > 0) umma_ts_w(tmem_base + p.n0, a + k * 8, b_lo + second + k * 2, dhi, idesc1, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(&sm.empty[s]);
        }
        __syncwarp();
      }
      if (ok && elect_one()) umma_commit(sm.tfull);
      __syncwarp();
    }
    if (!ok && lane == 0) raise(sm, p.status, kDevTimeoutMma);
  } else if (warp < CTRL_WARPS + EPI_WARPS) {
    const int quad = warp & 3, half = (warp - CTRL_WARPS) >> 2;   // lanes (vocab rows); every other 32-token chunk
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    float* turn = sm.turn + (warp - CTRL_WARPS) * TURN_FLOATS;
    uint32_t tile = 0;
    bool ok = true;
    TileWalk w(p);
    while (!w.done(p) && ok) {
      const int u = w.u, split = u / p.groups, row0 = (u % p.groups) * p.gsz;
      const int row1 = min(row0 + p.gsz, p.n_rows);
      float m[CHUNKS], s[CHUNKS], t[CHUNKS];
      long long target[CHUNKS];   // relative to the launch's first vocab row
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
        m[i] = -INFINITY;
        s[i] = t[i] = 0.f;
        target[i] = -1;
        const int row = row0 + (2 * i + half) * 32 + lane;
        if (row < row1) {
          const long long tg = p.targets[row];
          if (tg != p.ignore_index) target[i] = tg - p.vocab_id0;
        }
      }
      for (; w.u == u; w.next(p), ++tile) {
        if (!mbar_wait_warp(sm.tfull, tile & 1, sm.abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const int v0 = w.vt * VROWS + quad * 32;           // vocab row of lane 0
        const int nv = min(32, p.v_rows - v0);             // rows that exist (may be <= 0)
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) {
          const int c = 2 * i + half;
          if (c * 32 < p.gsz) {
            uint32_t r[32];
            tmem_ld_x32(taddr + c * 32, r);
            tmem_wait_ld();
            tmem_regs_ready(r);
            __syncwarp();   // the previous block has been read
#pragma unroll
            for (int j = 0; j < 32; ++j) turn[lane * 33 + j] = __uint_as_float(r[j]);
            __syncwarp();
            if (nv > 0) {
              float x[32];
#pragma unroll
              for (int j = 0; j < 32; ++j) x[j] = j < nv ? turn[j * 33 + lane] : -INFINITY;
              float mx4[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
              for (int j = 4; j < 32; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], x[j]);
              // finite: row v0 exists and logits are
              const float nm = fmaxf(m[i], fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * kLog2e);
              float a4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
              for (int j = 0; j < 32; ++j) a4[j & 3] += fast_exp2(fmaf(x[j], kLog2e, -nm));
              s[i] = s[i] * fast_exp2(m[i] - nm) + ((a4[0] + a4[1]) + (a4[2] + a4[3]));
              m[i] = nm;
              const long long rel = target[i] - v0;
              if (rel >= 0 && rel < nv) t[i] = turn[static_cast<int>(rel) * 33 + lane];
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.tempty);
      }
      if (!ok) raise(sm, p.status, kDevTimeoutEpilogue);
      // the quadrants' triples of a token meet in the turning buffers
      __syncwarp();
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
        turn[i * 32 + lane] = m[i];
        turn[(CHUNKS + i) * 32 + lane] = s[i];
        turn[(2 * CHUNKS + i) * 32 + lane] = t[i];
      }
      ok = !epilogue_any(!ok);   // all of them go on or none, so none is left at a barrier
      if (!ok) break;
      if (quad == 0) {
        const float* all = sm.turn + half * 4 * TURN_FLOATS;   // this half's four warps, in any order
#pragma unroll 1
        for (int i = 0; i < CHUNKS; ++i) {
          const int row = row0 + (2 * i + half) * 32 + lane;
          if (row >= row1) break;
          float mm = -INFINITY, ss = 0.f, tt = 0.f;
#pragma unroll
          for (int k = 0; k < 4; ++k) mm = fmaxf(mm, all[k * TURN_FLOATS + i * 32 + lane]);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float* f = all + k * TURN_FLOATS + i * 32 + lane;
            if (f[CHUNKS * 32] != 0.f) ss += f[CHUNKS * 32] * fast_exp2(f[0] - mm);
            tt += f[2 * CHUNKS * 32];
          }
          const size_t o = static_cast<size_t>(split) * p.n_rows + row;
          p.pm[o] = mm * kLn2;   // back to natural-log units
          p.ps[o] = ss;
          p.pt[o] = tt;
        }
        __syncwarp();
      }
      epilogue_any(false);   // read before the next unit writes
    }
  } else {
    // expanding warps: group g takes the k blocks with kb % 2 == g
    const int grp = (warp - CTRL_WARPS - EPI_WARPS) >> 2, quad = warp & 3;
    const int trow = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t swz = static_cast<uint32_t>((trow >> 1) & 3);
    const bool qp_f32 = p.qp_f32 != 0, qvec = p.qvec != 0;
    auto load8 = [&](int row, int kb, uint4& s8, uint4& b8) {   // parameters of k blocks [kb, kb + 8)
      if (row >= p.v_rows) return;
      const long long idx = static_cast<long long>(row) * p.kblocks + kb;
      s8 = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p.scales) + idx));
      b8 = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p.biases) + idx));
    };
    auto pick = [](const uint4& v, int k) -> uint32_t {   // k-th bf16 of eight
      const uint32_t lo = (k & 4) ? v.z : v.x, hi = (k & 4) ? v.w : v.y;
      return (((k & 2) ? hi : lo) >> ((k & 1) * 16)) & 0xFFFFu;
    };
    uint4 s_cur = make_uint4(0, 0, 0, 0), b_cur = s_cur, s_nxt = s_cur, b_nxt = s_cur;
    uint32_t it0 = 0, ci = 0;   // stage sequence number of the tile's first k block; code tile sequence number
    bool ok = true;
    TileWalk w(p);
    if (qvec && !w.done(p)) load8(w.vt * VROWS + trow, 0, s_nxt, b_nxt);
    for (; !w.done(p) && ok; w.next(p), it0 += p.kblocks) {
      const int row = w.vt * VROWS + trow;
      const bool valid = row < p.v_rows;
      for (int cb = 0; cb < cblocks; ++cb, ++ci) {
        const int kb = 2 * cb + grp;
        const bool mine = kb < p.kblocks;
        uint32_t sc = 0, bi = 0;
        if (qvec) {
          if ((cb & 3) == 0) {
            s_cur = s_nxt;
            b_cur = b_nxt;
            if (cb + 4 < cblocks) {
              load8(row, 2 * cb + 8, s_nxt, b_nxt);
            } else {
              TileWalk nx = w;
              nx.next(p);
              if (!nx.done(p)) load8(nx.vt * VROWS + trow, 0, s_nxt, b_nxt);
            }
          }
          sc = pick(s_cur, kb & 7);
          bi = pick(b_cur, kb & 7);
        } else if (valid && mine) {
          sc = dq_load_param(p.scales, static_cast<long long>(row) * p.kblocks + kb, qp_f32);
          bi = dq_load_param(p.biases, static_cast<long long>(row) * p.kblocks + kb, qp_f32);
        }
        const uint32_t cs = ci % CODE_SLOTS;
        ok = mbar_wait_warp(&sm.cfull[cs], (ci / CODE_SLOTS) & 1, sm.abort_flag);
        if (!ok) break;
        if (mine) {
          const uint32_t crow = smem_u32(sm.codes) + cs * CODE_BYTES + trow * 64;
          const uint4 lo = lds128(crow + (((2 * grp) ^ swz) << 4)), hi = lds128(crow + (((2 * grp + 1) ^ swz) << 4));
          const uint32_t cw[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
          uint32_t r[32];
          if (!valid) {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = 0u;
          } else if (!qp_f32 && dq_fast_ok(sc, bi)) {
            const uint32_t s2b = sc | (sc << 16), b2b = bi | (bi << 16);
            const __nv_bfloat162 s2 = *reinterpret_cast<const __nv_bfloat162*>(&s2b);
            const __nv_bfloat162 b2 = *reinterpret_cast<const __nv_bfloat162*>(&b2b);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const uint4 v = dq_word_fast(cw[c], s2, b2);
              r[4 * c] = v.x; r[4 * c + 1] = v.y; r[4 * c + 2] = v.z; r[4 * c + 3] = v.w;
            }
          } else {
            const float fs = __uint_as_float(qp_f32 ? sc : sc << 16), fb = __uint_as_float(qp_f32 ? bi : bi << 16);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const uint4 v = dq_word_f32(cw[c], fs, fb);
              r[4 * c] = v.x; r[4 * c + 1] = v.y; r[4 * c + 2] = v.z; r[4 * c + 3] = v.w;
            }
          }
          const uint32_t it = it0 + kb;
          const int s = it % STAGES;
          ok = mbar_wait_warp(&sm.empty[s], ((it / STAGES) & 1) ^ 1, sm.abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          tmem_st_x32(tmem_base + TMEM_A + s * (KB / 2) + lane_off, r);
          tmem_wait_st();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.full[s]);
        }
        // only now: an arrive right behind the shared-memory loads could pass them (see ce_logits_kernel)
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.cempty[cs]);
      }
    }
    if (!ok && lane == 0) raise(sm, p.status, kDevTimeoutProducer);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

std::atomic<int> g_configured[64];

int num_groups(int64_t n) { return static_cast<int>(ceil_div(n, kMostTokens)); }

}  // namespace

int ce_int4_fwd_splits(int64_t n, int64_t v_rows) {
  return ce_tc_choose_splits(num_groups(n), static_cast<int>(ceil_div(v_rows, VROWS)), sm_count());
}

int ce_int4_launch_fwd(const void* hidden, const QuantHead& q, int64_t v_rows, int64_t n, int d, int64_t vocab_id0,
                       const int64_t* targets, int64_t ignore_index, int splits, float* pm, float* ps, float* pt,
                       cudaStream_t stream, int* status) {
  int dev = 0;
  B200TP_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !g_configured[dev].load(std::memory_order_acquire)) {
    B200TP_CUDA_OK(cudaFuncSetAttribute(int4_logits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    if (dev >= 0 && dev < 64) g_configured[dev].store(1, std::memory_order_release);
  }
  Int4Params p{};
  p.n_rows = static_cast<int>(n);
  p.kblocks = d / KB;
  p.v_rows = static_cast<int>(v_rows);
  p.num_vt = static_cast<int>(ceil_div(v_rows, VROWS));
  p.splits = splits;
  p.groups = num_groups(n);
  p.gsz = static_cast<int>(align_up(ceil_div(n, p.groups), 16));
  // one MMA takes at most 256 columns
  p.boxes = p.gsz > 256 ? 2 : 1;
  p.n0 = p.boxes == 1 ? p.gsz : static_cast<int>(align_up(p.gsz / 2, 16));
  p.n1 = p.gsz - p.n0;
  p.vocab_id0 = vocab_id0;
  p.targets = reinterpret_cast<const long long*>(targets);
  p.ignore_index = ignore_index;
  p.pm = pm;
  p.ps = ps;
  p.pt = pt;
  p.scales = q.scales;
  p.biases = q.biases;
  p.qp_f32 = q.qp_f32;
  p.qvec = !q.qp_f32 && d % 512 == 0 &&
           ((reinterpret_cast<uintptr_t>(q.scales) | reinterpret_cast<uintptr_t>(q.biases)) & 15) == 0;
  p.status = status;
  CUtensorMap tmap_h, tmap_c;
  int rc = make_tmap_2d_bf16(&tmap_h, hidden, n, d, d, p.n0, KB);
  if (rc) return rc;
  rc = make_tmap_2d_u32(&tmap_c, q.wq, v_rows, d / 8, d / 8, VROWS, 16);
  if (rc) return rc;
  const int grid = std::min(sm_count(), p.groups * splits);
  int4_logits_kernel<<<grid, THREADS, SMEM_BYTES, stream>>>(tmap_h, tmap_c, p);
  B200TP_CUDA_OK(cudaGetLastError());
  return B200TP_OK;
}

}  // namespace b200tp
