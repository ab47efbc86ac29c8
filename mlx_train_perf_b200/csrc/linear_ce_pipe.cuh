// The scaffolding the tensor-core kernels of the linear cross-entropy share: tile sizes, the shared-memory ring and
// its barriers, CTA set-up and teardown, and what a timed-out wait does.
#pragma once

#include <algorithm>

#include "linear_ce_tc.h"
#include "ptx.cuh"

namespace b200tp {
namespace {

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int STAGES = 4;
constexpr int A_BYTES = BM * BK * 2;  // 16 KiB
constexpr int B_BYTES = BN * BK * 2;  // 32 KiB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
// CTA pairs: a CTA holds half of B's tile, so its ring has six stages in the same space
constexpr int PAIR_STAGES = 6;
constexpr int PAIR_STAGE_BYTES = A_BYTES + B_BYTES / 2;
static_assert(PAIR_STAGES * PAIR_STAGE_BYTES == STAGES * STAGE_BYTES, "one ring size");
constexpr int DQ_WARPS = 8;                       // dequantising warps of the QUANT kernels
constexpr int CODE_BYTES = 32 * 1024;             // QUANT: ring of packed-code tiles filled by TMA
constexpr int CODE_SLOTS_LOGITS = 2;              // 256 rows x 64 B (two k blocks) = 16 KiB each
constexpr int CODE_SLOTS_DH = 4;                  // 64 rows x 128 B (one k block, 256 columns) = 8 KiB each
constexpr int BAR_BYTES = 256;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + BAR_BYTES + 1024;  // + alignment slack
constexpr int SMEM_BYTES_Q = SMEM_BYTES + CODE_BYTES;
constexpr uint32_t TMEM_COLS = 512;                                  // two 256-column accumulators

struct SmemView {
  uint8_t* base;
  int stages, stage_bytes;
  uint64_t* full;
  uint64_t* empty;
  uint64_t* tfull;
  uint64_t* tempty;
  uint32_t* tmem_ptr;
  int* abort_flag;
  uint8_t* codes;       // QUANT only
  uint64_t* cfull;      // [4]
  uint64_t* cempty;     // [4]
  __device__ uint8_t* a(int s) const { return base + s * stage_bytes; }
  __device__ uint8_t* b(int s) const { return base + s * stage_bytes + A_BYTES; }
};

__device__ __forceinline__ SmemView carve_smem(uint8_t* raw, bool quant = false, bool pair = false) {
  const uint32_t addr = smem_u32(raw);
  const uint32_t aligned = (addr + 1023u) & ~1023u;
  SmemView v;
  v.base = raw + (aligned - addr);
  v.stages = pair ? PAIR_STAGES : STAGES;
  v.stage_bytes = pair ? PAIR_STAGE_BYTES : STAGE_BYTES;
  v.codes = v.base + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v.base + STAGES * STAGE_BYTES + (quant ? CODE_BYTES : 0));
  v.cfull = bars + 2 * STAGES + 6;
  v.cempty = bars + 2 * STAGES + 10;
  v.full = bars;
  v.empty = bars + v.stages;
  v.tfull = bars + 2 * v.stages;
  v.tempty = bars + 2 * v.stages + 2;
  v.tmem_ptr = reinterpret_cast<uint32_t*>(bars + 2 * v.stages + 4);
  v.abort_flag = reinterpret_cast<int*>(v.tmem_ptr + 1);
  return v;
}

__device__ __forceinline__ void raise_abort(const SmemView& sm, int* status, int code) {
  atomicExch(sm.abort_flag, 1);
  if (status != nullptr) atomicCAS(status, 0, code);
}

// Common prologue: barriers, TMEM allocation.  Returns the TMEM base address.
__device__ __forceinline__ uint32_t cta_setup(const SmemView& sm, int warp, uint32_t full_count = 1,
                                              uint32_t epi_warps = 4, bool pair = false) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < sm.stages; ++s) {
      mbar_init(&sm.full[s], full_count);   // the TMA producer's arrive.expect_tx (+ one per dequantising warp)
      mbar_init(&sm.empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sm.tfull[s], 1);
      mbar_init(&sm.tempty[s], epi_warps);  // one arrive per epilogue warp
    }
    if (full_count > 1) {
      for (int s = 0; s < 4; ++s) {
        mbar_init(&sm.cfull[s], 1);
        mbar_init(&sm.cempty[s], DQ_WARPS);
      }
    }
    *sm.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    if (pair) {
      tmem_alloc_pair(sm.tmem_ptr, TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(sm.tmem_ptr, TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  if (pair) cluster_sync();   // the other CTA's barriers are initialised too
  else __syncthreads();
  tc_fence_after_sync();
  return *reinterpret_cast<volatile uint32_t*>(sm.tmem_ptr);
}

// (A pair leaves together: until then the other CTA's MMAs, commits and arrivals may reach into this one.)
__device__ __forceinline__ void cta_teardown(const SmemView& sm, int warp, uint32_t tmem_base, bool pair = false) {
  tc_fence_before_sync();
  if (pair) cluster_sync();
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    if (pair) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// After an abort the producer may still have bulk copies in flight into this CTA's shared
// memory: wait (bounded) for every stage it armed before the CTA is allowed to retire.
__device__ __forceinline__ void producer_drain(const SmemView& sm, uint32_t it) {
  const uint32_t n = sm.stages, first = it > n ? it - n : 0;
  for (uint32_t j = first; j < it; ++j) mbar_wait_drain(&sm.full[j % n], (j / n) & 1);
}

template <bool PAIR>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                     uint32_t idesc, uint32_t accumulate) {
  if (PAIR) umma_ss_pair_w(tmem_d, a_lo, a_hi, b_lo, b_hi, idesc, accumulate);
  else umma_ss_w(tmem_d, a_lo, a_hi, b_lo, b_hi, idesc, accumulate);
}
template <bool PAIR>
__device__ __forceinline__ void commit(uint64_t* bar) {
  if (PAIR) umma_commit_pair(bar);
  else umma_commit(bar);
}
// An epilogue warp has read its accumulator: told to the CTA that issues the MMAs.
template <bool PAIR>
__device__ __forceinline__ void release_acc(uint64_t* bar) {
  if (PAIR) mbar_arrive_cluster(map_to_rank(bar, 0));
  else mbar_arrive(bar);
}

// `units` of work on pairs (`kernel` is a PAIR instantiation) or on single CTAs.  `pdl`: the kernel calls griddep_wait().
template <typename P>
int launch_units(void (*kernel)(CUtensorMap, CUtensorMap, P), int threads, bool pair, long long units,
                 cudaStream_t stream, const CUtensorMap& a, const CUtensorMap& b, const P& p, bool pdl = false) {
  cudaLaunchConfig_t cfg{};
  const long long most = pair ? sm_count() / 2 : sm_count();
  cfg.gridDim = dim3(static_cast<unsigned>(std::min(most, units) * (pair ? 2 : 1)));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  if (pair) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs++].val.clusterDim = {2, 1, 1};
  }
  if (pdl && pdl_enabled()) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  B200TP_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, a, b, p));
  return B200TP_OK;
}

}  // namespace
}  // namespace b200tp
