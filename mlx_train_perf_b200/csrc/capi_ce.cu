// C ABI of the fused linear cross-entropy: argument checks, workspace carving and the
// per-chunk launch sequences of the two implementations (tcgen05 and SIMT).
#include <string>

#include "common.h"
#include "linear_ce_grad.h"
#include "linear_ce_simt.h"
#include "linear_ce_split.h"
#include "linear_ce_tc.h"

namespace b200tp {
const char* last_error_cstr();

namespace {

// Default upper bound on the vocab rows per backward chunk: kTcChunkRowsMax, fewer when N is so large that
// the (N, chunk) bf16 matrix of g would exceed kTcScratchBytes.  Measured at N=8192, D=4096, V=151936
// (backward alone, ms / workspace): bound 4096 20.0 / 192 MB, 8192 18.3 / 256 MB, 16384 18.2 / 368 MB,
// 32768 17.5 / 604 MB, larger no faster.  Inside the power-capped forward + backward step the last gain
// disappears (24.73 against 24.81 ms per step), so the default stays at the smaller scratch.
constexpr int64_t kTcChunkRowsMax = 16384;
constexpr int64_t kTcChunkRowsMin = 2048;
constexpr int64_t kTcScratchBytes = 512ll << 20;
constexpr int64_t kSimtChunkRows = 4096;  // vocab rows per SIMT chunk
// fp32 on the tensor cores: bound of what a chunk's planes take (weight rows, in the backward g too), as much as
// the CUDA-core path's (N, 4096) fp32 tile at 8192 rows, and the chunk widths it may give
constexpr int64_t kSplitScratchBytes = 128ll << 20;
constexpr int64_t kSplitWorkMin = 1ll << 28;   // multiplications of a contraction (see pick_impl)
constexpr int64_t kSplitChunkRowsMin = 2048, kSplitChunkRowsMax = 16384;

// Vocab rows per tensor-core backward chunk for a shard of `v` rows.  The bound (the default above, or what
// the caller asked for in `reserved`) trades scratch for launches: the (N, chunk) bf16 matrix of g is the
// backward's main workspace.  The rows are spread evenly over the fewest chunks the bound allows (a
// short last chunk would keep the second GEMM's contraction too short to hide its fp32 accumulator
// round trip).
constexpr int kReservedInline = 0x10000;    // 4-bit head: expand inside the kernels whatever the row count
constexpr int kReservedChunked = 0x20000;   // 4-bit head: dequantise chunk by chunk whatever the row count
constexpr int kReservedSplit = 0x40000;     // fp32, dense head: the tensor cores whatever the size
constexpr int64_t kInlineMaxRows = 2048;    // default: the forward expands in the kernel up to this many rows of hidden

// `grow` (the forward that also forms the gradient): few rows take wider chunks, up to the scratch that
// 8192 rows use anyway.  A chunk ends in a partly filled wave of tiles and an fp32 round trip of d_hidden in each of
// its two GEMMs: at 1000 x 4096 x 151936 ten chunks make 40 tile times of logits out of 32.1 full waves, two make
// 34 (training step 2.63 -> 2.30 ms; 60 x 1024 x 32768 in one chunk instead of two: GPU time 94 -> 58 us).
// A 4-bit head's chunk is dequantised too: at most twice the rows of the default, within what both tiles take at 8192
// rows and D = 4096 (2048 x 4096 x 151936: training step 4.64 -> 4.46 ms).
constexpr int64_t kGrowScratchBytes = 256ll << 20;
constexpr int64_t kGrowQuantBytes = 384ll << 20, kGrowQuantRows = 2 * kTcChunkRowsMax;

int64_t tc_chunk_rows(const b200tp_ce_args* a, int64_t* num_chunks, bool grow = false) {
  int64_t bound = static_cast<int64_t>(a->reserved & 0xFFFF) * kCeTileCols;
  if (bound <= 0) {
    const int64_t fit = kTcScratchBytes / (2 * std::max<int64_t>(a->n, 1)) / kCeTileCols * kCeTileCols;
    bound = std::min(kTcChunkRowsMax, std::max(kTcChunkRowsMin, fit));
    if (grow) {
      const int64_t fits = a->quant_bits == 0 ? kGrowScratchBytes / (2 * a->n)
                                              : std::min(kGrowQuantRows, kGrowQuantBytes / (2 * (a->n + a->d)));
      bound = std::max(bound, fits / kCeTileCols * kCeTileCols);
    }
  }
  const int64_t nc = ceil_div(a->v_local, bound);
  *num_chunks = nc;
  return static_cast<int64_t>(align_up(static_cast<size_t>(ceil_div(a->v_local, nc)), kCeTileCols));
}

struct Bump {
  char* base;
  size_t off = 0;
  explicit Bump(void* p) : base(static_cast<char*>(p)) {}
  template <typename T>
  T* take(size_t count) {
    off = align_up(off, 256);
    T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
    off += count * sizeof(T);
    return p;
  }
};

int check_args(const b200tp_ce_args* a) {
  if (a == nullptr) return fail(B200TP_ERR_LOSS_INPUT, "args is null");
  if (a->n <= 0) return fail(B200TP_ERR_LOSS_INPUT, "hidden must have at least one row (n=" + std::to_string(a->n) + ")");
  if (a->d <= 0 || a->v_local <= 0) return fail(B200TP_ERR_LOSS_INPUT, "d and v_local must be positive");
  if (a->n > (1ll << 30) || a->v_local > (1ll << 30)) return fail(B200TP_ERR_LOSS_INPUT, "n / v_local too large");
  if (a->dtype != B200TP_F32 && a->dtype != B200TP_BF16)
    return fail(B200TP_ERR_UNSUPPORTED_HEAD, "only fp32 / bf16 hidden dtypes are supported");
  if (a->hidden == nullptr || a->targets == nullptr) return fail(B200TP_ERR_LOSS_INPUT, "hidden / targets is null");
  if (a->quant_bits == 0) {
    if (a->weight == nullptr) return fail(B200TP_ERR_LOSS_INPUT, "dense head without a weight pointer");
  } else if (a->quant_bits == 4) {
    if (a->group_size != 64)
      return fail(B200TP_ERR_UNSUPPORTED_HEAD, "only group_size=64 quantized heads are supported (got " +
                                                   std::to_string(a->group_size) + ")");
    if (a->d % 64 != 0)
      return fail(B200TP_ERR_UNSUPPORTED_HEAD, "a quantized head needs a hidden size that is a multiple of 64");
    if (a->w_q == nullptr || a->scales == nullptr || a->biases == nullptr)
      return fail(B200TP_ERR_LOSS_INPUT, "quantized head with a null w_q / scales / biases pointer");
    if (a->qparam_dtype != B200TP_F32 && a->qparam_dtype != B200TP_BF16)
      return fail(B200TP_ERR_UNSUPPORTED_HEAD, "scales / biases must be fp32 or bf16");
  } else {
    return fail(B200TP_ERR_UNSUPPORTED_HEAD,
                "only 4-bit quantized heads are supported (got bits=" + std::to_string(a->quant_bits) + ")");
  }
  if (a->impl != B200TP_IMPL_AUTO && a->impl != B200TP_IMPL_TC && a->impl != B200TP_IMPL_SIMT)
    return fail(B200TP_ERR_LOSS_INPUT, "unknown impl selector");
  if (a->reserved < 0 || (a->reserved & ~(0xFFFF | kReservedInline | kReservedChunked | kReservedSplit)) != 0 ||
      (a->reserved & (kReservedInline | kReservedChunked)) == (kReservedInline | kReservedChunked))
    return fail(B200TP_ERR_LOSS_INPUT,
                "reserved holds the backward chunk bound (low 16 bits, units of 256 vocab rows) and at most one of "
                "the 4-bit dequantisation selectors 0x10000 / 0x20000, and 0x40000");
  return B200TP_OK;
}

// Where a 4-bit head is expanded on the tensor-core path.
//   in the kernels: the weight operand never exists in global memory.  The forward's default kernel expands a code
//     once per 320 rows of hidden (linear_ce_int4.cu); the kernels that `reserved` selects (bit for bit the dense ones
//     on dequantised weights, and the only ones of the backward) once per 128;
//   chunk by chunk into a bf16 scratch (one pass over the codes per GEMM pass, 0.03 ms per 16384 x 4096
//     chunk) followed by the dense kernels.
// Default, from timings at D=4096, V=151936 (in-kernel / chunked, us): forward 260 / 692 at N=60, 304 / 884 at 257,
// 563 / 815 at 512, 1176 / 1344 at 1024, 2050 / 2245 at 2048, 4373 / 4194 at 4096 -- in the kernel up to
// kInlineMaxRows rows, with no weight scratch at all; backward 3.2 / 1.9 ms at N=128, 3.8 / 2.1 at 512 -- always
// chunked: with few row blocks the d_hidden GEMM has only D / 256 tiles, so a handful of CTAs would each expand their
// 256 columns of the whole head, while the dequantisation kernel spreads the same work over every SM.  `reserved`
// can force either form in both directions (in-kernel needs no weight scratch).  The in-kernel path
// needs a 16-byte aligned w_q (TMA).
bool quant_inline(const b200tp_ce_args* a, bool backward) {
  if (a->quant_bits != 4 || (reinterpret_cast<uintptr_t>(a->w_q) & 15) != 0) return false;
  if (a->reserved & kReservedInline) return true;
  if (a->reserved & kReservedChunked) return false;
  return !backward && a->n <= kInlineMaxRows;
}

QuantHead packed_head(const b200tp_ce_args* a) {
  QuantHead q{};
  q.wq = a->w_q;
  q.scales = a->scales;
  q.biases = a->biases;
  q.qp_f32 = a->qparam_dtype == B200TP_F32 ? 1 : 0;
  return q;
}

QuantHead quant_head(const b200tp_ce_args* a, bool backward) {
  return quant_inline(a, backward) ? packed_head(a) : QuantHead{};
}

// Whether a contraction is large enough for the planes to be the faster form (see pick_impl).
bool split_pays(const b200tp_ce_args* a) { return a->n * a->v_local >= kSplitWorkMin / a->d; }

// 1 = tcgen05, 2 = SIMT, 3 = tcgen05 over the three bf16 planes of fp32 operands, negative = refusal already
// recorded.  3 is the default for fp32 with a dense head: 2048 x 1024 x 32768 forward + backward 18.5 -> 1.65 ms, with
// a third of the CUDA-core path's distance to float64.  The CUDA cores keep the contraction of a trained head's
// gradient (its g comes from the planes like the forward's lse), D % 8 != 0 (TMA strides), a 4-bit head under fp32
// hidden states, and calls whose contraction is under 2^28 multiplications: there the CUDA cores need no longer than
// the split's extra launches take (forward / forward + backward, CUDA cores against split: 128 x 512 x 2000 65 / 259
// against 90 / 282 us, 32 x 1024 x 32000 1001 / 4151 against 173 / 430 us).
int pick_impl(const b200tp_ce_args* a) {
  const bool tc_ok = a->dtype == B200TP_BF16 && a->d % 8 == 0;
  if (a->impl == B200TP_IMPL_SIMT) return 2;
  if (a->impl == B200TP_IMPL_TC) {
    if (!tc_ok) {
      fail(B200TP_ERR_UNSUPPORTED_HEAD,
           "the tensor-core path needs bf16 operands and a hidden size that is a multiple of 8; use impl=simt");
      return -1;
    }
    if ((a->reserved & kReservedInline) && !quant_inline(a, false)) {
      fail(B200TP_ERR_UNSUPPORTED_HEAD, "in-kernel dequantisation needs a 4-bit head with a 16-byte aligned w_q");
      return -1;
    }
    return 1;
  }
  if (tc_ok) return 1;
  const bool large = (a->reserved & kReservedSplit) != 0 || split_pays(a);
  return a->dtype == B200TP_F32 && a->quant_bits == 0 && a->d % 8 == 0 && large ? 3 : 2;
}

int64_t split_chunk_rows(const b200tp_ce_args* a, int64_t bytes_per_row, int64_t* num_chunks) {
  int64_t bound = static_cast<int64_t>(a->reserved & 0xFFFF) * kCeTileCols;
  if (bound <= 0)
    bound = std::min(kSplitChunkRowsMax,
                     std::max(kSplitChunkRowsMin, kSplitScratchBytes / bytes_per_row / kCeTileCols * kCeTileCols));
  *num_chunks = ceil_div(a->v_local, bound);
  return static_cast<int64_t>(align_up(static_cast<size_t>(ceil_div(a->v_local, *num_chunks)), kCeTileCols));
}

size_t elem_size(int dtype) { return dtype == B200TP_BF16 ? 2 : 4; }

struct FwdPlan {
  int impl;
  int64_t chunk;        // vocab rows per launch (tc dense: all)
  int64_t num_chunks;
  int64_t total_splits; // tc only
  bool int4;            // tc: the head is expanded into tensor memory (linear_ce_int4.cu)
  // workspace pointers
  float* pm; float* ps; float* pt;
  void* deq;
  float* logits;
  // fp32 on the tensor cores: the planes; `logits` overlays the weight's, `simt_chunk` columns of it fit
  int* flag;
  void* h3; void* w3;
  int64_t simt_chunk;
  size_t bytes;
};

FwdPlan plan_fwd(const b200tp_ce_args* a, void* ws) {
  FwdPlan p{};
  p.impl = pick_impl(a);
  if (p.impl < 0) return p;
  Bump b(ws);
  if (p.impl == 1) {
    if (a->quant_bits == 0 || quant_inline(a, false)) {
      // one launch over the whole shard (a 4-bit head is expanded inside the kernel, tile by tile)
      p.chunk = a->v_local;
      p.num_chunks = 1;
      p.int4 = a->quant_bits != 0 && (a->reserved & kReservedInline) == 0;
      p.total_splits = p.int4 ? ce_int4_fwd_splits(a->n, a->v_local) : ce_tc_fwd_splits(a->n, a->d, a->v_local);
    } else {
      // 4-bit head, chunked: dequantise a chunk of vocab rows, run the dense kernel over it
      p.chunk = tc_chunk_rows(a, &p.num_chunks);
      p.total_splits = 0;
      for (int64_t c = 0; c < p.num_chunks; ++c) {
        const int64_t w = std::min<int64_t>(p.chunk, a->v_local - c * p.chunk);
        p.total_splits += ce_tc_fwd_splits(a->n, a->d, w);
      }
      p.deq = b.take<char>(static_cast<size_t>(p.chunk) * a->d * 2);
    }
    p.pm = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
    p.ps = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
    p.pt = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
  } else if (p.impl == 3) {
    p.chunk = split_chunk_rows(a, 6ll * a->d, &p.num_chunks);
    for (int64_t c = 0; c < p.num_chunks; ++c)
      p.total_splits += 2 * ce_split_splits(a->n, std::min<int64_t>(p.chunk, a->v_local - c * p.chunk));
    p.flag = b.take<int>(1);
    p.h3 = b.take<char>(static_cast<size_t>(a->n) * a->d * 6);
    const size_t planes = static_cast<size_t>(p.chunk) * a->d * 6;
    const size_t least = static_cast<size_t>(a->n) * std::min<int64_t>(kSimtChunkRows, a->v_local) * 4;
    p.w3 = b.take<char>(std::max(planes, least));
    p.logits = static_cast<float*>(p.w3);
    p.simt_chunk = std::min<int64_t>(a->v_local, static_cast<int64_t>(std::max(planes, least) / 4) / a->n);
    p.pm = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
    p.ps = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
    p.pt = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
  } else {
    p.chunk = std::min<int64_t>(kSimtChunkRows, a->v_local);
    p.num_chunks = ceil_div(a->v_local, p.chunk);
    p.logits = b.take<float>(static_cast<size_t>(a->n) * p.chunk);
    p.simt_chunk = p.chunk;
    if (a->quant_bits != 0) p.deq = b.take<char>(static_cast<size_t>(p.chunk) * a->d * elem_size(a->dtype));
  }
  p.bytes = align_up(b.off, 256);
  return p;
}

struct BwdPlan {
  int impl;
  int64_t chunk, num_chunks;
  int ldg;
  void* g;        // tc: bf16 (n, ldg)
  float* logits;  // simt: f32 (n, chunk)
  float* acc;     // f32 (n, d) when the output is bf16 and must be accumulated in fp32
  void* deq;
  // fp32 on the tensor cores: the planes, `shares` partial sums of d_hidden; `logits` overlays g's planes
  int* flag;
  void* h3; void* w3; void* g3;
  float* shares_acc;
  int shares;
  int64_t simt_chunk;
  size_t bytes;
};

BwdPlan plan_bwd(const b200tp_ce_args* a, int out_dtype, void* ws) {
  BwdPlan p{};
  p.impl = pick_impl(a);
  if (p.impl < 0) return p;
  Bump b(ws);
  if (p.impl == 1) {
    p.chunk = tc_chunk_rows(a, &p.num_chunks);
    p.ldg = static_cast<int>(p.chunk);
    p.g = b.take<char>(static_cast<size_t>(a->n) * p.ldg * 2);
    if (out_dtype == B200TP_BF16 && p.num_chunks > 1) p.acc = b.take<float>(static_cast<size_t>(a->n) * a->d);
    if (a->quant_bits != 0 && !quant_inline(a, true)) p.deq = b.take<char>(static_cast<size_t>(p.chunk) * a->d * 2);
  } else if (p.impl == 3) {
    p.chunk = split_chunk_rows(a, 6ll * (a->n + a->d), &p.num_chunks);
    p.ldg = static_cast<int>(p.chunk);
    p.shares = ce_split_dh_shares(a->n, a->d, p.chunk);
    p.flag = b.take<int>(1);
    p.h3 = b.take<char>(static_cast<size_t>(a->n) * a->d * 6);
    p.w3 = b.take<char>(static_cast<size_t>(p.chunk) * a->d * 6);
    p.g3 = b.take<char>(static_cast<size_t>(a->n) * p.chunk * 6);
    p.shares_acc = b.take<float>(static_cast<size_t>(p.shares) * a->n * a->d);
    p.logits = static_cast<float*>(p.g3);
    p.simt_chunk = std::min<int64_t>(a->v_local, p.chunk * 6 / 4);
  } else {
    p.chunk = std::min<int64_t>(kSimtChunkRows, a->v_local);
    p.num_chunks = ceil_div(a->v_local, p.chunk);
    p.logits = b.take<float>(static_cast<size_t>(a->n) * p.chunk);
    p.simt_chunk = p.chunk;
    if (out_dtype == B200TP_BF16) p.acc = b.take<float>(static_cast<size_t>(a->n) * a->d);
    if (a->quant_bits != 0) p.deq = b.take<char>(static_cast<size_t>(p.chunk) * a->d * elem_size(a->dtype));
  }
  p.bytes = align_up(b.off, 256);
  return p;
}

// Forward that also forms the gradient: what it leaves for the backward (`state`) and its scratch.  The scratch
// is like the recomputing backward's: one (N, chunk) bf16 tile, one dequantised chunk of a 4-bit head, plus the
// forward's partial triples.
struct GradPlan {
  bool ok;
  int impl;              // 1 or 3, as pick_impl's
  int64_t chunk, num_chunks;
  int shares;            // partial sums of d_hidden (see ce_tc_dh_ksplit)
  int64_t total_splits;
  // state
  int* overflow;         // [0]: the sums are void; fp32: [1]: an operand had no planes; [2]: that, or g's own had none
  float* ref2;           // (n), log2 units; fp32: natural units
  float* acc;            // (shares, n, d)
  size_t state_bytes;
  // scratch
  void* g;
  void* deq;
  float* pm; float* ps; float* pt;
  size_t bytes;          // forward
  float* ct;             // (n): the cotangents of a reduced loss
  size_t bwd_bytes;      // backward: g, deq and ct
  // fp32: planes; `logits` overlays g's
  void* h3; void* w3;
  float* logits;
  int64_t simt_chunk;
  // fp32: void sums are computed again from planes, by the CUDA cores only where a value has none -- or where these are
  // the faster form anyway.  One row of 2048 x 1024 x 32768 at 100 nats: 3.0 ms a step (2.1 without such a row), on the
  // CUDA cores 19.9.
  bool planes_again;
};

GradPlan plan_grad(const b200tp_ce_args* a, void* state, void* ws) {
  GradPlan p{};
  p.impl = pick_impl(a);
  p.ok = p.impl == 3 || (p.impl == 1 && (a->reserved & kReservedInline) == 0);
  if (!p.ok) return p;
  if (p.impl == 3) {
    p.chunk = split_chunk_rows(a, 6ll * (a->n + a->d), &p.num_chunks);
    p.shares = ce_split_dh_shares(a->n, a->d, p.chunk);
    p.planes_again = split_pays(a);
    Bump st(state);
    p.overflow = st.take<int>(3);
    p.ref2 = st.take<float>(a->n);
    p.acc = st.take<float>(static_cast<size_t>(p.shares) * a->n * a->d);
    p.state_bytes = align_up(st.off, 256);
    Bump b(ws);
    p.g = b.take<char>(static_cast<size_t>(a->n) * p.chunk * 6);
    p.logits = static_cast<float*>(p.g);
    p.simt_chunk = std::min<int64_t>(a->v_local, p.chunk * 6 / 4);
    p.ct = b.take<float>(a->n);
    if (!p.planes_again) p.bwd_bytes = align_up(b.off, 256);
    p.h3 = b.take<char>(static_cast<size_t>(a->n) * a->d * 6);
    p.w3 = b.take<char>(static_cast<size_t>(p.chunk) * a->d * 6);
    if (p.planes_again) p.bwd_bytes = align_up(b.off, 256);
    for (int64_t c = 0; c < p.num_chunks; ++c)
      p.total_splits += 2 * ce_split_splits(a->n, std::min<int64_t>(p.chunk, a->v_local - c * p.chunk));
    p.pm = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
    p.ps = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
    p.pt = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
    p.bytes = align_up(b.off, 256);
    return p;
  }
  p.chunk = tc_chunk_rows(a, &p.num_chunks, true);
  p.shares = ce_tc_dh_ksplit(a->n, a->d, static_cast<int>(p.chunk));
  Bump st(state);
  p.overflow = st.take<int>(1);
  p.ref2 = st.take<float>(a->n);
  p.acc = st.take<float>(static_cast<size_t>(p.shares) * a->n * a->d);
  p.state_bytes = align_up(st.off, 256);
  Bump b(ws);
  p.g = b.take<char>(static_cast<size_t>(a->n) * p.chunk * 2);
  if (a->quant_bits != 0) p.deq = b.take<char>(static_cast<size_t>(p.chunk) * a->d * 2);
  p.ct = b.take<float>(a->n);
  p.bwd_bytes = align_up(b.off, 256);
  for (int64_t c = 0; c < p.num_chunks; ++c)
    p.total_splits += ce_tc_fwd_splits(a->n, a->d, std::min<int64_t>(p.chunk, a->v_local - c * p.chunk));
  p.pm = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
  p.ps = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
  p.pt = b.take<float>(static_cast<size_t>(p.total_splits) * a->n);
  p.bytes = align_up(b.off, 256);
  return p;
}

int check_grad_args(const b200tp_ce_args* a) {
  int rc = check_args(a);
  if (rc) return rc;
  if (a->v_offset != 0)
    return fail(B200TP_ERR_LOSS_INPUT, "the forward with gradient needs the whole vocabulary (v_offset = 0)");
  return B200TP_OK;
}

// The bf16 row kernels around the forward that forms the gradient read whole 16-byte words ahead of any tensor map.
int check_grad_alignment(const b200tp_ce_args* a, const GradPlan& p, const void* d_hidden) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(a->hidden) | reinterpret_cast<uintptr_t>(d_hidden) |
                        (a->quant_bits == 0 ? reinterpret_cast<uintptr_t>(a->weight) : 0);
  if (p.impl == 1 && (all & 15) != 0)
    return fail(B200TP_ERR_LOSS_INPUT, "tensor base address must be 16-byte aligned for TMA");
  return B200TP_OK;
}

int check_workspace(void* ws, size_t have, size_t need) {
  if (need == 0) return B200TP_OK;
  if (ws == nullptr) return fail(B200TP_ERR_WORKSPACE, "workspace is null but " + std::to_string(need) + " bytes are needed");
  if ((reinterpret_cast<uintptr_t>(ws) & 255) != 0) return fail(B200TP_ERR_WORKSPACE, "workspace must be 256-byte aligned");
  if (have < need)
    return fail(B200TP_ERR_WORKSPACE,
                "workspace too small: have " + std::to_string(have) + ", need " + std::to_string(need) + " bytes");
  return B200TP_OK;
}

}  // namespace
}  // namespace b200tp

using namespace b200tp;

extern "C" {

size_t b200tp_linear_ce_fwd_workspace_bytes(const b200tp_ce_args* a) {
  if (check_args(a) != B200TP_OK) return 0;
  FwdPlan p = plan_fwd(a, nullptr);
  return p.impl < 0 ? 0 : p.bytes;
}

int b200tp_linear_ce_fwd(const b200tp_ce_args* a, float* row_max, float* row_sumexp, float* tgt_logit, float* lse,
                         float* nll, void* workspace, size_t workspace_bytes, void* stream_v, int* status) {
  int rc = check_args(a);
  if (rc) return rc;
  if (row_max == nullptr || row_sumexp == nullptr || tgt_logit == nullptr)
    return fail(B200TP_ERR_LOSS_INPUT, "row_max / row_sumexp / tgt_logit outputs are required");
  rc = require_sm100();
  if (rc) return rc;
  FwdPlan p = plan_fwd(a, workspace);
  if (p.impl < 0) return B200TP_ERR_UNSUPPORTED_HEAD;
  rc = check_workspace(workspace, workspace_bytes, p.bytes);
  if (rc) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);

  if (p.impl == 1) {
    if (p.deq == nullptr) {
      const int splits = static_cast<int>(p.total_splits);
      const QuantHead q = quant_head(a, false);
      if (p.int4)
        rc = ce_int4_launch_fwd(a->hidden, q, a->v_local, a->n, a->d, a->v_offset, a->targets,
                                a->ignore_index, splits, p.pm, p.ps, p.pt, stream, status);
      else
        rc = ce_tc_launch_fwd(a->hidden, a->weight, a->v_local, a->n, a->d, 0, a->v_local, a->v_offset, a->targets,
                              a->ignore_index, splits, p.pm, p.ps, p.pt, &q, stream, status);
      if (rc) return rc;
    } else {
      int64_t slot = 0;
      for (int64_t c = 0; c < p.num_chunks; ++c) {
        const int64_t r0 = c * p.chunk;
        const int64_t w = std::min<int64_t>(p.chunk, a->v_local - r0);
        rc = launch_dequant_int4(a->w_q, a->scales, a->biases, a->qparam_dtype, r0, w, a->d, a->group_size, p.deq,
                                 B200TP_BF16, stream);
        if (rc) return rc;
        const int splits = ce_tc_fwd_splits(a->n, a->d, w);
        rc = ce_tc_launch_fwd(a->hidden, p.deq, w, a->n, a->d, 0, w, a->v_offset + r0, a->targets, a->ignore_index,
                              splits, p.pm + slot * a->n, p.ps + slot * a->n, p.pt + slot * a->n, nullptr, stream,
                              status);
        if (rc) return rc;
        slot += splits;
      }
    }
    return launch_combine(p.pm, p.ps, p.pt, a->n, static_cast<int>(p.total_splits), a->n, a->targets,
                          a->ignore_index, row_max, row_sumexp, tgt_logit, lse, nll, stream);
  }

  if (p.impl == 3) {
    B200TP_CUDA_OK(cudaMemsetAsync(p.flag, 0, sizeof(int), stream));
    rc = ce_split_planes(static_cast<const float*>(a->hidden), a->n * a->d, p.h3, p.flag, stream);
    if (rc) return rc;
    int64_t slot = 0;
    for (int64_t c = 0; c < p.num_chunks; ++c) {
      const int64_t r0 = c * p.chunk;
      const int64_t w = std::min<int64_t>(p.chunk, a->v_local - r0);
      rc = ce_split_planes(static_cast<const float*>(a->weight) + r0 * a->d, w * a->d, p.w3, p.flag, stream);
      if (rc) return rc;
      const int splits = ce_split_splits(a->n, w);
      rc = ce_split_fwd(p.h3, p.w3, a->n, a->d, w, a->v_offset + r0, a->targets, a->ignore_index, splits,
                        p.pm + slot * a->n, p.ps + slot * a->n, p.pt + slot * a->n, stream, status);
      if (rc) return rc;
      slot += 2 * splits;
    }
    rc = launch_combine(p.pm, p.ps, p.pt, a->n, static_cast<int>(p.total_splits), a->n, a->targets, a->ignore_index,
                        row_max, row_sumexp, tgt_logit, lse, nll, stream);
    if (rc) return rc;
  }

  // SIMT: running triples live directly in the caller's output arrays.  After the split path: only where it met
  // values its planes cannot hold.
  for (int64_t r0 = 0; r0 < a->v_local; r0 += p.simt_chunk) {
    const int64_t w = std::min<int64_t>(p.simt_chunk, a->v_local - r0);
    const void* wc;
    if (a->quant_bits == 0) {
      wc = static_cast<const char*>(a->weight) + static_cast<size_t>(r0) * a->d * elem_size(a->dtype);
    } else {
      rc = launch_dequant_int4(a->w_q, a->scales, a->biases, a->qparam_dtype, r0, w, a->d, a->group_size, p.deq,
                               a->dtype, stream);
      if (rc) return rc;
      wc = p.deq;
    }
    rc = ce_simt_fwd_chunk(a->hidden, wc, a->dtype, a->n, a->d, w, a->v_offset + r0, a->targets, a->ignore_index,
                           p.logits, row_max, row_sumexp, tgt_logit, r0 == 0 ? 1 : 0, stream, p.flag);
    if (rc) return rc;
  }
  return launch_combine(row_max, row_sumexp, tgt_logit, a->n, 1, a->n, a->targets, a->ignore_index, nullptr, nullptr,
                        tgt_logit, lse, nll, stream, p.flag);
}

int b200tp_linear_ce_combine(const float* parts, int32_t num_parts, int64_t n, const int64_t* targets,
                             int64_t ignore_index, float* lse, float* nll, float* tgt_logit, void* stream) {
  if (parts == nullptr || num_parts <= 0 || n <= 0)
    return fail(B200TP_ERR_LOSS_INPUT, "combine needs at least one part and one row");
  return launch_combine(parts, parts + n, parts + 2 * n, 3 * n, num_parts, n, targets, ignore_index, nullptr, nullptr,
                        tgt_logit, lse, nll, static_cast<cudaStream_t>(stream));
}

int b200tp_linear_ce_reduce(const float* nll, const int64_t* targets, int64_t n, int64_t ignore_index, float* out3,
                            void* stream) {
  if (nll == nullptr || out3 == nullptr || n <= 0)
    return fail(B200TP_ERR_LOSS_INPUT, "reduce needs nll, an output triple and at least one row");
  return launch_loss_reduce(nll, targets, n, ignore_index, out3, static_cast<cudaStream_t>(stream));
}

int b200tp_linear_ce_cotangent(const int64_t* targets, int64_t n, int64_t ignore_index, const float* upstream,
                               const float* count, float* cotangent, void* stream) {
  if (upstream == nullptr || cotangent == nullptr || n <= 0)
    return fail(B200TP_ERR_LOSS_INPUT, "cotangent needs the upstream scalar, an output vector and at least one row");
  return launch_loss_cotangent(targets, n, ignore_index, upstream, count, cotangent,
                               static_cast<cudaStream_t>(stream));
}

size_t b200tp_linear_ce_bwd_workspace_bytes(const b200tp_ce_args* a, int32_t d_hidden_dtype) {
  if (check_args(a) != B200TP_OK) return 0;
  BwdPlan p = plan_bwd(a, d_hidden_dtype, nullptr);
  return p.impl < 0 ? 0 : p.bytes;
}

// Stages: the tensor-core backward can be issued in `num_stages` calls.  Stage 0 launches everything
// up to and including the first slab of the LAST chunk's d_hidden GEMM; stage s > 0 launches slab s of
// it.  The slabs are whole waves of the row-block-major tile order, so their launches cost what the
// single launch costs, and the leading `*rows_done` rows of d_hidden are final once a stage's work has
// run.  num_stages == 1 is the plain backward.
static int bwd_impl(const b200tp_ce_args* a, const float* lse, const float* cotangent, void* d_hidden,
                    int32_t d_hidden_dtype, int32_t accumulate, void* d_weight, int num_stages, int stage,
                    int64_t* rows_done, void* workspace, size_t workspace_bytes, void* stream_v, int* status) {
  int rc = check_args(a);
  if (rc) return rc;
  if (d_weight != nullptr && a->quant_bits != 0)
    return fail(B200TP_ERR_UNSUPPORTED_HEAD, "a quantized head is frozen: it has no d_weight");
  if (lse == nullptr || cotangent == nullptr || d_hidden == nullptr)
    return fail(B200TP_ERR_LOSS_INPUT, "lse / cotangent / d_hidden is null");
  if (d_hidden_dtype != B200TP_F32 && d_hidden_dtype != a->dtype)
    return fail(B200TP_ERR_LOSS_INPUT, "d_hidden dtype must be the hidden dtype or fp32");
  if (accumulate && d_hidden_dtype != B200TP_F32)
    return fail(B200TP_ERR_LOSS_INPUT, "accumulate is only defined for an fp32 d_hidden");
  if (num_stages < 1 || num_stages > 64 || stage < 0 || stage >= num_stages)
    return fail(B200TP_ERR_LOSS_INPUT, "stage must lie in [0, num_stages) with 1 <= num_stages <= 64");
  rc = require_sm100();
  if (rc) return rc;
  BwdPlan p = plan_bwd(a, d_hidden_dtype, workspace);
  if (p.impl < 0) return B200TP_ERR_UNSUPPORTED_HEAD;
  rc = check_workspace(workspace, workspace_bytes, p.bytes);
  if (rc) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  const bool out_f32 = d_hidden_dtype == B200TP_F32;

  if (p.impl == 1) {
    const QuantHead q = quant_head(a, true);
    // slab `stage` of the last chunk's d_hidden tiles: whole waves of the persistent grid
    const int tiles = ce_tc_dh_tiles(a->n, a->d);
    const int ctas = sm_count();
    const int waves = static_cast<int>(ceil_div(tiles, ctas));
    auto slab_begin = [&](int s) { return std::min<int64_t>(tiles, static_cast<int64_t>(ctas) * (waves * s / num_stages)); };
    const int tile0 = static_cast<int>(slab_begin(stage));
    const int tile1 = stage + 1 == num_stages ? tiles : static_cast<int>(slab_begin(stage + 1));
    if (rows_done != nullptr) *rows_done = ce_tc_dh_rows_done(a->n, a->d, tile1);
    for (int64_t c = stage == 0 ? 0 : p.num_chunks - 1; c < p.num_chunks; ++c) {
      const int64_t r0 = c * p.chunk;
      const int64_t w = std::min<int64_t>(p.chunk, a->v_local - r0);
      const bool first = c == 0, last = c == p.num_chunks - 1;
      // weight operand of this chunk: rows [row0, row0 + w) of `wmat` (the dense head, the packed head, or
      // the chunk's dequantised copy, which stays valid for every stage's d_hidden launches of the chunk)
      const void* wmat = a->weight;
      int64_t wrows = a->v_local, row0 = r0, vocab_id0 = a->v_offset;
      const QuantHead* qp = &q;
      if (p.deq != nullptr) {
        if (stage == 0) {
          rc = launch_dequant_int4(a->w_q, a->scales, a->biases, a->qparam_dtype, r0, w, a->d, a->group_size, p.deq,
                                   B200TP_BF16, stream);
          if (rc) return rc;
        }
        wmat = p.deq;
        wrows = w;
        row0 = 0;
        vocab_id0 = a->v_offset + r0;
        qp = nullptr;
      }
      if (stage == 0) {
        rc = ce_tc_launch_bwd_g(a->hidden, wmat, wrows, a->n, a->d, row0, row0 + w, vocab_id0, a->targets,
                                a->ignore_index, lse, cotangent, p.g, p.ldg, qp, LaunchGuard{}, stream, status);
        if (rc) return rc;
      }
      const int k_total = static_cast<int>(align_up(w, kCeTileCols));
      const float* acc_in;
      float* acc_out;
      void* out_bf16;
      if (out_f32) {
        acc_in = (first && !accumulate) ? nullptr : static_cast<const float*>(d_hidden);
        acc_out = static_cast<float*>(d_hidden);
        out_bf16 = nullptr;
      } else {
        acc_in = first ? nullptr : p.acc;
        acc_out = last ? nullptr : p.acc;
        out_bf16 = last ? d_hidden : nullptr;
      }
      rc = ce_tc_launch_dh(p.g, p.ldg, k_total, a->n, wmat, wrows, a->d, row0, acc_in, acc_out, out_bf16,
                           last ? tile0 : -1, last ? tile1 : -1, 1, qp, LaunchGuard{}, stream, status);
      if (rc) return rc;
      if (d_weight != nullptr) {
        void* block = static_cast<char*>(d_weight) + static_cast<size_t>(r0) * a->d * elem_size(a->dtype);
        rc = ce_tc_launch_dw(p.g, p.ldg, w, a->n, a->hidden, a->d, block, stream, status);
        if (rc) return rc;
      }
    }
    return B200TP_OK;
  }

  // The other two paths are not staged (everything runs in stage 0).
  if (rows_done != nullptr) *rows_done = a->n;
  if (stage > 0) return B200TP_OK;
  if (p.impl == 3) {
    B200TP_CUDA_OK(cudaMemsetAsync(p.flag, 0, sizeof(int), stream));
    rc = ce_split_planes(static_cast<const float*>(a->hidden), a->n * a->d, p.h3, p.flag, stream);
    if (rc) return rc;
    for (int64_t c = 0; c < p.num_chunks; ++c) {
      const int64_t r0 = c * p.chunk;
      const int64_t w = std::min<int64_t>(p.chunk, a->v_local - r0);
      rc = ce_split_planes(static_cast<const float*>(a->weight) + r0 * a->d, w * a->d, p.w3, p.flag, stream);
      if (rc) return rc;
      rc = ce_split_bwd_g(p.h3, p.w3, a->n, a->d, w, a->v_offset + r0, a->targets, a->ignore_index, lse, cotangent,
                          ce_split_splits(a->n, w), p.g3, p.ldg, p.flag, stream, status);
      if (rc) return rc;
      rc = ce_split_dh(p.g3, p.ldg, p.w3, a->n, a->d, w, p.shares, p.shares_acc, c > 0, stream, status);
      if (rc) return rc;
      if (d_weight != nullptr) {
        // g from the same logits as the forward's lse, whose errors cancel in exp(z - lse); the contraction over the
        // rows on the CUDA cores
        rc = ce_simt_dw_planes(p.g3, p.ldg, w, static_cast<const float*>(a->hidden), a->n, a->d,
                               static_cast<float*>(d_weight) + r0 * a->d, p.flag, stream);
        if (rc) return rc;
      }
    }
    // d_hidden is only touched once it is known that the planes held every value
    rc = ce_split_sum(p.shares_acc, p.shares, a->n * a->d, static_cast<float*>(d_hidden), accumulate,
                      SplitGuard{nullptr, p.flag}, stream);
    if (rc) return rc;
  }
  float* acc = out_f32 ? static_cast<float*>(d_hidden) : p.acc;
  for (int64_t r0 = 0; r0 < a->v_local; r0 += p.simt_chunk) {
    const int64_t w = std::min<int64_t>(p.simt_chunk, a->v_local - r0);
    const void* wc;
    if (a->quant_bits == 0) {
      wc = static_cast<const char*>(a->weight) + static_cast<size_t>(r0) * a->d * elem_size(a->dtype);
    } else {
      rc = launch_dequant_int4(a->w_q, a->scales, a->biases, a->qparam_dtype, r0, w, a->d, a->group_size, p.deq,
                               a->dtype, stream);
      if (rc) return rc;
      wc = p.deq;
    }
    const int acc_flag = (r0 > 0 || (out_f32 && accumulate)) ? 1 : 0;
    rc = ce_simt_bwd_chunk(a->hidden, wc, a->dtype, a->n, a->d, w, a->v_offset + r0, a->targets, a->ignore_index, lse,
                           cotangent, p.logits, acc, acc_flag, stream, p.flag);
    if (rc) return rc;
    if (d_weight != nullptr) {
      void* block = static_cast<char*>(d_weight) + static_cast<size_t>(r0) * a->d * elem_size(a->dtype);
      rc = ce_simt_dw_chunk(p.logits, w, a->hidden, a->dtype, a->n, a->d, block, stream, p.flag);
      if (rc) return rc;
    }
  }
  if (!out_f32) return launch_cast_f32_to_bf16(acc, d_hidden, a->n * a->d, stream);
  return B200TP_OK;
}

int b200tp_linear_ce_bwd(const b200tp_ce_args* a, const float* lse, const float* cotangent, void* d_hidden,
                         int32_t d_hidden_dtype, int32_t accumulate, void* workspace, size_t workspace_bytes,
                         void* stream_v, int* status) {
  return bwd_impl(a, lse, cotangent, d_hidden, d_hidden_dtype, accumulate, nullptr, 1, 0, nullptr, workspace,
                  workspace_bytes, stream_v, status);
}

int b200tp_linear_ce_bwd_stage(const b200tp_ce_args* a, const float* lse, const float* cotangent, void* d_hidden,
                               int32_t d_hidden_dtype, int32_t accumulate, int32_t num_stages, int32_t stage,
                               int64_t* rows_done, void* workspace, size_t workspace_bytes, void* stream_v,
                               int* status) {
  return bwd_impl(a, lse, cotangent, d_hidden, d_hidden_dtype, accumulate, nullptr, num_stages, stage, rows_done,
                  workspace, workspace_bytes, stream_v, status);
}

int b200tp_linear_ce_bwd_train(const b200tp_ce_args* a, const float* lse, const float* cotangent, void* d_hidden,
                               int32_t d_hidden_dtype, int32_t accumulate, void* d_weight, void* workspace,
                               size_t workspace_bytes, void* stream_v, int* status) {
  if (d_weight == nullptr) return fail(B200TP_ERR_LOSS_INPUT, "d_weight is null");
  return bwd_impl(a, lse, cotangent, d_hidden, d_hidden_dtype, accumulate, d_weight, 1, 0, nullptr, workspace,
                  workspace_bytes, stream_v, status);
}

size_t b200tp_linear_ce_grad_state_bytes(const b200tp_ce_args* a) {
  return check_grad_args(a) == B200TP_OK ? plan_grad(a, nullptr, nullptr).state_bytes : 0;
}

size_t b200tp_linear_ce_fwd_grad_workspace_bytes(const b200tp_ce_args* a) {
  return check_grad_args(a) == B200TP_OK ? plan_grad(a, nullptr, nullptr).bytes : 0;
}

size_t b200tp_linear_ce_bwd_grad_workspace_bytes(const b200tp_ce_args* a) {
  return check_grad_args(a) == B200TP_OK ? plan_grad(a, nullptr, nullptr).bwd_bytes : 0;
}

int b200tp_linear_ce_fwd_grad(const b200tp_ce_args* a, float* tgt_logit, float* lse, float* nll, void* state,
                              size_t state_bytes, void* workspace, size_t workspace_bytes, void* stream_v,
                              int* status) {
  int rc = check_grad_args(a);
  if (rc) return rc;
  if (tgt_logit == nullptr || lse == nullptr || nll == nullptr)
    return fail(B200TP_ERR_LOSS_INPUT, "tgt_logit / lse / nll outputs are required");
  rc = require_sm100();
  if (rc) return rc;
  const GradPlan p = plan_grad(a, state, workspace);
  if (!p.ok)
    return fail(B200TP_ERR_UNSUPPORTED_HEAD, "the forward with gradient runs on the tensor-core path, 4-bit heads chunk-wise");
  rc = check_grad_alignment(a, p, nullptr);
  if (rc) return rc;
  rc = check_workspace(state, state_bytes, p.state_bytes);
  if (rc) return rc;
  rc = check_workspace(workspace, workspace_bytes, p.bytes);
  if (rc) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (p.impl == 3) {
    const float* hidden = static_cast<const float*>(a->hidden);
    const float* weight = static_cast<const float*>(a->weight);
    int *void_sums = p.overflow, *bad = p.overflow + 1;
    B200TP_CUDA_OK(cudaMemsetAsync(p.overflow, 0, 2 * sizeof(int), stream));
    rc = ce_split_reference(hidden, weight, a->n, a->d, a->v_local, a->targets, a->ignore_index, p.ref2, stream);
    if (rc) return rc;
    rc = ce_split_planes(hidden, a->n * a->d, p.h3, bad, stream);
    if (rc) return rc;
    int64_t slot = 0;
    for (int64_t c = 0; c < p.num_chunks; ++c) {
      const int64_t r0 = c * p.chunk;
      const int64_t w = std::min<int64_t>(p.chunk, a->v_local - r0);
      rc = ce_split_planes(weight + r0 * a->d, w * a->d, p.w3, bad, stream);
      if (rc) return rc;
      const int splits = ce_split_splits(a->n, w);
      rc = ce_split_fwd_grad(p.h3, p.w3, a->n, a->d, w, r0, a->targets, a->ignore_index, p.ref2, splits,
                             p.pm + slot * a->n, p.ps + slot * a->n, p.pt + slot * a->n, p.g,
                             static_cast<int>(p.chunk), bad, void_sums, stream, status);
      if (rc) return rc;
      slot += 2 * splits;
      // once the flag is set the sums are void: no need to go on with them
      rc = ce_split_dh(p.g, static_cast<int>(p.chunk), p.w3, a->n, a->d, w, p.shares, p.acc, c > 0, stream, status,
                       SplitGuard{nullptr, void_sums});
      if (rc) return rc;
    }
    rc = launch_combine(p.pm, p.ps, p.pt, a->n, static_cast<int>(p.total_splits), a->n, a->targets, a->ignore_index,
                        nullptr, nullptr, tgt_logit, lse, nll, stream);
    if (rc) return rc;
    // the CUDA cores, here and in the backward (which wants lse from the same logits as its own); the partials' space
    // holds their running triples
    const int* on_cores = p.planes_again ? bad : void_sums;
    for (int64_t r0 = 0; r0 < a->v_local; r0 += p.simt_chunk) {
      const int64_t w = std::min<int64_t>(p.simt_chunk, a->v_local - r0);
      rc = ce_simt_fwd_chunk(hidden, weight + r0 * a->d, a->dtype, a->n, a->d, w, r0, a->targets, a->ignore_index,
                             p.logits, p.pm, p.ps, tgt_logit, r0 == 0 ? 1 : 0, stream, on_cores);
      if (rc) return rc;
    }
    return launch_combine(p.pm, p.ps, tgt_logit, a->n, 1, a->n, a->targets, a->ignore_index, nullptr, nullptr,
                          tgt_logit, lse, nll, stream, on_cores);
  }
  const QuantHead q = packed_head(a);
  rc = launch_ce_reference(a->hidden, a->weight, a->quant_bits != 0 ? &q : nullptr, a->n, a->d, a->v_local, a->targets,
                           a->ignore_index, p.ref2, p.overflow, stream);
  if (rc) return rc;
  int64_t slot = 0;
  for (int64_t c = 0; c < p.num_chunks; ++c) {
    const int64_t r0 = c * p.chunk;
    const int64_t w = std::min<int64_t>(p.chunk, a->v_local - r0);
    const void* wmat = a->weight;
    int64_t wrows = a->v_local, row0 = r0, vocab_id0 = 0;
    if (p.deq != nullptr) {
      rc = launch_dequant_int4(a->w_q, a->scales, a->biases, a->qparam_dtype, r0, w, a->d, a->group_size, p.deq,
                               B200TP_BF16, stream);
      if (rc) return rc;
      wmat = p.deq;
      wrows = w;
      row0 = 0;
      vocab_id0 = r0;
    }
    const int splits = ce_tc_fwd_splits(a->n, a->d, w);
    rc = ce_tc_launch_fwd_grad(a->hidden, wmat, wrows, a->n, a->d, row0, row0 + w, vocab_id0, a->targets,
                               a->ignore_index, p.ref2, p.overflow, splits, p.pm + slot * a->n, p.ps + slot * a->n,
                               p.pt + slot * a->n, p.g, static_cast<int>(p.chunk), stream, status);
    if (rc) return rc;
    slot += splits;
    // once the flag is set the sums are void: no need to go on with them
    rc = ce_tc_launch_dh(p.g, static_cast<int>(p.chunk), static_cast<int>(align_up(w, kCeTileCols)), a->n, wmat, wrows,
                         a->d, row0, c == 0 ? nullptr : p.acc, p.acc, nullptr, -1, -1, p.shares, nullptr,
                         LaunchGuard{p.overflow, 0}, stream, status);
    if (rc) return rc;
  }
  return launch_combine(p.pm, p.ps, p.pt, a->n, static_cast<int>(p.total_splits), a->n, a->targets, a->ignore_index,
                        nullptr, nullptr, tgt_logit, lse, nll, stream);
}

// The rows' cotangents are `cotangent`, or formed here from `upstream` and `count`.
static int bwd_grad_impl(const b200tp_ce_args* a, const float* lse, const float* tgt_logit, const float* cotangent,
                         const float* upstream, const float* count, void* state, size_t state_bytes, void* d_hidden,
                         void* workspace, size_t workspace_bytes, void* stream_v, int* status) {
  int rc = check_grad_args(a);
  if (rc) return rc;
  if (lse == nullptr || tgt_logit == nullptr || (cotangent == nullptr && upstream == nullptr) || d_hidden == nullptr)
    return fail(B200TP_ERR_LOSS_INPUT, "lse / tgt_logit / cotangent / d_hidden is null");
  rc = require_sm100();
  if (rc) return rc;
  const GradPlan p = plan_grad(a, state, workspace);
  if (!p.ok)
    return fail(B200TP_ERR_UNSUPPORTED_HEAD, "the forward with gradient runs on the tensor-core path, 4-bit heads chunk-wise");
  rc = check_grad_alignment(a, p, d_hidden);
  if (rc) return rc;
  rc = check_workspace(state, state_bytes, p.state_bytes);
  if (rc) return rc;
  rc = check_workspace(workspace, workspace_bytes, p.bwd_bytes);
  if (rc) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (cotangent == nullptr) {
    rc = launch_loss_cotangent(a->targets, a->n, a->ignore_index, upstream, count, p.ct, stream);
    if (rc) return rc;
    cotangent = p.ct;
  }
  if (p.impl == 3) {
    const float* weight = static_cast<const float*>(a->weight);
    float* out = static_cast<float*>(d_hidden);
    rc = ce_split_finish(p.acc, p.shares, p.ref2, p.overflow, weight, a->n, a->d, a->v_local, a->targets,
                         a->ignore_index, lse, tgt_logit, cotangent, out, stream);
    if (rc) return rc;
    if (p.planes_again) {   // as bwd_impl; the void sums' space serves the shares
      const SplitGuard again{p.overflow, p.overflow + 1};
      const int ldg = static_cast<int>(p.chunk);
      int* flag = p.overflow + 2;
      rc = ce_split_planes(static_cast<const float*>(a->hidden), a->n * a->d, p.h3, flag, stream, again);
      if (rc) return rc;
      for (int64_t c = 0; c < p.num_chunks; ++c) {
        const int64_t r0 = c * p.chunk;
        const int64_t w = std::min<int64_t>(p.chunk, a->v_local - r0);
        rc = ce_split_planes(weight + r0 * a->d, w * a->d, p.w3, flag, stream, again);
        if (rc) return rc;
        rc = ce_split_bwd_g(p.h3, p.w3, a->n, a->d, w, r0, a->targets, a->ignore_index, lse, cotangent,
                            ce_split_splits(a->n, w), p.g, ldg, flag, stream, status, again);
        if (rc) return rc;
        rc = ce_split_dh(p.g, ldg, p.w3, a->n, a->d, w, p.shares, p.acc, c > 0, stream, status, again);
        if (rc) return rc;
      }
      rc = ce_split_sum(p.acc, p.shares, a->n * a->d, out, 0, SplitGuard{p.overflow, flag}, stream);
      if (rc) return rc;
    }
    const int* on_cores = p.planes_again ? p.overflow + 2 : p.overflow;
    for (int64_t r0 = 0; r0 < a->v_local; r0 += p.simt_chunk) {
      const int64_t w = std::min<int64_t>(p.simt_chunk, a->v_local - r0);
      rc = ce_simt_bwd_chunk(a->hidden, weight + r0 * a->d, a->dtype, a->n, a->d, w, r0, a->targets, a->ignore_index,
                             lse, cotangent, p.logits, out, r0 > 0, stream, on_cores);
      if (rc) return rc;
    }
    return B200TP_OK;
  }
  const QuantHead q = packed_head(a);
  rc = launch_ce_grad_finish(p.acc, p.shares, p.ref2, p.overflow, a->weight, a->quant_bits != 0 ? &q : nullptr, a->n,
                             a->d, a->v_local, a->targets, a->ignore_index, lse, tgt_logit, cotangent, d_hidden, stream);
  if (rc) return rc;
  // Overflowed references: recompute the logits chunk by chunk.  The sums in `state` are void then, so their
  // first share serves as the fp32 accumulator.  (1000 x 4096 x 151936, steps without such a row / with one / all of
  // them: 1.86 / 2.68 / 2.75 ms; 8192 rows 16.1 / 25.3 / 24.4; a forward and a recomputing backward took 3.16 and 25.5.)
  const LaunchGuard guard{p.overflow, 1};
  for (int64_t c = 0; c < p.num_chunks; ++c) {
    const int64_t r0 = c * p.chunk;
    const int64_t w = std::min<int64_t>(p.chunk, a->v_local - r0);
    const void* wmat = a->weight;
    int64_t wrows = a->v_local, row0 = r0, vocab_id0 = 0;
    if (p.deq != nullptr) {
      rc = launch_dequant_int4(a->w_q, a->scales, a->biases, a->qparam_dtype, r0, w, a->d, a->group_size, p.deq,
                               B200TP_BF16, stream, p.overflow);
      if (rc) return rc;
      wmat = p.deq;
      wrows = w;
      row0 = 0;
      vocab_id0 = r0;
    }
    rc = ce_tc_launch_bwd_g(a->hidden, wmat, wrows, a->n, a->d, row0, row0 + w, vocab_id0, a->targets, a->ignore_index,
                            lse, cotangent, p.g, static_cast<int>(p.chunk), nullptr, guard, stream, status);
    if (rc) return rc;
    const bool last = c == p.num_chunks - 1;
    rc = ce_tc_launch_dh(p.g, static_cast<int>(p.chunk), static_cast<int>(align_up(w, kCeTileCols)), a->n, wmat, wrows,
                         a->d, row0, c == 0 ? nullptr : p.acc, p.acc, last ? d_hidden : nullptr, -1, -1,
                         1, nullptr, guard, stream, status);
    if (rc) return rc;
  }
  return B200TP_OK;
}

int b200tp_linear_ce_bwd_grad(const b200tp_ce_args* a, const float* lse, const float* tgt_logit, const float* cotangent,
                              void* state, size_t state_bytes, void* d_hidden, void* workspace, size_t workspace_bytes,
                              void* stream, int* status) {
  return bwd_grad_impl(a, lse, tgt_logit, cotangent, nullptr, nullptr, state, state_bytes, d_hidden, workspace,
                       workspace_bytes, stream, status);
}

int b200tp_linear_ce_bwd_grad_reduced(const b200tp_ce_args* a, const float* lse, const float* tgt_logit,
                                      const float* upstream, const float* count, void* state, size_t state_bytes,
                                      void* d_hidden, void* workspace, size_t workspace_bytes, void* stream,
                                      int* status) {
  return bwd_grad_impl(a, lse, tgt_logit, nullptr, upstream, count, state, state_bytes, d_hidden, workspace,
                       workspace_bytes, stream, status);
}

int b200tp_linear_ce_fwd_grad_reduced(const b200tp_ce_args* a, float* tgt_logit, float* lse, float* nll, float* out3,
                                      void* state, size_t state_bytes, void* workspace, size_t workspace_bytes,
                                      void* stream, int* status) {
  if (out3 == nullptr) return fail(B200TP_ERR_LOSS_INPUT, "the reduced forward needs its output triple");
  const int rc = b200tp_linear_ce_fwd_grad(a, tgt_logit, lse, nll, state, state_bytes, workspace, workspace_bytes,
                                           stream, status);
  if (rc) return rc;
  return launch_loss_reduce(nll, a->targets, a->n, a->ignore_index, out3, static_cast<cudaStream_t>(stream));
}

int b200tp_dequant_int4(const uint32_t* w_q, const void* scales, const void* biases, int32_t qparam_dtype, int64_t row0,
                        int64_t rows, int32_t d, int32_t group_size, void* out, int32_t out_dtype, void* stream) {
  if (w_q == nullptr || scales == nullptr || biases == nullptr || out == nullptr)
    return fail(B200TP_ERR_LOSS_INPUT, "null pointer passed to dequant");
  if (group_size <= 0 || d % 8 != 0 || d % group_size != 0)
    return fail(B200TP_ERR_UNSUPPORTED_HEAD, "d must be a multiple of 8 and of group_size");
  if ((reinterpret_cast<uintptr_t>(out) & 15) != 0)
    return fail(B200TP_ERR_LOSS_INPUT, "out must be 16-byte aligned");
  return launch_dequant_int4(w_q, scales, biases, qparam_dtype, row0, rows, d, group_size, out, out_dtype,
                             static_cast<cudaStream_t>(stream));
}

}  // extern "C"
