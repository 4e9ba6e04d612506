// Shared host-side plumbing of the pair-stack library: context, scratch arena,
// resident weights, error reporting.  No torch types anywhere in this library.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/localfold_pairstack.h"

typedef __nv_bfloat16 bf16;
// Operand type of the tensor-core kernels: fp16 (11-bit significand) for the bounded
// intermediates (normalised activations, gated projections, probabilities); products
// accumulate in float32.  The pair stream itself is float32 or bf16.
typedef __half op16;

struct lf_context {
  int device = 0;
  // Pinned staging of weight uploads: filled from the front, the stream is waited for when it is full.
  char* pinned = nullptr;
  size_t pinned_used = 0;
  cudaStream_t stream = nullptr;
  bool owns_stream = false;
  std::string error;
  // Scratch arena: one device allocation, bump-allocated per operator call.
  char* arena = nullptr;
  size_t arena_bytes = 0;
  size_t arena_peak = 0;
  size_t arena_limit = 0;      // 0 = none; otherwise requests above it are refused without asking the driver (lf_context_limit_scratch)
  uint64_t launches = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaEvent_t inputs = nullptr;      // lf_context_await
  void* status_host = nullptr;       // pinned copy of *tc_status
  int sm_count = 148;
  void* tc_status = nullptr;   // device word the tensor-core kernels set when a bounded wait expires
  // Optional per-kernel-family timing (CUDA events on the context's stream).
  bool profiling = false;
  struct Timed { int family; cudaEvent_t start, stop; };
  std::vector<Timed> timed;
  double family_ms[LF_KERNEL_FAMILY_COUNT] = {0};
  uint64_t family_launches[LF_KERNEL_FAMILY_COUNT] = {0};
};

static inline void lf_prof_begin(lf_context* ctx, int family) {
  if (!ctx->profiling) return;
  lf_context::Timed t{family, nullptr, nullptr};
  cudaEventCreate(&t.start);
  cudaEventCreate(&t.stop);
  cudaEventRecord(t.start, ctx->stream);
  ctx->timed.push_back(t);
}
static inline void lf_prof_end(lf_context* ctx) {
  if (!ctx->profiling || ctx->timed.empty()) return;
  cudaEventRecord(ctx->timed.back().stop, ctx->stream);
}

// Kernels follow one another with programmatic dependent launch: the next kernel of the stream is set up as the last block of the
// one before leaves, and every kernel opens with lf_chain(), before it touches global memory, which waits until the one before is complete
// and visible.  Two to three microseconds between dependent launches are gone (26 launches of a 384 x 384 pair block 1530 -> 1478 us).
// Nothing asks for the next kernel earlier (griddepcontrol.launch_dependents): its blocks, waiting on the multiprocessors, slowed
// the running kernel by more than the set-up is worth (1550 us).
__device__ __forceinline__ void lf_chain() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... P, typename... A>
static inline void lf_launch(lf_context* ctx, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
  cudaLaunchAttribute chain{};
  chain.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  chain.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = ctx->stream;
  config.attrs = &chain;
  config.numAttrs = 1;
  cudaLaunchKernelEx(&config, kernel, std::forward<A>(args)...);
}

// Slots of lf_weights::f per operator kind.
enum { TRI_LN_G, TRI_LN_B, TRI_W4, TRI_B4, TRI_LNO_G, TRI_LNO_B, TRI_WZ, TRI_BZ, TRI_WG, TRI_BG, TRI_COUNT };
enum { ATT_LN_G, ATT_LN_B, ATT_W4, ATT_B4, ATT_WO, ATT_BO, ATT_PLN_G, ATT_PLN_B, ATT_WB, ATT_COUNT };
enum { TRN_LN_G, TRN_LN_B, TRN_W1, TRN_B1, TRN_W2, TRN_B2, TRN_COUNT };
enum { OPM_LN_G, OPM_LN_B, OPM_WL, OPM_BL, OPM_WR, OPM_BR, OPM_WOUT, OPM_BOUT, OPM_COUNT };
// global column attention: W3 = (key | value | gate) columns, B3 their biases (zero but for the gate)
enum { GLB_LN_G, GLB_LN_B, GLB_WQ, GLB_W3, GLB_B3, GLB_WO, GLB_BO, GLB_COUNT };

// A float32 matrix as three bf16 terms that add up to it: term t at p + t * term_stride, rows of ld, batch entries batch_stride
// apart (strides in elements, multiples of 8).
struct SplitMatrix {
  const bf16* p = nullptr;
  int64_t ld = 0, batch_stride = 0, term_stride = 0;
  bool pieces = false;      // in pieces of eight columns: element (i, j) of a term at (j / 8) * rows * 8 + i * 8 + j % 8
};

// Operands of the float32 GEMM, [n_out][k] terms, kept with the weights.  Operators that use them in either mode get them when the
// weights are prepared, others at the first float32 call (a pair stack's all at once), in room that small ones keep in their own block.
//   triangle: fused projection, output projection, output gate; attention: fused projection with heads padded to
//   head_width (and the pair bias columns when the bias comes from the normalised input), output projection, and at
//   g[2].p the projection's bias (float32); MSA averaging: values | gate, output projection;
//   transition: both projections; global attention: key | value | gate, output projection
constexpr int head_width(int d) { return d <= 32 ? (d + 7) / 8 * 8 : d <= 48 ? 48 : 64; }      // the attention core's instances
struct lf_f32_operands {
  bool made = false;               // with the mutex of f32_operands (api.cu) held
  lf_context* ctx = nullptr;       // whose stream made them
  cudaEvent_t ready = nullptr;     // null when they were made with the weights
  size_t bytes = 0;                // 0: the kind has none
  char* room = nullptr;            // in the weights' block, or
  void* block = nullptr;           // a block of their own
  size_t block_bytes = 0;
  SplitMatrix g[3];
};
constexpr size_t kF32RoomLimit = (size_t)1 << 20;      // the operators of a 128-channel pair block: 0.5 to 0.8 MiB each

// Canonical device-resident weights.  Every linear is stored (in,out) row-major
// float32 in `f[...]`; tensor-core kernels keep extra fp16 repacks (swizzled operand images) in `h[...]`.
struct lf_weights {
  lf_context* ctx = nullptr;
  int kind = 0;
  lf_weight_dims dims{};
  std::vector<float*> f;     // named by the per-kind enums above
  std::vector<void*> h;      // fp16 repacks (tensor-core path)
  std::vector<void*> g;      // fp16 [n_out][k] operands of the plain tensor-core GEMM (widths the fused kernels do not take)
  int device = 0;
  void* block = nullptr;     // the one device allocation behind all of them (weight_block_take)
  size_t block_bytes = 0;
  mutable lf_f32_operands f32;
  cudaEvent_t ready = nullptr;   // recorded on the creating context's stream when they have been prepared
  bool has_gate_bias = false, has_out_bias = false, has_pair_norm = false, has_pair_proj = false;
};

static inline lf_status lf_fail(lf_context* ctx, lf_status code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (ctx) ctx->error = buf;
  return code;
}

#define LF_CUDA(ctx, expr)                                                             \
  do {                                                                                 \
    cudaError_t e_ = (expr);                                                           \
    if (e_ != cudaSuccess)                                                             \
      return lf_fail((ctx), e_ == cudaErrorMemoryAllocation ? LF_ERR_MEMORY : LF_ERR_CUDA, \
                     "%s failed: %s", #expr, cudaGetErrorString(e_));                  \
  } while (0)

#define LF_TRY(expr)                  \
  do {                                \
    lf_status s_ = (expr);            \
    if (s_ != LF_OK) return s_;       \
  } while (0)

// Bump allocation out of the arena.  Sizing happens before any kernel of the
// call is enqueued (see Arena::plan in api.cu): the arena is never reallocated
// while work that uses it may still be in flight on the stream.
static inline size_t lf_align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct ArenaCursor {
  lf_context* ctx;
  size_t offset;
  // Planning pass: only adds sizes up.  Its addresses are stand-ins, aligned and distinct as the real ones are, so that whatever a call decides by
  // address - where a residual lives, how an output is aligned - it decides alike in both passes.
  bool dry;
  size_t peak = 0;   // high-water mark (callers may rewind `offset` between operators)
  template <typename T>
  T* take(size_t count) {
    size_t bytes = lf_align_up(count * sizeof(T), 256);
    T* p = dry ? reinterpret_cast<T*>((uintptr_t)256 + offset) : reinterpret_cast<T*>(ctx->arena + offset);
    offset += bytes;
    if (offset > peak) peak = offset;
    return p;
  }
};

// The same over a weights object's own allocation.
struct WeightCursor {
  char* base;
  size_t offset;
  bool dry;
  template <typename T>
  T* take(size_t count) {
    T* p = dry ? nullptr : reinterpret_cast<T*>(base + offset);
    offset += lf_align_up(count * sizeof(T) + 4, 256);
    return p;
  }
};

lf_status lf_arena_ensure(lf_context* ctx, size_t bytes);
// Work on `ctx`'s stream that reads `w` comes after the preparation of w on another context's stream.
static inline void lf_weights_await(lf_context* ctx, const lf_weights* w) {
  if (w && w->ctx != ctx && w->ready) cudaStreamWaitEvent(ctx->stream, w->ready, 0);
}
// The pair stack with the pair left in host memory (pair_spill.cu).
lf_status lf_pair_stack_spilled(lf_context* ctx, const lf_pair_stack_desc* d, lf_result* r);

static inline bool lf_aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
// Whether the fused 128-channel kernels take the caller's activations where they lie (the general path takes any address): they load 16
// bytes at a time and store by TMA, but rows that leave by threads' stores - bfloat16 ones, and float32 ones whose residual lives
// elsewhere - take 32-byte accesses.
static inline bool lf_fused_takes(const void* act, const void* resid, const void* out, int act_dtype) {
  const uintptr_t low = act_dtype == LF_DTYPE_F32 && (!resid || resid == out) ? 15 : 31;
  return lf_aligned16(act) && (((uintptr_t)resid | (uintptr_t)out) & low) == 0;
}

static inline int lf_ceil_div(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }
