// tcgen05 / TMEM / TMA kernels for sm_100a.
#include "tc_kernels.cuh"

#include <cuda.h>
#include <cuda_fp16.h>

#include <cmath>
#include <mutex>
#include <vector>

#include "tc05.cuh"

namespace tc {

using namespace tc05;

// ---------------------------------------------------------------------------
// host helpers

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn g_encode = nullptr;
static std::once_flag g_once;

lf_status make_map_f16_3d(lf_context* ctx, CUtensorMap* map, const void* base, uint64_t d0, uint64_t d1, uint64_t d2,
                          uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1, uint32_t b2) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
  cuuint32_t box[3] = {b0, b1, b2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return LF_OK;
}

// Attention activations q, k, v, gate, o: fp16 [batch][ldq][128] stored as 8-row x 8-channel pieces of 128
// contiguous bytes (element (b, q, c) at b*ldq*128 + (q/8)*1024 + (c/8)*64 + (q%8)*8 + c%8).  A warp whose
// threads own consecutive rows then writes whole 128-byte lines with 16-byte stores, and a piece is exactly
// one core matrix of the tensor core's unswizzled operand format.  The map's dimensions are (position in four
// neighbouring pieces, group of four pieces, piece along rows, batch row), and a box of `rows` rows x 64 channels lands in
// shared memory as [rows/8][8 pieces][8 rows][16 B].  (The innermost dimension is what a copy moves at a time: with the 16 bytes of
// a piece's row there, a store of 128 x 256 took 9000 cycles.)
lf_status make_map_tiled_act(lf_context* ctx, CUtensorMap* map, const void* base, int ldq, int batch, int rows) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[4] = {256, 4, (cuuint64_t)(ldq / 8), (cuuint64_t)batch};
  cuuint64_t strides[3] = {512, 2048, (cuuint64_t)ldq * 256};
  cuuint32_t box[4] = {256, 2, (cuuint32_t)(rows / 8), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (pieces) failed with code %d", (int)r);
  return LF_OK;
}

// The three bf16 terms of a float32 matrix, seen as (d0 contiguous, d1 rows, batch, term); boxes of 64 x b1 x 1 x all three terms
lf_status make_map_terms(lf_context* ctx, CUtensorMap* map, const SplitMatrix& a, uint64_t d0, uint64_t d1, uint64_t batch, uint32_t b1) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[4] = {d0, d1, batch, 3};
  cuuint64_t strides[3] = {(cuuint64_t)a.ld * 2, (cuuint64_t)(a.batch_stride ? a.batch_stride : a.ld * (int64_t)d1) * 2, (cuuint64_t)a.term_stride * 2};
  cuuint32_t box[4] = {64, b1, 1, 3};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(a.p), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (terms) failed with code %d", (int)r);
  return LF_OK;
}

// Terms in pieces of eight columns over rows (batch, Q), seen as (8-byte halves of a row's piece, batch row, piece, term): as 8-byte elements, 128 rows
// fit a box, and what lies past the end of a batch row arrives as zeros.  Boxes of `rows` rows of `batch_rows` batch rows, `pieces` and `terms`.
lf_status make_map_term_pieces(lf_context* ctx, CUtensorMap* map, const SplitMatrix& a, int Q, int batch, uint32_t rows, uint32_t batch_rows,
                               uint32_t pieces, uint32_t terms) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[4] = {(cuuint64_t)Q * 2, (cuuint64_t)batch, (cuuint64_t)a.ld / 8, 3};
  cuuint64_t strides[3] = {(cuuint64_t)Q * 16, (cuuint64_t)batch * Q * 16, (cuuint64_t)a.term_stride * 2};
  cuuint32_t box[4] = {rows * 2, batch_rows, pieces, terms};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<bf16*>(a.p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (term pieces) failed with code %d", (int)r);
  return LF_OK;
}

// float32 rows of 128 channels seen as (channel, d1, d2); boxes of 32 channels (one 128-byte swizzled row) x b1 x b2
lf_status make_map_f32_rows(lf_context* ctx, CUtensorMap* map, const void* base, uint64_t d1, uint64_t d2, uint64_t stride1_bytes,
                            uint64_t stride2_bytes, uint32_t b1, uint32_t b2) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[3] = {128, d1, d2};
  cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
  cuuint32_t box[3] = {32, b1, b2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (float32 rows) failed with code %d", (int)r);
  return LF_OK;
}

// the same with boxes of 16 channels (64-byte rows, 64-byte swizzle): the staging tiles of the triangle output
lf_status make_map_f32_rows_half(lf_context* ctx, CUtensorMap* map, const void* base, uint64_t d1, uint64_t d2, uint64_t stride1_bytes,
                                 uint64_t stride2_bytes, uint32_t b1, uint32_t b2) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[3] = {128, d1, d2};
  cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
  cuuint32_t box[3] = {16, b1, b2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (float32 rows, 16 channels, 3-d) failed with code %d", (int)r);
  return LF_OK;
}

// float32 rows of 128 channels as a 2-d map (channel, row) with boxes of 16 channels x 32 rows (64-byte rows,
// 64-byte swizzle): the staging tiles of the transition's output
lf_status make_map_f32_rows16(lf_context* ctx, CUtensorMap* map, const void* base, uint64_t rows) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[2] = {128, rows};
  cuuint64_t strides[1] = {512};
  cuuint32_t box[2] = {16, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (float32 rows, 16 channels) failed with code %d", (int)r);
  return LF_OK;
}

// float32 rows of any width, 128-byte swizzled boxes of 32 channels
lf_status make_map_f32_any(lf_context* ctx, CUtensorMap* map, const void* base, const uint64_t (&dims)[3], const uint64_t (&strides)[2], const uint32_t (&box)[3]) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t d[3] = {dims[0], dims[1], dims[2]}, st[2] = {strides[0], strides[1]};
  cuuint32_t b[3] = {box[0], box[1], box[2]}, estr[3] = {1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), d, st, b, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (float32, any width) failed with code %d", (int)r);
  return LF_OK;
}

// the outer product mean's sums grouped per pair, fp16 [cnt i][n j][32 a][32 b] seen as (b, a, j, i): boxes of one i, two j (64-byte swizzle)
lf_status make_map_grouped(lf_context* ctx, CUtensorMap* map, const void* base, uint64_t n, uint64_t cnt) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[4] = {32, 32, n, cnt}, strides[3] = {64, 2048, n * 2048};
  cuuint32_t box[4] = {32, 32, 2, 1}, estr[4] = {1, 1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (grouped sums) failed with code %d", (int)r);
  return LF_OK;
}

// fp16 operand planes [planes][plane_rows][ld] seen as (k, i, plane); boxes of 32 k (64 bytes, 64-byte swizzle) x 1 x box_h
// planes: what an epilogue warp of the triangle projection stores per pass
lf_status make_map_plane_runs(lf_context* ctx, CUtensorMap* map, const void* base, uint64_t n, uint64_t plane_rows, uint64_t planes,
                              uint64_t ld, uint32_t box_h) {
  if (!g_encode) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[3] = {n, plane_rows, planes};
  cuuint64_t strides[2] = {ld * 2, plane_rows * ld * 2};
  cuuint32_t box[3] = {32, 1, box_h};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lf_fail(ctx, LF_ERR_CUDA, "cuTensorMapEncodeTiled (operand planes) failed with code %d", (int)r);
  return LF_OK;
}

// Waits for the context's stream; the status word comes back behind its work, in the same wait.
lf_status check_status(lf_context* ctx) {
  Status st{};
  if (ctx->tc_status) {
    Status* to = ctx->status_host ? static_cast<Status*>(ctx->status_host) : &st;
    LF_CUDA(ctx, cudaMemcpyAsync(to, ctx->tc_status, sizeof st, cudaMemcpyDeviceToHost, ctx->stream));
    LF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    st = *to;
  } else LF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (st.code != 0) {
    cudaMemset(ctx->tc_status, 0, sizeof st);
    if (st.code == kStatusAlignment)
      return lf_fail(ctx, LF_ERR_CUDA, "a kernel's shared memory is not on the boundary that it needs (%u, block %u): nothing was computed", st.where, st.block);
    return lf_fail(ctx, LF_ERR_TIMEOUT, "a bounded wait expired in a tensor-core kernel (wait %u, block %u)", st.where, st.block);
  }
  return LF_OK;
}

bool ln_gemm_supported(const lf_weights* w) { return w && !w->h.empty() && w->h[0] != nullptr; }
bool pair_bias_supported(const lf_weights* w) { return w && w->h.size() >= 6 && w->h[4] != nullptr; }

// ---------------------------------------------------------------------------
// Triangle contraction.
//
// One 128 x 256 output tile of one channel per work item, K stepped by 64 through
// a 4-stage TMA ring, float32 accumulators double-buffered in TMEM (2 x 256
// columns) so the epilogue of a tile overlaps the main loop of the next.
// Warp roles: 0 = TMA producer, 1 = MMA issuer (owns TMEM), 2..5 = epilogue.
// MAJOR 0: both operands K-major (outgoing).  MAJOR 1: both MN-major (incoming),
// fetched as 64 x 64 boxes whose rows are k.

constexpr int CT_BM = 128, CT_BN = 256, CT_BK = 64, CT_STAGES = 4;
constexpr int CT_A_BYTES = CT_BM * CT_BK * 2;   // 16 KiB
constexpr int CT_B_BYTES = CT_BN * CT_BK * 2;   // 32 KiB
constexpr int CT_STAGE_BYTES = CT_A_BYTES + CT_B_BYTES;
constexpr int CT_OUT_STAGE = 32 * 256;          // per epilogue warp: 32 rows x 128 fp16 columns, for stores into a peer's memory
// EW epilogue warps: 4 for the triangle contraction (long k loops hide the epilogue), 8 for the grouped outer product, whose k
// loop of 4 to 16 blocks is shorter than a 4-warp epilogue of the 128 x 256 tile; the 8-warp form gives a stage
// of the operand ring to the four extra staging areas.
constexpr int ct_stages(int ew) { return ew == 8 ? 3 : CT_STAGES; }
constexpr int ct_smem(int ew) { return ct_stages(ew) * CT_STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/ + ew * CT_OUT_STAGE; }
constexpr int ct_threads(int ew) { return 64 + 32 * ew; }

// The outer product mean's use: with `group_c` > 0 rows are (i, a) and columns (j, b) with a, b < group_c, and element (i, a, j, b) is stored at
// ((i * group_n + j) * group_c + a) * group_c + b - the sums grouped per pair (i, j), which a warp writes as whole
// 2 * group_c^2-byte runs.
struct ContractExtra { int group_c; int group_n; };

template <int MAJOR, int EW = 4>
__global__ void __launch_bounds__(ct_threads(EW), 1)
contract_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                op16* __restrict__ x, int m_rows, int n_rows, int k_len, int ldx, int64_t x_plane, int col0, int c,
                float scale, Status* status, const __grid_constant__ PeerPtrs xpeer, int rows_per_rank, int ch0,
                const ContractExtra ex) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  constexpr int ST = EW == 8 ? 3 : CT_STAGES;      // = ct_stages(EW)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ST * CT_STAGE_BYTES);
  uint64_t* full = bars;                       // [STAGES]
  uint64_t* empty = bars + ST;                 // [STAGES]
  uint64_t* tmem_full = bars + 2 * ST;         // [2]
  uint64_t* tmem_empty = tmem_full + 2;        // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* out_stage = smem + ST * CT_STAGE_BYTES + 256;     // [EW epilogue warps][CT_OUT_STAGE]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // x[h][i][col0 + j] for i < m_rows, j < n_rows; the contraction index runs over k_len
  const int tiles_m = (m_rows + CT_BM - 1) / CT_BM, tiles_n = (n_rows + CT_BN - 1) / CT_BN;
  const int tiles_per_h = tiles_m * tiles_n;
  const int total = c * tiles_per_h;
  const int kblocks = (k_len + CT_BK - 1) / CT_BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], EW); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  lf_chain();

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tensormap(&mapA);
      prefetch_tensormap(&mapB);
      int stage = 0; uint32_t phase = 0;
      for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const int h = t / tiles_per_h, rem = t % tiles_per_h, mi = rem / tiles_n, nj = rem % tiles_n;
        bool ok = true;
        for (int kb = 0; kb < kblocks && ok; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, status, 1)) { ok = false; break; }
          uint8_t* sA = smem + stage * CT_STAGE_BYTES;
          uint8_t* sB = sA + CT_A_BYTES;
          mbar_expect_tx(&full[stage], CT_STAGE_BYTES);
          if (MAJOR == 0) {
            tma_load_3d(sA, &mapA, &full[stage], kb * CT_BK, mi * CT_BM, h);
            tma_load_3d(sB, &mapB, &full[stage], kb * CT_BK, nj * CT_BN, h);
          } else {
#pragma unroll
            for (int q = 0; q < CT_BM / 64; ++q) tma_load_3d(sA + q * 8192, &mapA, &full[stage], mi * CT_BM + q * 64, kb * CT_BK, h);
#pragma unroll
            for (int q = 0; q < CT_BN / 64; ++q) tma_load_3d(sB + q * 8192, &mapB, &full[stage], nj * CT_BN + q * 64, kb * CT_BK, h);
          }
          if (++stage == ST) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_f16(CT_BM, CT_BN, MAJOR, MAJOR);
      int stage = 0; uint32_t phase = 0;
      int it = 0;
      for (int t = blockIdx.x; t < total; t += gridDim.x, ++it) {
        const int buf = it & 1;
        if (!mbar_wait(&tmem_empty[buf], ((it >> 1) & 1) ^ 1, abort_flag, status, 2)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * CT_BN;
        bool ok = true;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag, status, 3)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + stage * CT_STAGE_BYTES);
          const uint32_t b_addr = a_addr + CT_A_BYTES;
#pragma unroll
          for (int kk = 0; kk < CT_BK / 16; ++kk) {
            uint64_t adesc, bdesc;
            if (MAJOR == 0) {
              adesc = make_smem_desc(a_addr + kk * 32, 16, 1024);
              bdesc = make_smem_desc(b_addr + kk * 32, 16, 1024);
            } else {
              adesc = make_smem_desc(a_addr + kk * 2048, 8192, 1024);
              bdesc = make_smem_desc(b_addr + kk * 2048, 8192, 1024);
            }
            umma_f16(d_tmem, adesc, bdesc, idesc, (kb | kk) != 0 ? 1u : 0u);
          }
          umma_commit(&empty[stage]);
          if (++stage == ST) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(&tmem_full[buf]);
      }
    }
  } else {
    const int q = warp & 3;                 // TMEM lane quadrant this warp may read
    const int chalf = (warp - 2) >> 2;      // EW == 8: the half of the tile's 256 columns this warp takes
    const int row = q * 32 + lane;
    int it = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x, ++it) {
      const int h = t / tiles_per_h, rem = t % tiles_per_h, mi = rem / tiles_n, nj = rem % tiles_n;
      const int buf = it & 1;
      if (!mbar_wait(&tmem_full[buf], (it >> 1) & 1, abort_flag, status, 4)) break;
      tc_fence_after();
      const int gi = mi * CT_BM + row;
      op16* dst_row;
      if (rows_per_rank > 0) {
        // row gi of the product belongs to rank gi / rows_per_rank: stored into that rank's
        // [channels][rows_per_rank][ldx] buffer (x_plane = rows_per_rank * ldx)
        int owner = gi / rows_per_rank;
        if (gi >= m_rows) owner = 0;      // not stored
        dst_row = reinterpret_cast<op16*>(xpeer.p[owner]) + (int64_t)(ch0 + h) * x_plane + (int64_t)(gi - owner * rows_per_rank) * ldx + col0;
      } else {
        dst_row = x + (int64_t)h * x_plane + (int64_t)gi * ldx + col0;
      }
      const int col_limit = (n_rows + 15) / 16 * 16 < ldx - col0 ? (n_rows + 15) / 16 * 16 : ldx - col0;
      if (rows_per_rank > 0) {
        // Rows bound for another GPU leave in 256-byte runs: a thread holds a row of the accumulator, so its
        // own stores would be 16-byte pieces 32 rows apart, which NVLink carries as 32 small packets.  The
        // warp's 32 rows x 128 columns are turned round in shared memory (16-byte pieces swizzled by row)
        // and written two rows per instruction, 16 lanes x 16 bytes each.
        uint8_t* stage = out_stage + (warp - 2) * CT_OUT_STAGE;
        const int g_row0 = mi * CT_BM + q * 32;            // the warp's rows share an owner: rows_per_rank % 128 == 0
        const int owner = g_row0 < m_rows ? g_row0 / rows_per_rank : 0;
        op16* owner_base = reinterpret_cast<op16*>(xpeer.p[owner]) + (int64_t)(ch0 + h) * x_plane + col0;
#pragma unroll 1
        for (int half = (EW == 8 ? chalf : 0); half < (EW == 8 ? chalf + 1 : 2); ++half) {
#pragma unroll 1
          for (int cc = 0; cc < 4; ++cc) {
            uint32_t r[32];
            tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + buf * CT_BN + half * 128 + cc * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float o[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = __uint_as_float(r[v * 8 + e]) * scale;
              uint4 pk;
              pk.x = pack_half2(o[0], o[1]);
              pk.y = pack_half2(o[2], o[3]);
              pk.z = pack_half2(o[4], o[5]);
              pk.w = pack_half2(o[6], o[7]);
              *reinterpret_cast<uint4*>(stage + lane * 256 + (((cc * 4 + v) ^ (lane & 15)) << 4)) = pk;
            }
          }
          __syncwarp();
#pragma unroll 4
          for (int rr = 0; rr < 16; ++rr) {
            const int srow = rr * 2 + (lane >> 4), piece = lane & 15;
            const uint4 pk = *reinterpret_cast<const uint4*>(stage + srow * 256 + ((piece ^ (srow & 15)) << 4));
            const int grow = g_row0 + srow, gj = nj * CT_BN + half * 128 + piece * 8;
            if (grow < m_rows && gj < col_limit)
              *reinterpret_cast<uint4*>(owner_base + (int64_t)(grow - owner * rows_per_rank) * ldx + gj) = pk;
          }
          __syncwarp();
        }
      } else
#pragma unroll 1
      for (int cc = (EW == 8 ? chalf * 4 : 0); cc < (EW == 8 ? chalf * 4 + 4 : CT_BN / 32); ++cc) {
        uint32_t r[32];
        tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + buf * CT_BN + cc * 32, r);
        tmem_ld_wait();
        const int gj0 = nj * CT_BN + cc * 32;   // column inside the window
        if (gi < m_rows) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const int gj = gj0 + v * 8;
            if (gj < col_limit) {
              float o[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = __uint_as_float(r[v * 8 + e]) * scale;
              uint4 pk;
              pk.x = pack_half2(o[0], o[1]);
              pk.y = pack_half2(o[2], o[3]);
              pk.z = pack_half2(o[4], o[5]);
              pk.w = pack_half2(o[6], o[7]);
              if (ex.group_c) {
                const int gc = ex.group_c;
                *reinterpret_cast<uint4*>(x + ((((int64_t)(gi / gc) * ex.group_n + gj / gc) * gc + gi % gc) * gc + gj % gc)) = pk;
              } else {
                *reinterpret_cast<uint4*>(dst_row + gj) = pk;
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[buf]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) drain_after_abort();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// Kernel attributes belong to a device (context), the driver entry point to the process.
void configure_once() {
  std::call_once(g_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<EncodeTiledFn>(fn);
    else
      cudaGetLastError();
  });
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return; }
  static std::once_flag per_device[64];
  std::call_once(per_device[dev], [] {
    cudaFuncSetAttribute(contract_kernel<0, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, ct_smem(4));
    cudaFuncSetAttribute(contract_kernel<1, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, ct_smem(4));
    cudaFuncSetAttribute(contract_kernel<1, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, ct_smem(8));
    configure_ln_gemm();
    configure_attention();
    configure_transition();
    configure_gemm3();
    configure_gemm();
    cudaGetLastError();
  });
}

bool contract_supported(int n, int c) { return n >= 1 && c >= 1 && g_encode != nullptr; }

static lf_status contract_impl(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, op16* x, int m_rows, int n_rows,
                               int k_len, int ld_ab, int ldx, int64_t x_plane, int col0, int c, int incoming, float scale,
                               const PeerPtrs* peers, int rows_per_rank, int ch0,
                               ContractExtra ex = ContractExtra{0, 0});

lf_status contract_rect(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, op16* x, int m_rows, int n_rows,
                        int k_len, int ld_ab, int ldx, int64_t x_plane, int col0, int c, int incoming, float scale) {
  return contract_impl(ctx, cur, a, b, x, m_rows, n_rows, k_len, ld_ab, ldx, x_plane, col0, c, incoming, scale, nullptr, 0, 0);
}

lf_status contract_scatter(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, int n, int ld, int c, int incoming,
                           float scale, const PeerPtrs& x_peers, int rows_per_rank, int total_channels, int ch0) {
  (void)total_channels;
  // the product's planes at the row owners hold rows_per_rank rows of ld elements
  return contract_impl(ctx, cur, a, b, nullptr, n, n, n, ld, ld, (int64_t)rows_per_rank * ld, 0, c, incoming, scale, &x_peers,
                       rows_per_rank, ch0);
}

lf_status contract_outer(lf_context* ctx, ArenaCursor& cur, const op16* left, const op16* right, op16* out, int cnt, int n, int c,
                         int k_len, float scale) {
  if (c % 8 != 0) return lf_fail(ctx, LF_ERR_UNSUPPORTED, "the grouped outer product needs c in whole groups of 8");
  if (c == 32) return gemm_outer32(ctx, cur, left, right, out, cnt, n, k_len, scale);
  // x[(i, a)][(j, b)] = scale * sum_s left[s][(i, a)] right[s][(j, b)]: both operands MN-major, the kernel's "b" is its M operand
  return contract_impl(ctx, cur, right, left, out, cnt * c, n * c, k_len, n * c, n * c, 0, 0, 1, 1, scale, nullptr, 0, 0,
                       ContractExtra{c, n});
}

static lf_status contract_impl(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, op16* x, int m_rows, int n_rows,
                               int k_len, int ld_ab, int ldx, int64_t x_plane, int col0, int c, int incoming, float scale,
                               const PeerPtrs* peers, int rows_per_rank, int ch0, ContractExtra ex) {
  if (cur.dry) return LF_OK;
  // a row of an operand holds k (K-major form) or the M / N index (MN-major form)
  const int row_len = incoming ? (m_rows > n_rows ? m_rows : n_rows) : k_len;
  if (ld_ab % 8 != 0 || ld_ab < row_len || ldx % 8 != 0 || col0 % 8 != 0)
    return lf_fail(ctx, LF_ERR_ARGUMENT, "contraction strides must be multiples of 8 and cover the row");
  CUtensorMap mapA, mapB;
  const uint64_t row_bytes = (uint64_t)ld_ab * 2;
  if (!incoming) {
    LF_TRY(make_map_f16_3d(ctx, &mapA, a, k_len, m_rows, c, row_bytes, (uint64_t)m_rows * row_bytes, CT_BK, CT_BM, 1));
    LF_TRY(make_map_f16_3d(ctx, &mapB, b, k_len, n_rows, c, row_bytes, (uint64_t)n_rows * row_bytes, CT_BK, CT_BN, 1));
  } else {
    // A(i,k) = b[h][k][i], B(j,k) = a[h][k][j]: boxes of 64 (i or j) x 64 (k)
    LF_TRY(make_map_f16_3d(ctx, &mapA, b, m_rows, k_len, c, row_bytes, (uint64_t)k_len * row_bytes, 64, CT_BK, 1));
    LF_TRY(make_map_f16_3d(ctx, &mapB, a, n_rows, k_len, c, row_bytes, (uint64_t)k_len * row_bytes, 64, CT_BK, 1));
  }
  const int tiles = c * ((m_rows + CT_BM - 1) / CT_BM) * ((n_rows + CT_BN - 1) / CT_BN);
  const int grid = tiles < ctx->sm_count ? tiles : ctx->sm_count;
  lf_prof_begin(ctx, LF_KERNEL_TRIANGLE_CONTRACT);
#define CT_LAUNCH(MAJ, EWN) \
  lf_launch(ctx, contract_kernel<MAJ, EWN>, grid, ct_threads(EWN), ct_smem(EWN), mapA, mapB, x, m_rows, n_rows, k_len, ldx, x_plane, col0, c, \
      scale, (Status*)ctx->tc_status, peers ? *peers : PeerPtrs{}, rows_per_rank, ch0, ex)
  if (ex.group_c) CT_LAUNCH(1, 8);      // (always incoming)
  else if (incoming) CT_LAUNCH(1, 4);
  else CT_LAUNCH(0, 4);
#undef CT_LAUNCH
  lf_prof_end(ctx);
  ctx->launches++;
  return LF_OK;
}

lf_status contract(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, op16* x, int n, int ld, int c,
                   int incoming, float scale) {
  // Up to about eight k blocks a tile the epilogue decides, and the GEMM kernel's sixteen warps win (N = 384, 128 channels: 37 -> 31 us);
  // from there on the contraction kernel's deeper ring does (N = 701: 101 against 111 us, N = 2048: 1.68 against 1.79 ms).
  if (n < 512) return gemm_planes(ctx, cur, a, b, x, n, ld, c, incoming, scale);
  return contract_rect(ctx, cur, a, b, x, n, n, n, ld, ld, (int64_t)n * ld, 0, c, incoming, scale);
}

}  // namespace tc
