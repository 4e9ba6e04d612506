// Plain fp16 GEMM on tcgen05 with its output layouts in the epilogue: fp16 rows, attention pieces, float32 rows added in
// place, the outer product mean's sums grouped per pair, the triangle contraction's planes.
#include <cuda.h>

#include "tc05.cuh"
#include "tc_kernels.cuh"

namespace tc {

using namespace tc05;

// One 128 x 256 tile of one batch entry per work item, k stepped by 64 through a three-stage TMA ring, accumulators
// double-buffered in TMEM.  Most uses have one to four k blocks, so the epilogue is what bounds them: sixteen warps (four per TMEM
// lane quadrant, 64 columns each) take a whole share into registers with one wait, hand the accumulator back at once,
// and send 4 KiB staging tiles off by TMA in whatever layout the next kernel reads - no thread stores to global memory,
// rows and columns past the ends are clipped by the tensor map, and columns past n are not even read.
// 147 456 x 264 x 64: 91 us with eight warps and stores by threads.
// Warp roles: 0 = TMA producer, 1 = MMA issuer (owns TMEM), 2..17 = epilogue.
constexpr int GM_BM = 128, GM_BN = 256, GM_BK = 64, GM_STAGES = 3, GM_EPI = 16;
constexpr int GM_A_BYTES = GM_BM * GM_BK * 2, GM_B_BYTES = GM_BN * GM_BK * 2, GM_STAGE = GM_A_BYTES + GM_B_BYTES;
constexpr int GM_OUT = 4096;                  // per epilogue warp: 32 rows x 128 bytes
constexpr int GM_SHARE = GM_BN / 4;           // columns of an epilogue warp
constexpr int GM_SMEM = GM_STAGES * GM_STAGE + GM_EPI * (GM_OUT + GM_SHARE * 4) + 256 + 1024;
constexpr int GM_THREADS = 64 + 32 * GM_EPI;

enum { GM_HALF = 0, GM_PIECES = 1, GM_F32 = 2, GM_GROUPED = 3 };

struct GemmParams {
  int m, n, k, batch;
  float scale;
  const float* bias;          // [n] or null
  int relu;
  int a_pieces;               // A arrives in 8-row x 8-channel pieces of groups of 128 channels ([group][batch][..])
  int add;                    // GM_F32: add to the rows instead of writing them
  int transposed;             // GM_F32: output coordinates (channel, batch, row) instead of (channel, row, batch)
  int width;                  // GM_PIECES: columns of one of q, k, v, gate (a multiple of 128)
  float qscale;
  Status* status;
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int MAJOR, int EPI>
__global__ void __launch_bounds__(GM_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const __grid_constant__ CUtensorMap mapO,
            const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  uint8_t* out_stage = smem + GM_STAGES * GM_STAGE;
  float* bias_s = reinterpret_cast<float*>(out_stage + GM_EPI * GM_OUT);      // [epilogue warp][its columns]
  uint64_t* bars = reinterpret_cast<uint64_t*>(bias_s + GM_EPI * GM_SHARE);
  uint64_t* full = bars;                       // [STAGES]
  uint64_t* empty = bars + GM_STAGES;          // [STAGES]
  uint64_t* tmem_full = empty + GM_STAGES;     // [2]
  uint64_t* tmem_empty = tmem_full + 2;        // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (p.m + GM_BM - 1) / GM_BM, tiles_n = (p.n + GM_BN - 1) / GM_BN, per = tiles_m * tiles_n;
  const int total = p.batch * per;
  const int kblocks = (p.k + GM_BK - 1) / GM_BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < GM_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], GM_EPI); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  lf_chain();
  // Work item t: N tiles of one M tile are neighbours (their A tile is read once from memory), shifted from M tile to M tile so
  // that no block keeps one N tile (the gate columns of the pieces cost more than the others).
  auto locate = [&](int t, int& h, int& mi, int& nj) {
    const int row = t / tiles_n;
    h = row / tiles_m;
    mi = row - h * tiles_m;
    nj = (t - row * tiles_n + row) % tiles_n;
  };

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tensormap(&mapA);
      prefetch_tensormap(&mapB);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int h, mi, nj;
        locate(t, h, mi, nj);
        const int hb = EPI == GM_HALF && MAJOR == 0 && p.batch > 1 && !p.a_pieces ? h : 0;      // B of the plane (weights have one)
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status, 111)) { ok = false; break; }
          uint8_t* sA = smem + stage * GM_STAGE;
          uint8_t* sB = sA + GM_A_BYTES;
          mbar_expect_tx(&full[stage], GM_STAGE);
          if (MAJOR == 0) {
            if (p.a_pieces) tma_load_4d(sA, &mapA, &full[stage], 0, (kb & 1) * 2, mi * (GM_BM / 8), (kb >> 1) * p.batch + h);
            else tma_load_3d(sA, &mapA, &full[stage], kb * GM_BK, mi * GM_BM, h);
            tma_load_3d(sB, &mapB, &full[stage], kb * GM_BK, nj * GM_BN, hb);
          } else {
#pragma unroll
            for (int q = 0; q < GM_BM / 64; ++q) tma_load_3d(sA + q * 8192, &mapA, &full[stage], mi * GM_BM + q * 64, kb * GM_BK, h);
#pragma unroll
            for (int q = 0; q < GM_BN / 64; ++q) tma_load_3d(sB + q * 8192, &mapB, &full[stage], nj * GM_BN + q * 64, kb * GM_BK, h);
          }
          if (++stage == GM_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x, ++it) {
        int h, mi, nj;
        locate(t, h, mi, nj);
        const int left = p.n - nj * GM_BN;
        const uint32_t idesc = make_idesc_f16(GM_BM, left >= GM_BN ? GM_BN : (left + 15) / 16 * 16, MAJOR, MAJOR);
        if (!mbar_wait(&tmem_empty[it & 1], ((it >> 1) & 1) ^ 1, abort_flag, p.status, 112)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + (it & 1) * GM_BN;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag, p.status, 113)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a0 = smem_u32(smem + stage * GM_STAGE), b0 = a0 + GM_A_BYTES;
#pragma unroll
          for (int kk = 0; kk < GM_BK / 16; ++kk) {
            const uint64_t adesc = MAJOR ? make_smem_desc(a0 + kk * 2048, 8192, 1024)
                                         : p.a_pieces ? make_smem_desc_plain(a0 + kk * 256, 128, 1024) : make_smem_desc(a0 + kk * 32, 16, 1024);
            const uint64_t bdesc = MAJOR ? make_smem_desc(b0 + kk * 2048, 8192, 1024) : make_smem_desc(b0 + kk * 32, 16, 1024);
            umma_f16(d, adesc, bdesc, idesc, (kb | kk) != 0 ? 1u : 0u);
          }
          umma_commit(&empty[stage]);
          if (++stage == GM_STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit(&tmem_full[it & 1]);
      }
    }
  } else {
    const int q = warp & 3, part = (warp - 2) >> 2;      // TMEM lane quadrant, 64 of the tile's 256 columns
    uint8_t* stage = out_stage + (warp - 2) * GM_OUT;
    float* bias = bias_s + (warp - 2) * GM_SHARE;
    uint32_t it = 0;
    int held = -1;      // first column of the bias share in shared memory
    if (lane == 0) prefetch_tensormap(&mapO);
    for (int t = blockIdx.x; t < total; t += gridDim.x, ++it) {
      int h, mi, nj;
      locate(t, h, mi, nj);
      const int col0 = nj * GM_BN + part * GM_SHARE, row0 = mi * GM_BM + q * 32;
      const bool mine = col0 < p.n && row0 < p.m;
      // of the pieces: q is scaled, the gate's exponent is -log2(e) (acc + bias)
      const int kind = EPI == GM_PIECES ? col0 / p.width : 0;
      const float scale = EPI != GM_PIECES ? p.scale : kind == 0 ? p.qscale : kind == 3 ? -1.4426950408889634f : 1.0f;
      if (mine && held != col0) {
        held = col0;
        __syncwarp();
#pragma unroll
        for (int e = 0; e < GM_SHARE; e += 32) {
          const int c = col0 + e + lane;
          bias[e + lane] = p.bias && c < p.n ? __ldg(p.bias + c) * (EPI == GM_PIECES ? scale : 1.0f) : 0.f;
        }
        __syncwarp();
      }
      if (!mbar_wait(&tmem_full[it & 1], (it >> 1) & 1, abort_flag, p.status, 114)) break;
      tc_fence_after();
      uint32_t r[2][32];
      if (mine) {
        const uint32_t d = tmem_base + ((uint32_t)(q * 32) << 16) + (it & 1) * GM_BN + part * GM_SHARE;
        tmem_ld32(d, r[0]);
        tmem_ld32(d + 32, r[1]);
        tmem_ld_wait();
        tie32(r[0]);
        tie32(r[1]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[it & 1]);      // the share is in registers: the accumulator may be overwritten
      if (!mine) continue;
      auto value = [&](int half, int e) { return __uint_as_float(r[half][e]); };
      if (EPI == GM_F32) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (col0 + half * 32 >= p.n) break;
          if (lane == 0) bulk_wait_read();      // the previous copy has read the staging rows
          __syncwarp();
#pragma unroll
          for (int k4 = 0; k4 < 8; ++k4) {
            const float4 b = *reinterpret_cast<const float4*>(bias + half * 32 + k4 * 4);
            *reinterpret_cast<float4*>(stage + lane * 128 + ((k4 ^ (lane & 7)) << 4)) =
                make_float4(fmaf(value(half, k4 * 4), scale, b.x), fmaf(value(half, k4 * 4 + 1), scale, b.y), fmaf(value(half, k4 * 4 + 2), scale, b.z),
                            fmaf(value(half, k4 * 4 + 3), scale, b.w));
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int y = p.transposed ? h : row0, z = p.transposed ? row0 : h;
            if (p.add) tma_reduce_add_3d(&mapO, stage, col0 + half * 32, y, z);
            else tma_store_3d(&mapO, stage, col0 + half * 32, y, z);
            bulk_commit();
          }
        }
      } else {
        if (lane == 0) bulk_wait_read();
        __syncwarp();
#pragma unroll
        for (int c8 = 0; c8 < 8; ++c8) {      // 16-byte pieces of eight columns
          uint32_t w[4];
          const int half = c8 >> 2, e0 = (c8 & 3) * 8;
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; e += 4) {
            const float4 b = *reinterpret_cast<const float4*>(bias + c8 * 8 + e);
            v[e] = fmaf(value(half, e0 + e), scale, b.x);
            v[e + 1] = fmaf(value(half, e0 + e + 1), scale, b.y);
            v[e + 2] = fmaf(value(half, e0 + e + 2), scale, b.z);
            v[e + 3] = fmaf(value(half, e0 + e + 3), scale, b.w);
          }
          if (EPI == GM_PIECES && kind == 3) {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = rcp_approx(1.0f + ex2_approx(v[e]));
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) w[e] = pack_half2(v[2 * e], v[2 * e + 1]);
          if (EPI == GM_HALF && p.relu) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __half2 m = __hmax2(*reinterpret_cast<const __half2*>(&w[e]), __float2half2_rn(0.f));
              w[e] = *reinterpret_cast<const uint32_t*>(&m);
            }
          }
          uint32_t off;
          if (EPI == GM_PIECES) off = (lane >> 3) * 1024 + c8 * 128 + (lane & 7) * 16;                         // [row / 8][piece][row % 8]
          else if (EPI == GM_GROUPED) off = (c8 >> 2) * 2048 + lane * 64 + (((c8 & 3) ^ ((lane >> 1) & 3)) << 4);      // [j][a][b], 64-byte swizzle
          else off = lane * 128 + ((c8 ^ (lane & 7)) << 4);                                                   // rows, 128-byte swizzle
          *reinterpret_cast<uint4*>(stage + off) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (EPI == GM_PIECES) {
            const int groups = p.width / 128, inner = col0 % p.width;
            tma_store_4d(&mapO, stage, 0, (inner % 128) / 32, row0 / 8, (kind * groups + inner / 128) * p.batch + h);
          } else if (EPI == GM_GROUPED) {
            tma_store_4d(&mapO, stage, 0, 0, col0 / 32, row0 / 32);
          } else {
            tma_store_3d(&mapO, stage, col0, row0, h);
          }
          bulk_commit();
        }
      }
    }
    if (lane == 0) bulk_wait_all();      // this thread's stores have landed
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) drain_after_abort();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

void configure_gemm() {
  cudaFuncSetAttribute(gemm_kernel<0, GM_HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM);
  cudaFuncSetAttribute(gemm_kernel<1, GM_HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM);
  cudaFuncSetAttribute(gemm_kernel<0, GM_PIECES>, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM);
  cudaFuncSetAttribute(gemm_kernel<0, GM_F32>, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM);
  cudaFuncSetAttribute(gemm_kernel<1, GM_GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM);
}

lf_status make_map_f16_3d(lf_context* ctx, CUtensorMap* map, const void* base, uint64_t d0, uint64_t d1, uint64_t d2,
                          uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1, uint32_t b2 = 1);
lf_status make_map_tiled_act(lf_context* ctx, CUtensorMap* map, const void* base, int ldq, int batch, int rows);
lf_status make_map_f32_any(lf_context* ctx, CUtensorMap* map, const void* base, const uint64_t (&dims)[3], const uint64_t (&strides)[2], const uint32_t (&box)[3]);
lf_status make_map_grouped(lf_context* ctx, CUtensorMap* map, const void* base, uint64_t n, uint64_t cnt);

template <int MAJOR, int EPI>
static lf_status launch(lf_context* ctx, int family, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo, GemmParams p) {
  p.status = (Status*)ctx->tc_status;
  const int64_t tiles = (int64_t)p.batch * ((p.m + GM_BM - 1) / GM_BM) * ((p.n + GM_BN - 1) / GM_BN);
  const int grid = (int)(tiles < ctx->sm_count ? tiles : ctx->sm_count);
  lf_prof_begin(ctx, family);
  lf_launch(ctx, gemm_kernel<MAJOR, EPI>, grid, GM_THREADS, GM_SMEM, ma, mb, mo, p);
  lf_prof_end(ctx);
  ctx->launches++;
  return LF_OK;
}

// out[m][n] = act(sum_k a[m][k] w[n][k] + bias[n]) on fp16 rows
lf_status contract_gemm(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* w, op16* out, int m_rows, int n_out, int k_len,
                        const float* bias, int relu) {
  if (cur.dry) return LF_OK;
  if (k_len % 8 || n_out % 8) return lf_fail(ctx, LF_ERR_ARGUMENT, "GEMM rows must be whole groups of eight");
  CUtensorMap ma, mb, mo;
  LF_TRY(make_map_f16_3d(ctx, &ma, a, k_len, m_rows, 1, (uint64_t)k_len * 2, (uint64_t)m_rows * k_len * 2, GM_BK, GM_BM));
  LF_TRY(make_map_f16_3d(ctx, &mb, w, k_len, n_out, 1, (uint64_t)k_len * 2, (uint64_t)n_out * k_len * 2, GM_BK, GM_BN));
  LF_TRY(make_map_f16_3d(ctx, &mo, out, n_out, m_rows, 1, (uint64_t)n_out * 2, (uint64_t)m_rows * n_out * 2, 64, 32));
  GemmParams p{};
  p.m = m_rows; p.n = n_out; p.k = k_len; p.batch = 1; p.scale = 1.0f; p.bias = bias; p.relu = relu;
  return launch<0, GM_HALF>(ctx, LF_KERNEL_TRIANGLE_CONTRACT, ma, mb, mo, p);
}

lf_status gemm_pieces(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* w, op16* out, int batch, int Q, int ldq, int k_len, int width,
                      const float* bias, float qscale) {
  if (cur.dry) return LF_OK;
  CUtensorMap ma, mb, mo;
  LF_TRY(make_map_f16_3d(ctx, &ma, a, k_len, Q, batch, (uint64_t)k_len * 2, (uint64_t)Q * k_len * 2, GM_BK, GM_BM));
  LF_TRY(make_map_f16_3d(ctx, &mb, w, k_len, 4 * width, 1, (uint64_t)k_len * 2, (uint64_t)4 * width * k_len * 2, GM_BK, GM_BN));
  LF_TRY(make_map_tiled_act(ctx, &mo, out, ldq, batch * 4 * (width / 128), 32));
  GemmParams p{};
  p.m = Q; p.n = 4 * width; p.k = k_len; p.batch = batch; p.scale = 1.0f; p.bias = bias; p.width = width; p.qscale = qscale;
  return launch<0, GM_PIECES>(ctx, LF_KERNEL_TRIANGLE_CONTRACT, ma, mb, mo, p);
}

lf_status gemm_rows_f32(lf_context* ctx, ArenaCursor& cur, const op16* a, int a_pieces, const op16* w, float* out, int add, int batch, int Q, int ldq,
                        int transposed, int n_out, int k_len, const float* bias) {
  if (cur.dry) return LF_OK;
  if (!a_pieces && !transposed) { Q *= batch; batch = 1; }      // rows one after the other
  CUtensorMap ma, mb, mo;
  if (a_pieces) LF_TRY(make_map_tiled_act(ctx, &ma, a, ldq, batch * (k_len / 128), GM_BM));
  else LF_TRY(make_map_f16_3d(ctx, &ma, a, k_len, Q, batch, (uint64_t)k_len * 2, (uint64_t)Q * k_len * 2, GM_BK, GM_BM));
  LF_TRY(make_map_f16_3d(ctx, &mb, w, k_len, n_out, 1, (uint64_t)k_len * 2, (uint64_t)n_out * k_len * 2, GM_BK, GM_BN));
  const uint64_t row = (uint64_t)n_out * 4;
  if (transposed) LF_TRY(make_map_f32_any(ctx, &mo, out, {(uint64_t)n_out, (uint64_t)batch, (uint64_t)Q}, {row, row * batch}, {32, 1, 32}));
  else LF_TRY(make_map_f32_any(ctx, &mo, out, {(uint64_t)n_out, (uint64_t)Q, (uint64_t)batch}, {row, row * Q}, {32, 32, 1}));
  GemmParams p{};
  p.m = Q; p.n = n_out; p.k = k_len; p.batch = batch; p.scale = 1.0f; p.bias = bias; p.a_pieces = a_pieces; p.add = add; p.transposed = transposed;
  return launch<0, GM_F32>(ctx, LF_KERNEL_TRIANGLE_CONTRACT, ma, mb, mo, p);
}

lf_status gemm_rows_half(lf_context* ctx, ArenaCursor& cur, const op16* a_pieces, const op16* w, op16* out, int batch, int Q, int ldq, int n_out, int k_len) {
  if (cur.dry) return LF_OK;
  CUtensorMap ma, mb, mo;
  LF_TRY(make_map_tiled_act(ctx, &ma, a_pieces, ldq, batch * (k_len / 128), GM_BM));
  LF_TRY(make_map_f16_3d(ctx, &mb, w, k_len, n_out, 1, (uint64_t)k_len * 2, (uint64_t)n_out * k_len * 2, GM_BK, GM_BN));
  LF_TRY(make_map_f16_3d(ctx, &mo, out, n_out, Q, batch, (uint64_t)n_out * 2, (uint64_t)Q * n_out * 2, 64, 32));
  GemmParams p{};
  p.m = Q; p.n = n_out; p.k = k_len; p.batch = batch; p.scale = 1.0f; p.a_pieces = 1;
  return launch<0, GM_HALF>(ctx, LF_KERNEL_TRIANGLE_CONTRACT, ma, mb, mo, p);
}

// x[(i, a)][(j, b)] = scale * sum_s left[s][(i, a)] right[s][(j, b)], stored [(i, j)][(a, b)], a, b < 32
lf_status gemm_outer32(lf_context* ctx, ArenaCursor& cur, const op16* left, const op16* right, op16* out, int cnt, int n, int k_len, float scale) {
  if (cur.dry) return LF_OK;
  CUtensorMap ma, mb, mo;
  const uint64_t row = (uint64_t)n * 64;      // both operands have rows of n * 32 values
  LF_TRY(make_map_f16_3d(ctx, &ma, left, (uint64_t)cnt * 32, k_len, 1, row, row * k_len, 64, GM_BK));
  LF_TRY(make_map_f16_3d(ctx, &mb, right, (uint64_t)n * 32, k_len, 1, row, row * k_len, 64, GM_BK));
  LF_TRY(make_map_grouped(ctx, &mo, out, n, cnt));
  GemmParams p{};
  p.m = cnt * 32; p.n = n * 32; p.k = k_len; p.batch = 1; p.scale = scale;
  return launch<1, GM_GROUPED>(ctx, LF_KERNEL_TRIANGLE_CONTRACT, ma, mb, mo, p);
}

// The triangle contraction (see contract): planes of c channels.
lf_status gemm_planes(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, op16* x, int n, int ld, int c, int incoming, float scale) {
  if (cur.dry) return LF_OK;
  CUtensorMap ma, mb, mo;
  const uint64_t row = (uint64_t)ld * 2, plane = row * n;
  if (!incoming) {
    LF_TRY(make_map_f16_3d(ctx, &ma, a, n, n, c, row, plane, GM_BK, GM_BM));
    LF_TRY(make_map_f16_3d(ctx, &mb, b, n, n, c, row, plane, GM_BK, GM_BN));
  } else {
    LF_TRY(make_map_f16_3d(ctx, &ma, b, n, n, c, row, plane, 64, GM_BK));
    LF_TRY(make_map_f16_3d(ctx, &mb, a, n, n, c, row, plane, 64, GM_BK));
  }
  LF_TRY(make_map_f16_3d(ctx, &mo, x, n, n, c, row, plane, 64, 32));
  GemmParams p{};
  p.m = n; p.n = n; p.k = n; p.batch = c; p.scale = scale;
  return incoming ? launch<1, GM_HALF>(ctx, LF_KERNEL_TRIANGLE_CONTRACT, ma, mb, mo, p) : launch<0, GM_HALF>(ctx, LF_KERNEL_TRIANGLE_CONTRACT, ma, mb, mo, p);
}

}  // namespace tc
