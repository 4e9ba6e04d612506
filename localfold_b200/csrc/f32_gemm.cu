// Float32 GEMM on tcgen05: operands taken apart into three bf16 terms (8 + 8 + 8 significand bits, nothing is lost), a
// product of two values into the six term products above 2^-24, float32 accumulation.
#include <cuda.h>

#include "tc05.cuh"
#include "tc_kernels.cuh"

namespace tc {

using namespace tc05;

// One 128 x 128 output tile of one batch entry per work item.  A k block of 64 holds the three terms of both operands
// (96 KiB a stage, two stages); the leading product goes into one TMEM accumulator and the five others into a second
// one (2 x 128 columns, double-buffered), so the tensor core's own additions, which truncate, act on the correction apart
// from the sum.  The epilogue adds the two and keeps the sum of the k blocks in its registers, in round-to-nearest, while the
// accumulators start afresh: errors against float64 are at or below those of a float32 FMA chain (1.9e-7 against
// 3.1e-7 to 4.8e-7 for the triangle update at 203 to 700; with all of k in TMEM 1.3e-6 for a transition of 384 channels).
// Warp roles: 0 = TMA producer, 1 = MMA issuer (owns TMEM), 2..17 = epilogue (lane quadrant = warp % 4, a quarter of the columns).
// With two k blocks a tile (K = 128) the epilogue is what bounds it - eight warps and scalar bias loads took 41 us a launch on average for
// the float32 pair block at N = 203, sixteen 35 - and the operands' way from L2 into shared memory (96 KiB per 1560 cycles of tensor work) with
// more.  An instance per form of output: what a shared epilogue left to passes of their own (triangle gates 38 us, ends of operators 10, bias columns)
// is done here, and 16 launches of the same block take 25 to 46 us, 456 in all, against 486 before with 190 of such passes beside them.
constexpr int G3_BM = 128, G3_BN = 128, G3_BK = 64, G3_STAGES = 2, G3_EPI = 16;
constexpr int G3_PLANE = G3_BM * G3_BK * 2;            // 16 KiB: one term of one operand
constexpr int G3_STAGE = 6 * G3_PLANE;
constexpr int G3_OUT = 2048;                           // per epilogue warp: 32 rows x 64 bytes
constexpr int G3_SMEM = G3_STAGES * G3_STAGE + G3_EPI * G3_OUT + 256 + 1024;
constexpr int G3_THREADS = 64 + 32 * G3_EPI;

struct Gemm3Params {
  int m, n, k, batch;
  float* out;                  // [batch][m][ldo] float32, or null
  bf16* terms;                 // ... or its three terms, [3][batch][m][ldo]
  int64_t ldo, batch_stride, term_stride;
  const float* bias;           // or null
  int bias_n, relu, sigmoid_col0, sigmoid_col1;
  float* gate;                 // behind terms in pieces (Gemm3Out)
  float* pair_bias;
  int bias_q, bias_ld, bias_swap;
  float* act;                  // the end of an operator (Gemm3Out)
  const float* factor;
  int act_add, act_batch, act_q;
  const float* plane_mask;     // or null; see Gemm3Out
  void* plane[2];
  int plane_n, plane_c, plane_half;
  Status* status;
};

// kind::f16 with bf16 operands
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, int major) {
  return make_idesc_f16(M, N, major, major) | (1u << 7) | (1u << 10);
}

// 1 / (1 + e^-v): the quotient by Newton's iteration on the approximate reciprocal, without the branches of the correctly rounded one.
// The bound keeps infinity out of the iteration (a result below 2^-126 is 0) and lets a NaN through, which fminf would drop.
__device__ __forceinline__ float g3_sigmoid(float v) {
  float y, r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(1.0f + expf(-v)), "f"(3e38f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return fmaf(r, fmaf(-y, r, 1.0f), r);
}

enum { G3_FLOAT, G3_TERMS, G3_TERM_PIECES, G3_PLANES, G3_ACT };      // what the epilogue writes (Gemm3Out)

// MAJOR 0: k contiguous in both operands; 1: the row index contiguous in both.  PIECES: A in pieces of eight k, the unswizzled operand format
template <int MAJOR, bool PIECES, int OUT>
__global__ void __launch_bounds__(G3_THREADS, 1)
gemm3_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const Gemm3Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  uint8_t* out_stage = smem + G3_STAGES * G3_STAGE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage + G3_EPI * G3_OUT);
  uint64_t* full = bars;                       // [STAGES]
  uint64_t* empty = bars + G3_STAGES;          // [STAGES]
  uint64_t* tmem_full = empty + G3_STAGES;     // [2]
  uint64_t* tmem_empty = tmem_full + 2;        // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (p.m + G3_BM - 1) / G3_BM, tiles_n = (p.n + G3_BN - 1) / G3_BN, per = tiles_m * tiles_n;
  const int total = p.batch * per;
  const int kblocks = (p.k + G3_BK - 1) / G3_BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < G3_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], G3_EPI); }
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
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        const int h = t / per, rem = t - h * per, mi = rem / tiles_n, nj = rem - mi * tiles_n;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status, 101)) { ok = false; break; }
          uint8_t* sA = smem + stage * G3_STAGE;
          uint8_t* sB = sA + 3 * G3_PLANE;
          mbar_expect_tx(&full[stage], G3_STAGE);
          if (MAJOR == 0) {      // [term][128 rows][64 k], or [term][8 pieces][128 rows]
            if (PIECES) tma_load_4d(sA, &mapA, &full[stage], mi * G3_BM * 2, 0, kb * (G3_BK / 8), 0);
            else tma_load_4d(sA, &mapA, &full[stage], kb * G3_BK, mi * G3_BM, h, 0);
            tma_load_4d(sB, &mapB, &full[stage], kb * G3_BK, nj * G3_BN, h, 0);
          } else {               // per 64 rows: [term][64 k][64 rows]
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              tma_load_4d(sA + q * 3 * (G3_PLANE / 2), &mapA, &full[stage], mi * G3_BM + q * 64, kb * G3_BK, h, 0);
              tma_load_4d(sB + q * 3 * (G3_PLANE / 2), &mapB, &full[stage], nj * G3_BN + q * 64, kb * G3_BK, h, 0);
            }
          }
          if (++stage == G3_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        // a last tile of few columns (a pair bias's) takes as many
        const int nj = t % per % tiles_n, columns = (min(G3_BN, p.n - nj * G3_BN) + 15) / 16 * 16;
        const uint32_t idesc = make_idesc_bf16(G3_BM, columns, MAJOR);
        for (int kb = 0; kb < kblocks; ++kb) {
          const uint32_t d = tmem_base + (it & 1) * 256;
          if (!mbar_wait(&tmem_empty[it & 1], ((it >> 1) & 1) ^ 1, abort_flag, p.status, 102) ||
              !mbar_wait(&full[stage], phase, abort_flag, p.status, 103)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a0 = smem_u32(smem + stage * G3_STAGE), b0 = a0 + 3 * G3_PLANE;
#pragma unroll
          for (int kk = 0; kk < G3_BK / 16; ++kk) {
            // operand descriptor of one term
            auto desc = [&](uint32_t base, int term) {
              return MAJOR == 0 ? make_smem_desc(base + term * G3_PLANE + kk * 32, 16, 1024)
                                : make_smem_desc(base + term * (G3_PLANE / 2) + kk * 2048, 3 * (G3_PLANE / 2), 1024);
            };
            auto adesc = [&](int term) { return PIECES ? make_smem_desc_plain(a0 + term * G3_PLANE + kk * 2 * G3_BM * 16, G3_BM * 16, 128) : desc(a0, term); };
            const uint32_t more = kk != 0 ? 1u : 0u;
            umma_f16(d + 128, adesc(2), desc(b0, 0), idesc, more);
            umma_f16(d + 128, adesc(1), desc(b0, 1), idesc, 1u);
            umma_f16(d + 128, adesc(0), desc(b0, 2), idesc, 1u);
            umma_f16(d + 128, adesc(1), desc(b0, 0), idesc, 1u);
            umma_f16(d + 128, adesc(0), desc(b0, 1), idesc, 1u);
            umma_f16(d, adesc(0), desc(b0, 0), idesc, more);
          }
          umma_commit(&empty[stage]);
          if (++stage == G3_STAGES) { stage = 0; phase ^= 1; }
          umma_commit(&tmem_full[it & 1]);
          ++it;
        }
      }
    }
  } else {
    const int q = warp & 3, part = (warp - 2) >> 2;      // TMEM lane quadrant, 32 of the tile's columns
    uint8_t* stage = out_stage + (warp - 2) * G3_OUT;
    uint32_t it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      const int h = t / per, rem = t - h * per, mi = rem / tiles_n, nj = rem - mi * tiles_n;
      const int col0 = nj * G3_BN + part * 32;
      float v[32];
#pragma unroll 1
      for (int kb = 0; kb < kblocks; ++kb, ++it) {
        if (!mbar_wait(&tmem_full[it & 1], (it >> 1) & 1, abort_flag, p.status, 104)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + ((uint32_t)(q * 32) << 16) + (it & 1) * 256 + part * 32;
#pragma unroll
        for (int c16 = 0; c16 < 2; ++c16) {
          uint32_t lead[16], rest[16];
          tmem_ld16(d + c16 * 16, lead);
          tmem_ld16(d + 128 + c16 * 16, rest);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float x = __uint_as_float(lead[e]) + __uint_as_float(rest[e]);
            v[c16 * 16 + e] = kb ? v[c16 * 16 + e] + x : x;
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[it & 1]);
      }
      if (!ok) break;
      const int row0 = mi * G3_BM + q * 32;
      if (col0 >= (OUT == G3_TERMS ? (int)p.ldo : p.n) || row0 >= p.m) continue;
      if (OUT == G3_PLANES) {
        // 16 channels of a projection and their gates; a lane's pair is its neighbour's next, so a channel leaves as a run of 32 values
        const int groups = p.n / 64, group = col0 / 32, which = group >= groups, h0 = (group - (which ? groups : 0)) * 16;
        const int left = p.plane_c - h0;      // channels there are
        float* bias = reinterpret_cast<float*>(stage);
        bias[lane] = p.bias && (lane & 15) < left ? __ldg(p.bias + (which * 2 + (lane >> 4)) * p.plane_c + h0 + (lane & 15)) : 0.f;
        __syncwarp();
        const int row = row0 + lane;
        if (row < p.m) {
          const float m = __ldg(p.plane_mask + row);
#pragma unroll
          for (int e = 0; e < 16; e += 4) {
            const float4 bp = *reinterpret_cast<const float4*>(bias + e), bg = *reinterpret_cast<const float4*>(bias + 16 + e);
            const float b4[4] = {bp.x, bp.y, bp.z, bp.w}, g4[4] = {bg.x, bg.y, bg.z, bg.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) v[e + u] = (v[e + u] + b4[u]) * g3_sigmoid(v[16 + e + u] + g4[u]) * m;
          }
        }
        const int64_t step = (int64_t)p.plane_n * p.ldo;
        if (p.plane_n % 8 == 0) {
          // eight pairs of a channel never straddle two pair rows: turned round in shared memory, they leave 16 bytes at a time
#pragma unroll 1
          for (int term = 0; term < (p.plane_half ? 1 : 3); ++term) {
            __syncwarp();
            uint16_t* turn = reinterpret_cast<uint16_t*>(stage) + lane;
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              if (p.plane_half) turn[e * 32] = __half_as_ushort(__float2half_rn(v[e]));
              else if (e % 2 == 0) {
                const uint32_t w = split_bf16(v[e], v[e + 1]);
                turn[e * 32] = (uint16_t)w;
                turn[e * 32 + 32] = (uint16_t)(w >> 16);
              }
            }
            __syncwarp();
            const int first = row0 + (lane & 3) * 8, i = first / p.plane_n, k = first - i * p.plane_n;
            uint16_t* dst = reinterpret_cast<uint16_t*>(p.plane[which]) + term * p.term_stride + (h0 + (lane >> 2)) * step + (int64_t)i * p.ldo + k;
#pragma unroll
            for (int u = 0; u < 2; ++u)
              if (first < p.m && (lane >> 2) + u * 8 < left) *reinterpret_cast<uint4*>(dst + u * 8 * step) = *reinterpret_cast<const uint4*>(stage + (u * 32 + lane) * 16);
          }
        } else if (row < p.m) {
          const int i = row / p.plane_n, k = row - i * p.plane_n;
          uint16_t* dst = reinterpret_cast<uint16_t*>(p.plane[which]) + h0 * step + (int64_t)i * p.ldo + k;
          for (int term = 0; term < (p.plane_half ? 1 : 3); ++term, dst += p.term_stride) {
            uint16_t* to = dst;
#pragma unroll
            for (int e = 0; e < 16; ++e, to += step) {
              if (e >= left) break;
              if (p.plane_half) *to = __half_as_ushort(__float2half_rn(v[e]));
              else {
                const bf16 b = __float2bfloat16_rn(v[e]);
                *to = __bfloat16_as_ushort(b);
                v[e] -= __bfloat162float(b);
              }
            }
          }
        }
        __syncwarp();
        continue;
      }
      if (p.bias && col0 < p.bias_n) {      // through the staging rows: four at a time, the same for every lane
        float* bias = reinterpret_cast<float*>(stage);
        bias[lane] = col0 + lane < p.bias_n ? __ldg(p.bias + col0 + lane) : 0.f;
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const float4 b = *reinterpret_cast<const float4*>(bias + e);
          v[e] += b.x; v[e + 1] += b.y; v[e + 2] += b.z; v[e + 3] += b.w;
        }
        __syncwarp();
      }
      if (p.relu) {
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = fmaxf(v[e], 0.f);
      }
      if (col0 >= p.sigmoid_col0 && col0 + 32 <= p.sigmoid_col1) {
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = g3_sigmoid(v[e]);
      } else if (col0 + 32 > p.sigmoid_col0 && col0 < p.sigmoid_col1) {
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = col0 + e >= p.sigmoid_col0 && col0 + e < p.sigmoid_col1 ? g3_sigmoid(v[e]) : v[e];
      }
      if (OUT == G3_ACT) {
        // as below, added where the activations live (no residual is read here: loads in the epilogue took 56 us where this and a pass of its own took 41).
        // The reduction flushes subnormal operands and sums to zero, where an addition in registers keeps them.
        int64_t to[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t r = (uint32_t)(row0 + i * 8 + (lane >> 2));
          to[i] = (p.act_q ? (int64_t)(r % (uint32_t)p.act_q) * p.act_batch + r / (uint32_t)p.act_q : (int64_t)r) * p.n;
        }
#pragma unroll
        for (int c16 = 0; c16 < 2; ++c16) {
          const int piece = lane & 3, col = col0 + c16 * 16 + piece * 4;
          float4 f[4];
          if (p.factor) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int r = row0 + i * 8 + (lane >> 2);
              f[i] = r < p.m && col < p.n ? __ldg(reinterpret_cast<const float4*>(p.factor + (int64_t)r * p.n + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
          }
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4)
            *reinterpret_cast<float4*>(stage + lane * 64 + ((k4 ^ ((lane >> 1) & 3)) << 4)) =
                make_float4(v[c16 * 16 + k4 * 4], v[c16 * 16 + k4 * 4 + 1], v[c16 * 16 + k4 * 4 + 2], v[c16 * 16 + k4 * 4 + 3]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = i * 8 + (lane >> 2);
            float4 x = *reinterpret_cast<const float4*>(stage + r * 64 + ((piece ^ ((r >> 1) & 3)) << 4));
            if (p.factor) { x.x *= f[i].x; x.y *= f[i].y; x.z *= f[i].z; x.w *= f[i].w; }
            if (row0 + r < p.m && col < p.n) {
              float* dst = p.act + to[i] + col;
              if (p.act_add) asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w) : "memory");
              else *reinterpret_cast<float4*>(dst) = x;
            }
          }
          __syncwarp();
        }
      } else if (OUT == G3_FLOAT) {
        // the warp's 32 x 32 values turned round in shared memory, 16 columns at a time (16-byte pieces swizzled by row): 64-byte runs leave
#pragma unroll
        for (int c16 = 0; c16 < 2; ++c16) {
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4)
            *reinterpret_cast<float4*>(stage + lane * 64 + ((k4 ^ ((lane >> 1) & 3)) << 4)) =
                make_float4(v[c16 * 16 + k4 * 4], v[c16 * 16 + k4 * 4 + 1], v[c16 * 16 + k4 * 4 + 2], v[c16 * 16 + k4 * 4 + 3]);
          __syncwarp();
          const int piece = lane & 3, col = col0 + c16 * 16 + piece * 4;
          float* dst = p.out + (int64_t)h * p.batch_stride + (int64_t)(row0 + (lane >> 2)) * p.ldo + col;
          const bool whole = col + 4 <= p.n && (p.ldo & 3) == 0;
#pragma unroll
          for (int i = 0; i < 4; ++i, dst += 8 * p.ldo) {
            const int r = i * 8 + (lane >> 2);
            const float4 x = *reinterpret_cast<const float4*>(stage + r * 64 + ((piece ^ ((r >> 1) & 3)) << 4));
            if (row0 + r < p.m) {
              if (whole) *reinterpret_cast<float4*>(dst) = x;
              else {
                if (col < p.n) dst[0] = x.x;
                if (col + 1 < p.n) dst[1] = x.y;
                if (col + 2 < p.n) dst[2] = x.z;
                if (col + 3 < p.n) dst[3] = x.w;
              }
            }
          }
          __syncwarp();
        }
      } else if (OUT == G3_TERM_PIECES) {
        const int row = row0 + lane;
        const int terms = (int)p.ldo, gates = terms / 3 * 4;      // first column of the gate, of the pair bias
        if (row < p.m && col0 + 32 > terms) {
#pragma unroll
          for (int k8 = 0; k8 < 4; ++k8) {
            const int col = col0 + k8 * 8;
            if (col >= terms && col < gates) {
              float* dst = p.gate + ((int64_t)((col - terms) / 8) * p.m + row) * 8;
              *reinterpret_cast<float4*>(dst) = make_float4(v[k8 * 8], v[k8 * 8 + 1], v[k8 * 8 + 2], v[k8 * 8 + 3]);
              *reinterpret_cast<float4*>(dst + 4) = make_float4(v[k8 * 8 + 4], v[k8 * 8 + 5], v[k8 * 8 + 6], v[k8 * 8 + 7]);
            }
          }
          if (col0 + 32 > gates && gates < p.n) {
            const int i = row / p.bias_q, j = row - i * p.bias_q;
            float* dst = p.pair_bias + (p.bias_swap ? (int64_t)j * p.bias_ld + i : (int64_t)i * p.bias_ld + j);
            const int64_t head = (int64_t)p.bias_q * p.bias_ld;
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (col0 + e >= gates && col0 + e < p.n) dst[(col0 + e - gates) * head] = v[e];
          }
        }
        if (row < p.m && col0 < terms) {
          // a lane's eight columns are 16 bytes and its neighbour's row follows: whole lines leave without a turn through shared memory
          bf16* dst = p.terms + ((int64_t)(col0 / 8) * p.m + row) * 8;
          const int64_t next = (int64_t)p.m * 8;
#pragma unroll
          for (int term = 0; term < 3; ++term, dst += p.term_stride) {
            bf16* to = dst;
#pragma unroll
            for (int k8 = 0; k8 < 4; ++k8, to += next) {
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) w[e] = split_bf16(v[k8 * 8 + 2 * e], v[k8 * 8 + 2 * e + 1]);
              if (col0 + k8 * 8 < terms) *reinterpret_cast<uint4*>(to) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      } else {
        // ... or their terms, 64-byte runs a row and term (ldo a multiple of 8)
        const int piece = lane & 3, col = col0 + piece * 8;
        bf16* dst = p.terms + (int64_t)h * p.batch_stride + (int64_t)(row0 + (lane >> 2)) * p.ldo + col;
#pragma unroll 1
        for (int term = 0; term < 3; ++term, dst += p.term_stride) {
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = split_bf16(v[k4 * 8 + 2 * e], v[k4 * 8 + 2 * e + 1]);
            *reinterpret_cast<uint4*>(stage + lane * 64 + ((k4 ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
          __syncwarp();
          bf16* to = dst;
#pragma unroll
          for (int i = 0; i < 4; ++i, to += 8 * p.ldo) {
            const int r = i * 8 + (lane >> 2);
            const uint4 x = *reinterpret_cast<const uint4*>(stage + r * 64 + ((piece ^ ((r >> 1) & 3)) << 4));
            if (row0 + r < p.m && col < p.ldo) *reinterpret_cast<uint4*>(to) = x;
          }
          __syncwarp();
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) drain_after_abort();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

void configure_gemm3() {
#define G3_CONFIGURE(...) cudaFuncSetAttribute(gemm3_kernel<__VA_ARGS__>, cudaFuncAttributeMaxDynamicSharedMemorySize, G3_SMEM)
  G3_CONFIGURE(0, false, G3_FLOAT);
  G3_CONFIGURE(0, false, G3_TERMS);
  G3_CONFIGURE(0, false, G3_TERM_PIECES);
  G3_CONFIGURE(0, false, G3_PLANES);
  G3_CONFIGURE(0, false, G3_ACT);
  G3_CONFIGURE(0, true, G3_ACT);
  G3_CONFIGURE(0, true, G3_FLOAT);
  G3_CONFIGURE(1, false, G3_FLOAT);
#undef G3_CONFIGURE
}

lf_status make_map_term_pieces(lf_context* ctx, CUtensorMap* map, const SplitMatrix& a, int Q, int batch, uint32_t rows, uint32_t batch_rows, uint32_t pieces, uint32_t terms);
lf_status make_map_terms(lf_context* ctx, CUtensorMap* map, const SplitMatrix& a, uint64_t d0, uint64_t d1, uint64_t batch, uint32_t b1);

lf_status gemm_f32(lf_context* ctx, ArenaCursor& cur, int major, const SplitMatrix& a, const SplitMatrix& b, int m, int n, int k, int batch,
                   const Gemm3Out& o) {
  if (cur.dry) return LF_OK;
  if (a.ld % 8 || b.ld % 8 || a.batch_stride % 8 || b.batch_stride % 8 || a.term_stride % 8 || b.term_stride % 8 || (o.terms && o.ld % 8))
    return lf_fail(ctx, LF_ERR_ARGUMENT, "split operands need strides of whole groups of eight");
  // What no instance below does: another output of an operand in pieces or of the row-contiguous form, a batch of what is laid out for one product
  const int outputs = (o.out != nullptr) + (o.terms != nullptr) + (o.act != nullptr) + (o.plane_mask != nullptr);
  if (outputs != 1 || b.pieces || (a.pieces && (major || !(o.out || o.act))) || (major && !o.out) || (batch != 1 && (a.pieces || o.pieces || o.act || o.plane_mask)) ||
      (o.pieces && (!o.terms || !o.gate || (n > o.ld / 3 * 4 && !o.pair_bias))) || (o.act && (n % 4 || !lf_aligned16(o.act))) ||
      (o.plane_mask && (m != (int64_t)o.plane_n * o.plane_n || n != gated_columns(o.plane_c))))
    return lf_fail(ctx, LF_ERR_UNSUPPORTED, "float32 GEMM: no kernel of this form (%d x %d x %d, batch %d)", m, n, k, batch);
  CUtensorMap ma, mb;
  if (major == 0) {
    if (a.pieces) LF_TRY(make_map_term_pieces(ctx, &ma, a, m, 1, G3_BM, 1, G3_BK / 8, 3));
    else LF_TRY(make_map_terms(ctx, &ma, a, k, m, batch, G3_BM));
    LF_TRY(make_map_terms(ctx, &mb, b, k, n, batch, G3_BN));
  } else {
    LF_TRY(make_map_terms(ctx, &ma, a, m, k, batch, G3_BK));
    LF_TRY(make_map_terms(ctx, &mb, b, n, k, batch, G3_BK));
  }
  Gemm3Params p{};
  p.m = m; p.n = n; p.k = k; p.batch = batch;
  p.out = o.out; p.terms = o.terms; p.ldo = o.ld; p.batch_stride = o.batch_stride; p.term_stride = o.term_stride;
  p.bias = o.bias; p.bias_n = o.bias_n; p.relu = o.relu; p.sigmoid_col0 = o.sigmoid_col0; p.sigmoid_col1 = o.sigmoid_col1;
  p.gate = o.gate; p.pair_bias = o.pair_bias; p.bias_q = o.bias_q; p.bias_ld = o.bias_ld; p.bias_swap = o.bias_swap;
  p.act = o.act; p.factor = o.factor; p.act_add = o.act_add; p.act_batch = o.act_batch; p.act_q = o.act_q;
  p.plane_mask = o.plane_mask; p.plane[0] = o.plane[0]; p.plane[1] = o.plane[1]; p.plane_n = o.plane_n; p.plane_c = o.plane_c; p.plane_half = o.plane_half;
  p.status = (Status*)ctx->tc_status;
  const int64_t tiles = (int64_t)batch * ((m + G3_BM - 1) / G3_BM) * ((n + G3_BN - 1) / G3_BN);
  if (tiles > INT32_MAX - ctx->sm_count) return lf_fail(ctx, LF_ERR_UNSUPPORTED, "float32 GEMM: %d x %d x %d tiles exceed the work index", batch, m, n);
  const int grid = (int)(tiles < ctx->sm_count ? tiles : ctx->sm_count);
  lf_prof_begin(ctx, LF_KERNEL_SIMT);
#define G3_LAUNCH(...) lf_launch(ctx, gemm3_kernel<__VA_ARGS__>, grid, G3_THREADS, G3_SMEM, ma, mb, p)
  if (a.pieces && o.act) G3_LAUNCH(0, true, G3_ACT);
  else if (a.pieces) G3_LAUNCH(0, true, G3_FLOAT);
  else if (o.act) G3_LAUNCH(0, false, G3_ACT);
  else if (major == 1) G3_LAUNCH(1, false, G3_FLOAT);
  else if (o.plane_mask) G3_LAUNCH(0, false, G3_PLANES);
  else if (o.pieces) G3_LAUNCH(0, false, G3_TERM_PIECES);
  else if (o.terms) G3_LAUNCH(0, false, G3_TERMS);
  else G3_LAUNCH(0, false, G3_FLOAT);
#undef G3_LAUNCH
  lf_prof_end(ctx);
  ctx->launches++;
  return LF_OK;
}

}  // namespace tc
