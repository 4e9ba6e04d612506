// Gated float32 attention core for any head width, its products on the tensor cores: every operand is taken apart into three
// bf16 terms (8 + 8 + 8 significand bits, so nothing of it is lost) and a product into the six term products above 2^-24,
// accumulated in float32.  Float32 mode, and 16-bit mode for the heads that the tcgen05 core does not take; few logits, and the head widths that
// f32_attention.cu does not have.
#pragma once

#include "common.cuh"

namespace mma_attention {

constexpr float kLog2E = 1.4426950408889634f;
// 2^x (relative error 2^-22).  exp(l - m) is taken as 2^(l log2(e) - m log2(e)) with one rounding of the exponent, as
// l - m would have; the factor that the rounding of m log2(e) makes is common to a row and divides out.
__device__ __forceinline__ float exp2_(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {      // round to nearest
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// (x, y) = sum over the three terms; the remainders are exact
__device__ __forceinline__ void split3(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[i] = pack_bf16(x, y);
    x -= __uint_as_float(t[i] << 16);
    y -= __uint_as_float(t[i] & 0xffff0000u);
  }
}
// The same by truncation, for probabilities (no conversion instruction).
__device__ __forceinline__ void split3_cut(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[i] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    if (i < 2) {
      x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
      y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
    }
  }
}

__device__ __forceinline__ void mma16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(b0));
}
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const void* row) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(row);
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
template <bool TRANS>
__device__ __forceinline__ void ldmatrix2(uint32_t& r0, uint32_t& r1, const void* row) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(row);
  if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
  else asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}

// global -> shared without passing through registers; bytes 0 writes zeros
__device__ __forceinline__ void copy_async16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

struct AttentionShape {
  int batch, Q, heads;
  int transpose, mask_mode, clamp;      // mask_mode 0: logit += 1e9 (m - 1); 1: logit += m > 0 ? 0 : -1e9
  float scale;
  int64_t rows, term_stride;            // rows and terms of q | k | v in pieces of eight channels: [3][channels / 8][rows][8]
  int ldb;                              // rows of the bias
  int64_t out_stride;                   // terms of the output
  int wb, wq;                           // warps of a block: wb batch rows x wq groups of 16 queries
  int kt;                               // keys of a staged tile, a multiple of 32
  int mk;                               // keys whose mask terms are held at a time, a multiple of kt
};

constexpr int AT_STEP = 32;                                                   // keys of one step of a warp
__host__ __device__ constexpr int at_pitch(int D) { return 8 * ((D / 8) | 1); }      // odd in 16-byte units: ldmatrix rows spread over the banks
constexpr int AT_TERMS = 3;
__host__ __device__ constexpr size_t attention_smem(int D, int wb, int kt, int mk) {
  return (size_t)wb * (2 * 2 * AT_TERMS * kt * at_pitch(D) * 2 + mk * 4);
}

//   qkv: terms of (q | k | v) in pieces and logical row order, a head of each D channels wide, gate: sigmoid(gate) likewise in
//        float32 (the projection's weights are padded to the instance's width, so nothing here is conditional on the true one)
//   bias: float32 [H][Q][ldb] or null; mask: indexed b * Q + j, or j * batch + b when transpose
//   out:  softmax(.) v * gate as terms in pieces, the operand of the output projection
// A warp owns 16 queries of one (batch row, head); Q and the running output stay in registers in the tensor core's
// fragment layout, and probabilities become the A operand of P V without leaving them.  The warps of a block share K and
// V tiles of kt keys, copied a tile ahead as the projection wrote them, and step through them 32 keys at a time; mask terms
// are fetched mk keys at a time (a fetch per tile had the block wait for it at every barrier).  A row's reference is the maximum of its first
// 32 logits, raised only when exponentials overflow 2^60: no maximum is searched otherwise.  P V of a tile goes into
// fresh accumulators (the leading term product apart from the others) that are added to the output outside the tensor
// core, so that whatever the tensor core's own additions lose is of a tile's share, not of the running sum: 2e-7
// relative against float64, as the float32 form on the FMA pipe.
// Bound by the latency of a warp's chain (a third of the tensor pipe, half of the issue slots, 16 warps an SM).  Measured,
// 384 x 384 with 4 heads of 16: 0.51 ms, against 5.06 ms with a warp per query and a shuffle per key and 0.68 ms with
// four queries a thread on packed FMAs; 203 x 203, 4 x 32: 0.19 ms against 0.98 and 0.24.
template <int D, bool BIAS>
__global__ void __launch_bounds__(256, D > 32 ? 1 : 2)
attention_kernel(const uint16_t* __restrict__ qkv, const float* __restrict__ gates, const float* __restrict__ bias, const float* __restrict__ mask, const AttentionShape s,
                 uint16_t* __restrict__ out) {
  lf_chain();
  constexpr int TERMS = AT_TERMS, TOP = TERMS - 1;                    // highest order of a term product that is kept: i + j <= TOP
  constexpr int KT = AT_STEP, PITCH = at_pitch(D), NK = D / 16, TAIL = (D / 8) & 1, ND = D / 8;
  const int plane = s.kt * PITCH;                   // elements of one term of one staged tile
  extern __shared__ uint4 at_sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int wb = warp / s.wq, wq = warp % s.wq;
  const int Q = s.Q, HD = s.heads * D;
  const int64_t piece = s.rows * 8;
  const int h = blockIdx.z, b0 = blockIdx.y * s.wb, b = b0 + wb;
  const int q0 = (blockIdx.x * s.wq + wq) * 16;
  // [2 buffers][wb][K: TERMS | V: TERMS][kt][PITCH], then [wb][mk] mask terms
  uint16_t* kv_s = reinterpret_cast<uint16_t*>(at_sm);
  float* mask_s = reinterpret_cast<float*>(kv_s + 2 * s.wb * 2 * TERMS * plane);
  const int tiles = (Q + s.kt - 1) / s.kt;
  const bool active = b < s.batch && q0 < Q;        // of the warp as a whole

  // ---- staging: 16-byte copies of eight channels of one term ----
  auto stage = [&](int tile) {
    const int j0 = tile * s.kt, buf = tile & 1;
    for (int u = threadIdx.x; u < s.kt * ND; u += blockDim.x) {      // (key, eight channels), then every batch row, K or V and term
      const int e = (u % ND) * 8, j = u / ND;
      for (int bb = 0; bb < s.wb; ++bb) {
        const bool ok = j0 + j < Q && b0 + bb < s.batch;
        const uint16_t* src = ok ? qkv + (HD + h * D + e) / 8 * piece + ((int64_t)(b0 + bb) * Q + j0 + j) * 8 : qkv;
        uint16_t* dst = kv_s + (buf * s.wb + bb) * 2 * TERMS * plane + j * PITCH + e;
#pragma unroll
        for (int which = 0; which < 2; ++which)
#pragma unroll
          for (int i = 0; i < TERMS; ++i)
            copy_async16(dst + (which * TERMS + i) * plane, ok ? src + which * (HD / 8) * piece + i * s.term_stride : src, ok ? 16 : 0);
      }
    }
    copy_async_commit();
  };
  auto fetch_mask = [&](int j0) {
    for (int u = threadIdx.x; u < s.wb * s.mk; u += blockDim.x) {
      const int j = j0 + u % s.mk, bb = b0 + u / s.mk;
      float term = 0.f;
      if (j < Q && bb < s.batch) {
        const float m = __ldg(mask + (s.transpose ? (int64_t)j * s.batch + bb : (int64_t)bb * Q + j));
        term = s.mask_mode == 0 ? 1e9f * (m - 1.0f) : (m > 0.f ? 0.f : -1e9f);
      }
      mask_s[u] = term;
    }
  };
  stage(0);

  // ---- Q as A fragments of its terms ----
  uint32_t qa[TERMS][NK > 0 ? NK : 1][4], qt[TERMS][2];      // qt: the last 8 channels of an odd number of them
  const int row0 = q0 + g, row1 = q0 + g + 8;
  auto q_pair = [&](int row, int term, int e) {
    return active && row < Q ? *reinterpret_cast<const uint32_t*>(qkv + term * s.term_stride + (h * D + e) / 8 * piece + ((int64_t)b * Q + row) * 8 + (e & 7)) : 0u;
  };
#pragma unroll
  for (int i = 0; i < TERMS; ++i) {
#pragma unroll
    for (int kk = 0; kk < NK; ++kk)
#pragma unroll
      for (int r = 0; r < 4; ++r) qa[i][kk][r] = q_pair((r & 1) ? row1 : row0, i, kk * 16 + 2 * t + (r >> 1) * 8);
    if (TAIL) {
#pragma unroll
      for (int r = 0; r < 2; ++r) qt[i][r] = q_pair(r ? row1 : row0, i, NK * 16 + 2 * t);
    }
  }

  // the bias of a tile's keys: this thread's two rows, eight columns each
  const bool pairs = (s.ldb & 1) == 0;
  const float* bias0 = BIAS ? bias + ((int64_t)h * Q + (row0 < Q ? row0 : 0)) * s.ldb + 2 * t : nullptr;
  const float* bias1 = BIAS ? bias + ((int64_t)h * Q + (row1 < Q ? row1 : 0)) * s.ldb + 2 * t : nullptr;
  float bv[4][4];
  auto load_bias = [&](int j0) {
    if (!BIAS) return;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int j = j0 + n * 8;
      if (pairs && j + 2 * t + 1 < Q) {
        const float2 x = __ldg(reinterpret_cast<const float2*>(bias0 + j)), y = __ldg(reinterpret_cast<const float2*>(bias1 + j));
        bv[n][0] = x.x; bv[n][1] = x.y; bv[n][2] = y.x; bv[n][3] = y.y;
      } else {
        bv[n][0] = j + 2 * t < Q ? __ldg(bias0 + j) : 0.f;
        bv[n][1] = j + 2 * t + 1 < Q ? __ldg(bias0 + j + 1) : 0.f;
        bv[n][2] = j + 2 * t < Q ? __ldg(bias1 + j) : 0.f;
        bv[n][3] = j + 2 * t + 1 < Q ? __ldg(bias1 + j + 1) : 0.f;
      }
    }
  };

  float o[ND][4];
#pragma unroll
  for (int n = 0; n < ND; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
  bool far = false;
  int mask0 = 0;                                      // first key of the mask terms at hand
  float ref[2] = {0.f, 0.f}, ref2[2] = {0.f, 0.f}, sum[2] = {0.f, 0.f};      // of rows row0, row1; ref2 = ref log2(e)
  if (active) load_bias(0);
  for (int tile = 0; tile < tiles; ++tile) {
    copy_async_wait();
    __syncthreads();                                  // the tile is staged, and nobody reads the other buffer any more
    if (tile + 1 < tiles) stage(tile + 1);
    if (tile * s.kt % s.mk == 0) {
      mask0 = tile * s.kt;
      fetch_mask(mask0);
      __syncthreads();
    }
    if (!active) continue;
    const int buf = tile & 1;
#pragma unroll 1
    for (int step = 0; step < s.kt && tile * s.kt + step < Q; step += KT) {
    const int key0 = tile * s.kt + step;
    const uint16_t* k_s = kv_s + (buf * s.wb + wb) * 2 * TERMS * plane + step * PITCH;
    const uint16_t* v_s = k_s + TERMS * plane;
    const float* ms = mask_s + wb * s.mk + key0 - mask0;
    // ---- S = Q K^T for 32 keys (four accumulators in flight): small term products first, the leading one last ----
    float l[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) l[n][e] = 0.f;
    {
      uint32_t kb[TERMS][2][4];
      // matrices (keys 0-7, k 0-7), (keys 0-7, k 8-15), (keys 8-15, k 0-7), (keys 8-15, k 8-15) of each 16 keys
      const uint16_t* base = k_s + ((lane & 7) + (lane >> 4) * 8) * PITCH + ((lane >> 3) & 1) * 8;
      // the term products below the leading one first, over all channels; the leading ones last
#pragma unroll
      for (int pass = TOP; pass >= 0; pass -= 2) {
#pragma unroll
        for (int kk = 0; kk < NK; ++kk) {
#pragma unroll
          for (int i = 0; i <= pass; ++i)
#pragma unroll
            for (int grp = 0; grp < 2; ++grp) ldmatrix4<false>(kb[i][grp], base + i * plane + grp * 16 * PITCH + kk * 16);
#pragma unroll
          for (int order = pass; order >= (pass ? 1 : 0); --order)        // terms i and order - i
#pragma unroll
            for (int i = 0; i <= order; ++i)
#pragma unroll
              for (int n = 0; n < 4; ++n) mma16(l[n], qa[i][kk], kb[order - i][n >> 1][(n & 1) * 2], kb[order - i][n >> 1][(n & 1) * 2 + 1]);
        }
        if (TAIL) {
          // matrices: keys 0-7, 8-15, 16-23, 24-31 of the last eight channels
#pragma unroll
          for (int i = 0; i <= pass; ++i) ldmatrix4<false>(kb[i][0], k_s + i * plane + lane * PITCH + NK * 16);
#pragma unroll
          for (int order = pass; order >= (pass ? 1 : 0); --order)
#pragma unroll
            for (int i = 0; i <= order; ++i)
#pragma unroll
              for (int n = 0; n < 4; ++n) mma8(l[n], qt[i][0], qt[i][1], kb[order - i][0][n]);
        }
      }
    }
    // ---- logits ----
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const float2 m2 = *reinterpret_cast<const float2*>(ms + 2 * t + 8 * n);
      // the bias by way of registers of its own, or not: the compiler orders the wide heads better with them (32: 184 -> 180 us a launch, 203 x 203),
      // the narrow ones without (8: 995 -> 936 us, 1024 x 256)
      float add[4] = {0.f, 0.f, 0.f, 0.f};
      if constexpr (BIAS && D > 16) {
#pragma unroll
        for (int e = 0; e < 4; ++e) add[e] = bv[n][e];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        l[n][e] = fmaf(l[n][e], s.scale, (e & 1) ? m2.y : m2.x);
        if (BIAS) l[n][e] += D > 16 ? add[e] : bv[n][e];
        if (s.clamp) l[n][e] = fminf(fmaxf(l[n][e], -1e8f), 1e8f);
      }
    }
    if (key0 + KT > Q) {                           // past the end: not keys at all
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (key0 + 2 * t + 8 * n + (e & 1) >= Q) l[n][e] = -INFINITY;
    }
    if (BIAS && key0 + KT < Q) load_bias(key0 + KT);      // for the next step
    auto row_max = [&](int r) {
      float m = fmaxf(l[0][2 * r], l[0][2 * r + 1]);
#pragma unroll
      for (int n = 1; n < 4; ++n) m = fmaxf(m, fmaxf(l[n][2 * r], l[n][2 * r + 1]));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
      return fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    };
    // a reference of a masked row is near -1e9, where its product with log2(e) is rounded to whole powers of two: such
    // rows subtract first
    auto update_far = [&]() { far = __any_sync(0xffffffffu, fabsf(ref[0]) > 65536.f || fabsf(ref[1]) > 65536.f); };
    if (key0 == 0) {
#pragma unroll
      for (int r = 0; r < 2; ++r) { ref[r] = row_max(r); ref2[r] = ref[r] * kLog2E; }      // key 0 exists: finite
      update_far();
    }
    float p[4][4], ps[2];
    auto exponentials = [&]() {
      float a[4], c[4];
      // exponents: l log2(e) - ref2, or of rows near -1e9 (l - ref) log2(e) - a pass of its own in front
      float x[4][4], shift[2] = {-ref2[0], -ref2[1]};
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) x[n][e] = l[n][e];
      if (far) {
        shift[0] = shift[1] = 0.f;
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) x[n][e] -= ref[e >> 1];
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) p[n][e] = exp2_(fmaf(x[n][e], kLog2E, shift[e >> 1]));
        a[n] = p[n][0] + p[n][1];
        c[n] = p[n][2] + p[n][3];
      }
      ps[0] = (a[0] + a[1]) + (a[2] + a[3]);
      ps[1] = (c[0] + c[1]) + (c[2] + c[3]);
    };
    exponentials();
    constexpr float kBig = 1.1529215e18f;      // 2^60
    if (__any_sync(0xffffffffu, !(ps[0] <= kBig) || !(ps[1] <= kBig))) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float next = fmaxf(ref[r], row_max(r)), next2 = next * kLog2E;
        const float c = exp2_(far ? (ref[r] - next) * kLog2E : ref2[r] - next2);
        ref[r] = next;
        ref2[r] = next2;
        sum[r] *= c;
#pragma unroll
        for (int n = 0; n < ND; ++n) { o[n][2 * r] *= c; o[n][2 * r + 1] *= c; }
      }
      update_far();
      exponentials();
    }
    sum[0] += ps[0];
    sum[1] += ps[1];
    // ---- P V: the leading product and the others in accumulators of their own ----
    float f[ND][4], fc[ND][4];
#pragma unroll
    for (int n = 0; n < ND; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) f[n][e] = fc[n][e] = 0.f;
#pragma unroll
    for (int grp = 0; grp < 2; ++grp) {
      uint32_t pa[TERMS][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {      // (row0, keys 2t), (row1, same), then keys + 8
        const float x = p[grp * 2 + (r >> 1)][(r & 1) * 2], y = p[grp * 2 + (r >> 1)][(r & 1) * 2 + 1];
        uint32_t term[3];
        split3_cut(x, y, term);
#pragma unroll
        for (int i = 0; i < 3; ++i) pa[i][r] = term[i];
      }
#pragma unroll
      for (int np = 0; np < ND; np += 2) {
        uint32_t vb[TERMS][4];
#pragma unroll
        for (int i = 0; i < TERMS; ++i) {
          const uint16_t* base = v_s + i * plane + (grp * 16 + (lane & 15)) * PITCH + np * 8;
          if (np + 1 < ND) ldmatrix4<true>(vb[i], base + (lane >> 4) * 8);
          else ldmatrix2<true>(vb[i][0], vb[i][1], base);
        }
#pragma unroll
        for (int order = TOP; order >= 0; --order)
#pragma unroll
          for (int i = 0; i <= order; ++i) {
            mma16(order ? fc[np] : f[np], pa[i], vb[order - i][0], vb[order - i][1]);
            if (np + 1 < ND) mma16(order ? fc[np + 1] : f[np + 1], pa[i], vb[order - i][2], vb[order - i][3]);
          }
      }
    }
#pragma unroll
    for (int n = 0; n < ND; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[n][e] += f[n][e] + fc[n][e];
    }
  }
  if (!active) return;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    const int row = r ? row1 : row0;
    if (row >= Q) continue;
    const float inv = 1.0f / sum[r];
    const float* gate = gates + h * D / 8 * piece + ((int64_t)b * Q + row) * 8 + 2 * t;
    uint16_t* dst = out + h * D / 8 * piece + ((int64_t)b * Q + row) * 8 + 2 * t;
#pragma unroll
    for (int n = 0; n < ND; ++n) {
      const float2 gv = __ldg(reinterpret_cast<const float2*>(gate + n * piece));
      uint32_t term[3];
      split3(o[n][2 * r] * inv * gv.x, o[n][2 * r + 1] * inv * gv.y, term);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(dst + i * s.out_stride + n * piece) = term[i];
    }
  }
}

}  // namespace mma_attention
