// Row-wise kernels around the GEMMs: LayerNorm in its output forms, gating, residual addition, layout changes.  All of
// them are bound by memory: 16-byte accesses, several rows in flight per warp, one read of the input.
#pragma once

#include "simt_kernels.cuh"

namespace rows {

using simt::from_f;
using simt::sigmoidf_;
using simt::to_f;
using simt::warp_sum;

// x -> the three bf16 terms of x and y, packed
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
    t[i] = *reinterpret_cast<const uint32_t*>(&b);
    x -= __low2float(b);
    y -= __high2float(b);
  }
}
// four consecutive values into a [3][...] terms matrix
__device__ __forceinline__ void store_terms4(bf16* dst, int64_t term_stride, const float (&v)[4]) {
  uint32_t a[3], b[3];
  split_pair(v[0], v[1], a);
  split_pair(v[2], v[3], b);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(dst + i * term_stride) = make_uint2(a[i], b[i]);
}
template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&v)[4]) {
  if (sizeof(T) == 4) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const T* h = reinterpret_cast<const T*>(&u);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = to_f(h[e]);
  }
}
template <typename T>
__device__ __forceinline__ void store4(T* p, const float (&v)[4]) {
  if (sizeof(T) == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else {
    T h[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = from_f<T>(v[e]);
    *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
  }
}

enum LnOut { LN_F32, LN_HALF, LN_HALF_ONE, LN_TERMS };      // LN_HALF_ONE: rows are ch + 16 long, a one and fifteen zeros after the channels

// LayerNorm over rows of ch = 4 * NV * L channels, L lanes a row (a power of two up to 32), R rows a lane group in
// flight.  Logical row r = b * Q + i reads memory row i * batch + b when `transpose`.  variance: 1 two-pass, 2 fast.
// 147 456 rows of 64 channels: 49 us with a warp and two to three passes over memory a row.
template <typename TIn, int NV, int L, int OUT, int R>
__global__ void __launch_bounds__(256)
layer_norm_rows_kernel(const TIn* __restrict__ in, int64_t count, const float* __restrict__ gamma, const float* __restrict__ beta, float eps,
                       int variance, int transpose, int batch, int Q, void* __restrict__ out, int64_t term_stride) {
  lf_chain();
  constexpr int CH = 4 * NV * L, GROUPS = 256 / L;
  const int l = threadIdx.x % L;
  const int64_t first = (int64_t)blockIdx.x * (GROUPS * R) + threadIdx.x / L;
  float v[R][NV][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t row = first + r * GROUPS;
    int64_t src = row;
    if (transpose) { const uint32_t u = (uint32_t)row, uq = (uint32_t)Q; src = (int64_t)(u % uq) * batch + u / uq; }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if (row < count) load4(in + src * CH + (k * L + l) * 4, v[r][k]);
      else v[r][k][0] = v[r][k][1] = v[r][k][2] = v[r][k][3] = 0.f;
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) s += (v[r][k][0] + v[r][k][1]) + (v[r][k][2] + v[r][k][3]);
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float mean = s * (1.0f / CH);
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) { const float d = variance == 2 ? v[r][k][e] : v[r][k][e] - mean; q = fmaf(d, d, q); }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    const float var = variance == 2 ? q * (1.0f / CH) - mean * mean : q * (1.0f / CH);
    float inv = rsqrtf(var + eps);
    inv = inv * (1.5f - 0.5f * (var + eps) * inv * inv);      // one Newton step: rsqrtf is 2 ulp
    const int64_t row = first + r * GROUPS;
    const bool ok = row < count;      // (no lane leaves the loop: the row groups of a warp share its shuffles)
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if (!ok) break;
      const int c = (k * L + l) * 4;
      const float4 g = __ldg(reinterpret_cast<const float4*>(gamma + c)), b = __ldg(reinterpret_cast<const float4*>(beta + c));
      float y[4] = {(v[r][k][0] - mean) * inv * g.x + b.x, (v[r][k][1] - mean) * inv * g.y + b.y, (v[r][k][2] - mean) * inv * g.z + b.z,
                    (v[r][k][3] - mean) * inv * g.w + b.w};
      if (OUT == LN_F32) store4(reinterpret_cast<float*>(out) + row * CH + c, y);
      else if (OUT == LN_TERMS) store_terms4(reinterpret_cast<bf16*>(out) + row * CH + c, term_stride, y);
      else store4(reinterpret_cast<__half*>(out) + row * (OUT == LN_HALF_ONE ? CH + 16 : CH) + c, y);
    }
    if (OUT == LN_HALF_ONE && ok && l < 2)
      *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(out) + row * (CH + 16) + CH + l * 8) = make_uint4(l == 0 ? 0x3c00u : 0u, 0u, 0u, 0u);
  }
}

// ... of any width, a warp a row: float32 into terms with rows of ld (a multiple of 8; zeros past the channels)
template <typename TIn>
__global__ void layer_norm_terms_kernel(const TIn* __restrict__ in, int64_t count, int ch, int ld, const float* __restrict__ gamma,
                                        const float* __restrict__ beta, float eps, int variance, int transpose, int batch, int Q,
                                        bf16* __restrict__ out, int64_t term_stride) {
  lf_chain();
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= count) return;
  int64_t src = row;
  if (transpose) { const int64_t b = row / Q, i = row % Q; src = i * batch + b; }
  const TIn* x = in + src * ch;
  float s = 0.f, ss = 0.f;
  for (int c = lane; c < ch; c += 32) { const float v = to_f(x[c]); s += v; ss += v * v; }
  s = warp_sum(s);
  const float mean = s / ch;
  float var;
  if (variance == 2) var = warp_sum(ss) / ch - mean * mean;
  else {
    float acc = 0.f;
    for (int c = lane; c < ch; c += 32) { const float d = to_f(x[c]) - mean; acc += d * d; }
    var = warp_sum(acc) / ch;
  }
  float inv = rsqrtf(var + eps);
  inv = inv * (1.5f - 0.5f * (var + eps) * inv * inv);
  for (int c = lane * 2; c < ld; c += 64) {
    uint32_t t[3];
    split_pair(c < ch ? (to_f(x[c]) - mean) * inv * gamma[c] + beta[c] : 0.f,
               c + 1 < ch ? (to_f(x[c + 1]) - mean) * inv * gamma[c + 1] + beta[c + 1] : 0.f, t);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(out + i * term_stride + row * ld + c) = t[i];
  }
}

// float32 rows of `ch` -> terms with rows of ld
__global__ void to_terms_kernel(const float* __restrict__ in, int64_t count, int ch, int ld, bf16* __restrict__ out, int64_t term_stride) {
  lf_chain();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int l2 = ld >> 1;
  if (idx >= count * l2) return;
  const int64_t row = idx / l2;
  const int c = (int)(idx % l2) * 2;
  uint32_t t[3];
  split_pair(c < ch ? in[row * ch + c] : 0.f, c + 1 < ch ? in[row * ch + c + 1] : 0.f, t);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(out + i * term_stride + row * ld + c) = t[i];
}

// SwiGLU over [rows][2 inter] (gate half first) -> terms with rows of ld
__global__ void swiglu_terms_kernel(const float* __restrict__ wide, int64_t count, int inter, int ld, bf16* __restrict__ out, int64_t term_stride) {
  lf_chain();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int l2 = ld >> 1;
  if (idx >= count * l2) return;
  const int64_t row = idx / l2;
  const int c = (int)(idx % l2) * 2;
  float v[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float g = c + e < inter ? wide[row * 2 * inter + c + e] : 0.f, x = c + e < inter ? wide[row * 2 * inter + inter + c + e] : 0.f;
    v[e] = g * sigmoidf_(g) * x;
  }
  uint32_t t[3];
  split_pair(v[0], v[1], t);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(out + i * term_stride + row * ld + c) = t[i];
}

// ... on fp16 (inter a multiple of 8): silu(gate half) * value half, eight channels a thread
__global__ void swiglu_half_kernel(const __half* __restrict__ wide, int64_t count, int inter, __half* __restrict__ out) {
  lf_chain();
  const int c = (blockIdx.x * 32 + threadIdx.x) * 8;
  const int64_t row = (int64_t)blockIdx.y * 8 + threadIdx.y;
  if (c >= inter || row >= count) return;
  const uint4 g = *reinterpret_cast<const uint4*>(wide + row * 2 * inter + c), x = *reinterpret_cast<const uint4*>(wide + row * 2 * inter + inter + c);
  uint4 o;
  __half2* h = reinterpret_cast<__half2*>(&o);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 a = __half22float2(reinterpret_cast<const __half2*>(&g)[e]), b = __half22float2(reinterpret_cast<const __half2*>(&x)[e]);
    h[e] = __floats2half2_rn(a.x * sigmoidf_(a.x) * b.x, a.y * sigmoidf_(a.y) * b.y);
  }
  *reinterpret_cast<uint4*>(out + row * inter + c) = o;
}

// LayerNorm over the channels of a channel-major x[h][i][ld] -> terms with rows of ldc.  A block takes 32 pairs of one pair row; the
// tile [c][32] sits in shared memory.
template <typename TIn>
__global__ void __launch_bounds__(256)
center_norm_kernel(const TIn* __restrict__ x, int c, int n, int ld, const float* __restrict__ gamma, const float* __restrict__ beta,
                   float eps, int variance, float prescale, int ldc, bf16* __restrict__ xn, int64_t term_stride) {
  lf_chain();
  extern __shared__ float tile[];   // [c][33]
  const int tiles = (n + 31) / 32, i = blockIdx.x / tiles, k0 = (blockIdx.x % tiles) * 32;
  const int tx = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int h = w; h < c; h += 8) tile[h * 33 + tx] = k0 + tx < n ? to_f(x[((int64_t)h * n + i) * ld + k0 + tx]) * prescale : 0.f;
  __syncthreads();
  for (int r = w; r < 32 && k0 + r < n; r += 8) {
    float s = 0.f, ss = 0.f;
    for (int h = tx; h < c; h += 32) { const float v = tile[h * 33 + r]; s += v; ss += v * v; }
    s = warp_sum(s);
    const float mean = s / c;
    float var;
    if (variance == 2) var = warp_sum(ss) / c - mean * mean;
    else {
      float acc = 0.f;
      for (int h = tx; h < c; h += 32) { const float d = tile[h * 33 + r] - mean; acc += d * d; }
      var = warp_sum(acc) / c;
    }
    float inv = rsqrtf(var + eps);
    inv = inv * (1.5f - 0.5f * (var + eps) * inv * inv);
    const int64_t row = ((int64_t)i * n + k0 + r) * ldc;
    for (int h = tx * 2; h < ldc; h += 64) {
      const float v0 = h < c ? (tile[h * 33 + r] - mean) * inv * gamma[h] + beta[h] : 0.f;
      const float v1 = h + 1 < c ? (tile[(h + 1) * 33 + r] - mean) * inv * gamma[h + 1] + beta[h + 1] : 0.f;
      uint32_t t[3];
      split_pair(v0, v1, t);
#pragma unroll
      for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(xn + e * term_stride + row + h) = t[e];
    }
  }
}

// The same from fp16 for c <= 8 GROUPS, a multiple of 8 (wider ones do not fit the registers): a block takes 64 pairs of one pair row in
// 16-byte pieces, four threads a pair hold the channels in registers (channels 8 g + 2 part and the next), and the terms leave through
// shared memory in 16-byte pieces.  Bound by the passes over shared memory.
constexpr int kCenterPitch = 72;      // 64 pairs and 16 bytes: the four channel rows a warp reads at a time spread over the banks
constexpr size_t center_norm_half_smem(int c) { return ((size_t)c * kCenterPitch + (size_t)3 * 64 * (c + 8)) * sizeof(uint16_t); }
template <int GROUPS>
__global__ void __launch_bounds__(256)
center_norm_half_kernel(const __half* __restrict__ x, int c, int n, int ld, const float* __restrict__ gamma, const float* __restrict__ beta, float eps,
                        int variance, float prescale, bf16* __restrict__ xn, int64_t term_stride) {
  lf_chain();
  extern __shared__ uint4 center_s[];
  __half* tile = reinterpret_cast<__half*>(center_s);                        // [c][kCenterPitch]
  bf16* rows_s = reinterpret_cast<bf16*>(tile + c * kCenterPitch);           // [3 terms][64][c + 8]
  const int tiles = (n + 63) / 64, i = blockIdx.x / tiles, k0 = (blockIdx.x % tiles) * 64, pieces = c >> 3;
  for (int u = threadIdx.x; u < c * 8; u += 256) {
    const int h = u >> 3, k = (u & 7) * 8;
    *reinterpret_cast<uint4*>(tile + h * kCenterPitch + k) =
        k0 + k < ld ? *reinterpret_cast<const uint4*>(x + ((int64_t)h * n + i) * ld + k0 + k) : make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, pair = (threadIdx.x >> 5) * 8 + (lane & 7), part = lane >> 3;
  auto over_parts = [](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
  };
  float v[GROUPS][2], s = 0.f, ss = 0.f;
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    const int h = g * 8 + part * 2;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      v[g][e] = g < pieces ? __half2float(tile[(h + e) * kCenterPitch + pair]) * prescale : 0.f;
      s += v[g][e];
      ss = fmaf(v[g][e], v[g][e], ss);
    }
  }
  const float mean = over_parts(s) / c;
  float var;
  if (variance == 2) var = over_parts(ss) / c - mean * mean;
  else {
    float acc = 0.f;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g)
#pragma unroll
      for (int e = 0; e < 2; ++e) { const float d = g < pieces ? v[g][e] - mean : 0.f; acc = fmaf(d, d, acc); }
    var = over_parts(acc) / c;
  }
  float inv = rsqrtf(var + eps);
  inv = inv * (1.5f - 0.5f * (var + eps) * inv * inv);
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    const int h = g * 8 + part * 2;
    if (g < pieces) {
      uint32_t t[3];
      split_pair((v[g][0] - mean) * inv * __ldg(gamma + h) + __ldg(beta + h), (v[g][1] - mean) * inv * __ldg(gamma + h + 1) + __ldg(beta + h + 1), t);
#pragma unroll
      for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(rows_s + (e * 64 + pair) * (c + 8) + h) = t[e];
    }
  }
  __syncthreads();
  for (int u = threadIdx.x; u < 64 * pieces; u += 256) {
    const int r = u / pieces, h = (u % pieces) * 8;
    if (k0 + r >= n) continue;
#pragma unroll
    for (int e = 0; e < 3; ++e)
      *reinterpret_cast<uint4*>(xn + e * term_stride + ((int64_t)i * n + k0 + r) * c + h) = *reinterpret_cast<const uint4*>(rows_s + (e * 64 + r) * (c + 8) + h);
  }
}

// out[dst(r)][c] = (resid ? resid[dst(r)][c] : 0) + proj[r][c] * (factor ? factor[r][c] : 1), four channels a thread
// (ch a multiple of 4); dst(r) follows the transposed-orientation rule of the attention operator.
template <typename TAct>
__global__ void finish4_kernel(const float* __restrict__ proj, const float* __restrict__ factor, const TAct* __restrict__ resid, int64_t count,
                               int ch, int transpose, int batch, int Q, TAct* __restrict__ out) {
  lf_chain();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int c4 = ch >> 2;
  if (idx >= count * c4) return;
  const int64_t r = idx / c4;
  const int c = (int)(idx % c4) * 4;
  int64_t dst = r;
  if (transpose) { const uint32_t u = (uint32_t)r, uq = (uint32_t)Q; dst = (int64_t)(u % uq) * batch + u / uq; }
  float v[4];
  load4(proj + r * ch + c, v);
  if (factor) {
    float g[4];
    load4(factor + r * ch + c, g);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] *= g[e];
  }
  if (resid) {
    float x[4];
    load4(resid + dst * ch + c, x);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] += x[e];
  }
  store4(out + dst * ch + c, v);
}

// ---- AF3 MSA pair-weighted averaging: the weights do not depend on the sequence, so they are made once and the averages
// of all sequences are one GEMM per head ----

// key[t] = max over the sequences of mask[s][t]; one warp per 32 tokens and slice of the sequences, combined in shared memory
__global__ void __launch_bounds__(1024) key_mask_kernel(const float* __restrict__ mask, int sequences, int tokens, float* __restrict__ key) {
  lf_chain();
  __shared__ float part[32][33];
  const int t = blockIdx.x * 32 + threadIdx.x;
  float largest = 0.f;
  if (t < tokens)
    for (int s = threadIdx.y; s < sequences; s += 32) largest = fmaxf(largest, mask[(int64_t)s * tokens + t]);
  part[threadIdx.y][threadIdx.x] = largest;
  __syncthreads();
  if (threadIdx.y == 0 && t < tokens) {
    for (int w = 1; w < 32; ++w) largest = fmaxf(largest, part[w][threadIdx.x]);
    key[t] = largest;
  }
}

// softmax over j of bias[h][i][j] + 1e9 (key[j] - 1) -> terms of its transpose, [3][h][j][ld] with i contiguous
__global__ void __launch_bounds__(256)
average_weights_kernel(const float* __restrict__ bias, const float* __restrict__ key, int n, int ld, bf16* __restrict__ out, int64_t term_stride) {
  lf_chain();
  __shared__ float tile[32][33], top[32], inv[32];
  const int h = blockIdx.y, i0 = blockIdx.x * 32, tx = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float* b = bias + ((int64_t)h * n + i0) * n;
  for (int r = w; r < 32 && i0 + r < n; r += 8) {
    float m = -INFINITY, s = 0.f;
    for (int j = tx; j < n; j += 32) {
      const float v = 1e9f * (key[j] - 1.0f) + b[(int64_t)r * n + j], next = fmaxf(m, v);
      s = s * expf(m - next) + expf(v - next);
      m = next;
    }
    float all = m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) all = fmaxf(all, __shfl_xor_sync(0xffffffffu, all, o));
    s = warp_sum(m == -INFINITY ? 0.f : s * expf(m - all));
    if (tx == 0) { top[r] = all; inv[r] = 1.0f / s; }
  }
  __syncthreads();
  for (int j0 = 0; j0 < n; j0 += 32) {
    for (int r = w; r < 32; r += 8)
      tile[r][tx] = i0 + r < n && j0 + tx < n ? expf(1e9f * (key[j0 + tx] - 1.0f) + b[(int64_t)r * n + j0 + tx] - top[r]) * inv[r] : 0.f;
    __syncthreads();
    const int i2 = (threadIdx.x & 15) * 2;
    for (int jj = threadIdx.x >> 4; jj < 32; jj += 16) {
      if (j0 + jj >= n || i0 + i2 >= ld) continue;
      uint32_t t[3];
      split_pair(tile[i2][jj], tile[i2 + 1][jj], t);
#pragma unroll
      for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(out + e * term_stride + ((int64_t)h * n + j0 + jj) * ld + i0 + i2) = t[e];
    }
    __syncthreads();
  }
}

// values: rows (s, j) of `ld` floats, head h at columns h * d -> terms [3][h][j][lds], element s * d + e; consecutive
// threads take consecutive sequences of one (head, j)
__global__ void average_values_kernel(const float* __restrict__ v, int64_t ld, int S, int n, int heads, int d, int lds, bf16* __restrict__ out,
                                      int64_t term_stride) {
  lf_chain();
  const int s = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, h = blockIdx.z;
  if (s >= S) return;
  const float* src = v + ((int64_t)s * n + j) * ld + h * d;
  bf16* dst = out + ((int64_t)h * n + j) * lds + (int64_t)s * d;
  if ((d & 7) == 0) {
    for (int e = 0; e < d; e += 8) {
      const float4 a = *reinterpret_cast<const float4*>(src + e), b = *reinterpret_cast<const float4*>(src + e + 4);
      uint32_t t[4][3];
      split_pair(a.x, a.y, t[0]);
      split_pair(a.z, a.w, t[1]);
      split_pair(b.x, b.y, t[2]);
      split_pair(b.z, b.w, t[3]);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(dst + i * term_stride + e) = make_uint4(t[0][i], t[1][i], t[2][i], t[3][i]);
    }
  } else {
    for (int e = 0; e < d; ++e) {
      float x = src[e];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const bf16 t = __float2bfloat16_rn(x);
        dst[i * term_stride + e] = t;
        x -= __bfloat162float(t);
      }
    }
  }
}

// o[(s, i)][h * d + e] = x[h][i][s * d + e] * gate[(s, i)][h * d + e] -> terms with rows of ldo
__global__ void average_gate_kernel(const float* __restrict__ x, int64_t ldx, const float* __restrict__ gate, int64_t ldg, int S, int n, int heads,
                                    int d, int ldo, bf16* __restrict__ out, int64_t term_stride) {
  lf_chain();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int l2 = ldo >> 1;
  if (idx >= (int64_t)S * n * l2) return;
  const int64_t r = idx / l2;
  const int s = (int)(r / n), i = (int)(r % n);
  float v[2] = {0.f, 0.f};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int c = (int)(idx % l2) * 2 + e;
    if (c < heads * d) { const int h = c / d; v[e] = x[((int64_t)h * n + i) * ldx + (int64_t)s * d + c % d] * gate[r * ldg + c]; }
  }
  uint32_t t[3];
  split_pair(v[0], v[1], t);
#pragma unroll
  for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(out + e * term_stride + r * ldo + (idx % l2) * 2) = t[e];
}

// ---- global column attention (extra-MSA stack): one key and value head, a query per column ----

// Per column: the masked sums over the sequences of the standardised rows and of the mask (c <= 512).  Sixteen warps share a
// column's sequences; a row is read once.  1024 x 256, 64 channels: 230 us with
// a thread per channel adding up the sequences one after the other, after a LayerNorm pass of its own.
template <typename T>
__global__ void __launch_bounds__(512)
global_mean_kernel(const T* __restrict__ act, const float* __restrict__ mask, int S, int n, int c, float eps, int variance, float* __restrict__ sums) {
  lf_chain();
  extern __shared__ float part[];      // [16 warps][c + 1]
  const int col = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float acc[16], count = 0.f;          // channels lane, lane + 32, ... (c <= 512)
#pragma unroll
  for (int k = 0; k < 16; ++k) acc[k] = 0.f;
  for (int s = w; s < S; s += 16) {
    const float m = mask[(int64_t)s * n + col];
    count += m;
    if (m == 0.f) continue;
    const T* x = act + ((int64_t)s * n + col) * c;
    float v[16], sum = 0.f, sq = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int ch = k * 32 + lane;
      v[k] = ch < c ? to_f(x[ch]) : 0.f;
      sum += v[k];
      if (k * 32 + 32 >= c) break;
    }
    const float mean = warp_sum(sum) / c;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const float d = k * 32 + lane < c ? (variance == 2 ? v[k] : v[k] - mean) : 0.f;
      sq = fmaf(d, d, sq);
      if (k * 32 + 32 >= c) break;
    }
    const float var = warp_sum(sq) / c - (variance == 2 ? mean * mean : 0.f);
    float inv = rsqrtf(var + eps);
    inv = inv * (1.5f - 0.5f * (var + eps) * inv * inv);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      acc[k] = fmaf((v[k] - mean) * inv, m, acc[k]);
      if (k * 32 + 32 >= c) break;
    }
  }
#pragma unroll
  for (int k = 0; k < 16; ++k)
    if (k * 32 + lane < c) part[w * (c + 1) + k * 32 + lane] = acc[k];
  if (lane == 0) part[w * (c + 1) + c] = count;
  __syncthreads();
  for (int ch = threadIdx.x; ch <= c; ch += 512) {
    float total = 0.f;
    for (int k = 0; k < 16; ++k) total += part[k * (c + 1) + ch];
    sums[(int64_t)col * (c + 1) + ch] = total;
  }
}

// ... of rows of 4 * NV * L channels: L lanes a row, four rows of each lane group in flight
template <typename T, int NV, int L>
__global__ void __launch_bounds__(512)
global_mean_rows_kernel(const T* __restrict__ act, const float* __restrict__ mask, int S, int n, float eps, int variance, float* __restrict__ sums) {
  lf_chain();
  constexpr int CH = 4 * NV * L, GROUPS = 512 / L;
  __shared__ float part[GROUPS][CH + 1];
  const int col = blockIdx.x, l = threadIdx.x % L, g = threadIdx.x / L;
  float acc[NV][4], count = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[k][e] = 0.f;
  for (int base = 0; base < S; base += 4 * GROUPS) {      // (the same trips for both row groups of a warp: they share its shuffles)
    const int s0 = base + g;
    float v[4][NV][4], m[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int s = s0 + r * GROUPS;
      m[r] = s < S ? __ldg(mask + (int64_t)s * n + col) : 0.f;
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        if (s < S) load4(act + ((int64_t)s * n + col) * CH + (k * L + l) * 4, v[r][k]);
        else v[r][k][0] = v[r][k][1] = v[r][k][2] = v[r][k][3] = 0.f;
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float sum = 0.f, sq = 0.f;
#pragma unroll
      for (int k = 0; k < NV; ++k) sum += (v[r][k][0] + v[r][k][1]) + (v[r][k][2] + v[r][k][3]);
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      const float mean = sum * (1.0f / CH);
#pragma unroll
      for (int k = 0; k < NV; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float d = variance == 2 ? v[r][k][e] : v[r][k][e] - mean; sq = fmaf(d, d, sq); }
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      const float var = variance == 2 ? sq * (1.0f / CH) - mean * mean : sq * (1.0f / CH);
      float inv = rsqrtf(var + eps);
      inv = inv * (1.5f - 0.5f * (var + eps) * inv * inv) * m[r];
      count += m[r];
#pragma unroll
      for (int k = 0; k < NV; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[k][e] = fmaf(v[r][k][e] - mean, inv, acc[k][e]);
    }
  }
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) part[g][(k * L + l) * 4 + e] = acc[k][e];
  if (l == 0) part[g][CH] = count;
  __syncthreads();
  for (int ch = threadIdx.x; ch <= CH; ch += 512) {
    float total = 0.f;
#pragma unroll
    for (int k = 0; k < GROUPS; ++k) total += part[k][ch];
    sums[(int64_t)col * (CH + 1) + ch] = total;
  }
}

// ... of rows wider than that, from their normalised terms (gain and offset applied)
__global__ void __launch_bounds__(512)
global_mean_terms_kernel(const bf16* __restrict__ nrm, int64_t ld, int64_t term_stride, const float* __restrict__ mask, int S, int n, int c,
                         float* __restrict__ sums) {
  lf_chain();
  const int col = blockIdx.x;
  for (int ch = threadIdx.x; ch <= c; ch += 512) {
    float total = 0.f;
    for (int s = 0; s < S; ++s) {
      const bf16* x = nrm + ((int64_t)s * n + col) * ld + (ch < c ? ch : 0);
      const float v = ch < c ? to_f(x[0]) + to_f(x[term_stride]) + to_f(x[2 * term_stride]) : 1.f;
      total = fmaf(v, mask[(int64_t)s * n + col], total);
    }
    sums[(int64_t)col * (c + 1) + ch] = total;
  }
}

// q[col][slot] = scale * sum_ch mean[ch] wq[ch][slot], mean = (gamma sum + beta count) / (1e-10 + count), or sum / (1e-10 + count) without gamma
__global__ void global_query_kernel(const float* __restrict__ sums, const float* __restrict__ gamma, const float* __restrict__ beta, int c, int HD,
                                    float scale, const float* __restrict__ wq, float* __restrict__ q) {
  lf_chain();
  extern __shared__ float means[];
  const int col = blockIdx.x;
  const float count = sums[(int64_t)col * (c + 1) + c], denominator = 1e-10f + count;
  for (int ch = threadIdx.x; ch < c; ch += blockDim.x) {
    const float sum = sums[(int64_t)col * (c + 1) + ch];
    means[ch] = (gamma ? gamma[ch] * sum + beta[ch] * count : sum) / denominator;
  }
  __syncthreads();
  for (int slot = threadIdx.x; slot < HD; slot += blockDim.x) {
    float r = 0.f;
    for (int ch = 0; ch < c; ++ch) r = fmaf(means[ch], wq[(int64_t)ch * HD + slot], r);
    q[(int64_t)col * HD + slot] = r * scale;
  }
}

// Softmax over the sequences of q(column, head) . k(sequence, column), masked sequences at -1e9, applied to the values; k at
// columns 0 .. d - 1 and v at d .. 2d - 1 of rows of `ld` floats (a multiple of 4), d <= D.  One block per column and HB heads: a key and
// value row is read once for all of them, in 16-byte loads where d is whole groups of four; a thread keeps an online
// softmax of its sequences, the block combines them by shuffles.
template <int D, int HB>
__global__ void __launch_bounds__(256)
global_attend_kernel(const float* __restrict__ q, const float* __restrict__ kv, int64_t ld, const float* __restrict__ mask, int S, int n, int heads,
                     int d, float* __restrict__ attended) {
  lf_chain();
  __shared__ float part[8][HB][D + 2], q_s[HB][D];
  const int col = blockIdx.x, h0 = blockIdx.y * HB, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int u = threadIdx.x; u < HB * D; u += 256) {
    const int h = u / D, e = u % D;
    q_s[h][e] = e < d && h0 + h < heads ? q[((int64_t)col * heads + h0 + h) * d + e] : 0.f;
  }
  __syncthreads();
  float acc[HB][D], top[HB], den[HB];
#pragma unroll
  for (int h = 0; h < HB; ++h) {
    top[h] = -1e30f;
    den[h] = 0.f;
#pragma unroll
    for (int e = 0; e < D; ++e) acc[h][e] = 0.f;
  }
  const bool vec = (d & 3) == 0;
  for (int s = threadIdx.x; s < S; s += 256) {
    const float* row = kv + ((int64_t)s * n + col) * ld;
    float k[D], v[D];
    if (vec) {
#pragma unroll
      for (int e = 0; e < D; e += 4) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (e < d) { a = *reinterpret_cast<const float4*>(row + e); b = *reinterpret_cast<const float4*>(row + d + e); }
        k[e] = a.x; k[e + 1] = a.y; k[e + 2] = a.z; k[e + 3] = a.w;
        v[e] = b.x; v[e + 1] = b.y; v[e + 2] = b.z; v[e + 3] = b.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < D; ++e) { k[e] = e < d ? row[e] : 0.f; v[e] = e < d ? row[d + e] : 0.f; }
    }
    const bool masked = mask[(int64_t)s * n + col] == 0.f;
#pragma unroll
    for (int h = 0; h < HB; ++h) {
      float logit = 0.f;
#pragma unroll
      for (int e = 0; e < D; ++e) logit = fmaf(q_s[h][e], k[e], logit);
      if (masked) logit = -1e9f;
      const float next = fmaxf(top[h], logit), keep = __expf(top[h] - next), weight = __expf(logit - next);
      top[h] = next;
      den[h] = den[h] * keep + weight;
#pragma unroll
      for (int e = 0; e < D; ++e) acc[h][e] = fmaf(acc[h][e], keep, weight * v[e]);
    }
  }
#pragma unroll
  for (int h = 0; h < HB; ++h) {
    const float all = simt::warp_max(top[h]), keep = __expf(top[h] - all);
    const float total = warp_sum(den[h] * keep);
    if (lane == 0) { part[w][h][D] = all; part[w][h][D + 1] = total; }
#pragma unroll
    for (int e = 0; e < D; ++e) {
      const float x = warp_sum(acc[h][e] * keep);
      if (lane == 0) part[w][h][e] = x;
    }
  }
  __syncthreads();
  for (int u = threadIdx.x; u < HB * d; u += 256) {
    const int h = u / d, e = u % d;
    if (h0 + h >= heads) continue;
    float all = -1e30f, total = 0.f, num = 0.f;
    for (int k = 0; k < 8; ++k) all = fmaxf(all, part[k][h][D]);
    for (int k = 0; k < 8; ++k) {
      const float keep = __expf(part[k][h][D] - all);
      total += part[k][h][D + 1] * keep;
      num += part[k][h][e] * keep;
    }
    attended[((int64_t)col * heads + h0 + h) * d + e] = num / total;
  }
}

// gate[(s, col)][slot] (columns gate0.. of rows of `ld`) * attended[col][slot] -> terms with rows of ldo (a multiple of 8); `per` blocks a sequence
__global__ void global_gate_kernel(const float* __restrict__ kvg, int64_t ld, int gate0, const float* __restrict__ attended, int per, int n, int HD, int ldo,
                                   bf16* __restrict__ out, int64_t term_stride) {
  lf_chain();
  const uint32_t idx = blockIdx.x % per * blockDim.x + threadIdx.x, l4 = (uint32_t)ldo >> 2;
  if (idx >= (uint32_t)n * l4) return;
  const uint32_t col = idx / l4, c = idx % l4 * 4;
  const int64_t r = (int64_t)(blockIdx.x / per) * n + col;
  const float* g = kvg + r * ld + gate0 + c;
  const float* x = attended + (int64_t)col * HD + c;
  float v[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] = (int)c + e < HD ? g[e] * x[e] : 0.f;
  store_terms4(out + r * ldo + c, term_stride, v);
}

// The attention core reads keys and bias columns up to a whole group of 16 and masks what is past Q: it only has to be finite.  Zeros in
// rows Q .. ldq - 1 of k and v (8 x 8 pieces, [batch][ldq][128] each; or null) and columns Q .. ldq - 1 of the bias [heads * Q][ldq] (or null).
// Only the padding is written: clearing the whole tensors took 90 us at 701 x 701 pairs.
__global__ void attention_padding_kernel(uint16_t* __restrict__ k, uint16_t* __restrict__ v, uint16_t* __restrict__ bias, int batch, int heads, int Q, int ldq) {
  lf_chain();
  const int pad = ldq - Q;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k && idx < (int64_t)batch * pad * 16) {
    const int piece = (int)(idx & 15), row = Q + (int)((idx >> 4) % pad);
    const int64_t at = (idx >> 4) / pad * ldq * 128 + (int64_t)(row >> 3) * 1024 + piece * 64 + (row & 7) * 8;
    *reinterpret_cast<uint4*>(k + at) = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(v + at) = make_uint4(0u, 0u, 0u, 0u);
  }
  if (bias && idx < (int64_t)heads * Q * pad) bias[idx / pad * ldq + Q + idx % pad] = 0;
}

}  // namespace rows
