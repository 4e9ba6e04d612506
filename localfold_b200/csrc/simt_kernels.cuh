// Kernels on the FMA pipe: LayerNorm, residuals and pair bias for widths and addresses that the vectorised row kernels do not take,
// the float32 outer product mean, the distogram's GEMM, int5 decode, and glue of the fp16 GEMMs.  Accumulation in float32,
// statistics by warp shuffles.
#pragma once

#include "common.cuh"

namespace simt {

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(bf16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float sigmoidf_(float v) { return 1.0f / (1.0f + expf(-v)); }

// o[0..7] = v[0..7] (+ r[0..7] when r is given): 16-byte accesses for float32 activations
template <typename TAct>
__device__ __forceinline__ void add_store8(float (&v)[8], const TAct* r, TAct* o) {
  if (sizeof(TAct) == 4) {
    if (r) {
      const float4 r0 = *reinterpret_cast<const float4*>(r), r1 = *reinterpret_cast<const float4*>(r + 4);
      v[0] += r0.x; v[1] += r0.y; v[2] += r0.z; v[3] += r0.w;
      v[4] += r1.x; v[5] += r1.y; v[6] += r1.z; v[7] += r1.w;
    }
    *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    if (r) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] += to_f(r[e]);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = from_f<TAct>(v[e]);
  }
}

// ---------------------------------------------------------------------------
// LayerNorm over the last axis, one warp per row.  `rows` logical rows; logical
// row r = b*Q + i reads memory row i*batch + b when `transpose` (batch, Q > 0).
// variance: 1 two-pass, 2 fast (E[x^2]-E[x]^2, unclamped).
// PAD16: the output rows are ch + 16 long, a one and fifteen zeros after the channels (the k column through which a
// GEMM that follows adds its bias)
template <typename TIn, typename TOut = float, bool PAD16 = false>
__global__ void layer_norm_kernel(const TIn* __restrict__ in, int64_t rows, int ch,
                                  const float* __restrict__ gamma, const float* __restrict__ beta,
                                  float eps, int variance, int transpose, int batch, int Q,
                                  TOut* __restrict__ out) {
  lf_chain();
  int lane = threadIdx.x & 31;
  int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  int64_t src = row;
  if (transpose) { int64_t b = row / Q, i = row % Q; src = i * batch + b; }
  const TIn* x = in + src * ch;
  float s = 0.f, ss = 0.f;
  for (int c = lane; c < ch; c += 32) { float v = to_f(x[c]); s += v; ss += v * v; }
  s = warp_sum(s);
  float mean = s / ch, var;
  if (variance == 2) {
    ss = warp_sum(ss);
    var = ss / ch - mean * mean;
  } else {
    float acc = 0.f;
    for (int c = lane; c < ch; c += 32) { float d = to_f(x[c]) - mean; acc += d * d; }
    var = warp_sum(acc) / ch;
  }
  float inv = rsqrtf(var + eps);
  // one Newton step: rsqrtf is 2 ulp, the parity bar is tighter than that squared error allows
  inv = inv * (1.5f - 0.5f * (var + eps) * inv * inv);
  TOut* y = out + row * (PAD16 ? ch + 16 : ch);
  for (int c = lane; c < ch; c += 32) y[c] = from_f<TOut>((to_f(x[c]) - mean) * inv * gamma[c] + beta[c]);
  if (PAD16 && lane < 16) y[ch + lane] = from_f<TOut>(lane == 0 ? 1.f : 0.f);
}

// ---------------------------------------------------------------------------
// Tiled SGEMM:  C[m][n] = sum_k A(m,k) B[k*ldb + n] + bias[n],  A(m,k) = TA ? A[k*lda + m] : A[m*lda + k]
// 64x64x16 tile, 256 threads, 4x4 micro-tile, every load and store bounds-checked.
template <bool TA>
__global__ void __launch_bounds__(256)
sgemm_kernel(int M, int N, int K, const float* __restrict__ A, int64_t lda, const float* __restrict__ B, int64_t ldb, float* __restrict__ C,
             int64_t ldc, const float* __restrict__ bias) {
  lf_chain();
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ float As[BK][BM + 4];
  __shared__ float Bs[BK][BN + 4];
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int t = threadIdx.x;
  const int tx = t & 15, ty = t >> 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      int idx = t + 256 * r;
      int m, k;
      if (TA) { m = idx & 63; k = idx >> 6; } else { k = idx & 15; m = idx >> 4; }
      int gm = m0 + m, gk = k0 + k;
      float v = 0.f;
      if (gm < M && gk < K) v = TA ? A[(int64_t)gk * lda + gm] : A[(int64_t)gm * lda + gk];
      As[k][m] = v;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      int idx = t + 256 * r;
      int n = idx & 63, k = idx >> 6;
      int gn = n0 + n, gk = k0 + k;
      Bs[k][n] = gn < N && gk < K ? B[(int64_t)gk * ldb + gn] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + tx * 4 + j;
      if (gn < N) C[(int64_t)gm * ldc + gn] = acc[i][j] + (bias ? bias[gn] : 0.f);
    }
  }
}

// ---------------------------------------------------------------------------
// out[dst(r)][c] = (resid ? resid[dst(r)][c] : 0) + proj[r][c] * (factor ? factor[r][c] : 1)
// dst(r) follows the transposed-orientation rule of the attention operator.
template <typename TAct>
__global__ void finish_kernel(const float* __restrict__ proj, const float* __restrict__ factor,
                              const TAct* __restrict__ resid, int64_t rows, int ch, int transpose,
                              int batch, int Q, TAct* __restrict__ out) {
  lf_chain();
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t total = rows * ch;
  if (idx >= total) return;
  int64_t r = idx / ch;
  int c = (int)(idx % ch);
  int64_t dst = r;
  if (transpose) { int64_t b = r / Q, i = r % Q; dst = i * batch + b; }
  float v = proj[idx];
  if (factor) v *= factor[idx];
  if (resid) v += to_f(resid[dst * ch + c]);
  out[dst * ch + c] = from_f<TAct>(v);
}

// ---------------------------------------------------------------------------
// Pair bias: out[h][i][j] = LN(pair[p,:]) . W[:,h] for p = i*Q + j, [h][j][i] if swap; rows of ldo.
// One warp per pair row.
template <typename TIn>
__global__ void pair_bias_kernel(const TIn* __restrict__ pair, int Q, int ch, int heads,
                                 const float* __restrict__ gamma, const float* __restrict__ beta,
                                 const float* __restrict__ w, float eps, int variance, int swap,
                                 float* __restrict__ out, int ldo) {
  lf_chain();
  int lane = threadIdx.x & 31;
  int64_t pairs = (int64_t)Q * Q;
  int64_t p = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (p >= pairs) return;
  const TIn* x = pair + p * ch;
  float s = 0.f, ss = 0.f;
  for (int c = lane; c < ch; c += 32) { float v = to_f(x[c]); s += v; ss += v * v; }
  s = warp_sum(s);
  const float mean = s / ch;
  float var;
  if (variance == 2) { ss = warp_sum(ss); var = ss / ch - mean * mean; }
  else {
    float acc = 0.f;
    for (int c = lane; c < ch; c += 32) { float d = to_f(x[c]) - mean; acc += d * d; }
    var = warp_sum(acc) / ch;
  }
  float inv = rsqrtf(var + eps);
  inv = inv * (1.5f - 0.5f * (var + eps) * inv * inv);
  const int64_t i = p / Q, j = p % Q, dst = swap ? j * ldo + i : i * ldo + j;
  for (int h = 0; h < heads; ++h) {
    float acc = 0.f;
    for (int c = lane; c < ch; c += 32) {
      acc = fmaf((to_f(x[c]) - mean) * inv * gamma[c] + beta[c], w[c * heads + h], acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) out[(int64_t)h * Q * ldo + dst] = acc;
  }
}

// Glue of the 16-bit GEMM path.
// out[dst(r)][c] = (resid ? resid[dst(r)][c] : 0) + (proj[r][c] * scale + bias[c]) for an fp16 projection;
// eight channels per thread (ch a multiple of 8)
template <typename TAct>
__global__ void finish_half_kernel(const __half* __restrict__ proj, float scale, const float* __restrict__ bias,
                                   const TAct* __restrict__ resid, int64_t rows, int ch, int transpose,
                                   int batch, int Q, TAct* __restrict__ out) {
  lf_chain();
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int c8 = ch >> 3;
  if (idx >= rows * c8) return;
  int64_t r = idx / c8;
  int c = (int)(idx % c8) * 8;
  int64_t dst = r;
  if (transpose) { int64_t b = r / Q, i = r % Q; dst = i * batch + b; }
  const uint4 raw = *reinterpret_cast<const uint4*>(proj + r * ch + c);
  const __half* h = reinterpret_cast<const __half*>(&raw);
  float v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = __half2float(h[e]) * scale + (bias ? bias[c + e] : 0.f);
  const TAct* rs = resid ? resid + dst * ch + c : nullptr;
  TAct* o = out + dst * ch + c;
  add_store8<TAct>(v, rs, o);
}

// fp16 pair bias [heads][Q][ld] (rows padded to ld) -> float32 [heads][Q][ldo]
__global__ void widen_bias_kernel(const __half* __restrict__ in, int heads, int Q, int ld, float* __restrict__ out, int ldo) {
  lf_chain();
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t total = (int64_t)heads * Q * Q;
  if (idx >= total) return;
  int k = (int)(idx % Q);
  int64_t hq = idx / Q;
  out[hq * ldo + k] = __half2float(in[hq * ld + k]);
}

// out[i][j][b] = half[i][j][b] + half[j][i][b]: a sum over the two token orders, not a mean.
__global__ void symmetrise_sum_kernel(const float* __restrict__ half, int tokens, int bins, float* __restrict__ out) {
  lf_chain();
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t total = (int64_t)tokens * tokens * bins;
  if (idx >= total) return;
  int b = (int)(idx % bins);
  int64_t p = idx / bins;
  int i = (int)(p / tokens), j = (int)(p % tokens);
  out[idx] = half[idx] + half[((int64_t)j * tokens + i) * bins + b];
}

// ---------------------------------------------------------------------------
// Outer product mean glue.
// rows [S*N][c] times their mask values, into fp16 copies (operands of the tensor-core outer product)
__global__ void mask_rows_half_kernel(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ mask,
                                      int64_t rows, int c, __half* __restrict__ a16, __half* __restrict__ b16) {
  lf_chain();
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * c) return;
  float m = mask[idx / c];
  a16[idx] = __float2half_rn(a[idx] * m);
  b16[idx] = __float2half_rn(b[idx] * m);
}

// the fp16 projection lr [rows][2c] (left | right) + biases, masked, into the outer product's operands
__global__ void opm_split_half_kernel(const __half* __restrict__ lr, const float* __restrict__ bl, const float* __restrict__ br,
                                      const float* __restrict__ mask, int64_t rows, int c, __half* __restrict__ a16,
                                      __half* __restrict__ b16) {
  lf_chain();
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * c) return;
  int64_t r = idx / c;
  int a = (int)(idx % c);
  float m = mask[r];
  a16[idx] = __float2half_rn((__half2float(lr[r * 2 * c + a]) + bl[a]) * m);
  b16[idx] = __float2half_rn((__half2float(lr[r * 2 * c + c + a]) + br[a]) * m);
}

// out[i][j][z] = (proj[(i - i0) N + j][z] * scale + bout[z]) / (eps + counts[i][j]) (+ resid), or with the bias after
// the division by max(count, 1); fp16 projection
template <typename TAct>
__global__ void opm_finish_half_kernel(const __half* __restrict__ proj, float scale, const float* __restrict__ bout,
                                       const float* __restrict__ counts, int N, int cz, int i0, int cnt, float norm_eps,
                                       int bias_after_norm, const TAct* __restrict__ resid, TAct* __restrict__ out) {
  lf_chain();
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;      // eight channels per thread (cz a multiple of 8)
  const int z8 = cz >> 3;
  if (idx >= (int64_t)cnt * N * z8) return;
  const int z = (int)(idx % z8) * 8;
  const int64_t pr = idx / z8;                 // (i - i0) * N + j
  const int64_t pair = (int64_t)i0 * N + pr;
  const uint4 raw = *reinterpret_cast<const uint4*>(proj + pr * cz + z);
  const __half* h = reinterpret_cast<const __half*>(&raw);
  const float count = counts[pair];
  const float inv = bias_after_norm ? 1.0f / fmaxf(count, 1.0f) : 1.0f / (norm_eps + count);
  float v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float t = __half2float(h[e]) * scale;
    v[e] = bias_after_norm ? t * inv + bout[z + e] : (t + bout[z + e]) * inv;
  }
  const int64_t o = pair * cz + z;
  add_store8<TAct>(v, resid ? resid + o : nullptr, out + o);
}

// ... in place
__global__ void mask_rows_kernel(float* __restrict__ a, float* __restrict__ b, const float* __restrict__ mask,
                                 int64_t rows, int c) {
  lf_chain();
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * c) return;
  float m = mask[idx / c];
  a[idx] *= m;
  b[idx] *= m;
}

// outer: [(i - i0)*c + a][j*c + b] for i in [i0, i0+ni); out[i][j][z] =
// (sum_ab outer * wout[(a*c+b)][z] + bout[z]) / (eps + count(i,j)), + resid.
// One block per (i, group of JT columns j); thread z loops over the c*c products.
// (TOuter: float32 sums, or the tensor-core contraction's fp16 sums scaled by 1 / outer_scale)
template <typename TAct, int JT, typename TOuter>
__global__ void opm_output_kernel(const TOuter* __restrict__ outer, float outer_scale, const float* __restrict__ wout,
                                  const float* __restrict__ bout, const float* __restrict__ mask,
                                  int S, int N, int c, int cz, int i0, float norm_eps,
                                  int bias_after_norm, const TAct* __restrict__ resid,
                                  TAct* __restrict__ out) {
  lf_chain();
  extern __shared__ float sm[];     // [JT][c*c] + counts[JT]
  const int cc = c * c;
  float* tile = sm;
  float* counts = sm + JT * cc;
  const int i = i0 + blockIdx.y;
  const int j0 = blockIdx.x * JT;
  const int64_t ldo = (int64_t)N * c;
  for (int idx = threadIdx.x; idx < JT * cc; idx += blockDim.x) {
    int jj = idx / cc, ab = idx % cc, a = ab / c, b2 = ab % c;
    int j = j0 + jj;
    tile[idx] = j < N ? to_f(outer[((int64_t)(i - i0) * c + a) * ldo + (int64_t)j * c + b2]) * outer_scale : 0.f;
  }
  if (threadIdx.x < JT) {
    int j = j0 + threadIdx.x;
    float cnt = 0.f;
    if (j < N) for (int s = 0; s < S; ++s) cnt += mask[(int64_t)s * N + i] * mask[(int64_t)s * N + j];
    counts[threadIdx.x] = cnt;
  }
  __syncthreads();
  for (int z = threadIdx.x; z < cz; z += blockDim.x) {
    float acc[JT];
#pragma unroll
    for (int jj = 0; jj < JT; ++jj) acc[jj] = 0.f;
    for (int ab = 0; ab < cc; ++ab) {
      float wv = wout[(int64_t)ab * cz + z];
#pragma unroll
      for (int jj = 0; jj < JT; ++jj) acc[jj] = fmaf(tile[jj * cc + ab], wv, acc[jj]);
    }
#pragma unroll
    for (int jj = 0; jj < JT; ++jj) {
      int j = j0 + jj;
      if (j >= N) continue;
      float v;
      if (bias_after_norm) v = acc[jj] / fmaxf(counts[jj], 1.0f) + bout[z];
      else v = (acc[jj] + bout[z]) / (norm_eps + counts[jj]);
      int64_t o = ((int64_t)i * N + j) * cz + z;
      if (resid) v += to_f(resid[o]);
      out[o] = from_f<TAct>(v);
    }
  }
}

// int5 decode: one thread per value.  value = code*scale + zero.
__global__ void int5_decode_kernel(const uint8_t* __restrict__ codes, const __half* __restrict__ scales,
                                   const __half* __restrict__ zeros, int64_t elements, int block,
                                   float* __restrict__ out) {
  lf_chain();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= elements) return;
  int64_t g = i / block;
  int within = (int)(i % block);
  int bit = within * 5;
  const uint8_t* base = codes + g * (block * 5 / 8);
  unsigned two = base[bit >> 3] | ((unsigned)base[(bit >> 3) + 1] << 8);
  unsigned code = (two >> (bit & 7)) & 31u;
  out[i] = fmaf((float)code, __half2float(scales[g]), __half2float(zeros[g]));
}

}  // namespace simt
