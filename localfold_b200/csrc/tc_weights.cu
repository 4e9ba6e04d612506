// Tensor-core operands of an operator's weights: swizzled fp16 images, folded LayerNorm vectors and plain GEMM operands,
// derived on the device from the canonical float32 arrays.
#include "tc_kernels.cuh"

namespace tc {

namespace {

// One derived array.  All of an operator's jobs run in one launch (blockIdx.y = job): preparing a stack is bound by its
// launches and allocations, not by the few hundred KiB a job moves.  An AF3 pairformer block at 128 / 384 channels
// took 4.2 ms with a launch, and often an allocation, per array.
enum JobKind {
  JOB_IMAGE,      // W (in, out) [K][ld], columns col0 .. col0 + n_out -> fp16 image of W^T in the swizzled K-major layout ([K / 64][n_pad rows][128 B]) at row0
  JOB_OPERAND,    // ... -> fp16 [n_out][K] (the plain GEMM wants k contiguous in both operands)
  JOB_BIASED,     // ... -> fp16 [n_out][K + 16], bias in k column K and zeros after it (the activations carry a column of ones there)
  JOB_FOLD,       // float [n_out]: scale * (bias[c] + sum_k vec[k] W[k][col0 + c]): a LayerNorm offset folded into a bias
  JOB_TERMS,      // ... -> three bf16 terms [3][rows][n_pad] at row0, zeros past K (n_pad = K rounded up to 8)
  JOB_GATED,      // the fused triangle projection (four roles of n_out columns) as terms [3][n_fill][n_pad], rows as Gemm3Out's planes want them
  JOB_HEADS,      // the fused attention projection as terms, every head of d channels (row0) padded with zero rows to D (n_pad)
  JOB_HEADS_BIAS, // ... its bias vector, as float32
  JOB_HEADS_OUT,  // the output projection as terms, the k of every head padded likewise
  JOB_COLSUM      // float [n_out]: sum_k fp16(vec[k] W[k][col0 + c]): what the tensor core multiplies the mean by
};
struct Job {
  const float* w;
  const float* vec;      // IMAGE: gain of the LayerNorm before the projection, folded into the rows (may be null); FOLD, COLSUM: see above
  const float* bias;     // may be null
  void* out;
  float scale;
  int kind, K, ld, col0, n_out, n_fill, n_pad, row0;      // columns n_out .. n_fill - 1 are written as zeros
  int64_t term_stride;
};
constexpr int kMaxJobs = 26;      // 2.1 KiB of kernel parameters
struct JobList { Job j[kMaxJobs]; int count; };

__global__ void __launch_bounds__(256) weight_jobs_kernel(const __grid_constant__ JobList list) {
  const Job& j = list.j[blockIdx.y];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j.kind == JOB_FOLD || j.kind == JOB_COLSUM) {
    // a warp per column, its lanes along k: a thread per column is a serial chain of K loads and float64 additions (10 us)
    const int lane = threadIdx.x & 31;
    for (int64_t c = first >> 5; c < j.n_fill; c += stride >> 5) {
      double acc = 0.0;
      if (c < j.n_out)
        for (int k = lane; k < j.K; k += 32) {
          const float w = j.w[(int64_t)k * j.ld + j.col0 + c];
          acc += j.kind == JOB_FOLD ? (double)j.vec[k] * (double)w : (double)__half2float(__float2half_rn(j.vec[k] * w));
        }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) {
        if (j.bias && c < j.n_out) acc += (double)j.bias[c];
        reinterpret_cast<float*>(j.out)[c] = (float)(acc * j.scale);
      }
    }
    return;
  }
  const int d = j.row0, D = j.n_pad;      // of the head forms
  if (j.kind == JOB_HEADS_BIAS) {
    for (int64_t n = first; n < j.n_fill; n += stride)
      reinterpret_cast<float*>(j.out)[n] = n % D < d && n / D * d + n % D < j.n_out ? j.w[n / D * d + n % D] : 0.f;
    return;
  }
  if (j.kind == JOB_GATED) {
    for (int64_t i = first; i < (int64_t)j.n_pad * j.n_fill; i += stride) {
      const int k = (int)(i / j.n_fill), n = (int)(i % j.n_fill), half = j.n_fill / 2, which = n / half, in = n % half, h = in / 32 * 16 + in % 16;
      float v = k < j.K && h < j.n_out ? j.w[(int64_t)k * j.ld + (which * 2 + in % 32 / 16) * j.n_out + h] : 0.f;
      bf16* t = reinterpret_cast<bf16*>(j.out) + (int64_t)n * j.n_pad + k;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const bf16 b = __float2bfloat16_rn(v);
        t[e * j.term_stride] = b;
        v -= __bfloat162float(b);
      }
    }
    return;
  }
  if (j.kind == JOB_HEADS || j.kind == JOB_HEADS_OUT) {
    // [n_fill][ld8(K)] (heads along n) or [n_out][n_fill] (heads along k)
    const bool out_proj = j.kind == JOB_HEADS_OUT;
    const int kk = out_proj ? j.n_fill : (j.K + 7) / 8 * 8, nn = out_proj ? j.n_out : j.n_fill;
    for (int64_t i = first; i < (int64_t)kk * nn; i += stride) {
      const int k = (int)(i / nn), n = (int)(i % nn);
      float v = 0.f;
      if (out_proj) { if (k % D < d) v = j.w[(int64_t)(k / D * d + k % D) * j.ld + n]; }
      else if (k < j.K && n % D < d) v = j.w[(int64_t)k * j.ld + n / D * d + n % D];
      bf16* t = reinterpret_cast<bf16*>(j.out) + (int64_t)n * kk + k;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const bf16 b = __float2bfloat16_rn(v);
        t[e * j.term_stride] = b;
        v -= __bfloat162float(b);
      }
    }
    return;
  }
  // consecutive threads take consecutive columns of a row of W, so that the reads coalesce
  const int K2 = j.kind == JOB_BIASED ? j.K + 16 : j.kind == JOB_TERMS ? j.n_pad : j.K;
  op16* out = reinterpret_cast<op16*>(j.out);
  for (int64_t i = first; i < (int64_t)K2 * j.n_fill; i += stride) {
    const int k = (int)(i / j.n_fill), n = (int)(i % j.n_fill);
    float v = 0.f;
    if (n < j.n_out) v = k < j.K ? j.w[(int64_t)k * j.ld + j.col0 + n] : k == j.K && j.kind == JOB_BIASED ? j.bias[n] : 0.f;
    if (j.kind == JOB_TERMS) {
      bf16* t = reinterpret_cast<bf16*>(j.out) + (int64_t)(j.row0 + n) * K2 + k;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const bf16 b = __float2bfloat16_rn(v);
        t[e * j.term_stride] = b;
        v -= __bfloat162float(b);
      }
      continue;
    }
    if (j.kind == JOB_IMAGE) {
      v = v * j.scale * (j.vec ? j.vec[k] : 1.0f);
      const int row = j.row0 + n;
      const size_t off = (size_t)(k >> 6) * ((size_t)j.n_pad * 128) + (size_t)row * 128 + ((((k & 63) >> 3) ^ (row & 7)) << 4) + (k & 7) * 2;
      out[off / 2] = __float2half_rn(v);
    } else {
      out[(int64_t)n * K2 + k] = __float2half_rn(v);
    }
  }
}

struct Preparer {
  lf_context* ctx;
  bool dry;
  JobList list{};
  int64_t most = 0;      // elements of the largest job
  void push(const Job& j) {
    if (dry) return;
    list.j[list.count++] = j;
    const int64_t elements = (int64_t)(j.K ? j.K : 1) * j.n_fill;
    if (elements > most) most = elements;
    if (list.count == kMaxJobs) flush();
  }
  void image(const float* w, int K, int n_out, int n_pad, int col0, int ld, op16* img, int row0, float scale, const float* gain = nullptr, int n_fill = 0) {
    push(Job{w, gain, nullptr, img, scale, JOB_IMAGE, K, ld, col0, n_out, n_fill ? n_fill : n_out, n_pad, row0});
  }
  void operand(const float* w, int K, int ld, int n_out, op16* out) {
    push(Job{w, nullptr, nullptr, out, 1.0f, JOB_OPERAND, K, ld, 0, n_out, n_out, 0, 0});
  }
  void fold(const float* w, int K, int n_out, int col0, int ld, const float* offset, const float* bias, float scale, float* out, int n_fill = 0) {
    push(Job{w, offset, bias, out, scale, JOB_FOLD, K, ld, col0, n_out, n_fill ? n_fill : n_out, 0, 0});
  }
  void flush() {
    if (dry || list.count == 0) return;
    // eight elements a thread of the largest job
    const int blocks = most / 2048 < 16 ? 16 : most / 2048 > 592 ? 592 : (int)(most / 2048);
    weight_jobs_kernel<<<dim3(blocks, list.count), 256, 0, ctx->stream>>>(list);
    ctx->launches++;
    list.count = 0;
    most = 0;
  }
};

// The float32 GEMM's operands of w, out of `cur`; false: the kind (or a head width past the attention core's) has none.
bool f32_jobs(Preparer& prep, const lf_weights* w, WeightCursor& cur, SplitMatrix* g) {
  const auto& f = w->f;
  const auto& dims = w->dims;
  struct Part { const float* w; int ld, col0, n; };
  auto operand = [&](SplitMatrix& out, int K, std::initializer_list<Part> parts) {
    const int ld = (K + 7) / 8 * 8;
    int n = 0, row = 0;
    for (const Part& q : parts) n += q.n;
    bf16* p = cur.take<bf16>((size_t)3 * n * ld);
    out.p = p;
    out.ld = ld;
    out.batch_stride = 0;
    out.term_stride = (int64_t)n * ld;
    for (const Part& q : parts) {
      if (q.n) prep.push(Job{q.w, nullptr, nullptr, p, 1.0f, JOB_TERMS, K, q.ld, q.col0, q.n, q.n, ld, row, out.term_stride});
      row += q.n;
    }
  };
  const int c = dims.channels, HD = dims.heads * dims.head_dim;
  switch (w->kind) {
    case LF_WEIGHTS_TRIANGLE_AF2:
    case LF_WEIGHTS_TRIANGLE_AF3:
      {
        const int ld = (c + 7) / 8 * 8, rows = gated_columns(dims.hidden);
        bf16* p = cur.take<bf16>((size_t)3 * rows * ld);
        g[0] = SplitMatrix{p, ld, 0, (int64_t)rows * ld};
        prep.push(Job{f[TRI_W4], nullptr, nullptr, p, 1.0f, JOB_GATED, c, 4 * dims.hidden, 0, dims.hidden, rows, ld, 0, g[0].term_stride});
      }
      operand(g[1], dims.hidden, {{f[TRI_WZ], c, 0, c}});
      operand(g[2], c, {{f[TRI_WG], c, 0, c}});
      break;
    case LF_WEIGHTS_TRANSITION_AF2:
    case LF_WEIGHTS_TRANSITION_AF3: {
      const int wide = w->kind == LF_WEIGHTS_TRANSITION_AF3 ? 2 * dims.hidden : dims.hidden;
      operand(g[0], c, {{f[TRN_W1], wide, 0, wide}});
      operand(g[1], dims.hidden, {{f[TRN_W2], c, 0, c}});
      break;
    }
    case LF_WEIGHTS_GLOBAL_ATTENTION_AF2: {
      const int wide = 2 * dims.head_dim + HD;
      operand(g[0], c, {{f[GLB_W3], wide, 0, wide}});
      operand(g[1], HD, {{f[GLB_WO], c, 0, c}});
      break;
    }
    case LF_WEIGHTS_MSA_ATTENTION_AF3:
      operand(g[0], c, {{f[ATT_W4], 4 * HD, 2 * HD, 2 * HD}});
      operand(g[1], HD, {{f[ATT_WO], c, 0, c}});
      break;
    case LF_WEIGHTS_ATTENTION_AF2:
    case LF_WEIGHTS_GRID_ATTENTION_AF3:
    case LF_WEIGHTS_SINGLE_ATTENTION_AF3:
      {
        if (dims.head_dim > 64) return false;
        const int d = dims.head_dim, D = head_width(d), wide = 4 * dims.heads * D, own_bias = w->has_pair_proj && !w->has_pair_norm ? dims.heads : 0;
        const int ld = (c + 7) / 8 * 8;
        bf16* p = cur.take<bf16>((size_t)3 * (wide + own_bias) * ld);
        g[0] = SplitMatrix{p, ld, 0, (int64_t)(wide + own_bias) * ld};
        prep.push(Job{f[ATT_W4], nullptr, nullptr, p, 1.0f, JOB_HEADS, c, 4 * HD, 0, 4 * HD, wide, D, d, g[0].term_stride});
        if (own_bias) prep.push(Job{f[ATT_WB], nullptr, nullptr, p, 1.0f, JOB_TERMS, c, own_bias, 0, own_bias, own_bias, ld, wide, g[0].term_stride});
        bf16* po = cur.take<bf16>((size_t)3 * c * dims.heads * D);
        g[1] = SplitMatrix{po, (int64_t)dims.heads * D, 0, (int64_t)c * dims.heads * D};
        prep.push(Job{f[ATT_WO], nullptr, nullptr, po, 1.0f, JOB_HEADS_OUT, HD, c, 0, c, dims.heads * D, D, d, g[1].term_stride});
        float* bias = cur.take<float>(wide);
        g[2].p = reinterpret_cast<const bf16*>(bias);
        prep.push(Job{f[ATT_B4], nullptr, nullptr, bias, 1.0f, JOB_HEADS_BIAS, 0, 0, 0, 4 * HD, wide, D, d, 0});
      }
      break;
    default: return false;
  }
  return true;
}

}  // namespace

// h[0] = swizzled fp16 image of the fused projection W^T (plus the pair-bias projection rows for attention), h[1] = its
// bias vector, h[2], h[3] = the output kernel's; h[4], h[5] = the pair bias projection with a LayerNorm of its own; g =
// operands of the plain GEMM.  Runs twice: a dry pass that adds the sizes up, then the real one.
lf_status prepare_weights(lf_context* ctx, lf_weights* w, WeightCursor& cur) {
  const bool tri = w->kind == LF_WEIGHTS_TRIANGLE_AF2 || w->kind == LF_WEIGHTS_TRIANGLE_AF3;
  const bool att = w->kind == LF_WEIGHTS_ATTENTION_AF2 || w->kind == LF_WEIGHTS_GRID_ATTENTION_AF3;
  const auto& f = w->f;
  Preparer prep{ctx, cur.dry};
  w->h.clear();
  w->g.clear();
  if (tri && w->dims.channels == 128 && w->dims.hidden == 128) {
    // the input LayerNorm's gain goes into the rows of the images, its offset into the biases: the kernels' producers
    // hand the tensor core (x - mean) / std
    op16* img = cur.take<op16>(512 * 128);
    float* b4 = cur.take<float>(512);
    prep.image(f[TRI_W4], 128, 512, 512, 0, 512, img, 0, 1.0f, f[TRI_LN_G]);
    prep.fold(f[TRI_W4], 128, 512, 0, 512, f[TRI_LN_B], f[TRI_B4], 1.0f, b4);
    // output kernel: rows 0..127 = (diag(gain) Wz)^T, rows 128..255 = Wg^T; the centre LayerNorm folded into (s1 | t | gate bias):
    // s1[c] = sum_h fp16(gain[h] Wz[h][c]), t = offset through Wz + bz, and the input offset through Wg + bg
    op16* img2 = cur.take<op16>(256 * 128);
    float* fold = cur.take<float>(384);
    prep.image(f[TRI_WZ], 128, 128, 256, 0, 128, img2, 0, 1.0f, f[TRI_LNO_G]);
    prep.image(f[TRI_WG], 128, 128, 256, 0, 128, img2, 128, 1.0f, f[TRI_LN_G]);
    prep.push(Job{f[TRI_WZ], f[TRI_LNO_G], nullptr, fold, 1.0f, JOB_COLSUM, 128, 128, 0, 128, 128, 0, 0});
    prep.fold(f[TRI_WZ], 128, 128, 0, 128, f[TRI_LNO_B], f[TRI_BZ], 1.0f, fold + 128);
    prep.fold(f[TRI_WG], 128, 128, 0, 128, f[TRI_LN_B], f[TRI_BG], 1.0f, fold + 256);
    w->h = {img, b4, img2, fold};
  } else if (att && w->dims.channels == 128 && w->dims.heads * w->dims.head_dim == 128 && w->dims.heads <= 16 && !w->has_pair_norm) {
    op16* img = cur.take<op16>(528 * 128);
    float* bias = cur.take<float>(528);
    const float qs = 1.0f / sqrtf((float)w->dims.head_dim);      // the query columns carry the head_dim^-1/2 logit scale
    const int heads = w->has_pair_proj ? w->dims.heads : 0;      // rows past the heads are zeros
    prep.image(f[ATT_W4], 128, 128, 528, 0, 512, img, 0, qs, f[ATT_LN_G]);
    prep.image(f[ATT_W4], 128, 384, 528, 128, 512, img, 128, 1.0f, f[ATT_LN_G]);
    prep.fold(f[ATT_W4], 128, 128, 0, 512, f[ATT_LN_B], f[ATT_B4], qs, bias);
    prep.fold(f[ATT_W4], 128, 384, 128, 512, f[ATT_LN_B], f[ATT_B4] + 128, 1.0f, bias + 128);
    prep.image(f[ATT_WB], 128, heads, 528, 0, heads, img, 512, 1.0f, f[ATT_LN_G], 16);
    prep.fold(f[ATT_WB], 128, heads, 0, heads, f[ATT_LN_B], nullptr, 1.0f, bias + 512, 16);
    op16* img2 = cur.take<op16>(128 * 128);
    prep.image(f[ATT_WO], 128, 128, 128, 0, 128, img2, 0, 1.0f);
    w->h = {img, bias, img2, nullptr};
  }
  if (w->has_pair_norm && w->has_pair_proj && w->dims.pair_channels == 128 && w->dims.heads <= 16 &&
      (w->kind == LF_WEIGHTS_ATTENTION_AF2 || w->kind == LF_WEIGHTS_SINGLE_ATTENTION_AF3 || w->kind == LF_WEIGHTS_MSA_ATTENTION_AF3)) {
    // pair bias from a 128-channel pair with a LayerNorm of its own: a 16-row image of the projection (gain in its
    // rows, the offset's share as a bias) for the tensor-core projection kernel run with the bias chunk alone
    op16* img = cur.take<op16>(16 * 128);
    float* pb = cur.take<float>(16);
    prep.image(f[ATT_WB], 128, w->dims.heads, 16, 0, w->dims.heads, img, 0, 1.0f, f[ATT_PLN_G], 16);
    prep.fold(f[ATT_WB], 128, w->dims.heads, 0, w->dims.heads, f[ATT_PLN_B], nullptr, 1.0f, pb, 16);
    if (w->h.size() < 6) w->h.resize(6, nullptr);
    w->h[4] = img;
    w->h[5] = pb;
  }
  if (w->kind == LF_WEIGHTS_TRANSITION_AF2 && w->dims.channels == 128 && w->dims.hidden == 512) {
    // per 128-wide hidden chunk: W1 slice image (rows = hidden columns, K = 128 inputs), then W2 slice
    // image (rows = 128 outputs, K = the chunk's 128 hidden channels)
    op16* img = cur.take<op16>(4 * 32768);
    float* b1 = cur.take<float>(512);
    for (int c = 0; c < 4 && !cur.dry; ++c) {
      prep.image(f[TRN_W1], 128, 128, 128, c * 128, 512, img + c * 32768, 0, 1.0f, f[TRN_LN_G]);
      prep.image(f[TRN_W2] + (size_t)c * 128 * 128, 128, 128, 128, 0, 128, img + c * 32768 + 16384, 0, 1.0f);
    }
    prep.fold(f[TRN_W1], 128, 512, 0, 512, f[TRN_LN_B], f[TRN_B1], 1.0f, b1);
    w->h = {img, b1};
  }
  if (w->kind == LF_WEIGHTS_TRANSITION_AF3 && w->dims.channels == 128 && w->dims.hidden == 512) {
    // per 64-wide hidden chunk: W1 slice image of 128 rows (64 gate columns, then the matching 64 value
    // columns; K = 128 inputs: 32 KiB), then W2 slice image (rows = 128 outputs, K = 64 hidden: 16 KiB)
    op16* img = cur.take<op16>(8 * 24576);
    float* b1 = cur.take<float>(1024);
    for (int c = 0; c < 8 && !cur.dry; ++c) {
      op16* base = img + (size_t)c * 24576;
      prep.image(f[TRN_W1], 128, 64, 128, c * 64, 1024, base, 0, 1.0f, f[TRN_LN_G]);
      prep.image(f[TRN_W1], 128, 64, 128, 512 + c * 64, 1024, base, 64, 1.0f, f[TRN_LN_G]);
      prep.image(f[TRN_W2] + (size_t)c * 64 * 128, 64, 128, 128, 0, 128, base + 16384, 0, 1.0f);
    }
    prep.fold(f[TRN_W1], 128, 1024, 0, 1024, f[TRN_LN_B], f[TRN_B1], 1.0f, b1);
    w->h = {img, b1};
  }
  // Operands of the plain fp16 GEMM for the widths the fused kernels do not take: weights [k][n] -> fp16 [n][k]; attention: the heads
  // that the tcgen05 core takes four at a time
  if (att && (w->h.empty() || !w->h[0]) && w->dims.channels % 8 == 0 && w->dims.head_dim == 32 && w->dims.heads > 0 && w->dims.heads % 4 == 0 &&
      !(w->has_pair_proj && !w->has_pair_norm)) {
    const int c = w->dims.channels, HD = w->dims.heads * 32;
    op16 *w4 = cur.take<op16>((size_t)4 * HD * c), *wo = cur.take<op16>((size_t)c * HD);
    prep.operand(f[ATT_W4], c, 4 * HD, 4 * HD, w4);
    prep.operand(f[ATT_WO], HD, c, c, wo);
    w->g = {w4, wo};
  }
  if ((w->kind == LF_WEIGHTS_TRANSITION_AF2 || w->kind == LF_WEIGHTS_TRANSITION_AF3) && w->h.empty() &&
      w->dims.channels % 8 == 0 && w->dims.hidden % 8 == 0) {
    const int c = w->dims.channels, hd = w->dims.hidden, wide = w->kind == LF_WEIGHTS_TRANSITION_AF3 ? 2 * hd : hd;
    op16 *w1 = cur.take<op16>((size_t)wide * (c + 16)), *w2 = cur.take<op16>((size_t)c * hd);
    prep.push(Job{f[TRN_W1], nullptr, f[TRN_B1], w1, 1.0f, JOB_BIASED, c, wide, 0, wide, wide, 0, 0});
    prep.operand(f[TRN_W2], hd, c, c, w2);
    w->g = {w1, w2};
  }
  if (w->kind == LF_WEIGHTS_OPM_AF2 && w->dims.channels % 8 == 0 && w->dims.hidden % 8 == 0 && w->dims.out_channels % 8 == 0) {
    const int cm = w->dims.channels, c = w->dims.hidden, cz = w->dims.out_channels;
    op16 *wlr = cur.take<op16>((size_t)2 * c * cm), *wout = cur.take<op16>((size_t)cz * c * c);
    prep.operand(f[OPM_WL], cm, c, c, wlr);
    prep.operand(f[OPM_WR], cm, c, c, wlr + (int64_t)c * cm);
    prep.operand(f[OPM_WOUT], c * c, cz, cz, wout);
    w->g = {wlr, wout};
  }
  // Operands of the float32 GEMM: now for operators that run on it in 16-bit mode too, later (f32_operands in api.cu) for the others
  const bool fused = !w->h.empty() && w->h[0], transition = w->kind == LF_WEIGHTS_TRANSITION_AF2 || w->kind == LF_WEIGHTS_TRANSITION_AF3;
  const bool flash = (fused && w->dims.heads == 4 && w->dims.head_dim == 32) || (!w->g.empty() && (!w->has_pair_norm || pair_bias_supported(w)));
  const bool always = tri ? !fused : att ? !flash : transition ? !fused && w->g.empty() : true;
  lf_f32_operands& o = w->f32;
  Preparer none{ctx, true};
  WeightCursor size{nullptr, 0, true};
  o.bytes = f32_jobs(none, w, size, o.g) ? size.offset : 0;
  if (o.bytes && always) {
    f32_jobs(prep, w, cur, o.g);
    o.made = !cur.dry;
    o.ctx = ctx;
  } else if (o.bytes && o.bytes <= kF32RoomLimit) {
    o.room = cur.take<char>(o.bytes);
  }
  prep.flush();
  if (!cur.dry && cudaGetLastError() != cudaSuccess) return lf_fail(ctx, LF_ERR_CUDA, "weight preparation launch failed");
  return LF_OK;
}

lf_status prepare_f32_operands(lf_context* ctx, const lf_weights* const* w, int count) {
  Preparer prep{ctx, false};
  for (int i = 0; i < count; ++i) {
    lf_f32_operands& o = w[i]->f32;
    WeightCursor cur{o.room ? o.room : static_cast<char*>(o.block), 0, false};
    if (!f32_jobs(prep, w[i], cur, o.g)) return lf_fail(ctx, LF_ERR_UNSUPPORTED, "weights of kind %d have no float32 GEMM operands", w[i]->kind);
  }
  prep.flush();
  return cudaGetLastError() == cudaSuccess ? LF_OK : lf_fail(ctx, LF_ERR_CUDA, "weight preparation launch failed");
}

}  // namespace tc
