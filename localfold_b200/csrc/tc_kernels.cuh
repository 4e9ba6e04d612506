// Tensor-core (tcgen05 / TMEM / TMA) kernels for sm_100a: launchers used by api.cu.
// Each *_supported() says whether a kernel covers a shape; api.cu routes
// everything else to the general path.
#pragma once

#include "common.cuh"

namespace tc {

// Device buffers of the other ranks of a box as mapped into this process (entry `rank` = the local
// buffer).  Kernels only ever store to them: plain st.global, or TMA stores without multicast.
constexpr int kMaxPeers = 16;
struct PeerPtrs { void* p[kMaxPeers]; };

void configure_once();
// Tensor-core operands of the weights, out of the weights' own allocation (tc_weights.cu); a dry cursor only adds sizes up.
lf_status prepare_weights(lf_context* ctx, lf_weights* w, WeightCursor& cur);
// Waits for the stream and reads the device status word; LF_ERR_TIMEOUT if a bounded wait expired in a kernel.
lf_status check_status(lf_context* ctx);

// Float32 GEMM on the tensor cores (f32_gemm.cu), batched: out[b][i][j] = act(sum_k A(b, i, k) B(b, j, k) + bias[j]), both operands
// as bf16 terms; major 0: k contiguous (A [m][ld], or in pieces of eight columns over m rows when a.pieces, B [n][ld]); major 1: the row index
// contiguous (A [k][ld], B [k][ld]).
struct Gemm3Out {
  float* out;                  // float32 result, or null:
  bf16* terms;                 // its terms (ld a multiple of 8)
  int64_t ld, batch_stride, term_stride;
  const float* bias;           // or null; columns from bias_n on have none
  int bias_n, relu;
  int sigmoid_col0, sigmoid_col1;      // columns through a sigmoid (empty range: none)
  // Terms in pieces of eight columns, [3][ld / 8][m][8] (element (t, i, j) at t * term_stride + (j / 8) * m * 8 + i * 8 + j % 8), what
  // the attention cores read.  Columns from ld on (a multiple of 8; the projection has ld / 3 of them) are the gate then, float32 pieces [ld / 24][m][8]; the ones behind
  // a pair bias, row i * bias_q + j -> float32 pair_bias[column][i][bias_ld] at j, or [j] at i when bias_swap.
  int pieces = 0;
  float* gate = nullptr;
  float* pair_bias = nullptr;
  int bias_q = 0, bias_ld = 0, bias_swap = 0;
  // Or the operands of a triangle product: columns in groups of 32, 16 channels of a projection and the 16 of its gate (the fused projection's operand
  // is laid out so; all groups of a, then all of b, channels padded to whole groups), rows = pairs (i, k) of length plane_n:
  // planes[channel][i][k] = mask (projection + bias) sigmoid(gate + bias), rows of ld, fp16 when plane_half, else terms; bias = [4][plane_c]
  const float* plane_mask = nullptr;
  void* plane[2] = {nullptr, nullptr};
  int plane_n = 0, plane_c = 0, plane_half = 0;
  // Or the end of an operator in float32, rows of n (a multiple of 4) on 16-byte boundaries: act[dst(i)][j] (+)= value * (factor ? factor[i][j] : 1), added when
  // act_add; rows (b, q) go to row q * act_batch + b when act_q is not 0 (i = b * act_q + q)
  float* act = nullptr;
  const float* factor = nullptr;      // rows of n
  int act_add = 0, act_batch = 0, act_q = 0;
};
constexpr int gated_columns(int c) { return 4 * ((c + 15) / 16 * 16); }
void configure_gemm3();
lf_status gemm_f32(lf_context* ctx, ArenaCursor& cur, int major, const SplitMatrix& a, const SplitMatrix& b, int m, int n, int k, int batch,
                   const Gemm3Out& o);
// Attention core on split operands (f32_attention.cu): qkv = the terms of q | k | v in pieces over rows (batch, Q), heads of D channels, gate = sigmoid(gate) likewise in float32;
// bias float32 [heads][Q][ldb] (ldb a multiple of 4) or null; out = terms in pieces.
void configure_attention3();
bool attention3_wins(const lf_context* ctx, int D, int batch, int Q, int heads);      // over mma_attention.cuh
lf_status attention3(lf_context* ctx, ArenaCursor& cur, int D, const SplitMatrix& qkv, const float* gate, const float* bias, int ldb, const float* mask, int batch,
                     int Q, int heads, int transpose, int mask_mode, int clamp, float scale, const SplitMatrix& out);
// The weights' operands of the float32 GEMM (lf_f32_operands), into their room or block; as few launches as the jobs of all of them fit into.
lf_status prepare_f32_operands(lf_context* ctx, const lf_weights* const* w, int count);

// Triangle contraction, batched over the c channels of channel-major fp16
// operands a, b [c][n][ld] (ld a multiple of 8, elements past n never read):
//   outgoing: x[h][i][j] = scale * sum_k a[h][i][k] * b[h][j][k]
//   incoming: x[h][i][j] = scale * sum_k a[h][k][j] * b[h][k][i]
bool contract_supported(int n, int c);
lf_status contract(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, op16* x, int n, int ld, int c,
                   int incoming, float scale);
// Rectangular form for row shards: x[h][i][col0 + j] = scale * sum_k a[h][i][k] b[h][j][k], i < m_rows, j < n_rows,
// k < k_len; a, b have row stride ld_ab and dense planes, x has row stride ldx and plane stride x_plane.
lf_status contract_rect(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, op16* x, int m_rows, int n_rows,
                        int k_len, int ld_ab, int ldx, int64_t x_plane, int col0, int c, int incoming, float scale);

// Plain fp16 GEMMs (tc_gemm.cu), weights [n_out][k]:
void configure_gemm();
// q | k | v | gate of rows (b, q) as the attention core reads them: [q, k, v, gate][width / 128][batch][ldq * 128] in 8 x 8 pieces (see
// attention_project), value (acc + bias) * (qscale for q), gate through a sigmoid; rows Q .. ldq hold finite values
lf_status gemm_pieces(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* w, op16* out, int batch, int Q, int ldq, int k_len, int width,
                      const float* bias, float qscale);
// out[dst(b, q)][n_out] (+)= a w^T + bias in float32; a = rows (b, q), or pieces [k / 128][batch][ldq * 128] when a_pieces; dst is row q * batch + b
// when transposed; out on a 16-byte boundary, n_out a multiple of 4
lf_status gemm_rows_f32(lf_context* ctx, ArenaCursor& cur, const op16* a, int a_pieces, const op16* w, float* out, int add, int batch, int Q, int ldq,
                        int transposed, int n_out, int k_len, const float* bias);
lf_status gemm_rows_half(lf_context* ctx, ArenaCursor& cur, const op16* a_pieces, const op16* w, op16* out, int batch, int Q, int ldq, int n_out, int k_len);
lf_status gemm_outer32(lf_context* ctx, ArenaCursor& cur, const op16* left, const op16* right, op16* out, int cnt, int n, int k_len, float scale);
lf_status gemm_planes(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, op16* x, int n, int ld, int c, int incoming, float scale);
// fp16 rows: out[m][n] = act(sum_k a[m][k] w[n][k] + bias[n]) (k contiguous in both
// operands, k_len and n_out multiples of 8; bias may be null; act = ReLU when `relu`), fp16 result.
lf_status contract_gemm(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* w, op16* out, int m_rows, int n_out,
                        int k_len, const float* bias, int relu);
// ... and as the outer product mean's sum over the sequences, stored grouped per pair:
// out[((i * n + j) * c + a) * c + b] = scale * sum_s left[s][i*c + a] right[s][j*c + b] for i < cnt, j < n
// (left, right: k_len rows of n*c, left already offset to its first i), so that the c*c -> c_z projection that
// follows is a plain GEMM over rows (i, j).
lf_status contract_outer(lf_context* ctx, ArenaCursor& cur, const op16* left, const op16* right, op16* out, int cnt, int n, int c,
                         int k_len, float scale);

// Channel-sharded form for the GPUs of one box: a, b are this rank's `c` channels over all n rows
// ([c][n][ld]); row i of channel h of the product goes to rank i / rows_per_rank, into its buffer
// x_peers[...] laid out [all channels][rows_per_rank][ldx], at channel ch0 + h.
lf_status contract_scatter(lf_context* ctx, ArenaCursor& cur, const op16* a, const op16* b, int n, int ld, int c, int incoming,
                           float scale, const PeerPtrs& x_peers, int rows_per_rank, int total_channels, int ch0);

// LayerNorm + projection kernels for 128-channel activations (weights repacked by
// prepare_weights into lf_weights::h).
bool ln_gemm_supported(const lf_weights* w);
void configure_ln_gemm();
// a, b [c][n][ld] fp16 = mask * (LN(z) Wp + bp) * sigmoid(LN(z) Wg + bg)
// `rows` pair rows of length n (rows = n for the whole pair, fewer for a row shard)
lf_status triangle_project(lf_context* ctx, ArenaCursor& cur, const void* z, int act_dtype, const float* mask, int rows,
                           int n, int ld, int variance, float eps, const lf_weights* w, op16* a, op16* b);
// The same for a row shard whose operands are wanted channel-sharded: channel h of the shard's rows goes
// to rank h / (128 / ranks), into its buffers a_peers / b_peers laid out [128 / ranks][n][ld], at rows
// row0 .. row0 + rows (row0 = this rank's first pair row).
lf_status triangle_project_scatter(lf_context* ctx, ArenaCursor& cur, const void* z, int act_dtype, const float* mask, int rows,
                                   int n, int ld, int variance, float eps, const lf_weights* w, const PeerPtrs& a_peers,
                                   const PeerPtrs& b_peers, int ranks, int row0);
// q (pre-scaled by head_dim^-1/2), k, v, sigmoid(gate) as fp16 logical rows [batch][ld][128] stored in 8-row x
// 8-channel pieces (element (b, q, c) at b*ld*128 + (q/8)*1024 + (c/8)*64 + (q%8)*8 + c%8, ld = Q rounded up to 16) and the
// pair bias fp16 [heads][batch rows][ldb] (null = none) from the normalised input
lf_status pair_bias_project(lf_context* ctx, ArenaCursor& cur, const void* pair, int pair_dtype, int Q, int variance, float eps,
                            int heads, const lf_weights* w, op16* bias, int ldb);
bool pair_bias_supported(const lf_weights* w);
lf_status attention_project(lf_context* ctx, ArenaCursor& cur, const void* act, int act_dtype, int batch, int Q,
                            int transpose, int variance, float eps, int heads, int head_dim, int bias_swap,
                            const lf_weights* w, op16* q, op16* k, op16* v, op16* g, op16* bias, int ldb);
// The same for a row shard: its bias rows are written into every rank's copy of the whole bias
// [heads][bias_rows][ldb] at query rows row0 .. row0 + batch.  `transpose`: the shard is held as [Q][batch]
// (logical row (b, q) at memory row q*batch + b), as for a block of columns of the pair.
lf_status attention_project_scatter(lf_context* ctx, ArenaCursor& cur, const void* act, int act_dtype, int batch, int Q,
                                    int variance, float eps, int heads, const lf_weights* w, op16* q, op16* k, op16* v,
                                    op16* g, const PeerPtrs& bias_peers, int ranks, int bias_rows, int row0, int ldb,
                                    int transpose = 0);
lf_status attention_output(lf_context* ctx, ArenaCursor& cur, const op16* o, int batch, int Q, int transpose,
                           const lf_weights* w, const void* resid, void* out, int act_dtype);
// `x_plane_elems`: distance between the channel planes of x (0 = rows * ld, a dense shard; n * ld when x points at
// `rows` rows inside whole planes)
lf_status triangle_output(lf_context* ctx, ArenaCursor& cur, const op16* x, int rows, int n, int ld, float x_eps,
                          const void* z, int act_dtype, int variance, float eps, const lf_weights* w, const void* resid,
                          void* out, int64_t x_plane_elems = 0);
// out[b*Q+i][128] = (softmax_j(q_i.k_j + bias[h][i][j] + mask term_j) v_j) * gate, 4 heads x 32
void configure_attention();
// `bias`: fp16 [4][Q][ldb] (head, query, key; ldb a multiple of 16) or null
lf_status attention_core(lf_context* ctx, ArenaCursor& cur, const op16* q, const op16* k, const op16* v, const op16* g,
                         const op16* bias, int ldb, const float* mask, int batch, int Q, int transpose,
                         int mask_mode, int clamp, op16* out);

// Fused AF2 pair transition (128 channels, 512 hidden): out = resid + relu(LN(x) W1 + b1) W2 + b2
void configure_transition();
bool transition_supported(const lf_weights* w);
lf_status transition_run(lf_context* ctx, ArenaCursor& cur, const void* act, int act_dtype, int64_t rows, int variance,
                         float eps, const lf_weights* w, const void* resid, void* out);

}  // namespace tc
