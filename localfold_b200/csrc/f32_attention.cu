// Gated float32 attention core on tcgen05 for heads of 8, 16 or 32 channels: every operand as three bf16 terms (nothing of a
// float32 value is lost), a product of two values as the six term products above 2^-24, float32 accumulation.
//
// Work item = 128 queries of one head for four neighbouring batch rows, a stream each; the streams share the bias tiles.  Per key tile
// (32 keys): S = Q K^T; the stream's four softmax warps (a thread a query, so every reduction over keys is thread-local) take
// S into registers, add bias and mask terms, exponentiate and write the terms of P over S; P V runs with P as the A operand from
// tensor memory into fresh accumulators - the leading term product and the others apart - which the softmax warps add to the output
// in their registers during the next tile, in round-to-nearest: what the tensor core's own additions lose, since they truncate, is of a
// tile's share, not of the running sum.
//
// Operands lie in pieces of eight channels ([term][channels / 8][row][8], see Gemm3Out), so a tile of keys is one contiguous run a
// piece and term, and one tensor copy brings all of them in as the tensor core's unswizzled operand format, zeros past the end of the
// batch row, for the four streams at once.  (Beside sixteen busy warps a producer's step - a barrier's test, its arming, a copy - takes about
// 600 clocks: a copy a stream and operand, or a bulk copy a run, was the bound.)
//
// What bounds it: issue slots (65 % of them busy at 384 x 384) and the round trips of a tile; the exponents take a quarter of their unit's time, the tensor
// core a third.  An exponential costs its share of 17 instructions, six of them to take it apart and three to add the products up.  Two streams
// with tiles of 64 keys, two softmax warps a scheduler, took a tenth longer; with the next logits requested during the exponentials another tenth.
// Against the mma.sync kernel (mma_attention.cuh; a warp's chain of dependent MMAs): 384 x 384, 4 heads of 16: 465 -> 198 us; 203 x 203,
// 4 x 32: 184 -> 84; 1024 x 256, 8 x 8: 936 -> 485.
#include <cuda.h>

#include "tc05.cuh"
#include "tc_kernels.cuh"

namespace tc {

using namespace tc05;

constexpr int F3_STREAMS = 4;
constexpr int F3_THREADS = 20 * 32;       // sixteen softmax warps, two MMA issuers, two producers
// 20 warps start with 96 registers a thread; setmaxnreg trades inside the block's own allocation: 16 x 104 + 4 x 64 = 20 x 96.
constexpr uint32_t F3_REGS_SOFTMAX = 104, F3_REGS_SERVICE = 64;
constexpr int F3_QT = 128, F3_KT = 32;
constexpr int F3_BIAS_BYTES = F3_QT * F3_KT * 4;

// A product of heads of 8 channels fills half of the tensor core's k, so two products share a step, its halves from two term planes:
// (q0 q2)(k2 k0), (q1 q2)(k0 k1), (q0 q1)(k1 k2), (q0 q1)(k0 k1), for which the keys' first plane is there once more behind the third.
template <int D>
struct F3Form {
  static constexpr int PIECES = D / 8;
  static constexpr int K_PLANES = D == 8 ? 4 : 3;       // (of V a fourth that is only there to be multiplied: N is a multiple of 16)
  static constexpr int STAGES = D == 32 ? 2 : 3;        // of K, V and the bias
  static constexpr int Q_BUFFERS = D == 32 ? 1 : 2;
  static constexpr int MASKS = D == 32 ? 4 : 8;         // tiles whose mask terms are held: more than the K ring and the softmax warps are apart
  static constexpr int Q_BYTES = 3 * PIECES * F3_STREAMS * F3_QT * 16;
  static constexpr int K_BYTES = K_PLANES * PIECES * F3_STREAMS * F3_KT * 16;      // ... and of V
  // Columns of a stream's 128 of tensor memory: buffers of S, over each of them the first two terms of P (16 keys: eight columns of
  // each, over their logits); the third, of whichever tile is at it; P V.
  static constexpr int S_BUFFERS = D == 32 ? 1 : 2;
  static constexpr int THIRD = S_BUFFERS * F3_KT, O = THIRD + F3_KT / 2;
  static constexpr int BARRIERS = 2 * (Q_BUFFERS + 3 * STAGES + F3_STREAMS * S_BUFFERS) + F3_STREAMS;
  static constexpr int SMEM_USED = STAGES * F3_BIAS_BYTES + Q_BUFFERS * Q_BYTES + STAGES * 2 * K_BYTES + F3_STREAMS * MASKS * F3_KT * 4 + BARRIERS * 8 + 8 +
                                   F3_STREAMS * MASKS * 4;
  static constexpr int SMEM = SMEM_USED + (D == 32 ? 0 : 1024);      // the bias tiles want 1024-byte boundaries, which the allocation starts on in fact
};
static_assert(F3Form<32>::SMEM <= 232448 && F3Form<16>::SMEM <= 232448 && F3Form<8>::SMEM <= 232448, "shared memory of a block");

struct F3Params {
  int batch, Q, heads, qtiles, ktiles;
  int transpose, mask_mode, clamp;
  float scale;
  const float* gate;       // sigmoid(gate) in pieces of eight channels over `rows` rows
  int64_t rows;
  const float* mask;       // b*Q + j, or j*batch + b when transpose
  bf16* out;               // terms in pieces, out_stride apart
  int64_t out_stride;
  Status* status;
};

__device__ __forceinline__ float f3_ex2(float x) {      // relative error 2^-22
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// the leading bf16 terms of x, y by truncation
__device__ __forceinline__ uint32_t f3_pack(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }
__host__ __device__ constexpr uint32_t f3_idesc(int N, int b_major) {      // 128 x N, bf16 operands, A K-major
  return make_idesc_f16(F3_QT, N, 0, b_major) | (1u << 7) | (1u << 10);
}

template <int D, bool BIAS>
__global__ void __launch_bounds__(F3_THREADS, 1)
attention3_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapK1,
                  const __grid_constant__ CUtensorMap mapB, const F3Params p) {
  typedef F3Form<D> F;
  constexpr int NS = F3_STREAMS, ST = F::STAGES, PIECES = F::PIECES, QB = F::Q_BUFFERS, SB = F::S_BUFFERS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  if (D == 32 && smem != smem_raw) {      // never seen
    if (threadIdx.x == 0 && p.status && atomicCAS(&p.status->code, 0u, kStatusAlignment) == 0u) { p.status->where = 59; p.status->block = blockIdx.x; }
    return;
  }
  uint8_t* sBias = smem;                                  // [stage][128 queries][32 keys], 128-byte swizzle
  uint8_t* sQ = sBias + ST * F3_BIAS_BYTES;               // [buffer][plane][piece][stream][128][16 B]
  uint8_t* sK = sQ + QB * F::Q_BYTES;                     // [stage][plane][piece][stream][32][16 B]
  uint8_t* sV = sK + ST * F::K_BYTES;                     // likewise
  float* sMask = reinterpret_cast<float*>(sV + ST * F::K_BYTES);      // [stream][tile % MASKS][32]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sMask + NS * F::MASKS * F3_KT);
  uint64_t* q_full = bars;                  // [buffer]
  uint64_t* q_empty = q_full + QB;          // [buffer] a commit a stream
  uint64_t* k_full = q_empty + QB;          // [stage]: keys and mask terms
  uint64_t* k_empty = k_full + ST;          // [stage] a commit a stream
  uint64_t* v_full = k_empty + ST;
  uint64_t* v_empty = v_full + ST;
  uint64_t* s_full = v_empty + ST;    // [stream][buffer]
  uint64_t* p_full = s_full + NS * SB;      // [stream][buffer] count 4
  uint64_t* o_full = p_full + NS * SB;      // [stream], a phase a key tile
  uint64_t* b_full = o_full + NS;           // [stage]
  uint64_t* b_empty = b_full + ST;          // [stage] count 16
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(b_empty + ST);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* mask_flag = abort_flag + 1;      // [stream][tile % MASKS]: a term is not zero

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t items = (uint32_t)((p.batch + NS - 1) / NS) * p.heads * p.qtiles;
  const int T = p.ktiles;
  // query tiles change fastest: they read the same keys
  auto locate = [&](uint32_t item, int& b, int& h, int& tile) {
    const uint32_t r = item / (uint32_t)p.qtiles;
    tile = item - r * p.qtiles;
    b = NS * (int)(r / (uint32_t)p.heads);
    h = r % (uint32_t)p.heads;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < QB; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], NS); }
    for (int i = 0; i < ST; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], NS); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], NS); }
    for (int i = 0; i < NS * SB; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); }
    for (int i = 0; i < NS; ++i) mbar_init(&o_full[i], 1);
    for (int i = 0; i < ST; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 16); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 17) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  lf_chain();

  if (warp >= 16) {
  reg_dec<F3_REGS_SERVICE>();
  const int hp = p.heads * PIECES;       // pieces of q (of k, of v)
  if (warp == 16) {
    // ---------------- producer of K, V and the mask terms ----------------
    // coordinates: 8-byte halves of a row's piece, batch row, piece, term
    if (lane == 0) { prefetch_tensormap(&mapK); if (D == 8) prefetch_tensormap(&mapK1); }
    uint32_t n = 0;      // key tiles so far, the same of every stream
    int st = 0;
    uint32_t par = 1;
    bool ok = true;
    int b0, h, tile;
    float next[NS];      // mask value of a key a lane, of every stream: fetched a tile ahead
    auto fetch = [&](int b, int t) {
      const int j = t * F3_KT + lane;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const int row = b + s;
        next[s] = j < p.Q && row < p.batch ? p.mask[p.transpose ? (int64_t)j * p.batch + row : (int64_t)row * p.Q + j] : 1.f;
      }
    };
    locate(blockIdx.x, b0, h, tile);
    fetch(b0, 0);
    for (uint32_t item = blockIdx.x; item < items && ok; item += gridDim.x) {
      locate(item, b0, h, tile);
      for (int t = 0; t < T && ok; ++t, ++n) {
        float m[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) m[s] = next[s];
        if (t + 1 < T) fetch(b0, t + 1);
        else if (item + gridDim.x < items) {
          int nb, nh, nt;
          locate(item + gridDim.x, nb, nh, nt);
          fetch(nb, 0);
        }
        ok = __all_sync(0xffffffffu, mbar_wait(&k_empty[st], par, abort_flag, p.status, 61));
        if (!ok) break;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          const float term = p.mask_mode == 0 ? 1e9f * (m[s] - 1.0f) : (m[s] > 0.f ? 0.f : -1e9f);
          const int slot = s * F::MASKS + (n & (F::MASKS - 1));
          sMask[slot * F3_KT + lane] = term;
          const unsigned any = __ballot_sync(0xffffffffu, term != 0.f);
          if (lane == 0) mask_flag[slot] = any != 0;
        }
        __syncwarp();
        if (lane == 0) {
          mbar_expect_tx(&k_full[st], F::K_BYTES);      // publishes the terms too
          tma_load_4d(sK + st * F::K_BYTES, &mapK, &k_full[st], t * F3_KT * 2, b0, hp + h * PIECES, 0);
          if (D == 8) tma_load_4d(sK + st * F::K_BYTES + 3 * NS * F3_KT * 16, &mapK1, &k_full[st], t * F3_KT * 2, b0, hp + h, 0);
          ok = mbar_wait(&v_empty[st], par, abort_flag, p.status, 62);
          if (ok) {
            mbar_expect_tx(&v_full[st], 3 * PIECES * NS * F3_KT * 16);
            tma_load_4d(sV + st * F::K_BYTES, &mapK, &v_full[st], t * F3_KT * 2, b0, 2 * hp + h * PIECES, 0);
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (++st == ST) { st = 0; par ^= 1; }
      }
    }
  } else if (warp == 19) {
    // ---------------- producer of Q and the bias tiles (the streams share them) ----------------
    if (lane == 0) {
      prefetch_tensormap(&mapQ);
      if (BIAS) prefetch_tensormap(&mapB);
      uint32_t n_item = 0, par = 1;
      int st = 0;
      bool ok = true;
      for (uint32_t item = blockIdx.x; item < items && ok; item += gridDim.x, ++n_item) {
        int b0, h, tile;
        locate(item, b0, h, tile);
        const uint32_t qb = n_item % QB, q_par = (n_item / QB) & 1;
        ok = mbar_wait(&q_empty[qb], q_par ^ 1, abort_flag, p.status, 60);
        if (!ok) break;
        mbar_expect_tx(&q_full[qb], F::Q_BYTES);
        tma_load_4d(sQ + qb * F::Q_BYTES, &mapQ, &q_full[qb], tile * F3_QT * 2, b0, h * PIECES, 0);
        for (int t = 0; BIAS && t < T && ok; ++t) {
          ok = mbar_wait(&b_empty[st], par, abort_flag, p.status, 63);
          if (!ok) break;
          mbar_expect_tx(&b_full[st], F3_BIAS_BYTES);
          tma_load_3d(sBias + st * F3_BIAS_BYTES, &mapB, &b_full[st], t * F3_KT, tile * F3_QT, h);
          if (++st == ST) { st = 0; par ^= 1; }
        }
      }
    }
  } else {
    // ---------------- MMA issuers of two streams each ----------------
    // P V of a key tile once P is written, S of a tile once its operands are there and the P that lies in its place has had its P V
    // issued (the tensor pipe keeps the order): whichever comes first, so that operands that are late keep no product waiting.  A
    // lane looks at one barrier - (stream, operand) = (lane / 4, lane % 4) with the operands K, Q, P, V - and a ballot tells them all.
    // The whole warp runs the loop, one elected lane issues.
    const int w = __shfl_sync(0xffffffffu, warp - 17, 0);
    uint32_t my_items = 0;
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) ++my_items;
    const uint32_t U = my_items * (uint32_t)T;
    const int look_s = 2 * w + ((lane >> 2) & 1), look_kind = lane & 3;
    uint64_t* const look = look_kind == 0 ? k_full : look_kind == 1 ? q_full : look_kind == 2 ? p_full + look_s * SB : v_full;
    const int look_ring = look_kind == 1 ? QB : look_kind == 2 ? SB : ST;
    int look_at = 0;
    uint32_t look_par = 0;
    struct Stream { uint32_t qk, pv, qk_t, qk_st, qk_qb, pv_st; } str[2] = {};
    uint32_t idle = 0;
    uint64_t since = 0;
    auto qk_issue = [&](const Stream& x, int s) {
      constexpr uint32_t idesc = f3_idesc(F3_KT, 0);
      const uint32_t d = tmem_base + s * 128 + (x.qk % SB) * F3_KT;
      const uint64_t q0 = make_smem_desc_plain(smem_u32(sQ + x.qk_qb * F::Q_BYTES + s * F3_QT * 16), NS * F3_QT * 16, 128);
      const uint64_t k0 = make_smem_desc_plain(smem_u32(sK + x.qk_st * F::K_BYTES + s * F3_KT * 16), NS * F3_KT * 16, 128);
      auto qd = [&](int plane, int pc) { return q0 + (plane * PIECES + pc) * NS * F3_QT; };      // (address field: units of 16 bytes)
      auto kd = [&](int plane, int pc) { return k0 + (plane * PIECES + pc) * NS * F3_KT; };
      if (D == 8) {      // small term products first, the leading one last
        umma_f16(d, make_smem_desc_plain(smem_u32(sQ + x.qk_qb * F::Q_BYTES + s * F3_QT * 16), 2 * NS * F3_QT * 16, 128), kd(2, 0), idesc, 0);
        umma_f16(d, qd(1, 0), kd(0, 0), idesc, 1);
        umma_f16(d, qd(0, 0), kd(1, 0), idesc, 1);
        umma_f16(d, qd(0, 0), kd(0, 0), idesc, 1);
      } else {
#pragma unroll
        for (int kk = 0; kk < PIECES; kk += 2) {
          umma_f16(d, qd(0, kk), kd(2, kk), idesc, kk != 0);
          umma_f16(d, qd(1, kk), kd(1, kk), idesc, 1);
          umma_f16(d, qd(2, kk), kd(0, kk), idesc, 1);
          umma_f16(d, qd(0, kk), kd(1, kk), idesc, 1);
          umma_f16(d, qd(1, kk), kd(0, kk), idesc, 1);
        }
#pragma unroll
        for (int kk = 0; kk < PIECES; kk += 2) umma_f16(d, qd(0, kk), kd(0, kk), idesc, 1);
      }
      umma_commit(&s_full[s * SB + x.qk % SB]);
      umma_commit(&k_empty[x.qk_st]);
      if (x.qk_t + 1 == (uint32_t)T) umma_commit(&q_empty[x.qk_qb]);
    };
    auto pv_issue = [&](const Stream& x, int s) {
      const uint32_t d0 = tmem_base + s * 128, pb = d0 + (x.pv % SB) * F3_KT, d_o = d0 + F::O;
      // V as the MN-major operand: 16 keys a step, the terms' pieces one after the other along N
      const uint64_t v0 = make_smem_desc_plain(smem_u32(sV + x.pv_st * F::K_BYTES + s * F3_KT * 16), 128, NS * F3_KT * 16);
#pragma unroll
      for (int kk = 0; kk < F3_KT / 16; ++kk) {
        auto vd = [&](int term) { return v0 + term * PIECES * NS * F3_KT + kk * 16; };
        auto pt = [&](int term) { return term == 2 ? d0 + F::THIRD + kk * 8 : pb + kk * 16 + term * 8; };
        const uint32_t more = kk != 0;
        if (D == 8) {              // columns 0-7 p0 v0, 8-15 p0 v1, 16-23 p0 v2, 32-39 (p1 + p2) v0, 40-47 (p1 + p2) v1
          umma_f16_ts(d_o, pt(0), vd(0), f3_idesc(32, 1), more);
          umma_f16_ts(d_o + 32, pt(1), vd(0), f3_idesc(16, 1), more);
          umma_f16_ts(d_o + 32, pt(2), vd(0), f3_idesc(16, 1), 1);
        } else if (D == 16) {      // 0-15 p0 v0, 16-31 p0 v1 + p1 v0, 32-47 p0 v2 + p1 v1 + p2 v0
          umma_f16_ts(d_o, pt(0), vd(0), f3_idesc(48, 1), more);
          umma_f16_ts(d_o + 16, pt(1), vd(0), f3_idesc(32, 1), 1);
          umma_f16_ts(d_o + 32, pt(2), vd(0), f3_idesc(16, 1), 1);
        } else {                   // 0-31 p0 v0, 32-63 the others
          umma_f16_ts(d_o, pt(0), vd(0), f3_idesc(64, 1), more);
          umma_f16_ts(d_o + 32, pt(0), vd(2), f3_idesc(32, 1), 1);
          umma_f16_ts(d_o + 32, pt(1), vd(1), f3_idesc(32, 1), 1);
          umma_f16_ts(d_o + 32, pt(2), vd(0), f3_idesc(32, 1), 1);
          umma_f16_ts(d_o + 32, pt(1), vd(0), f3_idesc(32, 1), 1);
        }
      }
      umma_commit(&o_full[s]);
      umma_commit(&v_empty[x.pv_st]);
    };
    while (str[0].pv < U || str[1].pv < U) {
      const uint32_t there = __ballot_sync(0xffffffffu, mbar_test(look + look_at, look_par));
      __syncwarp();
      bool done = false;
      auto step = [&](Stream& x, int i) {
        const uint32_t bits = there >> (i * 4);
        uint32_t taken = 0;      // operands whose barriers move on
        if (x.pv < x.qk && (bits & 12u) == 12u) {
          tc_fence_after();
          if (elect_one()) pv_issue(x, 2 * w + i);
          __syncwarp();
          if (++x.pv_st == ST) x.pv_st = 0;
          ++x.pv;
          taken = 12u;
        }
        if (x.qk < U && x.qk < x.pv + SB && (bits & 1u) && (x.qk_t != 0 || (bits & 2u))) {
          tc_fence_after();
          if (elect_one()) qk_issue(x, 2 * w + i);
          __syncwarp();
          if (++x.qk_st == ST) x.qk_st = 0;
          if (++x.qk_t == (uint32_t)T) {
            x.qk_t = 0;
            if (++x.qk_qb == QB) x.qk_qb = 0;
            taken |= 2u;
          }
          ++x.qk;
          taken |= 1u;
        }
        if (((lane >> 2) & 1) == i && (taken >> look_kind & 1u)) {
          if (++look_at == look_ring) { look_at = 0; look_par ^= 1; }
        }
        done |= taken != 0;
      };
      step(str[0], 0);
      step(str[1], 1);
      if (done) { idle = 0; continue; }
      if ((++idle & 2047u) == 0) {      // bounded, as mbar_wait
        const uint64_t now = global_timer_ns();
        if (idle == 2048u) since = now;
        const bool late = now - since > kWaitLimitNs;
        if (late && *abort_flag == 0) {
          *abort_flag = 1;
          if (p.status && atomicCAS(&p.status->code, 0u, kStatusTimeout) == 0u) { p.status->where = 64; p.status->block = blockIdx.x; }
        }
        if (__any_sync(0xffffffffu, late || *abort_flag != 0)) break;
      }
    }
  }
  } else {
    reg_inc<F3_REGS_SOFTMAX>();
    // ---------------- softmax: one thread per query of one stream ----------------
    const int g = warp >> 2, q = warp & 3, row = q * 32 + lane;
    const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + g * 128;
    constexpr float L2E = 1.4426950408889634f;
    uint32_t n = 0;
    int st = 0, slot = 0;
    uint32_t b_par = 0;
    bool ok = true;
    for (uint32_t item = blockIdx.x; item < items && ok; item += gridDim.x) {
      float o[D];
#pragma unroll
      for (int e = 0; e < D; ++e) o[e] = 0.f;
      // p = 2^(l log2(e) - ref2) with a whole ref2, so that a change of it scales by a power of two, exactly.  A masked row's logits
      // are near -1e9, where their product with log2(e) is rounded to whole powers of two: such a query (far) subtracts ref first, so its
      // base is ref log2(e).  A query keeps the form that its own reference asks for, whatever the others of its warp do.
      float ref = 0.f, ref2 = 0.f, sum = 0.f, lost = 0.f;      // lost: what the additions to the sum have rounded away so far, negated
      bool far = false, any_far = false;                       // any_far: of the warp's queries
      // P V of tile m times c onto the output
      auto add_product = [&](uint32_t m, float c) -> bool {
        if (!mbar_wait(&o_full[g], m & 1, abort_flag, p.status, 70)) return false;
        tc_fence_after();
        auto f = [](uint32_t x) { return __uint_as_float(x); };
        constexpr int G = D == 8 ? 5 : D == 16 ? 3 : 2;      // accumulators of a channel, eight channels at a time
#pragma unroll
        for (int c0 = 0; c0 < D; c0 += 8) {
          uint32_t r[G][8];
#pragma unroll
          for (int i = 0; i < G; ++i) tmem_ld8(acc + F::O + (D == 8 ? (i < 3 ? i : i + 1) * 8 : i * D + c0), r[i]);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            float rest = f(r[1][e]);
            if (G > 2) rest += f(r[G > 2 ? 2 : 1][e]);
            if (G > 3) rest += f(r[G > 3 ? 3 : 1][e]) + f(r[G > 3 ? 4 : 1][e]);
            o[c0 + e] = fmaf(f(r[0][e]) + rest, c, o[c0 + e]);
          }
        }
        return true;
      };
      int b0, h, tile;
      locate(item, b0, h, tile);
      const int qi = tile * F3_QT + row;
      const bool live = b0 + g < p.batch && qi < p.Q;
      const int64_t r = (int64_t)(b0 + g) * p.Q + qi;
      for (int t = 0; t < T; ++t, ++n) {
        const uint32_t sbuf = acc + (n % SB) * F3_KT;
        if (!mbar_wait(&s_full[g * SB + n % SB], (n / SB) & 1, abort_flag, p.status, 68)) { ok = false; break; }
        tc_fence_after();
        float l[F3_KT];
        uint32_t(&u)[32] = reinterpret_cast<uint32_t(&)[32]>(l);
        tmem_ld32(sbuf, u);
        if (BIAS && !mbar_wait(&b_full[st], b_par, abort_flag, p.status, 69)) { ok = false; break; }
        // S being there implies the mask terms (published through k_full)
        const bool masked = mask_flag[g * F::MASKS + slot] != 0;
        const int left = p.Q - t * F3_KT;
        tmem_ld_wait();
        tie32(u);
        {
          const uint8_t* brow = sBias + st * F3_BIAS_BYTES + row * 128;
          auto bias4 = [&](int j4) {      // four keys' bias of this query
            return BIAS ? *reinterpret_cast<const float4*>(brow + ((j4 ^ (row & 7)) << 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
          };
          if (!masked) {
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              const float4 b = bias4(j4);
              const float2 lo = fma2(make_float2(l[j4 * 4], l[j4 * 4 + 1]), make_float2(p.scale, p.scale), make_float2(b.x, b.y));
              const float2 hi = fma2(make_float2(l[j4 * 4 + 2], l[j4 * 4 + 3]), make_float2(p.scale, p.scale), make_float2(b.z, b.w));
              l[j4 * 4] = lo.x; l[j4 * 4 + 1] = lo.y; l[j4 * 4 + 2] = hi.x; l[j4 * 4 + 3] = hi.y;
            }
          } else {
            const float* ms = sMask + (g * F::MASKS + slot) * F3_KT;
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              const float4 m = *reinterpret_cast<const float4*>(ms + j4 * 4), b = bias4(j4);
              l[j4 * 4] = fmaf(l[j4 * 4], p.scale, m.x) + b.x;
              l[j4 * 4 + 1] = fmaf(l[j4 * 4 + 1], p.scale, m.y) + b.y;
              l[j4 * 4 + 2] = fmaf(l[j4 * 4 + 2], p.scale, m.z) + b.z;
              l[j4 * 4 + 3] = fmaf(l[j4 * 4 + 3], p.scale, m.w) + b.w;
            }
          }
          if (left < F3_KT) {      // past the end: not keys at all
#pragma unroll
            for (int j = 0; j < F3_KT; ++j) l[j] = j < left ? l[j] : -INFINITY;
          }
        }
        auto row_max = [&]() {
          float m[4] = {l[0], l[1], l[2], l[3]};
#pragma unroll
          for (int j = 4; j < 32; j += 8) {
#pragma unroll
            for (int e = 0; e < 4; ++e) m[e] = j + 4 + e < 32 ? fmaxf(fmaxf(m[e], l[j + e]), l[j + 4 + e]) : fmaxf(m[e], l[j + e]);
          }
          return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
        };
        // the reference stays while every exponential is at most 2^60
        float top = row_max(), carry = 1.f;      // carry: factor of the product that is still to be added
        if (__any_sync(0xffffffffu, t == 0 || any_far || !(fmaf(top, L2E, -ref2) <= 60.f))) {
          if (p.clamp) {      // changes the result of such rows only: everywhere else what it raises has probability 0 with and without it
#pragma unroll
            for (int j = 0; j < F3_KT; ++j) l[j] = j < left ? fminf(fmaxf(l[j], -1e8f), 1e8f) : l[j];
            top = row_max();
          }
          if (t == 0) {
            ref = top;      // key 0 exists: finite
            ref2 = rintf(ref * L2E);
          } else if (!((far ? (top - ref) * L2E : fmaf(top, L2E, -ref2)) <= 60.f)) {
            const float next = fmaxf(ref, top), next2 = rintf(next * L2E);
            const bool next_far = fabsf(next) > 65536.f;
            // from the base that sum and output have to the one that they get
            carry = f3_ex2(far ? (next_far ? (ref - next) * L2E : fmaf(ref, L2E, -next2)) : next_far ? fmaf(-next, L2E, ref2) : ref2 - next2);
            ref = next;
            ref2 = next2;
            sum *= carry;
            lost *= carry;
#pragma unroll
            for (int e = 0; e < D; ++e) o[e] *= carry;
          }
          far = fabsf(ref) > 65536.f;
          any_far = __any_sync(0xffffffffu, far);
        }
        float shift = -ref2;
        if (any_far) {      // a pass of its own in front
          const float first = far ? ref : 0.f;
          if (far) shift = 0.f;
#pragma unroll
          for (int j = 0; j < F3_KT; ++j) l[j] -= first;
        }
        // exponentials, and the terms of the 16 keys before by truncation: keys 2i, 2i + 1 -> column i of each term
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (c < 2) {
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
              const float2 x = fma2(make_float2(l[c * 16 + j], l[c * 16 + j + 1]), make_float2(L2E, L2E), make_float2(shift, shift));
              l[c * 16 + j] = f3_ex2(x.x);
              l[c * 16 + j + 1] = f3_ex2(x.y);
            }
          }
          if (c == 1 && t > 0 && !add_product(n - 1, carry)) { ok = false; break; }
          if (c > 0) {
            float* x16 = l + (c - 1) * 16;
            float2 a = make_float2(x16[0], x16[1]), b = make_float2(x16[2], x16[3]);
#pragma unroll
            for (int j = 4; j < 16; j += 4) {
              a = add2(a, make_float2(x16[j], x16[j + 1]));
              b = add2(b, make_float2(x16[j + 2], x16[j + 3]));
            }
            a = add2(a, b);
            const float more = (a.x + a.y) - lost, next = sum + more;
            lost = (next - sum) - more;
            sum = next;
            uint32_t w[3][8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              float x = x16[2 * e], y = x16[2 * e + 1];
#pragma unroll
              for (int i = 0; i < 3; ++i) {
                w[i][e] = f3_pack(x, y);
                if (i < 2) bf16_rest(x, y, w[i][e]);
              }
            }
            tmem_st8(sbuf + (c - 1) * 16, w[0]);
            tmem_st8(sbuf + (c - 1) * 16 + 8, w[1]);
            tmem_st8(acc + F::THIRD + (c - 1) * 8, w[2]);      // P V of the tile before has landed: its product has been read
          }
        }
        if (!ok) break;
        __syncwarp();
        if (BIAS && lane == 0) mbar_arrive(&b_empty[st]);
        if (++st == ST) { st = 0; b_par ^= 1; }
        if (++slot == F::MASKS) slot = 0;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[g * SB + n % SB]);
      }
      if (!ok) break;
      // ---- gate and store: the terms of this query's D channels ----
      float4 gate[D / 4];
      if (live) {
        const float* src = p.gate + (int64_t)h * PIECES * p.rows * 8 + r * 8;
#pragma unroll
        for (int i = 0; i < D / 4; ++i) gate[i] = __ldg(reinterpret_cast<const float4*>(src + (i >> 1) * p.rows * 8 + (i & 1) * 4));
      }
      if (!add_product(n - 1, 1.f)) { ok = false; break; }
      if (live) {
        const float inv = 1.0f / sum;
        bf16* dst = p.out + ((int64_t)h * PIECES * p.rows + r) * 8;
#pragma unroll
        for (int pc = 0; pc < PIECES; ++pc) {
          uint32_t w[3][4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float4 g4 = gate[pc * 2 + (e >> 1)];
            float x = o[pc * 8 + 2 * e] * inv * (e & 1 ? g4.z : g4.x), y = o[pc * 8 + 2 * e + 1] * inv * (e & 1 ? g4.w : g4.y);
#pragma unroll
            for (int i = 0; i < 3; ++i) w[i][e] = split_bf16(x, y);
          }
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(dst + i * p.out_stride + pc * p.rows * 8) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
        }
      }
      tc_fence_before();      // the product's read is ordered before this warp's next "P written" arrive
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) drain_after_abort();
  if (warp == 17) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

void configure_attention3() {
#define F3_CASE(D_)                                                                                                          \
  cudaFuncSetAttribute(attention3_kernel<D_, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, F3Form<D_>::SMEM);           \
  cudaFuncSetAttribute(attention3_kernel<D_, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, F3Form<D_>::SMEM);
  F3_CASE(8)
  F3_CASE(16)
  F3_CASE(32)
#undef F3_CASE
}

// Terms in pieces of eight channels over rows (batch, Q), seen as (8-byte halves of a row's piece, batch row, piece, term)
lf_status make_map_term_pieces(lf_context* ctx, CUtensorMap* map, const SplitMatrix& a, int Q, int batch, uint32_t rows, uint32_t streams, uint32_t pieces, uint32_t terms);
lf_status make_map_f32_any(lf_context* ctx, CUtensorMap* map, const void* base, const uint64_t (&dims)[3], const uint64_t (&strides)[2], const uint32_t (&box)[3]);

// A round of the blocks takes a key tile in 1.7 us, with heads of 32 channels in 2.6, after 3 us of start-up, however few of them have work; the mma.sync kernel's
// time follows the number of logits, 1.75 / 2.05 / 5.5 us a million at 8 / 16 / 32 channels.  64 x 64, 4 heads of 32: 13.2 against its 9.5 us;
// 96 x 96: 16.5 against 23.0; 8 rows of 384, 4 x 16: 28.5 against 18.9; 32 rows: 27.6 against 43.4.
bool attention3_wins(const lf_context* ctx, int D, int batch, int Q, int heads) {
  if (D != 8 && D != 16 && D != 32) return false;
  const int64_t items = (int64_t)((batch + F3_STREAMS - 1) / F3_STREAMS) * heads * ((Q + F3_QT - 1) / F3_QT);
  const int64_t rounds = (items + ctx->sm_count - 1) / ctx->sm_count, tiles = (Q + F3_KT - 1) / F3_KT;
  const double here = 3.0 + (double)(rounds * tiles) * (D == 32 ? 2.6 : 1.7);
  const double there = 1e-6 * (double)batch * heads * Q * Q * (D == 8 ? 1.75 : D == 16 ? 2.05 : 5.5);
  return items <= INT32_MAX && here < there;
}

lf_status attention3(lf_context* ctx, ArenaCursor& cur, int D, const SplitMatrix& qkv, const float* gate, const float* bias, int ldb, const float* mask, int batch,
                     int Q, int heads, int transpose, int mask_mode, int clamp, float scale, const SplitMatrix& out) {
  if (cur.dry) return LF_OK;
  CUtensorMap mq, mk, mk1{}, mb{};
  const uint32_t pieces = D / 8;
  LF_TRY(make_map_term_pieces(ctx, &mq, qkv, Q, batch, F3_QT, F3_STREAMS, pieces, 3));
  LF_TRY(make_map_term_pieces(ctx, &mk, qkv, Q, batch, F3_KT, F3_STREAMS, pieces, 3));
  if (D == 8) LF_TRY(make_map_term_pieces(ctx, &mk1, qkv, Q, batch, F3_KT, F3_STREAMS, pieces, 1));
  if (bias)
    LF_TRY(make_map_f32_any(ctx, &mb, bias, {(uint64_t)ldb, (uint64_t)Q, (uint64_t)heads}, {(uint64_t)ldb * 4, (uint64_t)Q * ldb * 4}, {F3_KT, F3_QT, 1}));
  F3Params p{};
  p.batch = batch; p.Q = Q; p.heads = heads; p.qtiles = (Q + F3_QT - 1) / F3_QT; p.ktiles = (Q + F3_KT - 1) / F3_KT;
  p.transpose = transpose; p.mask_mode = mask_mode; p.clamp = clamp; p.scale = scale;
  p.gate = gate; p.rows = (int64_t)batch * Q;
  p.mask = mask; p.out = const_cast<bf16*>(out.p); p.out_stride = out.term_stride;
  p.status = (Status*)ctx->tc_status;
  const int64_t items = (int64_t)((batch + F3_STREAMS - 1) / F3_STREAMS) * heads * p.qtiles;
  const int grid = (int)(items < ctx->sm_count ? items : ctx->sm_count);
  lf_prof_begin(ctx, LF_KERNEL_SIMT);
#define F3_CASE(D_)                                                                                               \
  case D_:                                                                                                        \
    if (bias) lf_launch(ctx, attention3_kernel<D_, true>, grid, F3_THREADS, F3Form<D_>::SMEM, mq, mk, mk1, mb, p);             \
    else lf_launch(ctx, attention3_kernel<D_, false>, grid, F3_THREADS, F3Form<D_>::SMEM, mq, mk, mk1, mb, p);                 \
    break;
  switch (D) { F3_CASE(8) F3_CASE(16) F3_CASE(32) }
#undef F3_CASE
  lf_prof_end(ctx);
  ctx->launches++;
  return LF_OK;
}

}  // namespace tc
