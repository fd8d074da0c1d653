// Differential-attention forward for sm_100a: what the forward kernels share (arguments, tile geometry of the
// D <= 64 kernel).  The kernels themselves: fwd64.cuh (head dims 32 and 64), fwd128.cuh (head dim 128).
//
// A CTA works on one tile of 128 query rows of one (batch, head) at a time.  TMEM (512 columns of 128 lanes x 32 bit) at
// D <= 64: S1 two 64-column buffers [0,128), S2 likewise [128,256), O1 [256,384), O2 [384,512).  Scores are
// produced in sub-tiles of 64 key rows into alternating buffers, so the MMA for sub-tile t+1 runs while the
// softmax warps work on sub-tile t.  P_b (16-bit, two per column) overwrites the first 32 columns of its S
// buffer and is the TMEM A-operand of P_b V.
// Replaces the reference's Triton forward (src/kernel.py:21-207): same math (two online softmaxes,
// O = O1/l1 - lambda O2/l2, RMSNorm * (1 - lambda_init)), but saves lse1, lse2, rstd and A2 = P2 V
// instead of O1/O2.
#pragma once
#include "sm100.cuh"

namespace da {

struct FwdArgs {
  __half* y;          // [B*H, N, 2D] dense; "__half" stands for a 16-bit element here: fp16, or bf16 in the BF kernels
  __half* a2;         // [B*H, N, 2D] dense, branch-2 output P2 V (kept for the backward)
  float* lse1;        // [B*H, N] natural-log logsumexp of s Q1 K1^T
  float* lse2;
  float* rstd;        // [B*H, N] rsqrt(mean(A^2) + eps)   (written also when rms_norm is off)
  const void* lambda_ptr;
  int lambda_dtype;   // 0 = fp16, 1 = fp32, 2 = bf16
  float sm_scale;
  float out_scale;    // 1 - lambda_init
  float eps;
  int rms_norm;
  int n;              // sequence length
  int h;              // heads
  int d;              // real head dim: 64, or 32 (then the 64-wide tiles are zero-filled by TMA beyond column 32 / 64)
  int causal;         // 1: query row i sees key columns j <= i only
  uint32_t drop_thresh;   // dropout: 0 = off, else keep a probability iff its hash byte >= drop_thresh (see sm100.cuh)
  uint32_t seed_lo, seed_hi;
  float drop_scale;       // 256 / (256 - drop_thresh)
  const float* gain;      // NULL, or fp32 [2D]: learnable gain of the output norm; then yg = y * gain is written too
  __half* yg;             // [B*H, N, 2D] dense (only with gain)
  WorkArgs work;          // D <= 64: the tiles of a persistent CTA
};

// key/value tiles of 128 rows that query tile `tile` sees: with a causal mask the tiles right of the diagonal tile are skipped
// altogether.  (The last tile may reach past N: TMA fills those rows with zeros.)
__device__ __forceinline__ int key_tiles(int causal, int n, int tile) {
  const int all = (n + 127) / 128;
  return (causal && tile + 1 < all) ? tile + 1 : all;
}

__device__ __forceinline__ float load_lambda(const void* p, int dtype) {
  if (dtype == 0) return __half2float(*reinterpret_cast<const __half*>(p));
  if (dtype == 2) return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(p));
  return *reinterpret_cast<const float*>(p);
}


namespace fwd64 {
constexpr int BM = 128;            // query rows per CTA
constexpr int BN = 128;            // key/value rows per shared-memory tile
constexpr int SUB = 64;            // key/value rows per MMA sub-tile (one S buffer in TMEM)
constexpr int HD = 64;
constexpr int DV = 128;
constexpr int KS = 3;              // K ring depth
constexpr int VS = 2;              // V ring depth
constexpr int Q_BYTES = BM * HD * 2;            // 16 KB per Q
constexpr int K_BYTES = BN * HD * 2;            // 16 KB per K
constexpr int V_BYTES = BN * DV * 2;            // 32 KB (two 64-column boxes)
constexpr int OFF_Q1 = 0;
constexpr int OFF_Q2 = Q_BYTES;
constexpr int OFF_K = 2 * Q_BYTES;                       // stage s: K1 at +s*2*K_BYTES, K2 right after
constexpr int OFF_V = OFF_K + KS * 2 * K_BYTES;
constexpr int OFF_MISC = OFF_V + VS * V_BYTES;           // barriers, coefficients
constexpr int PRELOAD = 2;                               // key/value tiles requested before the setup barrier (<= KS, VS)
constexpr int STORE_TILE_BYTES = BM * 128;               // epilogue staging: 128 rows x 64 columns x 2 bytes
static_assert(4 * STORE_TILE_BYTES <= VS * V_BYTES && 2 * STORE_TILE_BYTES <= 2 * K_BYTES && KS >= 2,
              "the y / a2 staging tiles reuse the V ring, the gained-y tiles a K stage that the next tile's first load does not fill");
// TMEM columns: S_b buffer u at 128*b + 64*u; O1 at 256, O2 at 384
constexpr int T_O = 256;

}  // namespace fwd64

__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }

// ------------------------------------------------------------------------------------------------
// Softmax of one 64-column sub-tile of one branch.  Thread = query row.
//
// Two warpgroups per branch take alternate sub-tiles (score buffer u = sub-tile & 1 belongs to warpgroup u), so that
// one of them works on its exponentials while the other waits for scores, loads them or stores its probabilities.
// Both accumulate into the same O_b and must use one reference maximum: sub-tile t first finds its own row maximum,
// then takes over the running one that sub-tile t-1 published (`m_row` in shared memory),
// keeps it unless the tile exceeds it by more than 2^8 (always at t = 0, otherwise rare), publishes the result and only
// then starts its exponentials: the serial part between two sub-tiles is the short maximum pass.  Raising the
// maximum rescales O_b once P_b V of sub-tile t-1 has completed, so P never leaves fp16 range and the final division by
// l is exact.  Each warpgroup keeps its own share of the row sum l, relative to the maximum it last saw.
// ------------------------------------------------------------------------------------------------
struct SoftmaxState {
  float m = -INFINITY, l = 0.f;
};

// t_s: this thread's lane and the sub-tile's score columns in TMEM; t_p: where its probabilities go (two per column; may be
// t_s); t_o, O_COLS: the branch's accumulator; first: sub-tile 0; t: its index, only read with dropout; nv: visible columns of this row (the rest get -inf, probability 0); loaded:
// the scores are in registers; wait_m / publish_m: hand-over of the running maximum; wait_pv: P_b V of
// sub-tile t-1 has completed; mid: runs half way through the exponentials; p_free: the
// columns behind t_p may be overwritten.
template <bool BF, bool DROP, int O_COLS, class Loaded, class WaitM, class PublishM, class WaitPv, class Mid, class PFree>
__device__ __forceinline__ void softmax_subtile(SoftmaxState& st, uint32_t t_s, uint32_t t_p, uint32_t t_o, bool first, int t, int nv, float sl2,
                                                volatile float* m_row, const DropWalk& dr, Loaded loaded, WaitM wait_m, PublishM publish_m,
                                                WaitPv wait_pv, Mid mid, PFree p_free) {
  uint32_t sr[64];
  tmem_ld32(t_s, sr);
  tmem_ld32(t_s + 32, sr + 32);
  tc_wait_ld();
  loaded();
  if (nv < 64) {
#pragma unroll
    for (int i = 0; i < 64; ++i)
      if (i >= nv) sr[i] = 0xff800000u;
  }
  float mx[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) mx[c] = __uint_as_float(sr[c]);
#pragma unroll
  for (int i = 2; i < 32; ++i) mx[i & 3] = max3(mx[i & 3], __uint_as_float(sr[2 * i]), __uint_as_float(sr[2 * i + 1]));
  const float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
  float m_prev = -INFINITY;
  bool need = true;
  if (!first) {
    wait_m();
    m_prev = *m_row;
    need = (m_tile - m_prev) * sl2 > 8.f;
  }
  const float m = need ? m_tile : m_prev;
  if (need) *m_row = m;
  publish_m();
  if (__any_sync(0xffffffffu, need) && !first) {
    wait_pv();
    tc_fence_after();
    const float scale = need ? ex2((m_prev - m) * sl2) : 1.f;
#pragma unroll 1
    for (int c = 0; c < O_COLS / 16; ++c) {
      uint32_t o[16];
      tmem_ld16(t_o + c * 16, o);
      tc_wait_ld();
#pragma unroll
      for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * scale);
      tmem_st16(t_o + c * 16, o);
    }
  }
  if (m != st.m) {
    st.l *= ex2(fminf((st.m - m) * sl2, 0.f));        // (at first 0 times something finite, whatever the sign of the scale)
    st.m = m;
  }
  const f32x2 sl2_2 = pk2(sl2, sl2), neg_2 = pk2(-m * sl2, -m * sl2);
  f32x2 sum2[2] = {pk2(0.f, 0.f), pk2(0.f, 0.f)};
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if (i == 16) mid();
    const f32x2 x = fma2(pk2u(sr[2 * i], sr[2 * i + 1]), sl2_2, neg_2);
    float x0, x1;
    up2(x, x0, x1);
    const float p0 = ex2(x0), p1 = ex2(x1);
    sum2[i & 1] = add2(sum2[i & 1], pk2(p0, p1));          // the softmax denominator is taken before dropout
    sr[i] = pack2<BF>(p0, p1);
  }
  float sa, sb;
  up2(add2(sum2[0], sum2[1]), sa, sb);
  st.l += sa + sb;
  if constexpr (DROP) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      sr[i] &= drop_mask_pair(drop_at_col(dr, uint32_t(t * 32), i));
  }
  p_free();
  tmem_st32(t_p, sr);
  tc_wait_st();
  tc_fence_before();
}

}  // namespace da
