// Differential-attention backward for sm_100a, head dim D = 64 (value width 128).
//
// Three kernels (the default form of the backward) replace the reference's single Triton backward
// (src/kernel.py:221-458); bwd_fused64.cuh holds the optional form that merges 2 and 3:
//   1. bwd_pre      per row: dA = RMSNorm-backward(dY) (src/kernel.py:283-290), E1, E2 row sums
//                   (the reference's D1 and D2/(-lambda), :295-296), d(lambda) = -sum E2 with one
//                   atomic per CTA (division-free; the reference divides by lambda+eps, :293).
//   2. bwd_dkdv64   key/value-stationary: S^T, dP^T on tensor cores, dV += (P1-lam P2)^T dA,
//                   dK_b += dS_b^T Q_b (src/kernel.py:410-424).
//   3. bwd_dq64     query-stationary: dQ_b += dS_b K_b (src/kernel.py:426-436); every dQ tile has one
//                   owner CTA, so the accumulation is race-free and deterministic.
// Both tensor-core kernels recompute P_b = exp(s S_b - lse_b) from the saved logsumexp.
#pragma once
#include "sm100.cuh"
#include "fwd.cuh"

namespace da {

struct BwdArgs {
  const __half* y;      // [B*H, N, 2D]
  const __half* a2;     // [B*H, N, 2D]
  const __half* dy;     // [B*H, N, 2D] dense
  const float* lse1;
  const float* lse2;
  const float* rstd;
  __half* da;           // workspace [B*H, N, 2D]
  float4* stats;        // workspace, 16 bytes per row of [B*H, n_pad], NEGATED and interleaved by row pairs (see stat_row):
                        // x = -lse1*log2e, y = -(lse2*log2e - log2|lam|), z = -E1, w = -sg*E2 with sg = -sign(lam)
  __half* dq1; __half* dq2; __half* dk1; __half* dk2; __half* dv;   // dense
  float* dlambda;
  const void* lambda_ptr;
  int lambda_dtype;
  float sm_scale;
  float out_scale;      // 1 - lambda_init
  int rms_norm;
  int n;
  int h;
  int d;                // real head dim (64, or 32 with zero-filled padding in the 64-wide tiles)
  int causal;           // 1: query row i sees key columns j <= i only
  int n_pad;            // N rounded up to 128: row pitch of `stats` per (batch, head); rows N..n_pad-1 hold
                        // x = y = -inf, z = w = 0, which makes the probabilities of out-of-range query rows exactly 0
  long long rows;       // B*H*N
  uint32_t drop_thresh; // dropout: 0 = off (see sm100.cuh); must equal the forward's
  uint32_t seed_lo, seed_hi;
  float drop_scale;     // 256 / (256 - drop_thresh)
  const float* gain;    // NULL, or fp32 [2D]: then dy is the gradient of y * gain, and sum_rows(dy * y) is added to dgain
  float* dgain;         // fp32 [2D]
  float* dq_acc;        // NULL, or workspace fp32 [2][B*H][n_pad][64]: partial sums of dQ1, dQ2 of the single-pass kernel
                        // (bwd_fused64.cuh); zeroed by the preprocess kernel, converted by the finishing kernel
  long long dq_acc_f4;  // its size in float4 units
  WorkArgs qwork;       // D <= 64: the query tiles of a persistent dQ CTA
  WorkArgs kwork;       // D <= 64: the key tiles of a persistent dK/dV CTA
};

// Row statistics, interleaved by pairs of rows so that a kernel that walks two neighbouring rows (the key-side
// kernels: two query columns of a thread's 16) gets each quantity of both rows in one 64-bit register pair, the
// operand form of the packed fp32 instructions: rows 2q and 2q+1 occupy floats
//   [8q .. 8q+8) = { x(2q), x(2q+1), y(2q), y(2q+1), z(2q), z(2q+1), w(2q), w(2q+1) }.
// idx = (batch*head) * n_pad + row; n_pad is even, so a pair never straddles two heads.
__device__ __forceinline__ void stat_store(float4* stats, long long idx, float4 v) {
  float* f = reinterpret_cast<float*>(stats + (idx & ~1ll)) + (idx & 1);
  f[0] = v.x; f[2] = v.y; f[4] = v.z; f[6] = v.w;
}
__device__ __forceinline__ float4 stat_row(const float4* stats, size_t idx) {
  const float* f = reinterpret_cast<const float*>(stats + (idx & ~size_t(1))) + (idx & 1);
  return make_float4(f[0], f[2], f[4], f[6]);
}

// ------------------------------------------------------------------------------------------------
// 1. preprocess: HBM-bound (three [N, 2D] tensors in, one out).  A lane holds 8 elements (16-byte loads and stores), DV / 8
// lanes share a row, so a warp works on 4, 2 or 1 rows at head dims 32, 64, 128 and a row's sums take 3 to 5 shuffles.
// One such row set per warp and trip, four CTAs per SM: the other warps keep enough bytes in flight (two or four sets loaded before
// the first reduction cost registers and were slower: 60 / 70 / 93 us at B4 H16 N4096 D64).  Against a row per warp with 4, 8 and 16
// bytes per lane: B8 H16 N2048 D32 64 -> 31 us, B4 H16 N4096 D64 84 -> 60 (4.6 TB/s), B2 H8 N8192 D128 81 -> 67.
// ------------------------------------------------------------------------------------------------
template <int DV, bool BF>   // value width 64, 128, 256; BF: bf16 tensors
__global__ void __launch_bounds__(256, 4) diffattn_bwd_pre_kernel(const BwdArgs args) {
  constexpr int LANES = DV / 8, SETS = 32 / LANES;      // lanes per row, rows per warp
  griddep_launch();      // the first tensor-core kernel may set itself up; it waits for this one before it reads dA or the statistics
  constexpr float LOG2E = 1.4426950408889634f;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int sub = lane % LANES;                          // this lane's 8 columns: [8 sub, 8 sub + 8)
  const uint32_t rows = uint32_t(args.rows), n = uint32_t(args.n);      // (rows < 2^31: a row is at least 128 bytes)
  const float lam = load_lambda(args.lambda_ptr, args.lambda_dtype);
  const float c = args.out_scale;
  float dl_acc = 0.f;
  __shared__ float red[8];
  // learnable gain of the output norm: Y_out = Y * gain, so dY = dY_out * gain and d(gain) = sum over rows of dY_out * Y
  const bool has_gain = args.gain != nullptr;
  float gn[8], dg_acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) { gn[i] = has_gain ? args.gain[sub * 8 + i] : 1.f; dg_acc[i] = 0.f; }
  __shared__ float dg_red[8][DV];
  // the dQ partial sums of the single-pass backward start from zero
  if (args.dq_acc) {
    float4* z = reinterpret_cast<float4*>(args.dq_acc);
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < args.dq_acc_f4; t += (long long)gridDim.x * blockDim.x)
      z[t] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // rows N..n_pad-1 of every (batch, head) in `stats`: neutral values (see BwdArgs::n_pad)
  if (const int pad = args.n_pad - args.n) {
    const long long total = args.rows / args.n * pad;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
      const long long bh_i = i / pad;
      stat_store(args.stats, bh_i * args.n_pad + args.n + (i - bh_i * pad), make_float4(-INFINITY, -INFINITY, 0.f, 0.f));
    }
  }

  const uint32_t step = gridDim.x * (blockDim.x >> 5) * SETS;           // rows of one trip of the grid
  for (uint32_t row = (blockIdx.x * (blockDim.x >> 5) + warp) * SETS + lane / LANES; row - lane / LANES < rows; row += step) {
    uint4 vd, vy, va;
    float rstd = 1.f, lse1 = 0.f, lse2 = 0.f;
    vd = vy = va = make_uint4(0, 0, 0, 0);               // (lanes past the last row take part in the shuffles)
    if (row < rows) {
      const size_t off = size_t(row) * DV + sub * 8;
      vd = *reinterpret_cast<const uint4*>(args.dy + off);
      vy = *reinterpret_cast<const uint4*>(args.y + off);
      va = *reinterpret_cast<const uint4*>(args.a2 + off);
      rstd = args.rstd[row]; lse1 = args.lse1[row]; lse2 = args.lse2[row];
    }
    float dy[8], yv[8];
    const uint32_t wd[4] = {vd.x, vd.y, vd.z, vd.w}, wy[4] = {vy.x, vy.y, vy.z, vy.w};
    const uint32_t wa[4] = {va.x, va.y, va.z, va.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 fd = unpack2<BF>(wd[i]), fy = unpack2<BF>(wy[i]);
      dy[2 * i] = fd.x; dy[2 * i + 1] = fd.y;
      yv[2 * i] = fy.x; yv[2 * i + 1] = fy.y;
    }
    if (has_gain) {
#pragma unroll
      for (int i = 0; i < 8; ++i) { dg_acc[i] = fmaf(dy[i], yv[i], dg_acc[i]); dy[i] *= gn[i]; }
    }
    float k1 = 1.f, k2 = 0.f, k3 = 1.f;
    if (args.rms_norm) {
      // Y = c r A  =>  A = Y/(c r),  dA = r (c dY - Y (dY.Y) / (c Dv));  c == 0 gives dA = 0
      float t = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) t += dy[i] * yv[i];
#pragma unroll
      for (int o = LANES / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      const float inv_c = c != 0.f ? 1.f / c : 0.f;
      k1 = rstd * c; k2 = rstd * inv_c * t * (1.f / DV); k3 = inv_c / rstd;
    }
    // round dA to the 16-bit type first: the row sums below must agree with what the MMAs will see
    uint32_t hda[4];
    float e2 = 0.f, ea = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      hda[i] = args.rms_norm ? pack2<BF>(k1 * dy[2 * i] - k2 * yv[2 * i], k1 * dy[2 * i + 1] - k2 * yv[2 * i + 1])
                             : pack2<BF>(dy[2 * i], dy[2 * i + 1]);
      const float2 d = unpack2<BF>(hda[i]), a2 = unpack2<BF>(wa[i]);
      e2 += d.x * a2.x + d.y * a2.y;
      ea += d.x * (yv[2 * i] * k3) + d.y * (yv[2 * i + 1] * k3);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
      e2 += __shfl_xor_sync(0xffffffffu, e2, o);
      ea += __shfl_xor_sync(0xffffffffu, ea, o);
    }
    if (row < rows) {
      *reinterpret_cast<uint4*>(args.da + size_t(row) * DV + sub * 8) = make_uint4(hda[0], hda[1], hda[2], hda[3]);
      if (sub == 0) {
        // E1 - lam E2 = rowsum(dA * A).  lambda is folded into the branch-2 statistics so that the tensor-core
        // kernels need no multiply for it: with P2' = |lam| P2 = 2^(s S2 log2e - y) and sg = -sign(lam),
        // -lam P2 = sg P2' and -lam P2 (dP - E2) = P2' (sg dP - w).  lam = 0 gives y = +inf, P2' = 0.
        const float sg = lam < 0.f ? 1.f : -1.f;
        const uint32_t bh_i = row / n;
        stat_store(args.stats, (long long)bh_i * args.n_pad + (row - bh_i * n),
                   make_float4(-lse1 * LOG2E, log2f(fabsf(lam)) - lse2 * LOG2E, -(ea + lam * e2), -sg * e2));
        dl_acc -= e2;
      }
    }
  }
#pragma unroll
  for (int o = LANES; o < 32; o <<= 1) {       // the row sets of the warp
    dl_acc += __shfl_xor_sync(0xffffffffu, dl_acc, o);
    if (has_gain) {
#pragma unroll
      for (int i = 0; i < 8; ++i) dg_acc[i] += __shfl_xor_sync(0xffffffffu, dg_acc[i], o);
    }
  }
  if (lane == 0) red[warp] = dl_acc;
  if (has_gain && lane < LANES) {
#pragma unroll
    for (int i = 0; i < 8; ++i) dg_red[warp][sub * 8 + i] = dg_acc[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int i = 0; i < (blockDim.x >> 5); ++i) s += red[i];
    atomicAdd(args.dlambda, s);
  }
  if (has_gain && threadIdx.x < DV) {
    float s = 0.f;
    for (int i = 0; i < (blockDim.x >> 5); ++i) s += dg_red[i][threadIdx.x];
    atomicAdd(args.dgain + threadIdx.x, s);       // one atomic per column and CTA
  }
}

// ------------------------------------------------------------------------------------------------
// 2. dK1, dK2, dV: a CTA works on 128 key/value rows of one (batch, head) at a time; query tiles of 64 stream by.
// TMEM: dV [0,128) dK1 [128,192) dK2 [192,256) | scores S1^T [256,320) S2^T [320,384) dP^T [384,448) |
// fp16 A-operands dS1^T [448,480) dS2^T [480,512).  Thread = key row; four warpgroups, warpgroup g handles
// query columns [16g, 16g+16) (more resident warps per scheduler hide the exp-unit and TMEM latencies).  The warpgroups pull their scores into registers and release the score columns at once,
// so the MMAs of tile i+1 run under the elementwise work of tile i.  dS_b^T goes back to TMEM (A-operand of
// dK_b += dS_b^T Q_b); (P1 - lam P2)^T goes to a double-buffered K-major shared-memory tile (A-operand of
// dV += Pc^T dA) because TMEM has no columns left for it.
// ------------------------------------------------------------------------------------------------
// Per-column statistics are read from shared memory DA_PF columns ahead of their use, by volatile loads that keep
// that order: every thread of a warp reads the same 16 bytes per column, and left to the compiler the loads sat
// right before their consumers with the shared-memory pipe's loaded latency exposed 16 times per tile (at
// B4 H16 N4096 D64 the dK/dV kernel took 1.33 ms that way; 1.22 ms with two columns ahead, 1.23 with four).
#ifndef DA_PF
#define DA_PF 2
#endif
__device__ __forceinline__ float4 lds_v4(const float4* p) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_u32(p)));
  return v;
}
namespace dkdv64 {
// (ring depth 4 with a single Pc buffer, and depth 3 with a single buffer, measured within noise of this setting)
constexpr int BKV = 128, BQ = 64, HD = 64, DV = 128, ST = 3, PCBUF = 2;
constexpr int K_BYTES = BKV * HD * 2;       // 16 KB
constexpr int V_BYTES = BKV * DV * 2;       // 32 KB, two boxes of 16 KB
constexpr int Q_BYTES = BQ * HD * 2;        // 8 KB
constexpr int DA_BYTES = BQ * DV * 2;       // 16 KB, two boxes of 8 KB
constexpr int STAT_BYTES = BQ * 16;         // 1 KB
constexpr int STAGE_BYTES = 2 * Q_BYTES + DA_BYTES + STAT_BYTES;   // 33 KB
static_assert(STAGE_BYTES % 1024 == 0 && STAGE_BYTES >= V_BYTES && V_BYTES == 2 * K_BYTES && ST == 3, "two ring slots take the epilogue's tiles");
constexpr int PC_BYTES = BKV * BQ * 2;      // 16 KB per buffer
constexpr int OFF_K1 = 0, OFF_K2 = K_BYTES, OFF_V = 2 * K_BYTES;
constexpr int OFF_PC = OFF_V + V_BYTES;                            // 64 KB
constexpr int OFF_STAGE = OFF_PC + PCBUF * PC_BYTES;                   // 96 KB
constexpr int OFF_MISC = OFF_STAGE + ST * STAGE_BYTES;             // 195 KB
constexpr int MISC_BYTES = 1024;
constexpr int SMEM_BYTES = OFF_MISC + MISC_BYTES + 1024;
constexpr int NWG = 4;                      // elementwise warpgroups; warpgroup g owns query columns [16g, 16g+16)
constexpr int NUM_THREADS = NWG * 128 + 128;                      // + TMA warp and three MMA-issuing warps, one per scheduler
constexpr int WARP_TMA = NWG * 4, WARP_MMA = NWG * 4 + 1;         // issuers: WARP_MMA (S^T), +1 (dP^T), +2 (dV, dK)
// Named barriers: output operands of a tile written (+ tile & 1), its scores in registers, the accumulators of a key tile in
// registers, its gradients in shared memory.  (A wait on an mbarrier costs an
// issuer 110-300 clocks even when the phase is long complete, a named barrier a tenth.)
constexpr int NB_E = 1, NB_SFREE = 3, NB_ACC = 4, NB_STORE = 5;
constexpr int NB_E_THREADS = NWG * 128 + 32, NB_SFREE_THREADS = NWG * 128 + 64;
constexpr int T_DV = 0, T_DK1 = 128, T_DK2 = 192, T_S1 = 256, T_S2 = 320, T_DP = 384, T_DS1 = 448, T_DS2 = 480;
struct Misc {
  uint64_t bar_kv, kv_empty;
  uint64_t full[ST], empty[ST];
  uint64_t s_full;      // scores of a tile written (MMA -> warpgroups)
  uint64_t mma_done;    // dV/dK MMAs of a tile completed (operand buffers reusable)
  uint64_t acc_full;
  uint32_t tmem_slot;
  int abort_flag;
};
}  // namespace dkdv64

template <bool BF, bool DROP, bool LIST>
__global__ void __launch_bounds__(dkdv64::NUM_THREADS, 1)
diffattn_bwd_dkdv64_kernel(const __grid_constant__ CUtensorMap tm_q1, const __grid_constant__ CUtensorMap tm_q2,
                           const __grid_constant__ CUtensorMap tm_k1, const __grid_constant__ CUtensorMap tm_k2,
                           const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_da,
                           const __grid_constant__ CUtensorMap tm_dk1, const __grid_constant__ CUtensorMap tm_dk2,
                           const __grid_constant__ CUtensorMap tm_dv, const BwdArgs args) {
  using namespace dkdv64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Misc* misc = reinterpret_cast<Misc*>(smem + OFF_MISC);
  volatile int* abort_flag = &misc->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Persistent: this CTA works on the key tiles of its WorkList one after the other; rings and barriers run on from one to the
  // next (each role counts along by itself), so the next tile's operands arrive and its first scores are computed under this
  // tile's last pass and epilogue, and the gradients leave under the next tile's first passes.
  // Against one CTA per tile: B8 H16 N512 D64 63 -> 58 us, causal 49 -> 42, B32 H16 N128 D64 35 -> 29, B4 H16 N4096 unchanged.
  // (With dK1 and dK2 staged in the Pc buffers one more ring slot could be refilled early, B32 H16 N128 25 us, but the wait that
  // the first Pc stores then need sat in the loop over the query tiles and cost it 4 %.)
  WorkList<LIST> work(args.kwork);
  // the last query tiles may reach past N (zero dA, neutral statistics); under the causal mask only query tiles
  // from the diagonal on see a key tile: tiles i0 .. nq_all-1, visited with the local index i (tile i0 + i)
  const int nq_all = args.n_pad / BQ;
  auto first_q = [&](int kv_tile) { return args.causal ? kv_tile * (BKV / BQ) : 0; };

  if (warp == WARP_TMA && lane == 0) {
    mbar_init(&misc->bar_kv, 1);
    mbar_init(&misc->kv_empty, 2);
    for (int i = 0; i < ST; ++i) { mbar_init(&misc->full[i], 1); mbar_init(&misc->empty[i], 1); }
    mbar_init(&misc->s_full, 2);
    mbar_init(&misc->mma_done, 1);
    mbar_init(&misc->acc_full, 1);
    misc->abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == WARP_MMA) tmem_alloc(&misc->tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&misc->tmem_slot);

  // (Requesting the resident tiles and the first ring pass before the setup barrier, as the forward and the dQ
  // kernel do, measured 3 % slower here.)
  if (warp == WARP_TMA) {
    bool ok = true;
    int st = 0, it = 0;
    uint32_t par = 1;                    // parity of an "empty" wait of the ring (the first pass never waits)
    WorkItem last{0, 0};
    // Gradients leave through the TMA engine, from the ring slots that the next tile fills second (dK1, dK2) and third (dV).
    // The engine clips at the tensor's bounds: key rows past the sequence end and, for head dim 32, the padding columns are not
    // written.
    auto store = [&](int second) {
      named_bar_sync(NB_STORE, NB_E_THREADS);
      if (elect_one()) {
        if (!*abort_flag) {
          const uint8_t* dk = smem + OFF_STAGE + second * STAGE_BYTES;
          const uint8_t* dv = smem + OFF_STAGE + (second + 1) % ST * STAGE_BYTES;
          tma_store_4d(dv, &tm_dv, 0, last.tile * BKV, last.bh, 0);
          if (args.d > 32) tma_store_4d(dv + V_BYTES / 2, &tm_dv, 64, last.tile * BKV, last.bh, 0);
          tma_store_4d(dk, &tm_dk1, 0, last.tile * BKV, last.bh, 0);
          tma_store_4d(dk + K_BYTES, &tm_dk2, 0, last.tile * BKV, last.bh, 0);
          tma_store_commit();
          tma_store_wait_read();
        }
      }
      __syncwarp();
    };
    for (; work.valid(); ++it, work.next()) {
      const WorkItem wi = work.item();
      const int b_idx = wi.bh / args.h, h_idx = wi.bh % args.h, i0 = first_q(wi.tile), nq = nq_all - i0;
      if (it > 0) ok = ok && mbar_wait_warp(&misc->kv_empty, (it - 1) & 1, abort_flag, 402, it) && !*abort_flag;      // (as mbar_wait_free)
      if (ok && elect_one()) {
        mbar_expect_tx(&misc->bar_kv, 2 * K_BYTES + V_BYTES);
        tma_load_4d(smem + OFF_K1, &tm_k1, &misc->bar_kv, 0, wi.tile * BKV, h_idx, b_idx);
        tma_load_4d(smem + OFF_K2, &tm_k2, &misc->bar_kv, 0, wi.tile * BKV, h_idx, b_idx);
        tma_load_4d(smem + OFF_V, &tm_v, &misc->bar_kv, 0, wi.tile * BKV, h_idx, b_idx);
        tma_load_4d(smem + OFF_V + V_BYTES / 2, &tm_v, &misc->bar_kv, 64, wi.tile * BKV, h_idx, b_idx);
        if (it == 0) {
          tma_prefetch_desc(&tm_dv); tma_prefetch_desc(&tm_dk1); tma_prefetch_desc(&tm_dk2);
          griddep_wait();        // dA and the statistics come from the preprocess kernel
          griddep_launch();      // dQ CTAs may set themselves up on the SMs that this grid's last wave leaves idle
        }
      }
      __syncwarp();
      for (int i = 0; i < nq; ++i) {
        if (i == 1 && it > 0) store(st);     // (every tile has at least two query tiles)
        ok = ok && mbar_wait_warp(&misc->empty[st], par, abort_flag, 401, i) && !*abort_flag;
        if (ok && elect_one()) {
          uint8_t* sp = smem + OFF_STAGE + st * STAGE_BYTES;
          mbar_expect_tx(&misc->full[st], STAGE_BYTES);
          tma_load_4d(sp, &tm_q1, &misc->full[st], 0, (i0 + i) * BQ, h_idx, b_idx);
          tma_load_4d(sp + Q_BYTES, &tm_q2, &misc->full[st], 0, (i0 + i) * BQ, h_idx, b_idx);
          tma_load_4d(sp + 2 * Q_BYTES, &tm_da, &misc->full[st], 0, (i0 + i) * BQ, wi.bh, 0);
          tma_load_4d(sp + 2 * Q_BYTES + DA_BYTES / 2, &tm_da, &misc->full[st], 64, (i0 + i) * BQ, wi.bh, 0);
          bulk_load_1d(sp + 2 * Q_BYTES + DA_BYTES, args.stats + (size_t(wi.bh) * args.n_pad + size_t(i0 + i) * BQ), STAT_BYTES, &misc->full[st]);
        }
        __syncwarp();
        if (++st == ST) { st = 0; par ^= 1; }
      }
      last = wi;
    }
    store((st + 1) % ST);
  } else if (warp == WARP_MMA || warp == WARP_MMA + 1) {
    // ---- score issuers: warp WARP_MMA issues S1^T and S2^T of every tile, warp WARP_MMA + 1 issues dP^T.
    // MMA issue is spread over three warps on three schedulers (these two and the output issuer below): one warp
    // issuing all 32 MMAs of a tile takes ~300 clocks per tile from the elementwise warps of its scheduler, and
    // every tile waits for that slowest quarter.  One elected thread per warp; descriptors advance by 32-bit adds.
    // (Every trip makes its barrier calls, issues and commits whether or not a wait for a load gave up, see mbar_wait_issued.)
    const bool is_dp = warp == WARP_MMA + 1;
    constexpr uint32_t IDESC_S = make_idesc(BKV, BQ, 0, 0, BF);     // S^T = K Q^T, dP^T = V dA^T
    const uint32_t k1_lo = sdesc_lo(smem_u32(smem + OFF_K1)), k2_lo = sdesc_lo(smem_u32(smem + OFF_K2));
    const uint32_t v_lo = sdesc_lo(smem_u32(smem + OFF_V));
    const uint32_t st_lo0 = sdesc_lo(smem_u32(smem + OFF_STAGE));
    const uint32_t tb = tmem_base;
    const int kd = args.d >> 4;       // 16-deep MMA steps over the head dim (value width: twice as many): head dim 32 skips the zero padding
    auto issue_scores = [&](uint32_t sp_lo) {
      if (!is_dp) {
#pragma unroll
        for (int k = 0; k < HD / 16; ++k)
          if (k < kd) mma_ss_lo(tb + T_S1, k1_lo + k * 2, sp_lo + k * 2, IDESC_S, k > 0);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k)
          if (k < kd) mma_ss_lo(tb + T_S2, k2_lo + k * 2, sp_lo + (Q_BYTES >> 4) + k * 2, IDESC_S, k > 0);
      } else {
#pragma unroll
        for (int k = 0; k < DV / 16; ++k)
          if (k < 2 * kd)
            mma_ss_lo(tb + T_DP, v_lo + (k / 4) * ((V_BYTES / 2) >> 4) + (k % 4) * 2,
                      sp_lo + ((2 * Q_BYTES) >> 4) + (k / 4) * ((DA_BYTES / 2) >> 4) + (k % 4) * 2, IDESC_S, k > 0);
      }
      mma_commit(&misc->s_full);        // two arrivals per tile: this warp's and the other score issuer's
    };
    griddep_wait();
    bool ok = true;
    int st = 0;
    uint32_t par = 0;
    for (int it = 0; work.valid(); ++it, work.next()) {
      const int nq = nq_all - first_q(work.item().tile);
      ok = ok && mbar_wait_warp(&misc->bar_kv, it & 1, abort_flag, 501, it);
      for (int i = 0; i < nq; ++i) {
        ok = ok && mbar_wait_warp(&misc->full[st], par, abort_flag, 502, i);      // under the warpgroups' pass over the tile before
        if (it > 0 || i > 0) named_bar_sync(NB_SFREE, NB_SFREE_THREADS);          // the scores before these are in registers
        tc_fence_after();
        if (elect_one()) {
          issue_scores(st_lo0 + st * (STAGE_BYTES >> 4));
          if (i == nq - 1) mma_commit(&misc->kv_empty);
        }
        __syncwarp();
        if (++st == ST) { st = 0; par ^= 1; }
      }
    }
    named_bar_sync(NB_SFREE, NB_SFREE_THREADS);
  } else if (warp == WARP_MMA + 2) {
    // ---- output issuer: dV += Pc^T dA, dK_b += dS_b^T Q_b of tile i once the warpgroups have written their operands
    // head dim 32: only the real 64 value columns / 32 head columns are produced
    const uint32_t IDESC_DV = make_idesc(BKV, 2 * args.d, 0, 1, BF);    // dV += Pc^T dA   (Pc K-major smem, dA MN-major)
    const uint32_t IDESC_DK = make_idesc(BKV, args.d, 0, 1, BF);        // dK += dS^T Q    (dS^T in TMEM, Q MN-major)
    const uint32_t pc_lo0 = sdesc_lo(smem_u32(smem + OFF_PC));
    const uint32_t st_lo0 = sdesc_lo(smem_u32(smem + OFF_STAGE));
    constexpr uint32_t DA_MN_LBO = ((DA_BYTES / 2) >> 4) << 16;   // dA as MN-major B: 64-column atoms 8 KB apart
    const uint32_t tb = tmem_base;
    int st = 0;
    for (int it = 0; work.valid(); ++it, work.next()) {
      const int nq = nq_all - first_q(work.item().tile);
      for (int i = 0; i < nq; ++i) {
        const uint32_t sp_lo = st_lo0 + st * (STAGE_BYTES >> 4);
        const uint32_t pc_lo = pc_lo0 + (i % PCBUF) * (PC_BYTES >> 4);
        // operands of tile i written: stage i was loaded and the score MMAs reading it have completed
        if (it > 0 && i == 0) named_bar_sync(NB_ACC, NB_E_THREADS);      // the accumulators of the key tile before are in registers
        named_bar_sync(NB_E + (i & 1), NB_E_THREADS);
        tc_fence_after();
        if (elect_one()) {
          const uint32_t first = i > 0;
#pragma unroll
          for (int k = 0; k < BQ / 16; ++k)
            mma_ss_lo(tb + T_DV, pc_lo + k * 2, sp_lo + ((2 * Q_BYTES) >> 4) + DA_MN_LBO - (1u << 16) + k * (2048 >> 4), IDESC_DV,
                      k > 0 ? 1u : first);
#pragma unroll
          for (int k = 0; k < BQ / 16; ++k)
            mma_ts_lo(tb + T_DK1, tb + T_DS1 + k * 8, sp_lo + k * (2048 >> 4), IDESC_DK, k > 0 ? 1u : first);
#pragma unroll
          for (int k = 0; k < BQ / 16; ++k)
            mma_ts_lo(tb + T_DK2, tb + T_DS2 + k * 8, sp_lo + (Q_BYTES >> 4) + k * (2048 >> 4), IDESC_DK, k > 0 ? 1u : first);
          mma_commit(&misc->mma_done);
          mma_commit(&misc->empty[st]);
          if (i == nq - 1) mma_commit(&misc->acc_full);
        }
        __syncwarp();
        if (++st == ST) st = 0;
      }
    }
  } else {
    const int g = warp >> 2;                       // warpgroup: query columns [16g, 16g+16) of every tile
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
    const uint32_t tb = tmem_base + lane_base;
    const float sl2 = args.sm_scale * 1.4426950408889634f;
    const float sg = load_lambda(args.lambda_ptr, args.lambda_dtype) < 0.f ? 1.f : -1.f;   // -sign(lambda)
    const f32x2 dscale_2 = pk2(args.drop_scale, args.drop_scale), sgd_2 = pk2(sg * args.drop_scale, sg * args.drop_scale);     // DROP only
    const f32x2 sl2_2 = pk2(sl2, sl2), sg_2 = pk2(sg, sg);
    griddep_wait();
    uint32_t s_ready = 0;            // answers of the early probes (see mbar_probe)
    int st = 0;
    for (; work.valid(); work.next()) {
      {
        // (nq is even, so the per-tile barriers' phases have parity i & 1 in every key tile)
        const WorkItem wi = work.item();
        const int kv_tile = wi.tile, i0 = first_q(kv_tile), nq = nq_all - i0;
        // dropout: this thread owns key column kv_tile*BKV + row; a hash covers two consecutive query rows of it
        DropWalk dw1, dw2;
        if constexpr (DROP) {
          const uint32_t col2 = uint32_t(kv_tile * BKV + row) >> 1;
          dw1 = drop_walk_col(drop_key(args.seed_lo, args.seed_hi, uint32_t(wi.bh), 0u), col2, row & 1, args.drop_thresh);
          dw2 = drop_walk_col(drop_key(args.seed_lo, args.seed_hi, uint32_t(wi.bh), 1u), col2, row & 1, args.drop_thresh);
        }
        for (int i = 0; i < nq; ++i) {
          const float4* stats = reinterpret_cast<const float4*>(smem + OFF_STAGE + st * STAGE_BYTES + 2 * Q_BYTES + DA_BYTES) + g * 16;
          if (!__all_sync(0xffffffffu, s_ready)) mbar_wait_issued_warp(&misc->s_full, i & 1, abort_flag, 601 + g, i);
          tc_fence_after();
          uint32_t s1[16], s2[16], dp[16];
          tmem_ld16(tb + T_S1 + g * 16, s1);
          tmem_ld16(tb + T_S2 + g * 16, s2);
          tmem_ld16(tb + T_DP + g * 16, dp);
          tc_wait_ld();
          tc_fence_before();
          named_bar_arrive(NB_SFREE, NB_SFREE_THREADS);
          if (args.causal) {
            // this thread's key row sees query columns >= its own index only: the first c0 columns of its 16 are hidden
            const int c0 = row - (i * BQ + g * 16);          // kv_tile * BKV = i0 * BQ
            if (c0 > 0) {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (j < c0) { s1[j] = 0xff800000u; s2[j] = 0xff800000u; }
            }
          }
          uint32_t pc[8], d1[8], d2[8];
          // statistics of the next DA_PF / 2 column pairs (see lds_v4): {x0, x1, y0, y1} and {z0, z1, w0, w1}, negated
          float4 sva[DA_PF / 2], svb[DA_PF / 2];
#pragma unroll
          for (int j = 0; j < DA_PF / 2; ++j) { sva[j] = lds_v4(stats + 2 * j); svb[j] = lds_v4(stats + 2 * j + 1); }
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) {
            const float4 sa = sva[jj % (DA_PF / 2)], sb = svb[jj % (DA_PF / 2)];
            if (jj + DA_PF / 2 < 8) {
              sva[jj % (DA_PF / 2)] = lds_v4(stats + 2 * (jj + DA_PF / 2));
              svb[jj % (DA_PF / 2)] = lds_v4(stats + 2 * (jj + DA_PF / 2) + 1);
            }
            float x10, x11, x20, x21;
            up2(fma2(pk2u(s1[2 * jj], s1[2 * jj + 1]), sl2_2, pk2(sa.x, sa.y)), x10, x11);
            up2(fma2(pk2u(s2[2 * jj], s2[2 * jj + 1]), sl2_2, pk2(sa.z, sa.w)), x20, x21);
            const float p10 = ex2(x10), p11 = ex2(x11);
            const float p20 = ex2(x20), p21 = ex2(x21);     // |lam| P2
            float pcv[2], d1v[2], d2v[2];
            if constexpr (DROP) {
              // dropped positions contribute neither to dV nor to dP; kept ones carry the factor 1/(1-p)
              const uint32_t f1 = drop_at_row(dw1, uint32_t((i0 + i) * (BQ / 2) + g * 8), jj), f2 = drop_at_row(dw2, uint32_t((i0 + i) * (BQ / 2) + g * 8), jj);
              const uint32_t m10 = drop_mask_first(f1), m11 = drop_mask_second(f1), m20 = drop_mask_first(f2), m21 = drop_mask_second(f2);
              const uint32_t dp0 = dp[2 * jj], dp1 = dp[2 * jj + 1];
              up2(fma2(sgd_2, pk2u(__float_as_uint(p20) & m20, __float_as_uint(p21) & m21),
                       mul2(dscale_2, pk2u(__float_as_uint(p10) & m10, __float_as_uint(p11) & m11))), pcv[0], pcv[1]);
              up2(mul2(pk2(p10, p11), fma2(dscale_2, pk2u(dp0 & m10, dp1 & m11), pk2(sb.x, sb.y))), d1v[0], d1v[1]);
              up2(mul2(pk2(p20, p21), fma2(sgd_2, pk2u(dp0 & m20, dp1 & m21), pk2(sb.z, sb.w))), d2v[0], d2v[1]);
            } else {
              const f32x2 p1_2 = pk2(p10, p11), p2_2 = pk2(p20, p21), dp_2 = pk2u(dp[2 * jj], dp[2 * jj + 1]);
              up2(fma2(sg_2, p2_2, p1_2), pcv[0], pcv[1]);
              up2(mul2(p1_2, add2(dp_2, pk2(sb.x, sb.y))), d1v[0], d1v[1]);
              up2(mul2(p2_2, fma2(sg_2, dp_2, pk2(sb.z, sb.w))), d2v[0], d2v[1]);
            }
            pc[jj] = pack2<BF>(pcv[0], pcv[1]);
            d1[jj] = pack2<BF>(d1v[0], d1v[1]);
            d2[jj] = pack2<BF>(d2v[0], d2v[1]);
          }
          // The dS^T columns are free once the output MMAs of tile i-1 have completed (mma_done); the Pc buffer of this
          // tile was last read by tile i-2, whose completion the previous trip waited for.  So the Pc stores and their
          // proxy fence go first, under the latency of an early look at mma_done (see mbar_probe).
          static_assert(PCBUF == 2, "the Pc buffer of tile i must be the one tile i-2 used");
          const uint32_t md_ready = i > 0 ? mbar_probe(&misc->mma_done, (i - 1) & 1) : 1u;
          // Pc tile [128 key rows][64 query columns] fp16, 128-byte rows, 16-byte chunks XOR-swizzled by row
          {
            uint8_t* prow = smem + OFF_PC + (i % PCBUF) * PC_BYTES + row * 128;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int chunk = (g * 2 + c) ^ (row & 7);
              *reinterpret_cast<uint4*>(prow + chunk * 16) = make_uint4(pc[4 * c], pc[4 * c + 1], pc[4 * c + 2], pc[4 * c + 3]);
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          if (i > 0) {
            if (!__all_sync(0xffffffffu, md_ready)) mbar_wait_issued_warp(&misc->mma_done, (i - 1) & 1, abort_flag, 605 + g, i);
            tc_fence_after();
          }
          s_ready = i + 1 < nq ? mbar_probe(&misc->s_full, (i + 1) & 1) : 0u;
          // 8 packed columns per warpgroup: the 32x32b.x8 shape
          asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                       ::"r"(tb + T_DS1 + g * 8), "r"(d1[0]), "r"(d1[1]), "r"(d1[2]), "r"(d1[3]), "r"(d1[4]), "r"(d1[5]), "r"(d1[6]), "r"(d1[7]) : "memory");
          asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                       ::"r"(tb + T_DS2 + g * 8), "r"(d2[0]), "r"(d2[1]), "r"(d2[2]), "r"(d2[3]), "r"(d2[4]), "r"(d2[5]), "r"(d2[6]), "r"(d2[7]) : "memory");
          tc_wait_st();
          tc_fence_before();
          named_bar_arrive(NB_E + (i & 1), NB_E_THREADS);
          if (++st == ST) st = 0;
        }
      }
      work.forget();
      mbar_wait_issued_warp(&misc->acc_full, work.round & 1, abort_flag, 611 + g);
      tc_fence_after();
      // warpgroup g reads accumulator columns [64g, 64g+64): g = 0,1 -> the two halves of dV, g = 2 -> dK1, g = 3 -> dK2
      uint32_t acc[64];
      tmem_ld32(tb + g * 64, acc);
      tmem_ld32(tb + g * 64 + 32, acc + 32);
      tc_wait_ld();
      if (work.has_next()) {
        tc_fence_before();
        named_bar_arrive(NB_ACC, NB_E_THREADS);
      }
      // The gradients leave through shared memory and the TMA engine (row-per-thread global stores of 16-byte
      // pieces are several times slower): each warpgroup lays its 64 columns into a swizzled [128][64] tile over buffers that
      // no MMA reads any more and the next tile does not fill at once, and the TMA warp stores the tiles.
      {
        const float s = g < 2 ? 1.f : args.sm_scale;
        // g = 0, 1: the halves of dV in the ring slot that is filled third from here; 2, 3: dK1, dK2 in the one filled second
        uint8_t* tile = smem + OFF_STAGE + (st + (g < 2 ? 2 : 1)) % ST * STAGE_BYTES + (g & 1) * K_BYTES;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint4 v;
          v.x = pack2<BF>(__uint_as_float(acc[8 * i + 0]) * s, __uint_as_float(acc[8 * i + 1]) * s);
          v.y = pack2<BF>(__uint_as_float(acc[8 * i + 2]) * s, __uint_as_float(acc[8 * i + 3]) * s);
          v.z = pack2<BF>(__uint_as_float(acc[8 * i + 4]) * s, __uint_as_float(acc[8 * i + 5]) * s);
          v.w = pack2<BF>(__uint_as_float(acc[8 * i + 6]) * s, __uint_as_float(acc[8 * i + 7]) * s);
          st_swizzled_chunk(tile, row, i, v);
        }
        fence_proxy_async_smem();
        named_bar_arrive(NB_STORE, NB_E_THREADS);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------
// 3. dQ1, dQ2: a CTA works on 128 query rows at a time; key/value tiles of 128 rows stream by.  TMEM: S1 [0,128), S2 [128,256),
// dP [256,384), dQ1 [384,448), dQ2 [448,512).  Thread = query row.
//
// Score tiles are 128 columns wide: an M = 128, N = 128 step reads 8 KB of operands in its 64 clocks where two N = 64 steps
// read 12 KB in 96, and the tensor pipe with its operand reads is what bounds this kernel.  That leaves one buffer per score
// tile, and each is refilled while the pass that used it is still running: a warpgroup forms dS_b = +-P_b (dP - E_b)
// of BOTH branches for 32 of the 128 columns, branch 1 first, and writes each as 16-bit over the first 16 of its own score
// columns (TMEM A-operand of dS_b K_b); dP is read once and stays in registers for both.  So dP(j+1) is issued as soon as
// dP(j) is in registers, S1(j+1) behind dQ1(j) under branch 2, S2(j+1) behind dQ2(j) under branch 1 of the next tile.
// The warpgroups of columns 64.. (team 1) run half a branch behind the others, so that one team's exponentials
// cover the other's waits, loads and stores.
// B4 H16 N4096 D64: 0.81 -> 0.77 ms (1.9 GHz), 0.935 -> 0.889 ms sustained under the power cap; B8 H16 N2048 D32 418 -> 375 us.
// (64-column sub-tiles in two buffers, the teams on alternate sub-tiles and the same piecewise refill: 0.950 ms sustained, 390 us.)
// ------------------------------------------------------------------------------------------------
namespace dq64 {
constexpr int BM = 128, BN = 128, HD = 64, DV = 128, KS = 3, VS = 2;
constexpr int Q_BYTES = BM * HD * 2;        // 16 KB
constexpr int DA_BYTES = BM * DV * 2;       // 32 KB
constexpr int K_BYTES = BN * HD * 2;        // 16 KB
constexpr int V_BYTES = BN * DV * 2;        // 32 KB
constexpr int OFF_Q1 = 0, OFF_Q2 = Q_BYTES, OFF_DA = 2 * Q_BYTES;
constexpr int OFF_K = OFF_DA + DA_BYTES;             // 64 KB; stage s: K1 at +s*2*K_BYTES, K2 right after
constexpr int OFF_V = OFF_K + KS * 2 * K_BYTES;      // 160 KB
constexpr int OFF_MISC = OFF_V + VS * V_BYTES;       // 224 KB
constexpr int MISC_BYTES = 1024;
constexpr int SMEM_BYTES = OFF_MISC + MISC_BYTES + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "more shared memory than an SM gives one CTA");
constexpr int NWG = 4;                      // warpgroup w: columns [32w, 32w+32) of each tile
constexpr int NUM_THREADS = NWG * 128 + 64;
constexpr int WARP_TMA = NWG * 4, WARP_MMA = NWG * 4 + 1;
constexpr int T_S1 = 0, T_S2 = 128, T_DP = 256, T_DQ1 = 384, T_DQ2 = 448;
// Named barriers: all warpgroups arrive, the MMA warp syncs.  (An mbarrier wait costs the issuer 150-300 clocks while MMAs
// saturate shared memory; a named barrier a tenth of that.)  NB_START: team 1 waits for team 0's first half branch.  NB_ACC: the
// accumulators of a tile are in registers.
constexpr int NB_DP = 1, NB_DS1 = 2, NB_DS2 = 3, NB_START = 4, NB_ACC = 5, NB_THREADS = NWG * 128 + 32;
struct Misc {
  uint64_t bar_q, q_empty;
  uint64_t k_full[KS], k_empty[KS], v_full[VS], v_empty[VS];
  uint64_t s_full[2], acc_full;   // [branch]; branch 1 stands for dP too
  uint32_t tmem_slot;
  int abort_flag;
};
static_assert(sizeof(Misc) <= MISC_BYTES, "misc area too small");
}  // namespace dq64

template <bool BF, bool DROP, bool LIST>
__global__ void __launch_bounds__(dq64::NUM_THREADS, 1)
diffattn_bwd_dq64_kernel(const __grid_constant__ CUtensorMap tm_q1, const __grid_constant__ CUtensorMap tm_q2,
                         const __grid_constant__ CUtensorMap tm_k1, const __grid_constant__ CUtensorMap tm_k2,
                         const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_da,
                         const BwdArgs args) {
  using namespace dq64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Misc* misc = reinterpret_cast<Misc*>(smem + OFF_MISC);
  volatile int* abort_flag = &misc->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Persistent: this CTA works on the tiles of its WorkList one after the other; the rings and barriers run on from tile to tile
  // (each role counts along by itself), so the next tile's operands arrive and its first scores are computed under this
  // tile's last pass and epilogue.
  // Against one CTA per tile: B8 H16 N2048 D32 380 -> 353 us, B8 H16 N512 D64 47 -> 41, B4 H16 N4096 D64 886 -> 871 sustained.
  WorkList<LIST> work(args.qwork);
  // key / value tile j into its ring slot
  auto load_k = [&](int st, int j, int h_idx, int b_idx) {
    uint8_t* sp = smem + OFF_K + st * 2 * K_BYTES;
    mbar_expect_tx(&misc->k_full[st], 2 * K_BYTES);
    tma_load_4d(sp, &tm_k1, &misc->k_full[st], 0, j * BN, h_idx, b_idx);
    tma_load_4d(sp + K_BYTES, &tm_k2, &misc->k_full[st], 0, j * BN, h_idx, b_idx);
  };
  auto load_v = [&](int st, int j, int h_idx, int b_idx) {
    uint8_t* sp = smem + OFF_V + st * V_BYTES;
    mbar_expect_tx(&misc->v_full[st], V_BYTES);
    tma_load_4d(sp, &tm_v, &misc->v_full[st], 0, j * BN, h_idx, b_idx);
    tma_load_4d(sp + V_BYTES / 2, &tm_v, &misc->v_full[st], 64, j * BN, h_idx, b_idx);
  };
  auto load_da = [&](int q_tile, int bh) {
    tma_load_4d(smem + OFF_DA, &tm_da, &misc->bar_q, 0, q_tile * BM, bh, 0);
    tma_load_4d(smem + OFF_DA + DA_BYTES / 2, &tm_da, &misc->bar_q, 64, q_tile * BM, bh, 0);
  };
  auto load_q = [&](int q_tile, int h_idx, int b_idx) {
    mbar_expect_tx(&misc->bar_q, 2 * Q_BYTES + DA_BYTES);       // Q1, Q2 here, dA by load_da
    tma_load_4d(smem + OFF_Q1, &tm_q1, &misc->bar_q, 0, q_tile * BM, h_idx, b_idx);
    tma_load_4d(smem + OFF_Q2, &tm_q2, &misc->bar_q, 0, q_tile * BM, h_idx, b_idx);
  };
  if (warp == WARP_TMA && lane == 0) {
    mbar_init(&misc->bar_q, 1);
    mbar_init(&misc->q_empty, 1);
    for (int i = 0; i < KS; ++i) { mbar_init(&misc->k_full[i], 1); mbar_init(&misc->k_empty[i], 1); }
    for (int i = 0; i < VS; ++i) { mbar_init(&misc->v_full[i], 1); mbar_init(&misc->v_empty[i], 1); }
    for (int b = 0; b < 2; ++b) mbar_init(&misc->s_full[b], 1);
    mbar_init(&misc->acc_full, 1);
    misc->abort_flag = 0;
    mbar_init_fence();
    // what the caller gave (Q and the first pass over the rings) is requested before the CTA-wide setup barrier
    const WorkItem wi = work.item();
    const int nkv = key_tiles(args.causal, args.n, wi.tile), b_idx = wi.bh / args.h, h_idx = wi.bh % args.h;
    load_q(wi.tile, h_idx, b_idx);
    for (int j = 0; j < VS && j < nkv; ++j) {
      load_v(j, j, h_idx, b_idx);
      load_k(j, j, h_idx, b_idx);
    }
  }
  if (warp == WARP_MMA) tmem_alloc(&misc->tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&misc->tmem_slot);

  if (warp == WARP_TMA) {
    if (elect_one()) {
      bool ok = true;
      int ks = 0, vs = 0;                 // ring slots; the parity bits are those of an "empty" wait (a first pass never waits)
      uint32_t k_par = 1, v_par = 1;
      for (int it = 0; ok && work.valid(); ++it, work.next()) {
        const WorkItem wi = work.item();
        const int nkv = key_tiles(args.causal, args.n, wi.tile), b_idx = wi.bh / args.h, h_idx = wi.bh % args.h;
        if (it > 0) {
          ok = mbar_wait_free(&misc->q_empty, (it - 1) & 1, abort_flag, 703, it);
          if (!ok) break;
          load_q(wi.tile, h_idx, b_idx);
        } else {
          griddep_wait();        // dA comes from the preprocess kernel, for which the grid before this one has waited
        }
        load_da(wi.tile, wi.bh);
        for (int j = 0; j < nkv; ++j) {
          if (it > 0 || j >= VS) {
            ok = mbar_wait_free(&misc->v_empty[vs], v_par, abort_flag, 701, j);
            if (!ok) break;
            load_v(vs, j, h_idx, b_idx);
            ok = mbar_wait_free(&misc->k_empty[ks], k_par, abort_flag, 702, j);
            if (!ok) break;
            load_k(ks, j, h_idx, b_idx);
          }
          if (++ks == KS) { ks = 0; k_par ^= 1; }
          if (++vs == VS) { vs = 0; v_par ^= 1; }
        }
      }
    }
  } else if (warp == WARP_MMA) {
    // One warp issues every MMA.  Every trip makes its barrier calls, issues and commits whether or not a wait for a load gave up (see
    // mbar_wait_issued).
    constexpr uint32_t IDESC_S = make_idesc(BM, BN, 0, 0, BF);     // S = Q K^T, dP = dA V^T
    const uint32_t IDESC_DQ = make_idesc(BM, args.d, 0, 1, BF);    // dQ += dS K   (K MN-major); head dim 32: 32 columns
    const int kd = args.d >> 4;       // 16-deep MMA steps over the head dim: head dim 32 skips the zero padding
    const uint32_t q_lo = sdesc_lo(smem_u32(smem + OFF_Q1)), da_lo = sdesc_lo(smem_u32(smem + OFF_DA));
    const uint32_t k_lo0 = sdesc_lo(smem_u32(smem + OFF_K)), v_lo0 = sdesc_lo(smem_u32(smem + OFF_V));
    const uint32_t tb = tmem_base;
    auto issue_dp = [&](int vs) {
      const uint32_t v_lo = v_lo0 + vs * (V_BYTES >> 4);
#pragma unroll
      for (int k = 0; k < DV / 16; ++k)
        if (k < 2 * kd)
          mma_ss_lo(tb + T_DP, da_lo + (k / 4) * ((DA_BYTES / 2) >> 4) + (k % 4) * 2, v_lo + (k / 4) * ((V_BYTES / 2) >> 4) + (k % 4) * 2, IDESC_S,
                    k > 0);
      mma_commit(&misc->v_empty[vs]);
    };
    auto issue_s = [&](int br, int ks) {
      const uint32_t k_lo = k_lo0 + ks * ((2 * K_BYTES) >> 4) + br * (K_BYTES >> 4);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        if (k < kd) mma_ss_lo(tb + (br ? T_S2 : T_S1), q_lo + br * (Q_BYTES >> 4) + k * 2, k_lo + k * 2, IDESC_S, k > 0);
      mma_commit(&misc->s_full[br]);
    };
    auto issue_dq = [&](int br, int ks, uint32_t first) {
      const uint32_t k_lo = k_lo0 + ks * ((2 * K_BYTES) >> 4) + br * (K_BYTES >> 4);
#pragma unroll
      for (int k = 0; k < BN / 16; ++k)
        mma_ts_lo(tb + (br ? T_DQ2 : T_DQ1), tb + (br ? T_S2 : T_S1) + (k / 2) * 32 + (k % 2) * 8, k_lo + k * (2048 >> 4), IDESC_DQ,
                  k > 0 ? 1u : first);
    };
    griddep_wait();
    bool ok = true;
    int ks = 0, vs = 0;                // ring slots of tile j
    uint32_t k_par = 0, v_par = 0;     // parities of their passes over the rings
    for (int it = 0; work.valid(); ++it, work.next()) {
      const int nkv = key_tiles(args.causal, args.n, work.item().tile);
      ok = ok && mbar_wait_warp(&misc->bar_q, it & 1, abort_flag, 801, it);
      ok = ok && mbar_wait_warp(&misc->v_full[vs], v_par, abort_flag, 802, it);
      ok = ok && mbar_wait_warp(&misc->k_full[ks], k_par, abort_flag, 803, it);
      tc_fence_after();
      if (elect_one()) {
        issue_dp(vs);
        issue_s(0, ks);
        issue_s(1, ks);
        if (nkv == 1) mma_commit(&misc->q_empty);
      }
      __syncwarp();
      for (int j = 0; j < nkv; ++j) {
        const bool more = j + 1 < nkv;
        int ks_n = ks + 1, vs_n = vs + 1;
        if (ks_n == KS) { ks_n = 0; k_par ^= 1; }
        if (vs_n == VS) { vs_n = 0; v_par ^= 1; }
        if (more) {                      // tile j + 1 has landed (waited for under the warpgroups' pass)
          ok = ok && mbar_wait_warp(&misc->v_full[vs_n], v_par, abort_flag, 804, j);
          ok = ok && mbar_wait_warp(&misc->k_full[ks_n], k_par, abort_flag, 805, j);
        }
        if (j == 0 && it > 0) named_bar_sync(NB_ACC, NB_THREADS);        // the previous tile's accumulators are in registers
        named_bar_sync(NB_DP, NB_THREADS);                               // dP(j) is in registers
        tc_fence_after();
        if (more && elect_one()) issue_dp(vs_n);
        __syncwarp();
        named_bar_sync(NB_DS1, NB_THREADS);                              // dS1(j) written
        tc_fence_after();
        if (elect_one()) {
          issue_dq(0, ks, j > 0);
          if (more) issue_s(0, ks_n);
        }
        __syncwarp();
        named_bar_sync(NB_DS2, NB_THREADS);                              // dS2(j) written
        tc_fence_after();
        if (elect_one()) {
          issue_dq(1, ks, j > 0);
          mma_commit(&misc->k_empty[ks]);
          if (more) issue_s(1, ks_n);
          if (j == nkv - 2) mma_commit(&misc->q_empty);
          if (!more) mma_commit(&misc->acc_full);
        }
        __syncwarp();
        ks = ks_n;
        vs = vs_n;
      }
    }
  } else {
    const int g = warp >> 2;                       // columns [32g, 32g + 32) of every tile
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
    const uint32_t tb = tmem_base + lane_base;
    const float sl2 = args.sm_scale * 1.4426950408889634f;
    const float lam = load_lambda(args.lambda_ptr, args.lambda_dtype);
    const float sg = lam < 0.f ? 1.f : -1.f;       // branch 2: -sign(lambda) (|lambda| sits in its statistics, the sign in e)
    const float dscale = DROP ? args.drop_scale : 1.f;
    const f32x2 sl2_2 = pk2(sl2, sl2);
    const uint32_t t_s1 = tb + T_S1 + g * 32, t_s2 = tb + T_S2 + g * 32, t_dp = tb + T_DP + g * 32;
    // own 32 columns of one branch: dS over the first 16 of them
    auto branch = [&](uint32_t* s, const uint32_t* dp, int nv, int j, float neg_l, float neg_e, float sgn, const DropWalk& dw, auto mid) {
      if (nv < 32) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i >= nv) s[i] = 0xff800000u;
      }
      const f32x2 negl_2 = pk2(neg_l, neg_l), nege_2 = pk2(neg_e, neg_e), sg_2 = pk2(sgn * dscale, sgn * dscale);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i == 8) mid();
        float x0, x1;
        up2(fma2(pk2u(s[2 * i], s[2 * i + 1]), sl2_2, negl_2), x0, x1);
        const float p0 = ex2(x0), p1 = ex2(x1);
        uint32_t d0 = dp[2 * i], d1 = dp[2 * i + 1];
        if constexpr (DROP) {
          // dP reaches a probability only where it was kept, with the factor 1/(1-p)
          const uint32_t f = drop_at_col(dw, uint32_t(j * (BN / 2) + g * 16), i);
          d0 &= drop_mask_first(f);
          d1 &= drop_mask_second(f);
        }
        float r0, r1;
        up2(mul2(pk2(p0, p1), fma2(pk2u(d0, d1), sg_2, nege_2)), r0, r1);
        s[i] = pack2<BF>(r0, r1);
      }
    };
    griddep_wait();                                // the statistics come from the preprocess kernel
    if (g >= 2) named_bar_sync(NB_START, NWG * 128);
    uint32_t done = 0;                             // key tiles done: the phase of the score barriers
    for (; work.valid(); work.next()) {
      {
        const WorkItem wi = work.item();
        const int q_tile = wi.tile, bh = wi.bh, nkv = key_tiles(args.causal, args.n, q_tile);
        const float4 sv = stat_row(args.stats, size_t(bh) * args.n_pad + size_t(q_tile) * BM + row);
        DropWalk dw1, dw2;
        if constexpr (DROP) {
          const uint32_t row2 = uint32_t(q_tile * BM + row) >> 1;
          dw1 = drop_walk_row(drop_key(args.seed_lo, args.seed_hi, uint32_t(bh), 0u), row2, row & 1, args.drop_thresh);
          dw2 = drop_walk_row(drop_key(args.seed_lo, args.seed_hi, uint32_t(bh), 1u), row2, row & 1, args.drop_thresh);
        }
        for (int j = 0; j < nkv; ++j, ++done) {
          // key columns past the sequence end or (causal) right of the diagonal: score -inf, probability 0
          const int c_first = j * BN + g * 32;
          int nv = args.n - c_first;
          if (args.causal) nv = min(nv, q_tile * BM + row - c_first + 1);
          uint32_t s[32], dp[32];
          mbar_wait_issued_warp(&misc->s_full[0], done & 1, abort_flag, 901, j);
          tc_fence_after();
          tmem_ld32(t_dp, dp);
          tmem_ld32(t_s1, s);
          tc_wait_ld();
          tc_fence_before();
          named_bar_arrive(NB_DP, NB_THREADS);
          branch(s, dp, nv, j, sv.x, sv.z, 1.f, dw1, [&] { if (done == 0 && g < 2) named_bar_arrive(NB_START, NWG * 128); });
          tmem_st16(t_s1, s);
          tc_wait_st();
          tc_fence_before();
          named_bar_arrive(NB_DS1, NB_THREADS);
          mbar_wait_issued_warp(&misc->s_full[1], done & 1, abort_flag, 902, j);
          tc_fence_after();
          tmem_ld32(t_s2, s);
          tc_wait_ld();
          branch(s, dp, nv, j, sv.y, sv.w, sg, dw2, [] {});
          tmem_st16(t_s2, s);
          tc_wait_st();
          tc_fence_before();
          named_bar_arrive(NB_DS2, NB_THREADS);
        }
      }
      work.forget();
      mbar_wait_issued_warp(&misc->acc_full, work.round & 1, abort_flag, 911);
      tc_fence_after();
      const int u = g >> 1, half = g & 1;            // this warpgroup stores columns [32 half, 32 half + 32) of dQ of branch u
      uint32_t acc[32];
      tmem_ld32(tb + (u ? T_DQ2 : T_DQ1) + half * 32, acc);
      tc_wait_ld();
      if (work.has_next()) {
        tc_fence_before();
        named_bar_arrive(NB_ACC, NB_THREADS);
      }
      const WorkItem wi = work.item();
      const int q_tile = wi.tile;
      // (32 columns per thread: direct 16-byte stores; a shared-memory tile and a TMA store, as the other two
      // kernels use for their wider rows, measured 4 % slower here)
      if (!*abort_flag && half * 32 < args.d && q_tile * BM + row < args.n) {
        const float sc = args.sm_scale;
        const size_t grow = size_t(wi.bh) * args.n + size_t(q_tile) * BM + row;
        uint4* p = reinterpret_cast<uint4*>((u ? args.dq2 : args.dq1) + grow * args.d + half * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 v;
          v.x = pack2<BF>(__uint_as_float(acc[8 * i + 0]) * sc, __uint_as_float(acc[8 * i + 1]) * sc);
          v.y = pack2<BF>(__uint_as_float(acc[8 * i + 2]) * sc, __uint_as_float(acc[8 * i + 3]) * sc);
          v.z = pack2<BF>(__uint_as_float(acc[8 * i + 4]) * sc, __uint_as_float(acc[8 * i + 5]) * sc);
          v.w = pack2<BF>(__uint_as_float(acc[8 * i + 6]) * sc, __uint_as_float(acc[8 * i + 7]) * sc);
          p[i] = v;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace da
