// Differential-attention forward for head dim D = 128 (value width 256), sm_100a.
//
// Two 256-wide accumulators do not fit in TMEM next to the score buffers, so the two branches run in the two CTAs of a
// thread-block cluster (blockIdx.z = branch): with a single branch the whole accumulator fits and nothing is computed twice
// (12 units of B*H*N^2*D and 2 N^2 exponentials per head).  Softmax as in the D <= 64 kernel (softmax_subtile in fwd.cuh):
// two warpgroups on alternate 64-column sub-tiles, half a pass apart.  TMEM also holds the probabilities apart from the scores
// (S(t+2) is computed as soon as S(t) is in registers) and Q, the A operand of the score MMAs.  At the end branch 2 hands its
// A2 = O_2 / l_2 in fp32 to branch 1 through distributed shared memory, and branch 1 forms y and rstd.
// What bounds it: the tensor pipe needs 768 clocks per sub-tile (S 256, P V 512), and at B2 H8 N8192 D128 it executes
// 1377 TFLOP/s sustained, the rate a plain cuBLAS loop reaches under the 1 kW cap.  Against one softmax warpgroup with P over
// its scores and Q in shared memory: 1.44 -> 1.20 ms there, a call at B1 H8 N4096 causal 168 -> 126 us; both warpgroups in phase 1.29 ms.
// (An earlier form kept both branches in one CTA and made two passes over the keys, with the probabilities recomputed in
// the second: 1.97 ms.  A form without the cluster -- branch 1 writes A1 as 16-bit values into y, a second kernel
// combines -- lost accuracy where A1 - lambda A2 cancels: with bf16 tensors, lambda 0.8, a causal mask and rms_norm two of 400
// seeded cases left the tolerance.)
#pragma once
#include "fwd.cuh"
#include "sm100.cuh"

namespace da {

namespace fwd128 {
constexpr int BM = 128, SUB = 64, HD = 128, DV = 256;
constexpr int KS = 4, VS = 3;                   // ring depths: K is requested two sub-tiles ahead of V
constexpr int Q_BYTES = BM * HD * 2;            // 32 KB: two boxes [128 x 64]
constexpr int K_BYTES = SUB * HD * 2;           // 16 KB: two boxes [64 x 64]
constexpr int V_BYTES = SUB * DV * 2;           // 32 KB: four boxes [64 x 64]
constexpr int OFF_Q = 0, OFF_K = Q_BYTES, OFF_V = OFF_K + KS * K_BYTES;
constexpr int OFF_MISC = OFF_V + VS * V_BYTES;              // 192 KB
// epilogue, rings and Q idle: 64-column tiles of the outputs (16 KB each) from 0, the fp32 exchange tile (128 KB) behind them
constexpr int OUT_TILE_BYTES = BM * 128;
constexpr int OFF_OUT = 0, OFF_X = 4 * OUT_TILE_BYTES;
static_assert(OFF_X + BM * DV * 4 <= OFF_MISC, "epilogue tiles do not fit");
constexpr int MISC_BYTES = 6144;
constexpr int SMEM_BYTES = OFF_MISC + MISC_BYTES + 1024;
constexpr int NUM_SOFTMAX = 256;
constexpr int NUM_THREADS = NUM_SOFTMAX + 128;
constexpr int WARP_TMA = 8, WARP_PV = 9, WARP_S = 10, WARP_TMA_V = 11;
// TMEM: S two 64-column buffers | P likewise, 16-bit pairs | Q as 16-bit pairs | O
constexpr int T_S = 0, T_P = 128, T_Q = 192, T_O = 256;
constexpr int NB_P = 2, NB_SF = 4, NB_M = 6, NB_OUT = 9, NB_START = 11;     // named barriers, + sub-tile parity (1: the softmax warps)
struct Misc {
  uint64_t bar_q, q_ready;
  uint64_t k_full[KS], k_empty[KS], v_full[VS], v_empty[VS];
  uint64_t s_full[2], pv_done[2], o_full;
  uint64_t peer_ready, peer_data;     // arrivals come from the partner CTA of the cluster (the other branch)
  uint32_t tmem_slot;
  int abort_flag;
  float m_run[BM];                    // running row maximum
  float m_end[2][BM], l_end[2][BM];   // maximum and row sum of each warpgroup at the end
  float ssq[2][BM];
};
static_assert(sizeof(Misc) <= MISC_BYTES, "misc area too small");
}  // namespace fwd128

template <bool BF, bool DROP>
__global__ void __launch_bounds__(fwd128::NUM_THREADS, 1)
diffattn_fwd128_branch_kernel(const __grid_constant__ CUtensorMap tm_q1, const __grid_constant__ CUtensorMap tm_q2,
                              const __grid_constant__ CUtensorMap tm_k1, const __grid_constant__ CUtensorMap tm_k2,
                              const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_y,
                              const __grid_constant__ CUtensorMap tm_a2, const FwdArgs args) {
  using namespace fwd128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Misc* misc = reinterpret_cast<Misc*>(smem + OFF_MISC);
  volatile int* abort_flag = &misc->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // causal: the later a query tile, the more keys it sees -- the heaviest tiles are launched first so that the grid's tail is light
  const int q_tile = args.causal ? int(gridDim.x) - 1 - int(blockIdx.x) : int(blockIdx.x), bh = blockIdx.y, br = blockIdx.z;
  const int b_idx = bh / args.h, h_idx = bh % args.h;
  const int nsub_all = ((args.n + 127) / 128) * 2;     // 64-row sub-tiles, N rounded up to 128 (TMA zero-fills)
  const int nsub = (args.causal && 2 * (q_tile + 1) < nsub_all) ? 2 * (q_tile + 1) : nsub_all;   // causal: stop at the diagonal tile
  const CUtensorMap* tm_q = br ? &tm_q2 : &tm_q1;
  const CUtensorMap* tm_k = br ? &tm_k2 : &tm_k1;

  auto load_k = [&](int t) {
    const int s = t % KS;
    uint8_t* kp = smem + OFF_K + s * K_BYTES;
    mbar_expect_tx(&misc->k_full[s], K_BYTES);
    for (int c = 0; c < 2; ++c) tma_load_4d(kp + c * 8192, tm_k, &misc->k_full[s], c * 64, t * SUB, h_idx, b_idx);
  };
  auto load_v = [&](int t) {
    const int s = t % VS;
    uint8_t* vp = smem + OFF_V + s * V_BYTES;
    mbar_expect_tx(&misc->v_full[s], V_BYTES);
    for (int c = 0; c < 4; ++c) tma_load_4d(vp + c * 8192, &tm_v, &misc->v_full[s], c * 64, t * SUB, h_idx, b_idx);
  };
  if (warp == WARP_TMA && lane == 0) {
    mbar_init(&misc->bar_q, 1);
    mbar_init(&misc->q_ready, NUM_SOFTMAX);
    for (int i = 0; i < KS; ++i) { mbar_init(&misc->k_full[i], 1); mbar_init(&misc->k_empty[i], 1); }
    for (int i = 0; i < VS; ++i) { mbar_init(&misc->v_full[i], 1); mbar_init(&misc->v_empty[i], 1); }
    for (int u = 0; u < 2; ++u) { mbar_init(&misc->s_full[u], 1); mbar_init(&misc->pv_done[u], 1); }
    mbar_init(&misc->o_full, 1);
    mbar_init(&misc->peer_ready, 1);
    mbar_init(&misc->peer_data, NUM_SOFTMAX);
    misc->abort_flag = 0;
    mbar_init_fence();
    // the first loads go out before the setup barriers; the first pass over a ring needs no "empty" wait
    mbar_expect_tx(&misc->bar_q, Q_BYTES);
    for (int c = 0; c < 2; ++c) tma_load_4d(smem + OFF_Q + c * 16384, tm_q, &misc->bar_q, c * 64, q_tile * BM, h_idx, b_idx);
    load_k(0); load_k(1); load_v(0); load_v(1);                 // nsub >= 2
    tma_prefetch_desc(&tm_y); tma_prefetch_desc(&tm_a2);
  }
  if (warp == WARP_PV) tmem_alloc(&misc->tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // the partner's mbarriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&misc->tmem_slot);

  if (warp == WARP_TMA) {
    if (elect_one()) {
      for (int t = 2; t < nsub; ++t) {
        if (!mbar_wait_free(&misc->k_empty[t % KS], ((t / KS) & 1) ^ 1, abort_flag, 2101, t)) break;
        load_k(t);
      }
    }
  } else if (warp == WARP_TMA_V) {
    // (a producer warp per ring: the score MMAs run two sub-tiles ahead of P V, and with one warp for both rings the next
    // K waits behind a V whose stage is not free yet: 2.3 ms against 1.4 ms at B2 H8 N8192 D128)
    if (elect_one()) {
      for (int t = 2; t < nsub; ++t) {
        if (!mbar_wait_free(&misc->v_empty[t % VS], ((t / VS) & 1) ^ 1, abort_flag, 2102, t)) break;
        load_v(t);
      }
    }
  } else if (warp == WARP_S) {
    // S(t+2) = Q K^T once the scores of sub-tile t are in registers.  Scores and probabilities have TMEM columns of their
    // own, so a warpgroup finds its next scores ready when it has stored its probabilities, and the two kinds of MMAs need no
    // order between them: two issuing warps, so that one's waits run under the other's MMAs (1.198 ms against 1.207 ms
    // with one warp for both at B2 H8 N8192 D128).  Both run every trip, whether or not a wait for a load gave up (see mbar_wait_issued).
    constexpr uint32_t IDESC_S = make_idesc(BM, SUB, 0, 0, BF);
    const uint32_t k_lo0 = sdesc_lo(smem_u32(smem + OFF_K));
    bool ok = mbar_wait_warp(&misc->q_ready, 0, abort_flag, 2201);
    for (int t = 0; t < nsub; ++t) {
      const int ks = t % KS, u = t & 1;
      ok = ok && mbar_wait_warp(&misc->k_full[ks], (t / KS) & 1, abort_flag, 2202, t);
      if (t >= 2) named_bar_sync(NB_SF + u, 160);
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < HD / 16; ++k)
          mma_ts_lo(tmem_base + T_S + u * SUB, tmem_base + T_Q + k * 8, k_lo0 + ks * (K_BYTES >> 4) + (k / 4) * (8192 >> 4) + (k % 4) * 2, IDESC_S, k > 0);
        mma_commit(&misc->s_full[u]);
        mma_commit(&misc->k_empty[ks]);
      }
      __syncwarp();
    }
  } else if (warp == WARP_PV) {
    // O += P(t) V(t)
    constexpr uint32_t IDESC_O = make_idesc(BM, DV, 0, 1, BF);      // V as MN-major B: four 64-column atoms 8 KB apart
    const uint32_t v_lo0 = sdesc_lo(smem_u32(smem + OFF_V), 8192);
    bool ok = true;
    for (int t = 0; t < nsub; ++t) {
      const int vs = t % VS, u = t & 1;
      ok = ok && mbar_wait_warp(&misc->v_full[vs], (t / VS) & 1, abort_flag, 2203, t);
      named_bar_sync(NB_P + u, 160);
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < SUB / 16; ++k)
          mma_ts_lo(tmem_base + T_O, tmem_base + T_P + u * (SUB / 2) + k * 8, v_lo0 + vs * (V_BYTES >> 4) + k * (2048 >> 4), IDESC_O, (t > 0 || k > 0));
        mma_commit(&misc->pv_done[u]);
        mma_commit(&misc->v_empty[vs]);
      }
      __syncwarp();
    }
    if (elect_one()) mma_commit(&misc->o_full);
  } else {
    const int u = warp >> 2;                                // sub-tile parity of this warpgroup
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
    const uint32_t t_o = tmem_base + lane_base + T_O;
    const float sl2 = args.sm_scale * 1.4426950408889634f;
    const size_t grow = size_t(bh) * args.n + size_t(q_tile) * BM + row;
    // Q into TMEM, the A operand of S = Q K^T: this thread's row, the 64 columns of box u (128 bytes, swizzled in 16-byte
    // chunks) -> 32 columns.  The score MMAs then read only K from shared memory (with both operands there an N = 64 step
    // takes 48 clocks of shared-memory bandwidth for 32 of tensor time).
    mbar_wait_warp(&misc->bar_q, 0, abort_flag, 2300);
    {
      uint32_t qv[32];
      const uint8_t* qrow = smem + OFF_Q + u * 16384 + row * 128;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint4 v = *reinterpret_cast<const uint4*>(qrow + ((c ^ (row & 7)) << 4));
        qv[4 * c] = v.x; qv[4 * c + 1] = v.y; qv[4 * c + 2] = v.z; qv[4 * c + 3] = v.w;
      }
      tmem_st32(tmem_base + lane_base + T_Q + u * 32, qv);
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&misc->q_ready);
    }
    SoftmaxState st;
    {
      const uint32_t t_s = tmem_base + lane_base + T_S + u * SUB, t_p = tmem_base + lane_base + T_P + u * (SUB / 2);
      DropWalk dr;
      if constexpr (DROP)
        dr = drop_walk_row(drop_key(args.seed_lo, args.seed_hi, uint32_t(bh), uint32_t(br)), uint32_t(q_tile * BM + row) >> 1, row & 1, args.drop_thresh);
      int t = u;
      // Warpgroup 1 starts half a pass behind warpgroup 0: in phase, both would be at their exponentials together and
      // leave the exp unit idle together.
      if (u == 1) named_bar_sync(NB_START, 256);
      uint32_t s_ready = 0;             // answer of the early probe (see mbar_probe)
      for (; t < nsub; t += 2) {
        if (!s_ready) mbar_wait_issued(&misc->s_full[u], (t >> 1) & 1, abort_flag, 2301 + br, t);
        __syncwarp();
        tc_fence_after();
        int nv = args.n - t * SUB;             // visible key columns of this row in this sub-tile
        if (args.causal) nv = min(nv, q_tile * BM + row - t * SUB + 1);
        softmax_subtile<BF, DROP, DV>(
                 st, t_s, t_p, t_o, t == 0, t, nv, sl2, &misc->m_run[row], dr,
                 [&] { if (t + 2 < nsub) { tc_fence_before(); named_bar_arrive(NB_SF + u, 160); } },
                 [&] { named_bar_sync(NB_M + (u ^ 1), 256); }, [&] { if (t + 1 < nsub) named_bar_arrive(NB_M + u, 256); },
                 [&] { mbar_wait_issued_warp(&misc->pv_done[u ^ 1], ((t - 1) >> 1) & 1, abort_flag, 2305 + br, t); },
                 [&] {
                   if (t == 0) named_bar_arrive(NB_START, 256);
                   if (t + 2 < nsub) s_ready = mbar_probe(&misc->s_full[u], ((t + 2) >> 1) & 1);
                 },
                 [&] { if (t >= 2) mbar_wait_issued_warp(&misc->pv_done[u], ((t - 2) >> 1) & 1, abort_flag, 2303 + br, t); });
        named_bar_arrive(NB_P + u, 160);
      }
    }

    // ---- epilogue.  The two CTAs of a cluster hold A1 = O_1 / l_1 (branch 1) and A2 = O_2 / l_2 (branch 2) of the same 128
    // query rows.  Branch 2 writes a2 and hands its A2 in fp32 to branch 1 through distributed shared memory (into branch
    // 1's rings, idle by then); branch 1 forms y = RMSNorm(A1 - lambda A2) (1 - lambda_init) and rstd.  Warpgroup u has
    // value columns [128 u, 128 u + 128).  Every thread runs every barrier; only the global writes depend on the waits.
    mbar_wait_issued_warp(&misc->o_full, 0, abort_flag, 2311 + br);
    tc_fence_after();
    misc->m_end[u][row] = st.m;
    misc->l_end[u][row] = st.l;
    named_bar_sync(1, NUM_SOFTMAX);
    const float ma = misc->m_end[0][row], mb = misc->m_end[1][row], m_fin = misc->m_run[row];      // O is relative to the last running maximum
    const float l_fin = misc->l_end[0][row] * ex2((ma - m_fin) * sl2) + misc->l_end[1][row] * ex2((mb - m_fin) * sl2);
    const float inv_l = (DROP ? args.drop_scale : 1.f) / l_fin;
    const bool live = !*abort_flag && (q_tile * BM + row < args.n);
    uint8_t* out = smem + OFF_OUT + 2 * u * OUT_TILE_BYTES;      // this warpgroup's two 64-column tiles
    // stores the warpgroup's two tiles once all its threads have written them
    auto store_tiles = [&](const CUtensorMap* map, uint8_t* tiles) {
      fence_proxy_async_smem();
      named_bar_sync(NB_OUT + u, 128);
      if ((warp & 3) == 0 && elect_one()) {
        if (!*abort_flag)
          for (int c = 0; c < 2; ++c) tma_store_4d(tiles + c * OUT_TILE_BYTES, map, (2 * u + c) * 64, q_tile * BM, bh, 0);
        tma_store_commit();
        tma_store_wait_read();
      }
    };
    // exchange tile: 64 chunks of four floats per row, chunk-major (chunk c of row r at (c * 128 + r) * 16 bytes), so that
    // the 32 rows of a warp touch consecutive 16-byte words
    uint8_t* xtile = smem + OFF_X;
    if (br == 1) {
      const uint32_t x_remote = cluster_map(smem_u32(xtile), 0);
      mbar_wait_cluster(&misc->peer_ready, 0, abort_flag, 2313);       // branch 1's rings are idle
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld32(t_o + u * 128 + c * 32, o);
        tc_wait_ld();
        float f[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(o[i]) * inv_l;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          cluster_st_v4(x_remote + uint32_t(((u * 32 + c * 8 + i) * BM + row) * 16), f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          st_swizzled_chunk(out + (c >> 1) * OUT_TILE_BYTES, row, (c & 1) * 4 + i,
                            make_uint4(pack2<BF>(f[8 * i + 0], f[8 * i + 1]), pack2<BF>(f[8 * i + 2], f[8 * i + 3]),
                                       pack2<BF>(f[8 * i + 4], f[8 * i + 5]), pack2<BF>(f[8 * i + 6], f[8 * i + 7])));
      }
      cluster_mbar_arrive(cluster_map(smem_u32(&misc->peer_data), 0));
      store_tiles(&tm_a2, out);
      if (live && u == 0) args.lse2[grow] = m_fin * args.sm_scale + logf(l_fin);
    } else {
      if (threadIdx.x == 0) cluster_mbar_arrive(cluster_map(smem_u32(&misc->peer_ready), 1));
      const float lam = load_lambda(args.lambda_ptr, args.lambda_dtype);
      const bool ok = mbar_wait_cluster(&misc->peer_data, 0, abort_flag, 2314);
      const float4* xrow = reinterpret_cast<const float4*>(xtile) + u * 32 * BM + row;
      // A = A1 - lambda A2 of one 32-column chunk (the accumulator and the exchange tile are read twice with rms_norm)
      auto load_a = [&](int c, float (&a)[32]) {
        uint32_t o[32];
        tmem_ld32(t_o + u * 128 + c * 32, o);
        tc_wait_ld();
        float ssq = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 z = xrow[(c * 8 + i) * BM];
          const float zz[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            a[4 * i + k] = __uint_as_float(o[4 * i + k]) * inv_l - lam * zz[k];
            ssq += a[4 * i + k] * a[4 * i + k];
          }
        }
        return ssq;
      };
      float ys = 1.f, ssq = 0.f;
      auto row_rstd = [&] {
        misc->ssq[u][row] = ssq;
        named_bar_sync(1, NUM_SOFTMAX);
        return rsqrtf((misc->ssq[0][row] + misc->ssq[1][row]) * (1.f / DV) + args.eps);
      };
      float rstd = 0.f;
      if (args.rms_norm) {
        for (int c = 0; c < 4; ++c) {
          float a[32];
          ssq += load_a(c, a);
        }
        rstd = row_rstd();
        ys = args.out_scale * rstd;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float a[32];
        const float s2 = load_a(c, a);
        if (!args.rms_norm) ssq += s2;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float f[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = a[8 * i + k] * ys;
          st_swizzled_chunk(out + (c >> 1) * OUT_TILE_BYTES, row, (c & 1) * 4 + i,
                            make_uint4(pack2<BF>(f[0], f[1]), pack2<BF>(f[2], f[3]), pack2<BF>(f[4], f[5]), pack2<BF>(f[6], f[7])));
          if (args.gain && live && ok) {
            const int col = u * 128 + c * 32 + 8 * i;
            const float4 g0 = __ldg(reinterpret_cast<const float4*>(args.gain + col)), g1 = __ldg(reinterpret_cast<const float4*>(args.gain + col + 4));
            *reinterpret_cast<uint4*>(args.yg + grow * DV + col) =
                make_uint4(pack2<BF>(f[0] * g0.x, f[1] * g0.y), pack2<BF>(f[2] * g0.z, f[3] * g0.w), pack2<BF>(f[4] * g1.x, f[5] * g1.y), pack2<BF>(f[6] * g1.z, f[7] * g1.w));
          }
        }
      }
      if (!args.rms_norm) rstd = row_rstd();
      store_tiles(&tm_y, out);
      if (live && ok && !*abort_flag && u == 0) {
        args.lse1[grow] = m_fin * args.sm_scale + logf(l_fin);
        args.rstd[grow] = rstd;
      }
    }
  }

  // neither CTA leaves while its partner may still arrive on its barriers or write into its shared memory
  tc_fence_before();
  cluster_sync_all();
  __syncthreads();
  if (warp == WARP_PV) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace da
