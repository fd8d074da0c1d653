// Forward kernel for head dims 32 and 64 (tile sizes, rings and TMEM map: namespace fwd64 in fwd.cuh).
//
// Sixteen softmax warps in four warpgroups, two per branch on alternate sub-tiles (softmax_subtile in fwd.cuh): four warps
// per scheduler, so that the exp unit has work while others wait for scores, load them or store probabilities.
#pragma once
#include "fwd.cuh"

namespace da {
namespace fwd64 {
constexpr int MISC_BYTES = 8192;
constexpr int SMEM_BYTES = OFF_MISC + MISC_BYTES + 1024; // +1024 for manual alignment
// warps 0-15 softmax (branch = warp >> 3, sub-tile parity = (warp >> 2) & 1, thread = query row); 16 TMA producer; 17
// allocates TMEM and watches the loads; 18 issues every MMA; 19 completes the role warpgroup.  Registers: five warps per
// scheduler are launched with 96 per thread; the role warpgroup hands some to the softmax warpgroups (setmaxnreg), which
// hold a whole 64-column sub-tile of scores per thread.
// One issuing warp in the fixed order (branch 1, branch 2): S_b of sub-tile t+2 right behind P_b V of sub-tile t.  With an
// issuer per branch the two branches' MMAs interleave, both branches' scores complete late and together, and all sixteen
// softmax warps then run in phase.  "P written" and the hand-over of the running maximum go through named barriers (see
// the load watcher).  B4 H16 N4096 D64 against eight softmax warps taking turns on the exp unit: 0.84 -> 0.77 ms (1.9 GHz),
// 0.917 -> 0.875 ms in a sustained loop under the 1 kW cap; mbarriers instead of the named barriers 0.79, an issuer per branch 0.85;
// a quarter of the exponentials on the FMA pipe 0.80 (the pass is not bound by the exp unit, and it costs power).
constexpr int NUM_SOFTMAX = 512;
constexpr int NUM_THREADS = NUM_SOFTMAX + 128;
constexpr int REGS_LAUNCH = 96, REGS_SOFTMAX = 104, REGS_ROLE = 64;
static_assert(4 * REGS_SOFTMAX + REGS_ROLE <= 5 * REGS_LAUNCH, "register shares exceed the launch pool of a scheduler");
constexpr int NB_ALL = 1, NB_STORE = 2, NB_P = 4, NB_M = 8, NB_KV = 12, NB_O = 13;     // named barriers; STORE + branch; P, M + branch * 2 + parity
constexpr int WARP_TMA = 16, WARP_ALLOC = 17, WARP_MMA = 18, WARP_STORE = 19;
struct Misc {
  uint64_t bar_q, q_empty;
  uint64_t stored;           // the epilogue's tiles have left the V ring
  uint64_t k_full[KS], k_empty[KS];
  uint64_t v_full[VS], v_empty[VS];
  uint64_t s_full[2][2];     // [branch][buffer]: S sub-tile written by the MMA
  uint64_t pv_done[2][2];    // [branch][buffer]: P_b V of the sub-tile that used this buffer has completed
  uint64_t o_full;           // everything accumulated
  uint32_t tmem_slot;
  int abort_flag;
  float m_run[2][BM];        // running row maximum per branch
  float m_end[2][2][BM];     // [branch][parity]: maximum and row sum of each warpgroup at the end
  float l_end[2][2][BM];
  float ssq[4][BM];          // partial sums of squares per 32 value columns
};
static_assert(sizeof(Misc) <= MISC_BYTES, "misc area too small");
}  // namespace fwd64


template <bool BF, bool DROP, bool LIST>   // BF: tensors are bf16 instead of fp16; DROP: attention dropout on; LIST: several tiles per CTA
__global__ void __launch_bounds__(fwd64::NUM_THREADS, 1)
diffattn_fwd64_kernel(const __grid_constant__ CUtensorMap tm_q1, const __grid_constant__ CUtensorMap tm_q2,
                      const __grid_constant__ CUtensorMap tm_k1, const __grid_constant__ CUtensorMap tm_k2,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_y,
                      const __grid_constant__ CUtensorMap tm_a2, const __grid_constant__ CUtensorMap tm_yg,
                      const FwdArgs args) {
  using namespace fwd64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Misc* misc = reinterpret_cast<Misc*>(smem + OFF_MISC);
  volatile int* abort_flag = &misc->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // Persistent: this CTA works on the tiles of its WorkList one after the other.  The loads of the next tile's Q and K go out
  // as soon as the last scores of this one are issued, its first scores as soon as the last P V is, and y and a2 leave under
  // the next tile's first passes.  Every ring and barrier runs on from tile to tile; each role counts along by itself.
  // Against one CTA per tile: B8 H16 N2048 D32 405 -> 375 us, B8 H16 N512 D64 52 -> 46, B4 H16 N2048 D64 causal 156 -> 144,
  // B4 H16 N4096 D64 878 -> 862 in a sustained loop.
  WorkList<LIST> work(args.work);
  if (warp == WARP_TMA && lane == 0) {
    mbar_init(&misc->bar_q, 1);
    mbar_init(&misc->q_empty, 1);
    mbar_init(&misc->stored, 1);
    for (int i = 0; i < KS; ++i) { mbar_init(&misc->k_full[i], 1); mbar_init(&misc->k_empty[i], 1); }
    for (int i = 0; i < VS; ++i) { mbar_init(&misc->v_full[i], 1); mbar_init(&misc->v_empty[i], 1); }
    for (int b = 0; b < 2; ++b) {
      for (int u = 0; u < 2; ++u) { mbar_init(&misc->s_full[b][u], 1); }
      for (int u = 0; u < 2; ++u) mbar_init(&misc->pv_done[b][u], 1);
    }
    mbar_init(&misc->o_full, 1);
    misc->abort_flag = 0;
    mbar_init_fence();
    // The first loads go out before the CTA-wide setup barrier (TMEM allocation, everyone's arrival): the
    // barriers they complete on are initialised above, and the first pass over a ring needs no "empty" wait.
    const WorkItem wi = work.item();
    const int nkv = key_tiles(args.causal, args.n, wi.tile);
    const int b_idx = wi.bh / args.h, h_idx = wi.bh % args.h;
    mbar_expect_tx(&misc->bar_q, 2 * Q_BYTES);
    tma_load_4d(smem + OFF_Q1, &tm_q1, &misc->bar_q, 0, wi.tile * BM, h_idx, b_idx);
    tma_load_4d(smem + OFF_Q2, &tm_q2, &misc->bar_q, 0, wi.tile * BM, h_idx, b_idx);
    for (int j = 0; j < PRELOAD && j < nkv; ++j) {
      mbar_expect_tx(&misc->k_full[j], 2 * K_BYTES);
      tma_load_4d(smem + OFF_K + j * 2 * K_BYTES, &tm_k1, &misc->k_full[j], 0, j * BN, h_idx, b_idx);
      tma_load_4d(smem + OFF_K + j * 2 * K_BYTES + K_BYTES, &tm_k2, &misc->k_full[j], 0, j * BN, h_idx, b_idx);
      mbar_expect_tx(&misc->v_full[j], V_BYTES);
      tma_load_4d(smem + OFF_V + j * V_BYTES, &tm_v, &misc->v_full[j], 0, j * BN, h_idx, b_idx);
      tma_load_4d(smem + OFF_V + j * V_BYTES + V_BYTES / 2, &tm_v, &misc->v_full[j], 64, j * BN, h_idx, b_idx);
    }
    tma_prefetch_desc(&tm_y); tma_prefetch_desc(&tm_a2);
  }
  if (warp == WARP_ALLOC) {
    tmem_alloc(&misc->tmem_slot, 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&misc->tmem_slot);

  if (warp == WARP_TMA) {
    // ------------------------------- TMA producer -------------------------------
    reg_dec<REGS_ROLE>();
    if (elect_one()) {
      bool ok = true;
      int ks = 0, vs = 0;                 // ring slots; the parity bits are those of an "empty" wait (a first pass never waits)
      uint32_t k_par = 1, v_par = 1;
      for (int it = 0; ok && work.valid(); ++it, work.next()) {
        const WorkItem wi = work.item();
        const int nkv = key_tiles(args.causal, args.n, wi.tile);
        const int b_idx = wi.bh / args.h, h_idx = wi.bh % args.h;
        if (it > 0) {
          ok = mbar_wait_free(&misc->q_empty, (it - 1) & 1, abort_flag, 103, it);
          if (!ok) break;
          mbar_expect_tx(&misc->bar_q, 2 * Q_BYTES);
          tma_load_4d(smem + OFF_Q1, &tm_q1, &misc->bar_q, 0, wi.tile * BM, h_idx, b_idx);
          tma_load_4d(smem + OFF_Q2, &tm_q2, &misc->bar_q, 0, wi.tile * BM, h_idx, b_idx);
        }
        for (int j = 0; j < nkv; ++j) {
          const bool requested = it == 0 && j < PRELOAD;
          if (!requested) {
            ok = mbar_wait_free(&misc->k_empty[ks], k_par, abort_flag, 101, j);
            if (!ok) break;
            mbar_expect_tx(&misc->k_full[ks], 2 * K_BYTES);
            tma_load_4d(smem + OFF_K + ks * 2 * K_BYTES, &tm_k1, &misc->k_full[ks], 0, j * BN, h_idx, b_idx);
            tma_load_4d(smem + OFF_K + ks * 2 * K_BYTES + K_BYTES, &tm_k2, &misc->k_full[ks], 0, j * BN, h_idx, b_idx);
            // the previous tile's y and a2 (and its gained y, in the K slot after the one just requested) have to leave first
            if (it > 0 && j == 0) ok = mbar_wait_free(&misc->stored, (it - 1) & 1, abort_flag, 104, it);
            ok = ok && mbar_wait_free(&misc->v_empty[vs], v_par, abort_flag, 102, j);
            if (!ok) break;
            mbar_expect_tx(&misc->v_full[vs], V_BYTES);
            tma_load_4d(smem + OFF_V + vs * V_BYTES, &tm_v, &misc->v_full[vs], 0, j * BN, h_idx, b_idx);
            tma_load_4d(smem + OFF_V + vs * V_BYTES + V_BYTES / 2, &tm_v, &misc->v_full[vs], 64, j * BN, h_idx, b_idx);
          }
          if (++ks == KS) { ks = 0; k_par ^= 1; }
          if (++vs == VS) { vs = 0; v_par ^= 1; }
        }
      }
    }
  } else if (warp == WARP_MMA) {
    // ------------- MMA issuer: O_b += P_b(t) V(sub-tile t), S_b(t+2) = Q_b K_b(sub-tile t+2)^T, branch 1 then branch 2 -------------
    // The thread that issues is chosen by elect.sync.  (A thread picked by comparing the lane id issues
    // tcgen05.mma about three times slower: 152 against 48 clocks per instruction, measured.)
    // Every trip makes its barrier calls, issues and commits whether or not a wait for a load gave up (see mbar_wait_issued).
    reg_dec<REGS_ROLE>();
    const uint32_t IDESC_O = make_idesc(BM, 2 * args.d, 0, 1, BF);    // V is MN-major; head dim 32: the 64 real value columns only
    constexpr uint32_t IDESC_S = make_idesc(BM, SUB, 0, 0, BF);
    constexpr uint32_t HALF = (SUB * 128) >> 4;
    const uint32_t v_lo0 = sdesc_lo(smem_u32(smem + OFF_V), V_BYTES / 2);
    const int kd = args.d >> 4;
    const uint32_t q_lo = sdesc_lo(smem_u32(smem + OFF_Q1));
    const uint32_t k_lo0 = sdesc_lo(smem_u32(smem + OFF_K));
    auto issue_s = [&](uint32_t k_lo, int br, int u) {
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        if (k < kd)
          mma_ss_lo(tmem_base + br * 128 + u * SUB, q_lo + br * (Q_BYTES >> 4) + k * 2, k_lo + br * (K_BYTES >> 4) + u * HALF + k * 2, IDESC_S, k > 0);
      mma_commit(&misc->s_full[br][u]);
    };
    bool ok = true;
    int vs = 0, ks = 0;
    uint32_t k_par = 0;
    for (int it = 0; work.valid(); ++it, work.next()) {
      const int nkv = key_tiles(args.causal, args.n, work.item().tile);
      ok = ok && mbar_wait_warp(&misc->bar_q, it & 1, abort_flag, 201, it);
      ok = ok && mbar_wait_warp(&misc->k_full[ks], k_par, abort_flag, 202, it);
      tc_fence_after();
      if (elect_one()) {
        const uint32_t k_lo = k_lo0 + ks * ((2 * K_BYTES) >> 4);
        for (int u = 0; u < 2; ++u)
          for (int br = 0; br < 2; ++br) issue_s(k_lo, br, u);
        mma_commit(&misc->k_empty[ks]);
        if (nkv == 1) mma_commit(&misc->q_empty);
      }
      __syncwarp();
      if (++ks == KS) { ks = 0; k_par ^= 1; }
      for (int j = 0; j < nkv; ++j) {
        const uint32_t v_lo = v_lo0 + vs * (V_BYTES >> 4);
        const uint32_t k_lo = k_lo0 + ks * ((2 * K_BYTES) >> 4);       // key tile j+1
        const bool more = j + 1 < nkv;
        named_bar_sync(NB_KV, 64);               // V of tile j and K of tile j + 1 have landed (the watcher warp)
        if (j == 0 && it > 0) named_bar_sync(NB_O, NUM_SOFTMAX + 32);  // the previous tile's accumulators are in registers
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int u = i >> 1, br = i & 1;
          named_bar_sync(NB_P + br * 2 + u, 160);
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < SUB / 16; ++k)
              mma_ts_lo(tmem_base + T_O + br * 128, tmem_base + br * 128 + u * SUB + k * 8, v_lo + u * HALF + k * (2048 >> 4), IDESC_O,
                        (j > 0 || u > 0 || k > 0));
            mma_commit(&misc->pv_done[br][u]);
            if (more) issue_s(k_lo, br, u);
            if (i == 3) {
              if (more) mma_commit(&misc->k_empty[ks]);
              if (j == nkv - 2) mma_commit(&misc->q_empty);
              mma_commit(&misc->v_empty[vs]);
            }
          }
          __syncwarp();
        }
        if (more && ++ks == KS) { ks = 0; k_par ^= 1; }
        if (++vs == VS) vs = 0;
      }
      if (elect_one()) mma_commit(&misc->o_full);
      __syncwarp();
    }
  } else if (warp == WARP_ALLOC) {
    // Load watcher: waits for V of tile j and K of tile j + 1 on behalf of the MMA issuer.  A wait on an mbarrier costs
    // 150-300 clocks while MMAs saturate shared memory, even when the phase completed long ago; a named barrier costs
    // a tenth of that, and the issuer is the busiest thread of the CTA.
    reg_dec<REGS_ROLE>();
    bool ok = true;
    int vs = 0, ks = 0;
    uint32_t v_par = 0, k_par = 0;
    for (; work.valid(); work.next()) {
      const int nkv = key_tiles(args.causal, args.n, work.item().tile);
      for (int j = 0; j < nkv; ++j) {
        if (++ks == KS) { ks = 0; k_par ^= 1; }          // key tile j + 1 (the issuer waits for tile 0 itself)
        ok = ok && mbar_wait_warp(&misc->v_full[vs], v_par, abort_flag, 205, j);
        if (j + 1 < nkv) ok = ok && mbar_wait_warp(&misc->k_full[ks], k_par, abort_flag, 203, j);
        named_bar_sync(NB_KV, 64);
        if (++vs == VS) { vs = 0; v_par ^= 1; }
      }
    }
  } else if (warp == WARP_STORE) {
    // y and a2 leave through the TMA engine from the V ring (idle between a tile's last P V and the next tile's first), the gained
    // y from the K slot that the next tile fills second.  A warp of its own waits for the engine, so nobody else does.
    reg_dec<REGS_ROLE>();
    const int dv_real = 2 * args.d;
    int ks = 0;
    for (; work.valid(); work.next()) {
      const WorkItem wi = work.item();
      ks = (ks + key_tiles(args.causal, args.n, wi.tile)) % KS;
      for (int br = 0; br < 2; ++br) {
        named_bar_sync(NB_STORE + br, NUM_SOFTMAX / 2 + 32);
        if (elect_one() && !*abort_flag && br * 64 < dv_real) {
          const uint8_t* ytile = smem + OFF_V + br * (2 * STORE_TILE_BYTES);
          tma_store_4d(ytile, &tm_y, br * 64, wi.tile * BM, wi.bh, 0);
          tma_store_4d(ytile + STORE_TILE_BYTES, &tm_a2, br * 64, wi.tile * BM, wi.bh, 0);
          if (args.gain) tma_store_4d(smem + OFF_K + ((ks + 1) % KS) * 2 * K_BYTES + br * STORE_TILE_BYTES, &tm_yg, br * 64, wi.tile * BM, wi.bh, 0);
          tma_store_commit();
        }
        __syncwarp();
      }
      tma_store_wait_read();       // (every lane: the elected one of either half has the groups)
      __syncwarp();
      if (lane == 0) mbar_arrive(&misc->stored);
    }
  } else {
    // ------------------------- softmax warpgroups + epilogue -------------------------
    reg_inc<REGS_SOFTMAX>();
    const int br = warp >> 3;                       // branch
    const int u = (warp >> 2) & 1;                  // sub-tile parity = score buffer of this warpgroup
    const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
    // query row inside the tile = TMEM lane; computed anew where it is needed (the softmax pass leaves no register to keep it)
    auto softmax_row = [] {
      uint32_t t;
      asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
      return int(t & 127u);
    };
    const float sl2 = args.sm_scale * 1.4426950408889634f;
    int tc = u;                                     // sub-tiles, counted on from tile to tile: tc >> 1 is the phase of the buffers' barriers
    for (; work.valid(); work.next()) {
      SoftmaxState st;
      {
        const WorkItem wi = work.item();
        const int row = softmax_row();
        const int nsub = 2 * key_tiles(args.causal, args.n, wi.tile);
        const uint32_t t_s = tmem_base + lane_base + br * 128 + u * SUB;
        const uint32_t t_o = tmem_base + lane_base + T_O + br * 128;
        DropWalk dr;
        if constexpr (DROP)
          dr = drop_walk_row(drop_key(args.seed_lo, args.seed_hi, uint32_t(wi.bh), uint32_t(br)), uint32_t(wi.tile * BM + row) >> 1, row & 1,
                             args.drop_thresh);
        const int t0 = tc - u, t_first = u ? -1 : tc, t_end = t0 + nsub;
        int seen = args.n;                            // visible key columns: up to the sequence end, up to the diagonal
        if (args.causal) seen = min(seen, wi.tile * BM + row + 1);
        seen += t0 * SUB;
        for (; tc < t_end; tc += 2) {
          mbar_wait_issued_warp(&misc->s_full[br][u], (tc >> 1) & 1, abort_flag, 301 + br, tc);
          tc_fence_after();
          // P_b V of sub-tile tc - 1 used the other buffer
          softmax_subtile<BF, DROP, DV>(
              st, t_s, t_s, t_o, tc == t_first, tc - t0, seen - tc * SUB, sl2, &misc->m_run[br][row], dr, [] {},
              [&] { named_bar_sync(NB_M + br * 2 + (u ^ 1), 256); }, [&] { if (tc + 1 < t_end) named_bar_arrive(NB_M + br * 2 + u, 256); },
              [&] { mbar_wait_issued_warp(&misc->pv_done[br][u ^ 1], ((tc - 1) >> 1) & 1, abort_flag, 305 + br, tc); }, [] {}, [] {});
          named_bar_arrive(NB_P + br * 2 + u, 160);
        }
      }
      work.forget();
      const int row = softmax_row();
      // ---- epilogue: every thread runs every barrier; only the global writes depend on abort_flag
      mbar_wait_issued_warp(&misc->o_full, work.round & 1, abort_flag, 311 + br);
      tc_fence_after();
      misc->m_end[br][u][row] = st.m;
      misc->l_end[br][u][row] = st.l;
      named_bar_sync(NB_ALL, NUM_SOFTMAX);
      float m_fin[2], l_fin[2];         // both branches of this row: the last running maximum, to which O_b is relative; row sum relative to it
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const float ma = misc->m_end[b][0][row], mb = misc->m_end[b][1][row];
        m_fin[b] = misc->m_run[b][row];
        l_fin[b] = misc->l_end[b][0][row] * ex2((ma - m_fin[b]) * sl2) + misc->l_end[b][1][row] * ex2((mb - m_fin[b]) * sl2);
      }
      const float lam = load_lambda(args.lambda_ptr, args.lambda_dtype);
      const float keep = DROP ? args.drop_scale : 1.f;       // kept probabilities are scaled by 1 / (1 - p)
      const float c1 = keep / l_fin[0], c2 = keep / l_fin[1];
      // this warpgroup owns value columns [32 q, 32 q + 32) of both accumulators
      const int q = br * 2 + u;
      uint32_t o1[32], o2[32];
      tmem_ld32(tmem_base + lane_base + T_O + q * 32, o1);
      tmem_ld32(tmem_base + lane_base + T_O + 128 + q * 32, o2);
      tc_wait_ld();
      tc_fence_before();
      if (work.has_next()) named_bar_arrive(NB_O, NUM_SOFTMAX + 32);
      float ssq = 0.f;
      const int dv_real = 2 * args.d;                      // 128, or 64 when the head dim is 32 (upper columns are padding)
      const bool pad = q * 32 >= dv_real;                  // head dim 32: columns 64..127 of the accumulators were never written
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float a2v = pad ? 0.f : __uint_as_float(o2[i]) * c2;
        const float av = pad ? 0.f : __uint_as_float(o1[i]) * c1 - lam * a2v;
        ssq += av * av;
        o1[i] = __float_as_uint(av);
        o2[i] = __float_as_uint(a2v);
      }
      misc->ssq[q][row] = ssq;
      named_bar_sync(NB_ALL, NUM_SOFTMAX);
      const float rstd = rsqrtf(((misc->ssq[0][row] + misc->ssq[1][row]) + (misc->ssq[2][row] + misc->ssq[3][row])) / float(dv_real) + args.eps);
      const float yscale = args.rms_norm ? args.out_scale * rstd : 1.f;
      const WorkItem wi = work.item();
      const int q_tile = wi.tile;
      const size_t grow = size_t(wi.bh) * args.n + size_t(q_tile) * BM + row;
      const bool write = q_tile * BM + row < args.n;     // rows past the sequence end are computed on zero padding and dropped
      // y and a2 leave through shared memory and the TMA engine: each thread lays its 32 columns into a swizzled
      // [128 rows][64 columns] tile in the (now idle) V ring, and the store warp stores the tiles.
      // (Row-per-thread global stores of 16-byte pieces cost 3.6 us per CTA, 8 % of the kernel at N = 4096.)
      {
        uint8_t* ytile = smem + OFF_V + br * (2 * STORE_TILE_BYTES);
        uint8_t* atile = ytile + STORE_TILE_BYTES;
        uint8_t* gtile = smem + OFF_K + ((tc >> 1) + 1) % KS * 2 * K_BYTES + br * STORE_TILE_BYTES;          // y * gain, only with a gain
        const float4* gp = reinterpret_cast<const float4*>(args.gain + q * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float f[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = __uint_as_float(o1[8 * i + k]) * yscale;
          uint4 av;
          av.x = pack2<BF>(__uint_as_float(o2[8 * i + 0]), __uint_as_float(o2[8 * i + 1]));
          av.y = pack2<BF>(__uint_as_float(o2[8 * i + 2]), __uint_as_float(o2[8 * i + 3]));
          av.z = pack2<BF>(__uint_as_float(o2[8 * i + 4]), __uint_as_float(o2[8 * i + 5]));
          av.w = pack2<BF>(__uint_as_float(o2[8 * i + 6]), __uint_as_float(o2[8 * i + 7]));
          st_swizzled_chunk(ytile, row, u * 4 + i, make_uint4(pack2<BF>(f[0], f[1]), pack2<BF>(f[2], f[3]), pack2<BF>(f[4], f[5]), pack2<BF>(f[6], f[7])));
          st_swizzled_chunk(atile, row, u * 4 + i, av);
          if (args.gain && !pad) {
            const float4 g0 = __ldg(gp + 2 * i), g1 = __ldg(gp + 2 * i + 1);
            st_swizzled_chunk(gtile, row, u * 4 + i, make_uint4(pack2<BF>(f[0] * g0.x, f[1] * g0.y), pack2<BF>(f[2] * g0.z, f[3] * g0.w),
                                                        pack2<BF>(f[4] * g1.x, f[5] * g1.y), pack2<BF>(f[6] * g1.z, f[7] * g1.w)));
          }
        }
        fence_proxy_async_smem();
        named_bar_arrive(NB_STORE + br, NUM_SOFTMAX / 2 + 32);
      }
      if (write && !*abort_flag && u == 0) {
        if (br == 0) {
          args.lse1[grow] = m_fin[0] * args.sm_scale + logf(l_fin[0]);
          args.rstd[grow] = rstd;
        } else {
          args.lse2[grow] = m_fin[1] * args.sm_scale + logf(l_fin[1]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == WARP_ALLOC) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace da
