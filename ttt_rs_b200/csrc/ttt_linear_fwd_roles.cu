// Fused TTT-Linear forward scan with a stage's work split over three groups of four warps: the form for launches in which
// a stream has an SM to itself.  Same mathematics, layouts and saved state as ttt_linear_fwd_kernel (ttt_linear_fwd.cu),
// which keeps a stage in one group of four warps and lets two or three streams share an SM.
//
// Of a stage only W -> Z1 -> LayerNorm gradient -> W is a chain from one stage to the next; the output of the stage (its
// second product with W, the causal matrix, the second LayerNorm) hangs off it.  With one stream on an SM nothing else
// fills the chain's waits, and a group that does all of it adds the rest to every stage (64 stages, 12 to 148 streams, one group
// and three, inference: bf16 heads of 64 68 us and 58-60; pairs of 32-wide heads 74 and 61-62; f32 185 and 152-163; saving
// state for the backward: 73-74 and 66; 81-83 and 66-68; 191-193 and 163-171).  So:
//   chain  (warps 0..3): W^T in its accumulator registers; publishes the stage's W as operand fragments and the bias, forms
//          Z1, its LayerNorm gradient Gp, publishes Gp as operand fragments, updates W and the bias, saves what the backward reads;
//   output (warps 4..7): Zq = Q W + b from the published fragments, Zbar = Zq - M' Gp, the LayerNorm and the output tile --
//          about half a stage behind;
//   prepare (warps 8..11): the TMA loads, the split of float32 tiles into bf16 planes, M' = -te (1 + tril(Q K^T)) as operand
//          fragments -- a stage or two ahead.
// Groups meet on mbarriers only: full (a slot's copies have landed), ready (its planes and M' too), empty (chain and output
// have read the slot), given (the stage's W, bias and Gp fragments), taken (the output group has read them).  Every wait is
// bounded; a group agrees on a wait that ran out at its next exchange and leaves, and the others follow when theirs run out.
#include "ttt_kernels.h"
#include "ttt_stage.cuh"

namespace ttt {

constexpr int ROLE_THREADS = 3 * NTHREADS;

template <typename T, int SEG>
struct RoleSmem {
  using TF = TileFmt<T>;
  static constexpr int NP = TF::NP, NST = sizeof(T) == 2 ? 4 : 3, HPT = HD / SEG;
  static constexpr uint32_t SLOT = 3 * TF::BYTES;                       // q, k, v
  static constexpr uint32_t OFF_OUT = NST * SLOT;                       // staging (raw format): 2 x output, 2 x Gp
  static constexpr uint32_t OFF_W = OFF_OUT + 4 * TF::RAW_BYTES;        // 2 x [4 k-steps][NP][128 threads] uint4
  static constexpr uint32_t W_BYTES = 4 * NP * NTHREADS * 16;
  static constexpr uint32_t OFF_B = OFF_W + 2 * W_BYTES;                // 2 x [128 threads] float4: the bias
  static constexpr uint32_t OFF_G = OFF_B + 2 * NTHREADS * 16;          // 2 x [NP][128 threads] uint4
  static constexpr uint32_t G_BYTES = NP * NTHREADS * 16;
  static constexpr uint32_t OFF_M = OFF_G + 2 * G_BYTES;                // NST x [HPT][NP][32 lanes] uint4
  static constexpr uint32_t M_BYTES = HPT * NP * 32 * 16;
  static constexpr uint32_t LR_SLOT = (SEG == 32) ? 128 : 64;
  static constexpr uint32_t OFF_LR = OFF_M + NST * M_BYTES;
  static constexpr uint32_t OFF_XCH = OFF_LR + NST * LR_SLOT;           // 2 x Xch4 for the chain group, 2 for the output group
  static constexpr uint32_t OFF_BAR = OFF_XCH + 4 * sizeof(Xch4);       // full, ready, empty [NST]; given, taken [2]
  static constexpr uint32_t TOTAL = OFF_BAR + (3 * NST + 4) * 8;
  static constexpr uint32_t DYN_BYTES = TOTAL + 1024;  // slack for manual 1024-byte alignment
};

template <typename T, int SEG, int MB>
__global__ void __launch_bounds__(ROLE_THREADS, 1)
    ttt_linear_fwd_roles_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                                const __grid_constant__ CUtensorMap tm_g, const LinFwdParams p) {
  using TF = TileFmt<T>;
  using SM = RoleSmem<T, SEG>;
  constexpr int NP = TF::NP, NST = SM::NST, HPT = SM::HPT;
  constexpr bool TWO_PASS = (sizeof(T) == 4);
  constexpr float INV_F = 1.f / SEG;  // features per head (LayerNorm row length)

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u32 = smem_u32(smem_raw);
  const uint32_t base = (raw_u32 + 1023u) & ~1023u;
  uint8_t* const gbase = smem_raw + (base - raw_u32);
  const uint32_t bar_full = base + SM::OFF_BAR, bar_ready = bar_full + 8 * NST, bar_empty = bar_ready + 8 * NST,
                 bar_given = bar_empty + 8 * NST, bar_taken = bar_given + 16;

  const int role = __shfl_sync(0xffffffffu, threadIdx.x >> 7, 0);
  Lane L;  // the thread's place in its group
  L.tid &= NTHREADS - 1;
  L.warp &= 3;
  L.nb = L.warp * 16;
  const int tid = L.tid, lane = L.lane, g = L.g, t = L.t, nb = L.nb;
  const int warp = __shfl_sync(0xffffffffu, L.warp, 0);  // (known to be the same in all lanes)
  const int hsel = L.warp >> 1;              // SEG = 32: which head of the pair this warp's columns belong to
  const int khalf = (SEG == 32) ? hsel : -1;
  const int stream = blockIdx.x, head = stream % p.H, NS = p.NS;
  const int row_base = stream * p.T;  // first row of this stream in the [B*H*T, 64] view
  const bool save = (p.w_ckpt != nullptr);

  if (threadIdx.x == 0) {
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
    prefetch_tmap(&tm_o);
    prefetch_tmap(&tm_g);
    for (int i = 0; i < NST; ++i) {
      mbar_init(bar_full + 8 * i, 1);
      mbar_init(bar_ready + 8 * i, 4);
      mbar_init(bar_empty + 8 * i, 8);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_given + 8 * i, 4);
      mbar_init(bar_taken + 8 * i, 4);
    }
    fence_mbar_init();
  }
  if constexpr (MB < CS) {
    // padding rows of every tile of the ring, and the lr slots: zero once; the copies only ever write the first MB rows
    for (uint32_t e = threadIdx.x * 16; e < NST * SM::SLOT; e += ROLE_THREADS * 16)
      if (io_pad<T, SEG, MB>(e % TF::BYTES)) st_u4(base + e, 0u, 0u, 0u, 0u);
    for (uint32_t e = threadIdx.x * 4; e < NST * SM::LR_SLOT; e += ROLE_THREADS * 4)
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(base + SM::OFF_LR + e), "r"(0u) : "memory");
  }
  __syncthreads();
  pdl_join();

  const float te_row[2] = {ld_as_float<T>(p.token_eta, g), MB == CS ? ld_as_float<T>(p.token_eta, g + 8) : 0.f};
  const float te15 = ld_as_float<T>(p.token_eta, MB - 1);
  // The state is carried as What = W / wscale with wscale = -te15, so that the update W -= te15 Gp^T K becomes
  // What += Gp^T K, accumulated by the tensor cores straight into the registers.  (te15 == 0: W never changes.)
  const bool w_moves = (te15 != 0.f);
  const float wscale = w_moves ? -te15 : 1.f;
  Xch4* const xch = reinterpret_cast<Xch4*>(gbase + SM::OFF_XCH) + 2 * (role & 1);
  int xsel = 0, failed = 0;

  if (role == 2) {
    // ============================== prepare ==============================
    auto issue_loads = [&](int s) {  // one thread
      const int slot = s % NST;
      const uint32_t bar = bar_full + 8 * slot, tq = base + slot * SM::SLOT;
      constexpr uint32_t TILE = TF::RAW_BYTES * MB / CS;
      mbar_expect_tx(bar, 3 * TILE + HPT * MB * TF::ELT);
      tma_load_io<T, SEG>(tq + TF::BYTES, &tm_k, stream, s * MB, p.T, bar);
      tma_load_io<T, SEG>(tq + 2 * TF::BYTES, &tm_v, stream, s * MB, p.T, bar);
      tma_load_io<T, SEG>(tq, &tm_q, stream, s * MB, p.T, bar);
#pragma unroll
      for (int j = 0; j < HPT; ++j)  // ttt_lr_eta is [B, H, T]: the two heads of a pair are lr_ld elements apart
        bulk_load_1d(base + SM::OFF_LR + slot * SM::LR_SLOT + j * CS * TF::ELT,
                     static_cast<const uint8_t*>(p.lr) + ((size_t)(HPT * stream + j) * p.lr_ld + s * MB) * TF::ELT,
                     MB * TF::ELT, bar);
    };
    if (warp == 0 && elect_one())
      for (int s = 0; s < NST && s < NS; ++s) issue_loads(s);
    __syncwarp();
    for (int s = 0; s < NS; ++s) {
      const int slot = s % NST;
      const uint32_t tq = base + slot * SM::SLOT, tk = tq + TF::BYTES;
      int fail = mbar_wait_bounded(bar_full + 8 * slot, (s / NST) & 1) ? 0 : 1;
      if constexpr (NP == 3) {
        if (!fail) {
          split_tile_f32(tk, tid);
          split_tile_f32(tq, tid);
        }
      }
      failed = group_sync_or<3>(fail);
      if (failed) {  // the copies behind this stage's land before the block leaves
        for (int q = s + 1; q < NS && q <= max(NST - 1, s - 3 + NST); ++q) mbar_wait_bounded(bar_full + 8 * (q % NST), (q / NST) & 1);
        break;
      }
      // Q K^T: an n-tile per warp over all features (warps 0, 1), or per head over the head's own (warps 0..3)
      if (SEG == 32 || warp < 2) {
        const int nt = warp & 1;
        float at[4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ks += 2) {
          if (SEG == 32 && (ks >> 1) != hsel) continue;
          Pk<NP> ak[2][4], aq[2][4], b[2][2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            ldsm_np<NP>(ak[k], tk + TF::PLANE_OFF + lane_off_io<T, SEG>(lane, 16 * (ks + k)), TILE_BF16_BYTES, false);
            ldsm_np<NP>(aq[k], tq + TF::PLANE_OFF + lane_off_io<T, SEG>(lane, 16 * (ks + k)), TILE_BF16_BYTES, false);
            // the A fragments of K are also the B fragments of Q K^T (the same four 8x8 blocks in another order)
            b[k][0] = nt ? ak[k][1] : ak[k][0];
            b[k][1] = nt ? ak[k][3] : ak[k][2];
          }
          mma_np_n<NP, 2>({&at, &at}, {&aq[0], &aq[1]}, {&b[0], &b[1]});
        }
        Pk<NP> am[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int i = g + 8 * r, j = 8 * nt + 2 * t;
          const F2 m = f2fma(pr(at, r), f2(-te_row[r]), f2(-te_row[r]));
          am[r] = split_pack<NP>((j <= i) ? m.x : 0.f, (j + 1 <= i) ? m.y : 0.f);
        }
        const uint32_t dst = base + SM::OFF_M + slot * SM::M_BYTES + (SEG == 32 ? hsel * NP * 512 : 0) + lane * 16 + nt * 8;
#pragma unroll
        for (int pl = 0; pl < NP; ++pl)
          asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(dst + pl * 512), "r"(am[0].p[pl]), "r"(am[1].p[pl]) : "memory");
      }
      mbar_arrive_warp(bar_ready + 8 * slot);
      // the slot of the stage before last takes the next stage that is not on its way yet
      if (warp == 0) {
        const int sr = s - 2;
        if (sr >= 0 && sr + NST < NS && elect_one()) {
          if (mbar_wait_bounded(bar_empty + 8 * (sr % NST), (sr / NST) & 1)) issue_loads(sr + NST);
        }
        __syncwarp();
      }
    }
  } else if (role == 0) {
    // ============================== chain ==============================
    F2 gam[2], bet[2];
    float bias[4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const int c = nb + 8 * nt + 2 * t;
      gam[nt] = f2(ld_as_float<T>(p.ln_g, (size_t)head * HD + c), ld_as_float<T>(p.ln_g, (size_t)head * HD + c + 1));
      bet[nt] = f2(ld_as_float<T>(p.ln_b, (size_t)head * HD + c), ld_as_float<T>(p.ln_b, (size_t)head * HD + c + 1));
      bias[2 * nt] = ld_as_float<T>(p.b0, (size_t)stream * HD + c);
      bias[2 * nt + 1] = ld_as_float<T>(p.b0, (size_t)stream * HD + c + 1);
    }
    const float winv = 1.f / wscale;
    // state W^T[n][k], n in {nb+g, nb+g+8}: wt[kt][2*rn + e] = W[k = 8kt+2t+e][n = nb+g+8rn]
    float wt[8][4];
#pragma unroll
    for (int kt = 0; kt < 8; ++kt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = 8 * kt + 2 * t + (i & 1), n = nb + g + 8 * (i >> 1);
        if constexpr (SEG == 64) {
          wt[kt][i] = ld_as_float<T>(p.w0, (size_t)stream * HD * HD + k * HD + n) * winv;
        } else {
          // block-diagonal: head hsel's 32 x 32 state at rows / columns [32 hsel, 32 hsel + 32); zero elsewhere
          wt[kt][i] = ((kt >> 2) == hsel)
                          ? ld_as_float<T>(p.w0, (size_t)(2 * stream + hsel) * 32 * 32 + (k & 31) * 32 + (n & 31)) * winv
                          : 0.f;
        }
      }
    float4* ck_ptr = save ? reinterpret_cast<float4*>(p.w_ckpt + (size_t)stream * (p.NCK + 1) * HD * HD) : nullptr;
    float* bs_ptr = save ? p.b_stage + (size_t)stream * (NS + 1) * HD : nullptr;
    int ck_left = 0;

    int fail = mbar_wait_bounded(bar_ready, 0) ? 0 : 1;
    for (int s = 0, slot = 0; s < NS; ++s) {
      const int par = s & 1;
      const uint32_t tk = base + slot * SM::SLOT + TF::BYTES, tv = tk + TF::BYTES, pk = tk + TF::PLANE_OFF;
      // the stage's W as B operands, for this group's product and, through shared memory, for the output group's
      Pk<NP> bw[4][2][2];
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) bfrag_from_state<NP>(wt, ks, bw[ks]);
      float z1[2][4] = {};
#pragma unroll
      for (int ks = 0; ks < 4; ks += 2) {
        Pk<NP> ak[4], al[4];
        ldsm_np<NP>(ak, pk + lane_off_io<T, SEG>(lane, 16 * ks), TILE_BF16_BYTES, false);
        ldsm_np<NP>(al, pk + lane_off_io<T, SEG>(lane, 16 * ks + 16), TILE_BF16_BYTES, false);
        mma_np2x2<NP>(z1[0], z1[1], ak, bw[ks][0], bw[ks][1], al, bw[ks + 1][0], bw[ks + 1][1]);
      }
      // (under the products' latency)
      const float lr_row[2] = {
          ld_as_float<T>(gbase + SM::OFF_LR + slot * SM::LR_SLOT, (SEG == 32 ? hsel * CS : 0) + g),
          ld_as_float<T>(gbase + SM::OFF_LR + slot * SM::LR_SLOT, (SEG == 32 ? hsel * CS : 0) + g + 8)};
      F2 btg[2][2];
      beta_minus_target<T, SEG>(bet, tk, tv, L, btg);
      // saved state: W before the update of every K-th stage (as the threads hold it), the bias before every stage
      if (save) {
        if (ck_left == 0) {
#pragma unroll
          for (int kt = 0; kt < 8; ++kt)
            ck_ptr[kt * NTHREADS + tid] =
                make_float4(wt[kt][0] * wscale, wt[kt][1] * wscale, wt[kt][2] * wscale, wt[kt][3] * wscale);
          ck_ptr += HD * HD / 4;
          ck_left = p.K;
        }
        --ck_left;
        if (g == 0) {
#pragma unroll
          for (int j = 0; j < 4; ++j) bs_ptr[nb + 8 * (j >> 1) + 2 * t + (j & 1)] = bias[j];
        }
        bs_ptr += HD;
      }
      // products were taken with What: Z = wscale * acc + b
      F2 z1p[2][2];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int r = 0; r < 2; ++r) z1p[nt][r] = f2fma(pr(z1[nt], r), f2(wscale), f2(bias[2 * nt], bias[2 * nt + 1]));
      // LN statistics of Z1, then G = dL/dZ1 and Gp = lr[row] * G
      float mean[2], rstd[2];
      ln_row_stats<TWO_PASS, SEG, true, 1>(z1p, xch, xsel, L, p.eps, mean, rstd, fail);
      if (fail) {
        failed = 1;
        if (tid == 0) report_timeout(p.status, 2, s);
        break;
      }
      if (save && s > 0 && warp == 1) {  // the Gp tile of the stage before is complete behind this exchange
        if (elect_one()) {
          tma_store_tile<T>(&tm_g, row_base + (s - 1) * MB, base + SM::OFF_OUT + (2 + (par ^ 1)) * TF::RAW_BYTES);
          bulk_commit();
          bulk_wait_read<1>();
        }
        __syncwarp();
      }
      F2 gp[2][2];
      {
        F2 xh[2][2], gy[2][2], gx[2][2];
        float sa[2], sb[2];
        ln_l2_pieces(z1p, mean, rstd, gam, btg, xh, gy, gx, sa, sb);
        float2 a0, a1;
        int f2_ = 0;
        xch_rows2<SEG, false, 1>(&xch[xsel], L, sa[0], sb[0], sa[1], sb[1], a0, a1, f2_);
        xsel ^= 1;
        const float A[2] = {a0.x * INV_F, a1.x * INV_F}, Bv[2] = {a0.y * INV_F, a1.y * INV_F};
        const float rs[2] = {rstd[0] * lr_row[0], rstd[1] * lr_row[1]};
        g_from_pieces(gx, xh, A, Bv, rs, gp);
        if (save && t == 0 && (SEG == 64 ? warp == 0 : (warp & 1) == 0)) {
          // row statistics of Z1: the first of two float4 per token (SEG = 32: per token and head)
          float4* sp = p.stats + ((size_t)row_base + (size_t)s * MB) * (SEG == 64 ? 2 : 4);
          const int at0 = SEG == 64 ? 2 * g : 2 * (2 * g + hsel), step = SEG == 64 ? 16 : 32;
          sp[at0] = make_float4(mean[0], rstd[0], A[0], Bv[0]);
          if constexpr (MB == CS) sp[at0 + step] = make_float4(mean[1], rstd[1], A[1], Bv[1]);
        }
      }
      // (the barriers awaited at the end of the stage, asked now: the answer takes a hundred cycles that the chain need not wait)
      uint32_t taken = 1u, next_ready = 1u;
      const int next = slot + 1 == NST ? 0 : slot + 1;
      if (s >= 2) taken = mbar_try_wait(bar_taken + 8 * par, ((s >> 1) - 1) & 1);
      if (s + 1 < NS) next_ready = mbar_try_wait(bar_ready + 8 * next, ((s + 1) / NST) & 1);
      // Gp as tensor-core operands, transposed through movmatrix: gt[nt][r] = (Gp block rows 8r.., cols nb+8nt..)^T; the same
      // values go to the saved Gp tile (bf16: exactly the operand bits)
      const uint32_t sgt = base + SM::OFF_OUT + (2 + par) * TF::RAW_BYTES;
      Pk<NP> gt[2][2];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const Pk<NP> pkd = split_pack<NP>(gp[nt][r].x, gp[nt][r].y);
          gt[nt][r] = movm_t_np<NP>(pkd);
        }
      if (save) st_slab<T, 64>(sgt, lane, nb, gp);
      // state update: W^T[nb.., :] -= te15 * Gp^T K ; b -= te15 * colsum(Gp)
      {
        const Pk<NP> agt[4] = {gt[0][0], gt[1][0], gt[0][1], gt[1][1]};
        if (w_moves) state_update_direct<NP, SEG>(wt, agt, pk, lane, khalf);
      }
      // under its latency: the stage's fragments and bias to the output group, the next stage's tiles awaited
      if (!taken && !mbar_wait_bounded(bar_taken + 8 * par, ((s >> 1) - 1) & 1)) fail = 1;
      {
        const uint32_t dst = base + SM::OFF_W + par * SM::W_BYTES + tid * 16;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
          for (int pl = 0; pl < NP; ++pl)
            st_u4(dst + (ks * NP + pl) * NTHREADS * 16, bw[ks][0][0].p[pl], bw[ks][0][1].p[pl], bw[ks][1][0].p[pl], bw[ks][1][1].p[pl]);
        st_u4(base + SM::OFF_B + (par * NTHREADS + tid) * 16, __float_as_uint(bias[0]), __float_as_uint(bias[1]),
              __float_as_uint(bias[2]), __float_as_uint(bias[3]));
#pragma unroll
        for (int pl = 0; pl < NP; ++pl)
          st_u4(base + SM::OFF_G + par * SM::G_BYTES + (pl * NTHREADS + tid) * 16, gt[0][0].p[pl], gt[0][1].p[pl], gt[1][0].p[pl], gt[1][1].p[pl]);
        mbar_arrive_warp(bar_given + 8 * par);
      }
      if (save) fence_proxy_async_smem();  // (the Gp tile is stored behind the next stage's first exchange)
      if constexpr (NP == 1) {
        // column sums of the bf16 Gp tile as a product with a tile of ones (every row of the result is the sum)
        constexpr uint32_t ONES = 0x3F803F80u;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          float cs[4] = {0.f, 0.f, 0.f, 0.f};
          mma_bf16(cs, ONES, ONES, ONES, ONES, gt[nt][0].p[0], gt[nt][1].p[0]);
          bias[2 * nt] -= te15 * cs[0];
          bias[2 * nt + 1] -= te15 * cs[1];
        }
      } else {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const F2 cs = f2add(gp[nt][0], gp[nt][1]);
          bias[2 * nt] -= te15 * col_sum(cs.x);
          bias[2 * nt + 1] -= te15 * col_sum(cs.y);
        }
      }
      mbar_arrive_warp(bar_empty + 8 * slot);
      if (!next_ready && !mbar_wait_bounded(bar_ready + 8 * next, ((s + 1) / NST) & 1)) fail = 1;
      slot = next;
    }

    if (!failed) {
      // ---- final state (returned, and kept as the last checkpoint / last bias record for the backward)
      float4* wc = save ? reinterpret_cast<float4*>(p.w_ckpt + ((size_t)stream * (p.NCK + 1) + p.NCK) * HD * HD) : nullptr;
#pragma unroll
      for (int kt = 0; kt < 8; ++kt)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int idx = (8 * kt + 2 * t + (i & 1)) * HD + nb + g + 8 * (i >> 1);
          if constexpr (SEG == 64) {
            st_from_float<T>(p.w_out, (size_t)stream * HD * HD + idx, wt[kt][i] * wscale);
          } else if ((kt >> 2) == hsel) {
            // the head's own 32 x 32 block (rows and columns 32 hsel .. of the tile's state)
            st_from_float<T>(p.w_out, (size_t)(2 * stream + hsel) * 32 * 32 + ((idx >> 6) & 31) * 32 + (idx & 31),
                             wt[kt][i] * wscale);
          }
          if (save && i == 3)
            wc[kt * NTHREADS + tid] =
                make_float4(wt[kt][0] * wscale, wt[kt][1] * wscale, wt[kt][2] * wscale, wt[kt][3] * wscale);
        }
      if (g == 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = nb + 8 * (j >> 1) + 2 * t + (j & 1);
          st_from_float<T>(p.b_out, (size_t)stream * HD + c, bias[j]);
          if (save) p.b_stage[((size_t)stream * (NS + 1) + NS) * HD + c] = bias[j];
        }
      }
      if (save) {
        group_sync<1>();
        if (warp == 1 && elect_one()) {
          tma_store_tile<T>(&tm_g, row_base + (NS - 1) * MB, base + SM::OFF_OUT + (2 + ((NS - 1) & 1)) * TF::RAW_BYTES);
          bulk_commit();
        }
        __syncwarp();
      }
    }
    if (warp == 1 && elect_one()) bulk_wait_all<0>();
  } else {
    // ============================== output ==============================
    F2 gam[2], bet[2];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const int c = nb + 8 * nt + 2 * t;
      gam[nt] = f2(ld_as_float<T>(p.ln_g, (size_t)head * HD + c), ld_as_float<T>(p.ln_g, (size_t)head * HD + c + 1));
      bet[nt] = f2(ld_as_float<T>(p.ln_b, (size_t)head * HD + c), ld_as_float<T>(p.ln_b, (size_t)head * HD + c + 1));
    }
    auto store_out = [&](int s) {
      if (warp == 0) {
        if (elect_one()) {
          tma_store_io<T, SEG>(&tm_o, stream, s * MB, p.T, base + SM::OFF_OUT + (s & 1) * TF::RAW_BYTES);
          bulk_commit();
        }
        __syncwarp();
      }
    };
    for (int s = 0; s < NS; ++s) {
      const int slot = s % NST, par = s & 1;
      const uint32_t tq = base + slot * SM::SLOT, pq = tq + TF::PLANE_OFF;
      int fail = 0;
      if (warp == 0) {  // the staging tile this stage writes behind its exchange has left (the store of stage s - 2)
        if (elect_one()) bulk_wait_read<0>();
        __syncwarp();
      }
      // ---- Zq = Q W + b
      if (!mbar_wait_bounded(bar_ready + 8 * slot, (s / NST) & 1)) fail = 1;
      if (!mbar_wait_bounded(bar_given + 8 * par, (s >> 1) & 1)) fail = 1;
      float zq[2][4] = {};
      const uint32_t src = base + SM::OFF_W + par * SM::W_BYTES + tid * 16;
#pragma unroll
      for (int ks = 0; ks < 4; ks += 2) {
        Pk<NP> aq[2][4], b[2][2][2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          ldsm_np<NP>(aq[k], pq + lane_off_io<T, SEG>(lane, 16 * (ks + k)), TILE_BF16_BYTES, false);
#pragma unroll
          for (int pl = 0; pl < NP; ++pl) {
            const uint4 v = ld_u4(src + ((ks + k) * NP + pl) * NTHREADS * 16);
            b[k][0][0].p[pl] = v.x;
            b[k][0][1].p[pl] = v.y;
            b[k][1][0].p[pl] = v.z;
            b[k][1][1].p[pl] = v.w;
          }
        }
        mma_np2x2<NP>(zq[0], zq[1], aq[0], b[0][0], b[0][1], aq[1], b[1][0], b[1][1]);
      }
      {
        const uint4 b = ld_u4(base + SM::OFF_B + (par * NTHREADS + tid) * 16);
        const F2 bb[2] = {f2(__uint_as_float(b.x), __uint_as_float(b.y)), f2(__uint_as_float(b.z), __uint_as_float(b.w))};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const F2 z = f2fma(pr(zq[nt], r), f2(wscale), bb[nt]);
            zq[nt][2 * r] = z.x;
            zq[nt][2 * r + 1] = z.y;
          }
      }
      // ---- Zbar = Zq - M' Gp,  M'[i][j] = te[i] (1 + Attn[i][j]) for j <= i
      Pk<NP> am[4], gt[2][2];
#pragma unroll
      for (int pl = 0; pl < NP; ++pl) {
        const uint4 v = ld_u4(base + SM::OFF_M + slot * SM::M_BYTES + (SEG == 32 ? hsel * NP * 512 : 0) + pl * 512 + lane * 16);
        am[0].p[pl] = v.x;
        am[1].p[pl] = v.y;
        am[2].p[pl] = v.z;
        am[3].p[pl] = v.w;
      }
#pragma unroll
      for (int pl = 0; pl < NP; ++pl) {
        const uint4 v = ld_u4(base + SM::OFF_G + par * SM::G_BYTES + (pl * NTHREADS + tid) * 16);
        gt[0][0].p[pl] = v.x;
        gt[0][1].p[pl] = v.y;
        gt[1][0].p[pl] = v.z;
        gt[1][1].p[pl] = v.w;
      }
      mbar_arrive_warp(bar_taken + 8 * par);
      mma_np2<NP>(zq[0], am, gt[0], zq[1], am, gt[1]);
      // ---- out = Q + LN(Zbar)
      F2 zb[2][2];
      slab_pairs(zq, zb);
      float mean[2], rstd[2];
      ln_row_stats<TWO_PASS, SEG, true, 2>(zb, xch, xsel, L, p.eps, mean, rstd, fail);
      if (fail) {
        failed = 1;
        if (tid == 0) report_timeout(p.status, 3, s);
        break;
      }
      if (s > 0) store_out(s - 1);  // complete behind this exchange
      if (save && t == 0 && (SEG == 64 ? warp == 0 : (warp & 1) == 0)) {
        float4* sp = p.stats + ((size_t)row_base + (size_t)s * MB) * (SEG == 64 ? 2 : 4);
        const int at0 = (SEG == 64 ? 2 * g : 2 * (2 * g + hsel)) + 1, step = SEG == 64 ? 16 : 32;
        sp[at0] = make_float4(mean[0], rstd[0], 0.f, 0.f);
        if constexpr (MB == CS) sp[at0 + step] = make_float4(mean[1], rstd[1], 0.f, 0.f);
      }
      const uint32_t so = base + SM::OFF_OUT + par * TF::RAW_BYTES;
      F2 oo[2][2];
      ld_slab<T, SEG>(tq, lane, nb, oo);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const F2 x = f2mul(f2sub(zb[nt][r], f2(mean[r])), f2(rstd[r]));
          oo[nt][r] = f2add(oo[nt][r], f2fma(gam[nt], x, bet[nt]));
        }
      st_slab<T, SEG>(so, lane, nb, oo);
      mbar_arrive_warp(bar_empty + 8 * slot);
      fence_proxy_async_smem();  // (stored behind the next stage's exchange)
    }
    if (!failed) {
      group_sync<2>();
      store_out(NS - 1);
    }
    if (warp == 0 && elect_one()) bulk_wait_all<0>();
  }
  __syncthreads();
}

template <typename T, int SEG, int MB>
static cudaError_t launch_t(const CUtensorMap* m, const LinFwdParams& p, int nstreams, cudaStream_t st) {
  using SM = RoleSmem<T, SEG>;
  auto kfn = ttt_linear_fwd_roles_kernel<T, SEG, MB>;
  static DeviceValue ready;
  int bytes = 0;
  const cudaError_t e = ready.get(0, &bytes, [&](int* n) {
    *n = (int)SM::DYN_BYTES;
    return cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, *n);
  });
  if (e != cudaSuccess) return e;
  // (one block to an SM at most, so it does not matter which SMs the kernel before leaves first)
  return launch_dependent(kfn, nstreams, ROLE_THREADS, SM::DYN_BYTES, st, m[0], m[1], m[2], m[3], m[4], p);
}
template <typename T, int SEG>
static cudaError_t launch_mb(int mb, const CUtensorMap* m, const LinFwdParams& p, int nstreams, cudaStream_t st) {
  return mb == 8 ? launch_t<T, SEG, 8>(m, p, nstreams, st) : launch_t<T, SEG, 16>(m, p, nstreams, st);
}
cudaError_t launch_linear_fwd_roles(int dtype, int seg, int mb, const CUtensorMap* m, const LinFwdParams& p, int nstreams,
                                    cudaStream_t st) {
  if (seg == 32) return dtype == 1 ? launch_mb<__nv_bfloat16, 32>(mb, m, p, nstreams, st) : launch_mb<float, 32>(mb, m, p, nstreams, st);
  return dtype == 1 ? launch_mb<__nv_bfloat16, 64>(mb, m, p, nstreams, st) : launch_mb<float, 64>(mb, m, p, nstreams, st);
}

}  // namespace ttt
