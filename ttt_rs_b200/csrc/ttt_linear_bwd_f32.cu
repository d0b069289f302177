// Fused TTT-Linear backward scan of float32 tensors: a stage's work split over four groups of four warps, one stream on an SM.
// Same mathematics, layouts, saved state and order of operations as ttt_linear_bwd_kernel (ttt_linear_bwd.cu), which keeps a
// bf16 stage in one group of four warps and lets two streams share an SM.
//
// In float32 every product is six of the bf16 planes and a stage's operands fill the shared memory of an SM: one stream at a
// time, whose four warps left the tensor pipe idle for three quarters of a stage (6.4 us alone on an SM).  Walking back, only
// dW -> K dW -> second derivative of the LayerNorm gradient -> dZ1 -> dW is a chain from one stage to the next: what W
// gives runs ahead of it and the outputs behind it, each in a group of its own that keeps the tensor pipe busy meanwhile:
//   recover (warps 0..3): undoes the stage's update of W, Z1 = K W + b, Zbar, its LayerNorm backward dZbar, dGp' = -M'^T dZbar;
//   chain   (warps 4..7): K dW, the second derivative, dZ1, dW += dZbar^T Q + dZ1^T K, the bias gradient;
//   output  (warps 8..11): dq, dk, dv and the token_eta terms from the copies of W, dW, dZbar and dZ1 that the others leave;
//   prepare (warps 12..15): split of float32 tiles into bf16 planes and Q K^T (three warps), the copies (one lane).
// 64 stages, us, in one group / in four: 96 streams 419 / 309, 12 streams 411 / 297, 192 streams 617 / 537, 384 1134 / 995.
// The chain group is what the others wait for (9.0 k of 9.3 k cycles a stage, 550 mma.sync per scheduler among them).  The
// same split of a bf16 stage is slower than the one group from 12 streams (138 / 132 us) to 1024 (1185 / 667): its products
// take a sixth, and four programs of 25 KB together miss in the instruction cache (3.4 of 12.7 stalled warps).
//
// Groups meet on mbarriers only: full (a slot's copies have landed), ready (its planes and Q K^T too), empty (all have read the
// slot), and given / taken of three records: recover's (r), the copy of dW (d), chain's (z).  What a stage is -- stream,
// place in the sequence, end of the work item, end of the launch -- travels in its slot.  Every wait is bounded; a wait that
// runs out raises `stop`, which ends the others, and a group leaves where its next exchange has agreed on it.
#include "ttt_kernels.h"
#include "ttt_stage.cuh"

namespace ttt {

constexpr int BR_THREADS = 4 * NTHREADS;

template <int SEG>
struct BwdRoleSmem {
  using TF = TileFmt<float>;
  static constexpr int NP = TF::NP, NH = HD / SEG;
  static constexpr int NST = 2;  // stages' inputs
  static constexpr int NR = 2;   // recover -> chain, output
  static constexpr int ND = 1;   // dW copies, chain -> output
  static constexpr int NZ = 2;   // chain -> output
  static constexpr uint32_t PLANES = NP * TILE_BF16_BYTES;
  // a slot: q, k, gp (raw + operand planes), v, d_out (raw), then small records
  static constexpr uint32_t OFF_Q = 0, OFF_K = TF::BYTES, OFF_G = 2 * TF::BYTES, OFF_V = 3 * TF::BYTES;
  static constexpr uint32_t OFF_DO = OFF_V + TF::RAW_BYTES, OFF_STAT = OFF_DO + TF::RAW_BYTES;
  static constexpr uint32_t STAT_BYTES = NH * 512;
  static constexpr uint32_t OFF_BS = OFF_STAT + STAT_BYTES;  // 64 floats: the bias at the start of the stage
  static constexpr uint32_t OFF_LR = OFF_BS + 256;           // NH x 16 elements
  static constexpr uint32_t OFF_REC = OFF_LR + 128;          // int4: stream, stage, chunk, flags
  static constexpr uint32_t SLOT = OFF_STAT + (NH == 2 ? 2048 : 1024);
  static_assert(OFF_REC + 16 <= SLOT && SLOT % 1024 == 0, "");
  // recover's record: copy of What, dZbar tile, Z1, dGp' and the rows' sum of dZbar as the threads hold them
  static constexpr uint32_t R_W = 0, R_DZ = 4 * PLANES, R_Z1 = R_DZ + PLANES, R_DG = R_Z1 + NTHREADS * 32,
                            R_SUM = R_DG + NTHREADS * 32, R_LN = R_SUM + NTHREADS * 16, R_BYTES = R_LN + 1024;
  // chain's record: dZ1 tile, dT and a partial sum as the threads hold them
  static constexpr uint32_t Z_DZ1 = 0, Z_DT = PLANES, Z_PS = Z_DT + NTHREADS * 32, Z_BYTES = (Z_PS + NTHREADS * 4 + 1023) / 1024 * 1024;
  static constexpr uint32_t OFF_R = NST * SLOT;
  static constexpr uint32_t OFF_D = OFF_R + NR * R_BYTES;
  static constexpr uint32_t OFF_Z = OFF_D + ND * 4 * PLANES;
  static constexpr uint32_t OFF_AT = OFF_Z + NZ * Z_BYTES;
  static constexpr uint32_t AT_BYTES = NH * 2 * 32 * 16;     // Q K^T as accumulator fragments
  static constexpr uint32_t OFF_XCH = OFF_AT + NST * AT_BYTES;  // recover 2, chain 2
  static constexpr uint32_t OFF_OX = OFF_XCH + 4 * sizeof(Xch4);  // output: 2 x 4 floats
  static constexpr uint32_t OFF_BAR = OFF_OX + 32;
  static constexpr int NBAR = 3 * NST + 2 * NR + 2 * ND + 2 * NZ;
  static constexpr uint32_t OFF_STOP = OFF_BAR + NBAR * 8;
  static constexpr uint32_t TOTAL = OFF_STOP + 16;
  static constexpr uint32_t DYN_BYTES = TOTAL + 1024;
  static_assert(R_BYTES % 1024 == 0 && OFF_AT % 1024 == 0 && DYN_BYTES <= 232448, "");
};

// A wait that ends when its phase completes, when another wait of the block has run out, or when it runs out itself.
__device__ __forceinline__ bool mbar_wait_or_stop(uint32_t bar, uint32_t parity, uint32_t stop) {
  for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    uint32_t s;
    asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(s) : "r"(stop) : "memory");
    if (s != 0) return false;
  }
  asm volatile("st.volatile.shared.b32 [%0], %1;" ::"r"(stop), "r"(1u) : "memory");
  return false;
}
__device__ __forceinline__ void st_f4(uint32_t a, float x, float y, float z, float w) {
  asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ float4 ld_f4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

enum : int { BR_FIRST = 1, BR_LAST = 2, BR_END = 4 };  // a stage's place in its work item; no more stages

template <int SEG, int MB>
__global__ void __launch_bounds__(BR_THREADS, 1)
    ttt_linear_bwd_f32_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                                const __grid_constant__ CUtensorMap tm_g, const LinBwdParams p) {
  using T = float;
  using TF = TileFmt<T>;
  using SM = BwdRoleSmem<SEG>;
  constexpr int NP = TF::NP, NST = SM::NST, NR = SM::NR, ND = SM::ND, NZ = SM::NZ;
  constexpr uint32_t PL = TILE_BF16_BYTES;  // plane stride
  constexpr float INV_F = 1.f / SEG;        // features per head (LayerNorm row length)
  constexpr int NH = SM::NH;                // heads per tile
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u32 = smem_u32(smem_raw);
  const uint32_t base = (raw_u32 + 1023u) & ~1023u;
  uint8_t* const gbase = smem_raw + (base - raw_u32);
  const uint32_t b_full = base + SM::OFF_BAR, b_ready = b_full + 8 * NST, b_empty = b_ready + 8 * NST;
  const uint32_t b_rgiven = b_empty + 8 * NST, b_rtaken = b_rgiven + 8 * NR;
  const uint32_t b_dgiven = b_rtaken + 8 * NR, b_dtaken = b_dgiven + 8 * ND;
  const uint32_t b_zgiven = b_dtaken + 8 * ND, b_ztaken = b_zgiven + 8 * NZ;
  const uint32_t stop = base + SM::OFF_STOP;

  const int role = __shfl_sync(0xffffffffu, threadIdx.x >> 7, 0);
  Lane L;  // the thread's place in its group
  L.tid &= NTHREADS - 1;
  L.warp &= 3;
  L.nb = L.warp * 16;
  const int tid = L.tid, lane = L.lane, g = L.g, t = L.t, nb = L.nb;
  const int warp = __shfl_sync(0xffffffffu, L.warp, 0);  // (known to be the same in all lanes)
  const int hsel = L.warp >> 1;                // SEG = 32: which head of the pair this warp's columns belong to
  const int khalf = (SEG == 32) ? hsel : -1;   // and the k-range of W^T / dW^T that is its own block
  const int NS = p.NS;
  constexpr int PREP_WARPS = 3;  // (the fourth issues the copies)

  if (threadIdx.x == 0) {
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
    prefetch_tmap(&tm_do);
    prefetch_tmap(&tm_g);
    for (int i = 0; i < NST; ++i) {
      mbar_init(b_full + 8 * i, 1);
      mbar_init(b_ready + 8 * i, PREP_WARPS);
      mbar_init(b_empty + 8 * i, 12);
    }
    for (int i = 0; i < NR; ++i) {
      mbar_init(b_rgiven + 8 * i, 4);
      mbar_init(b_rtaken + 8 * i, 8);
    }
    for (int i = 0; i < ND; ++i) {
      mbar_init(b_dgiven + 8 * i, 4);
      mbar_init(b_dtaken + 8 * i, 4);
    }
    for (int i = 0; i < NZ; ++i) {
      mbar_init(b_zgiven + 8 * i, 4);
      mbar_init(b_ztaken + 8 * i, 4);
    }
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(stop), "r"(0u) : "memory");
    fence_mbar_init();
  }
  if constexpr (MB < CS) {
    // padding rows of every tile of the ring, and of the statistics and lr records: zero once; the copies only ever write the
    // first MB rows / records
    for (uint32_t e = threadIdx.x * 4; e < NST * SM::SLOT; e += BR_THREADS * 4) {
      const uint32_t o = e % SM::SLOT;
      bool pad = false;
      if (o < 2 * TF::BYTES) pad = io_pad<T, SEG, MB>(o % TF::BYTES);  // q, k
      else if (o < SM::OFF_V) pad = io_pad<T, 64, MB>(o - SM::OFF_G);  // gp: always in the 64-wide form
      else if (o < SM::OFF_STAT) pad = io_pad<T, SEG, MB>((o - SM::OFF_V) % TF::RAW_BYTES);  // v, d_out
      else if (o < SM::OFF_BS) pad = (o - SM::OFF_STAT) >= MB * 32 * NH;
      else if (o >= SM::OFF_LR && o < SM::OFF_REC) pad = true;
      if (pad) asm volatile("st.shared.b32 [%0], %1;" ::"r"(base + e), "r"(0u) : "memory");
    }
    fence_proxy_async_smem();
  }
  __syncthreads();
  pdl_go();  // (the reduction waits)

  const float te_row[2] = {ld_as_float<T>(p.token_eta, g), MB == CS ? ld_as_float<T>(p.token_eta, g + 8) : 0.f};
  const float te15 = ld_as_float<T>(p.token_eta, MB - 1);
  // as in the forward, the state is carried as What = W / wscale (wscale = -te15), which turns the reversal of a stage's
  // update into one tensor-core accumulation What -= Gp^T K
  const bool w_moves = (te15 != 0.f);
  const float wscale = w_moves ? -te15 : 1.f;
  const size_t HOFF = 2 * HD * HD + HD;
  // Of another chunk's hand-off: one lane per warp polls (bounded), the warp goes on behind it.
  auto await_handoff = [&](int stream, int crank, int stage) -> int {
    int ok = 1;
    if (lane == 0) {
      ok = 0;
      const volatile int* flag = p.sched + 1 + stream;
      for (uint32_t it = 0; it < p.handoff_polls; ++it) {
        if (*flag >= crank) {
          ok = 1;
          break;
        }
        __nanosleep(100);
      }
      __threadfence();
      if (!ok) {
        report_timeout(p.status, 15, stage);
        asm volatile("st.volatile.shared.b32 [%0], %1;" ::"r"(stop), "r"(1u) : "memory");
      }
    }
    return __shfl_sync(0xffffffffu, ok, 0);
  };

  if (role == 3) {
    // (shares of the registers: 80 + 3 x 144 = 4 x 128, what the launch has)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    if (warp == 3) {
      // ============================== copies ==============================
      if (elect_one()) {
        const int nitems = p.nstreams * p.NCH;
        int i = 0;  // stages issued
        bool ok = true;
        int item = p.sched != nullptr ? atomicAdd(&p.sched[0], 1) + p.item_base : (int)blockIdx.x;
        for (;;) {
          const bool end = item >= nitems;
          const int crank = item / p.nstreams, chunk = p.NCH - 1 - crank, stream = item - crank * p.nstreams;
          const int s_lo = end ? 0 : chunk * p.CH, s_hi = end ? 0 : min(s_lo + p.CH, NS) - 1;
          // (taken before this one is worked on: an item waits only for items with smaller numbers, and a block works on its
          // own in order)
          const int next = (end || p.sched == nullptr) ? nitems : atomicAdd(&p.sched[0], 1) + p.item_base;
          for (int s = s_hi; s >= s_lo; --s, ++i) {
            const int slot = i % NST;
            const uint32_t bar = b_full + 8 * slot, sl = base + slot * SM::SLOT;
            if (i >= NST && !mbar_wait_or_stop(b_empty + 8 * slot, ((i / NST) - 1) & 1, stop)) {
              ok = false;
              break;
            }
            const int flags = end ? BR_END : (s == s_hi ? BR_FIRST : 0) | (s == s_lo ? BR_LAST : 0);
            st_u4(sl + SM::OFF_REC, (uint32_t)stream, (uint32_t)s, (uint32_t)chunk, (uint32_t)flags);
            if (end) {
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
              break;
            }
            constexpr uint32_t TILE = TF::RAW_BYTES * MB / CS;
            const int r0 = stream * p.T + s * MB;
            mbar_expect_tx(bar, 5 * TILE + NH * MB * TF::ELT + 512u * NH * MB / CS + 256u);
            tma_load_tile<T>(sl + SM::OFF_G, &tm_g, r0, bar);  // saved tiles are kept in the packed 64-wide form
            tma_load_io<T, SEG>(sl + SM::OFF_K, &tm_k, stream, s * MB, p.T, bar);
            tma_load_io<T, SEG>(sl + SM::OFF_Q, &tm_q, stream, s * MB, p.T, bar);
            tma_load_io<T, SEG>(sl + SM::OFF_DO, &tm_do, stream, s * MB, p.T, bar);
            tma_load_io<T, SEG>(sl + SM::OFF_V, &tm_v, stream, s * MB, p.T, bar);
            bulk_load_1d(sl + SM::OFF_BS, p.b_stage + ((size_t)stream * (NS + 1) + s) * HD, 256u, bar);
            bulk_load_1d(sl + SM::OFF_STAT, p.stats + (size_t)r0 * 2 * NH, 512u * NH * MB / CS, bar);
#pragma unroll
            for (int j = 0; j < NH; ++j)  // ttt_lr_eta is [B, H, T]: the two heads of a pair are T elements apart
              bulk_load_1d(sl + SM::OFF_LR + j * CS * TF::ELT,
                           static_cast<const uint8_t*>(p.lr) + ((size_t)(NH * stream + j) * p.T + s * MB) * TF::ELT,
                           MB * TF::ELT, bar);
          }
          if (!ok || end) break;
          item = next;
        }
        // copies into this block's shared memory land before it leaves
        if (!ok)
          for (int j = max(0, i - NST); j < i; ++j) mbar_wait_bounded(b_full + 8 * (j % NST), (j / NST) & 1);
      }
      __syncwarp();
    } else if (warp < PREP_WARPS) {
      // ============================== prepare: operand planes of float32 tiles, Q K^T ==============================
      for (int n = 0;; ++n) {
        const int slot = n % NST;
        const uint32_t sl = base + slot * SM::SLOT, tq = sl + SM::OFF_Q, tk = sl + SM::OFF_K;
        const int4 rec0 = make_int4(0, 0, 0, BR_END);
        int fail = mbar_wait_or_stop(b_full + 8 * slot, (n / NST) & 1, stop) ? 0 : 1;
        const int4 rec = fail ? rec0 : *reinterpret_cast<const int4*>(gbase + slot * SM::SLOT + SM::OFF_REC);
        if (!(rec.w & BR_END)) {
          for (int c = tid; c < 3 * NTHREADS; c += 32 * PREP_WARPS) {
            const int which = c >> 7;
            split_tile_f32(which == 0 ? tk : which == 1 ? tq : sl + SM::OFF_G, c & (NTHREADS - 1));
          }
        }
        uint32_t any;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %1, 0;\n\tbar.red.or.pred p, 4, 96, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(any)
                     : "r"(fail)
                     : "memory");
        fail = (int)any;
        if (fail) break;
        if (rec.w & BR_END) {
          mbar_arrive_warp(b_ready + 8 * slot);
          break;
        }
        if (warp < 2) {
          // SEG = 64: an n-tile per warp; SEG = 32: a head per warp, over the head's own features
          float at[2][4] = {};
#pragma unroll
          for (int k0 = 0; k0 < (SEG == 64 ? 4 : 2); ++k0) {
            const int ks = SEG == 64 ? k0 : 2 * warp + k0;
            Pk<NP> ak[4], aq[4];
            ldsm_np<NP>(ak, tk + TF::PLANE_OFF + lane_off_io<T, SEG>(lane, 16 * ks), PL, false);
            ldsm_np<NP>(aq, tq + TF::PLANE_OFF + lane_off_io<T, SEG>(lane, 16 * ks), PL, false);
            // the A fragments of K are also the B fragments of Q K^T (the same four 8x8 blocks in another order)
            const Pk<NP> b0[2] = {ak[0], ak[2]}, b1[2] = {ak[1], ak[3]};
            if constexpr (SEG == 32) {
              mma_np2<NP>(at[0], aq, b0, at[1], aq, b1);
            } else {
              if (warp == 0) mma_np<NP>(at[0], aq, b0);
              else mma_np<NP>(at[0], aq, b1);
            }
          }
          const uint32_t dst = base + SM::OFF_AT + slot * SM::AT_BYTES + lane * 16;
          if constexpr (SEG == 32) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) st_f4(dst + (2 * warp + nt) * 512, at[nt][0], at[nt][1], at[nt][2], at[nt][3]);
          } else {
            st_f4(dst + warp * 512, at[0][0], at[0][1], at[0][2], at[0][3]);
          }
        }
        mbar_arrive_warp(b_ready + 8 * slot);
      }
    }
  } else if (role == 0) {
    // ============================== recover: W, Zbar, dZbar ==============================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    Xch4* const xch = reinterpret_cast<Xch4*>(gbase + SM::OFF_XCH);
    const float winv = 1.f / wscale;
    float wt[8][4];
#pragma unroll
    for (int kt = 0; kt < 8; ++kt)
#pragma unroll
      for (int i = 0; i < 4; ++i) wt[kt][i] = 0.f;
    F2 gam[2] = {}, dgam[2] = {}, dbet[2] = {};
    int ck_idx = 0, s_ck = 0, xsel = 0;
    int fail = 0;
    bool fresh = false;  // wt holds a checkpoint as it was read
    auto read_ckpt = [&](int stream) {
      const float4* wc = reinterpret_cast<const float4*>(p.w_ckpt + ((size_t)stream * (p.NCK + 1) + ck_idx) * HD * HD);
#pragma unroll
      for (int kt = 0; kt < 8; ++kt) {
        const float4 v = __ldcg(wc + kt * NTHREADS + tid);
        wt[kt][0] = v.x; wt[kt][1] = v.y; wt[kt][2] = v.z; wt[kt][3] = v.w;
      }
      fresh = true;
      --ck_idx;
      s_ck = ck_idx * p.K - 1;  // (the last interval of the sequence may be shorter than the others)
    };
    for (int n = 0;; ++n) {
      const int slot = n % NST, rb = n % NR;
      const uint32_t sl = base + slot * SM::SLOT;
      const uint32_t tdo = sl + SM::OFF_DO, pq = sl + SM::OFF_Q + TF::PLANE_OFF, pk = sl + SM::OFF_K + TF::PLANE_OFF,
                     pg = sl + SM::OFF_G + TF::PLANE_OFF;
      const uint8_t* gsl = gbase + slot * SM::SLOT;
      const uint32_t rr = base + SM::OFF_R + rb * SM::R_BYTES;
      if (!mbar_wait_or_stop(b_ready + 8 * slot, (n / NST) & 1, stop)) fail = 1;
      const int4 rec = fail ? make_int4(0, 0, 0, 0) : *reinterpret_cast<const int4*>(gsl + SM::OFF_REC);
      if (rec.w & BR_END) {
        group_sync_or<1>(1);
        break;
      }
      const int stream = rec.x, s = rec.y;
      if (rec.w & BR_FIRST) {
        const int head = stream % p.H;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const int c = nb + 8 * nt + 2 * t;
          gam[nt] = f2(ld_as_float<T>(p.ln_g, (size_t)head * HD + c), ld_as_float<T>(p.ln_g, (size_t)head * HD + c + 1));
          dgam[nt] = dbet[nt] = f2(0.f);
        }
        // the next stage (walking down) that ends a checkpoint interval, and the checkpoint that holds the state after it
        ck_idx = s / p.K + 1;
        s_ck = min(ck_idx * p.K, NS) - 1;
        if (s_ck == s) {
          read_ckpt(stream);
        } else {
          --ck_idx;
          s_ck = ck_idx * p.K - 1;
          // (a chunk that ends inside a checkpoint interval: the state comes from the later chunk)
          if (!await_handoff(stream, p.NCH - 1 - rec.z, s)) {
            fail = 1;
          } else {
            const float4* ho = reinterpret_cast<const float4*>(p.handoff + (size_t)stream * HOFF);
#pragma unroll
            for (int kt = 0; kt < 8; ++kt) {
              const float4 a = __ldcg(ho + kt * NTHREADS + tid);
              wt[kt][0] = a.x; wt[kt][1] = a.y; wt[kt][2] = a.z; wt[kt][3] = a.w;
            }
          }
        }
      }
      if (fresh) {
#pragma unroll
        for (int kt = 0; kt < 8; ++kt)
#pragma unroll
          for (int i = 0; i < 4; ++i) wt[kt][i] *= winv;
        fresh = false;
      }
      // ---- 1. W_s from W_{s+1}: undo the stage's update with the saved Gp; b_s as saved
      if (w_moves) {
        Pk<NP> agt[4];
        ldsm_np<NP>(agt, pg + lane_off_B_nk(lane, nb), PL, true);
        const Pk<NP> ngt[4] = {neg_pk<NP>(agt[0]), neg_pk<NP>(agt[1]), neg_pk<NP>(agt[2]), neg_pk<NP>(agt[3])};
        state_update_direct<NP, SEG>(wt, ngt, pk, lane, khalf);
      }
      // ---- 2. Z1 = K W + b, Zq = Q W + b  (products with What: Z = wscale * acc + b); the fragments of What also go to the record
      // (whose last readers are past it by now: the slot this stage came in was theirs)
      if (n >= NR && !mbar_wait_or_stop(b_rtaken + 8 * rb, ((n / NR) - 1) & 1, stop)) fail = 1;
      float z1[2][4] = {}, zq[2][4] = {};
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        Pk<NP> bw[2][2], ak[4], aq[4];
        bfrag_from_state<NP>(wt, ks, bw);
        stsm_np<NP>(rr + SM::R_W + warp * SM::PLANES + lane_off_A(lane, 16 * ks), bw[0][0], bw[1][0], bw[0][1], bw[1][1]);
        ldsm_np<NP>(ak, pk + lane_off_io<T, SEG>(lane, 16 * ks), PL, false);
        ldsm_np<NP>(aq, pq + lane_off_io<T, SEG>(lane, 16 * ks), PL, false);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) mma_np2<NP>(z1[nt], ak, bw[nt], zq[nt], aq, bw[nt]);
      }
      {
        const float2 b0 = *reinterpret_cast<const float2*>(gsl + SM::OFF_BS + (nb + 2 * t) * 4);
        const float2 b1 = *reinterpret_cast<const float2*>(gsl + SM::OFF_BS + (nb + 8 + 2 * t) * 4);
        const float bias[4] = {b0.x, b0.y, b1.x, b1.y};
        scale_add(z1, wscale, bias);
        scale_add(zq, wscale, bias);
      }
      // ---- 3. Zbar = Zq - M' Gp   (am holds -M')
      Pk<NP> am[4];
#pragma unroll
      for (int jt = 0; jt < 2; ++jt) {
        const float4 a4 = ld_f4(base + SM::OFF_AT + slot * SM::AT_BYTES + (SEG == 32 ? hsel * 1024 : 0) + jt * 512 + lane * 16);
        const F2 at[2] = {f2(a4.x, a4.y), f2(a4.z, a4.w)};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int i = g + 8 * r, jj = 8 * jt + 2 * t;
          const F2 m = f2fma(at[r], f2(-te_row[r]), f2(-te_row[r]));
          am[2 * jt + r] = split_pack<NP>((jj <= i) ? m.x : 0.f, (jj + 1 <= i) ? m.y : 0.f);
        }
      }
      {
        Pk<NP> bg[4];
        ldsm_np<NP>(bg, pg + lane_off_B_kn(lane, nb), PL, true);
        const Pk<NP> b0[2] = {bg[0], bg[1]}, b1[2] = {bg[2], bg[3]};
        mma_np2<NP>(zq[0], am, b0, zq[1], am, b1);
      }
      // ---- 4. LN backward of the output (row statistics of Zbar saved by the forward) -> dZbar
      F2 dzb[2][2];
      {
        const float4* stat = reinterpret_cast<const float4*>(gsl + SM::OFF_STAT);
        const int rg = (SEG == 32) ? 2 * g + hsel : g, rg8 = (SEG == 32) ? 2 * (g + 8) + hsel : g + 8;
        const float4 sb0 = stat[2 * rg + 1], sb1 = stat[2 * rg8 + 1];
        const float mean2[2] = {sb0.x, sb1.x}, rstd2[2] = {sb0.y, sb1.y};
        F2 xz[2][2], tt[2][2];
        F2 p1[2] = {f2(0.f), f2(0.f)}, p2[2] = {f2(0.f), f2(0.f)};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const F2 d = ld_io<T, SEG>(tdo, g + 8 * r, nb + 8 * nt + 2 * t);
            const F2 x = f2mul(f2sub(pr(zq[nt], r), f2(mean2[r])), f2(rstd2[r]));
            xz[nt][r] = x;
            dgam[nt] = f2fma(d, x, dgam[nt]);
            dbet[nt] = f2add(dbet[nt], d);
            const F2 tv_ = f2mul(d, gam[nt]);
            tt[nt][r] = tv_;
            p1[r] = f2add(p1[r], tv_);
            p2[r] = f2fma(tv_, x, p2[r]);
          }
        float2 a0, a1;
        xch_rows2<SEG, true, 1>(&xch[xsel], L, f2hsum(p1[0]), f2hsum(p2[0]), f2hsum(p1[1]), f2hsum(p2[1]), a0, a1, fail);
        xsel ^= 1;
        if (fail) {
          if (tid == 0) report_timeout(p.status, 11, s);
          break;
        }
        const float c1[2] = {a0.x * INV_F, a1.x * INV_F}, c2[2] = {a0.y * INV_F, a1.y * INV_F};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r)
            dzb[nt][r] = f2mul(f2fma(xz[nt][r], f2(-c2[r]), f2sub(tt[nt][r], f2(c1[r]))), f2(rstd2[r]));
      }
      // ---- 5. the rest of the record: dZbar as an operand tile, Z1, dGp' = -M'^T dZbar
      const uint32_t tDZ = rr + SM::R_DZ;
      stsm_np<NP>(tDZ + lane_off_A(lane, nb), split_pack<NP>(dzb[0][0].x, dzb[0][0].y), split_pack<NP>(dzb[0][1].x, dzb[0][1].y),
                  split_pack<NP>(dzb[1][0].x, dzb[1][0].y), split_pack<NP>(dzb[1][1].x, dzb[1][1].y));
      __syncwarp();
      float dgp[2][4] = {};
      {
        Pk<NP> bdz[4];
        ldsm_np<NP>(bdz, tDZ + lane_off_B_kn(lane, nb), PL, true);  // (this warp's own columns)
        const Pk<NP> amt[4] = {movm_t_np<NP>(am[0]), movm_t_np<NP>(am[2]), movm_t_np<NP>(am[1]), movm_t_np<NP>(am[3])};
        const Pk<NP> z0[2] = {bdz[0], bdz[1]}, zz1[2] = {bdz[2], bdz[3]};
        mma_np2<NP>(dgp[0], amt, z0, dgp[1], amt, zz1);
      }
      {
        const F2 d0 = f2add(dzb[0][0], dzb[0][1]), d1 = f2add(dzb[1][0], dzb[1][1]);
        st_f4(rr + SM::R_SUM + tid * 16, d0.x, d0.y, d1.x, d1.y);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          st_f4(rr + SM::R_Z1 + (nt * NTHREADS + tid) * 16, z1[nt][0], z1[nt][1], z1[nt][2], z1[nt][3]);
          st_f4(rr + SM::R_DG + (nt * NTHREADS + tid) * 16, dgp[nt][0], dgp[nt][1], dgp[nt][2], dgp[nt][3]);
        }
      }
      if (rec.w & BR_LAST) {
        // this group's part of the LayerNorm gradients of the item, and W for the chunk before where that needs it
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float a = col_sum(dgam[nt].x), b = col_sum(dgam[nt].y), c = col_sum(dbet[nt].x), d = col_sum(dbet[nt].y);
          if (g == 0) st_f4(rr + SM::R_LN + (nb / 2 + 4 * nt + t) * 16, a, b, c, d);
        }
        if (rec.z > 0 && s % p.K != 0) {
          float4* ho = reinterpret_cast<float4*>(p.handoff + (size_t)stream * HOFF);
#pragma unroll
          for (int kt = 0; kt < 8; ++kt) ho[kt * NTHREADS + tid] = make_float4(wt[kt][0], wt[kt][1], wt[kt][2], wt[kt][3]);
          __threadfence();
        }
      }
      mbar_arrive_warp(b_rgiven + 8 * rb);
      mbar_arrive_warp(b_empty + 8 * slot);
      if (!(rec.w & BR_LAST) && s - 1 == s_ck) read_ckpt(stream);  // (in flight until the next stage is there)
    }
  } else if (role == 1) {
    // ============================== chain: dW, dZ1 ==============================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    Xch4* const xch = reinterpret_cast<Xch4*>(gbase + SM::OFF_XCH) + 2;
    float dwt[8][4];
#pragma unroll
    for (int kt = 0; kt < 8; ++kt)
#pragma unroll
      for (int i = 0; i < 4; ++i) dwt[kt][i] = 0.f;
    F2 gam[2] = {}, bet[2] = {}, dgam[2] = {}, dbet[2] = {}, dbias[2] = {};
    int xsel = 0, fail = 0;
    for (int n = 0;; ++n) {
      const int slot = n % NST, rb = n % NR, db = n % ND, zb = n % NZ;
      const uint32_t sl = base + slot * SM::SLOT;
      const uint32_t tk = sl + SM::OFF_K, tv = sl + SM::OFF_V, pq = sl + SM::OFF_Q + TF::PLANE_OFF, pk = tk + TF::PLANE_OFF;
      const uint8_t* gsl = gbase + slot * SM::SLOT;
      const uint32_t rr = base + SM::OFF_R + rb * SM::R_BYTES, rd = base + SM::OFF_D + db * 4 * SM::PLANES,
                     rz = base + SM::OFF_Z + zb * SM::Z_BYTES;
      if (!mbar_wait_or_stop(b_ready + 8 * slot, (n / NST) & 1, stop)) fail = 1;
      const int4 rec = fail ? make_int4(0, 0, 0, 0) : *reinterpret_cast<const int4*>(gsl + SM::OFF_REC);
      if (rec.w & BR_END) {
        group_sync_or<2>(1);
        break;
      }
      const int stream = rec.x, s = rec.y, chunk = rec.z, crank = p.NCH - 1 - chunk;
      float* const ho = p.handoff + (size_t)stream * HOFF;
      if (rec.w & BR_FIRST) {
        const int head = stream % p.H;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const int c = nb + 8 * nt + 2 * t;
          gam[nt] = f2(ld_as_float<T>(p.ln_g, (size_t)head * HD + c), ld_as_float<T>(p.ln_g, (size_t)head * HD + c + 1));
          bet[nt] = f2(ld_as_float<T>(p.ln_b, (size_t)head * HD + c), ld_as_float<T>(p.ln_b, (size_t)head * HD + c + 1));
          dgam[nt] = dbet[nt] = dbias[nt] = f2(0.f);
        }
        if (crank == 0) {
          // gradient flowing into the final state: zero (the reference's behaviour) unless the caller supplies it
#pragma unroll
          for (int kt = 0; kt < 8; ++kt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int k = 8 * kt + 2 * t + (i & 1), nn = nb + g + 8 * (i >> 1);
              if constexpr (SEG == 64) {
                dwt[kt][i] = (p.dw_in == nullptr) ? 0.f : ld_as_float<T>(p.dw_in, (size_t)stream * HD * HD + k * HD + nn);
              } else {
                // the head's own 32 x 32 block of the pair's block-diagonal dW^T; zero elsewhere
                dwt[kt][i] = (p.dw_in == nullptr || (kt >> 2) != hsel)
                                 ? 0.f
                                 : ld_as_float<T>(p.dw_in, (size_t)(2 * stream + hsel) * 32 * 32 + (k & 31) * 32 + (nn & 31));
              }
            }
          if (p.db_in != nullptr) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              const size_t o = (size_t)stream * HD + nb + 8 * nt + 2 * t;
              dbias[nt] = f2(ld_as_float<T>(p.db_in, o), ld_as_float<T>(p.db_in, o + 1));
            }
          }
        } else if (!await_handoff(stream, crank, s)) {
          fail = 1;
        } else {
#pragma unroll
          for (int kt = 0; kt < 8; ++kt) {
            const float4 b = __ldcg(reinterpret_cast<const float4*>(ho + HD * HD) + kt * NTHREADS + tid);
            dwt[kt][0] = b.x; dwt[kt][1] = b.y; dwt[kt][2] = b.z; dwt[kt][3] = b.w;
          }
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) dbias[nt] = __ldcg(reinterpret_cast<const float2*>(ho + 2 * HD * HD + nb + 8 * nt + 2 * t));
        }
      }
      // ---- 1. dW^T as operand fragments, K dW, and dW's copy for the output group
      float kdw[2][4] = {};
#pragma unroll
      for (int ks = 0; ks < 4; ks += 2) {
        Pk<NP> bd[2][2][2], ak[4], al[4];
        bfrag_from_state<NP>(dwt, ks, bd[0]);
        bfrag_from_state<NP>(dwt, ks + 1, bd[1]);
        ldsm_np<NP>(ak, pk + lane_off_io<T, SEG>(lane, 16 * ks), PL, false);
        ldsm_np<NP>(al, pk + lane_off_io<T, SEG>(lane, 16 * ks + 16), PL, false);
        mma_np2x2<NP>(kdw[0], kdw[1], ak, bd[0][0], bd[0][1], al, bd[1][0], bd[1][1]);
        if (ks == 0 && n >= ND && !mbar_wait_or_stop(b_dtaken + 8 * db, ((n / ND) - 1) & 1, stop)) fail = 1;
#pragma unroll
        for (int j = 0; j < 2; ++j)
          stsm_np<NP>(rd + warp * SM::PLANES + lane_off_A(lane, 16 * (ks + j)), bd[j][0][0], bd[j][1][0], bd[j][0][1], bd[j][1][1]);
      }
      mbar_arrive_warp(b_dgiven + 8 * db);
      const float lr_row[2] = {ld_as_float<T>(gsl + SM::OFF_LR, (SEG == 32 ? hsel * CS : 0) + g),
                               ld_as_float<T>(gsl + SM::OFF_LR, (SEG == 32 ? hsel * CS : 0) + g + 8)};
      const float4* stat = reinterpret_cast<const float4*>(gsl + SM::OFF_STAT);
      const int rg = (SEG == 32) ? 2 * g + hsel : g, rg8 = (SEG == 32) ? 2 * (g + 8) + hsel : g + 8;
      const float4 sa0 = stat[2 * rg], sa1 = stat[2 * rg8];
      const float mean1[2] = {sa0.x, sa1.x}, rstd1[2] = {sa0.y, sa1.y}, A[2] = {sa0.z, sa1.z}, Bv1[2] = {sa0.w, sa1.w};
      F2 btg[2][2];
      beta_minus_target<T, SEG>(bet, tk, tv, L, btg);
      if (!mbar_wait_or_stop(b_rgiven + 8 * rb, (n / NR) & 1, stop)) fail = 1;
      // ---- 2. LN + L2 pieces of Z1 from the saved row statistics
      F2 xh[2][2], gy[2][2], gx[2][2], G[2][2];
      {
        F2 z1p[2][2];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float4 z = ld_f4(rr + SM::R_Z1 + (nt * NTHREADS + tid) * 16);
          z1p[nt][0] = f2(z.x, z.y);
          z1p[nt][1] = f2(z.z, z.w);
        }
        float sa[2], sb[2];
        ln_l2_pieces(z1p, mean1, rstd1, gam, btg, xh, gy, gx, sa, sb);
        g_from_pieces(gx, xh, A, Bv1, rstd1, G);
      }
      // ---- 3. gradient reaching Gp and the first pair of second-derivative sums
      F2 u[2][2], v[2][2];
      float s1t[2], s2t[2], pgb;
      {
        F2 p1[2] = {f2(0.f), f2(0.f)}, p2[2] = {f2(0.f), f2(0.f)}, pdl[2] = {f2(0.f), f2(0.f)}, pg_ = f2(0.f);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float4 d4 = ld_f4(rr + SM::R_DG + (nt * NTHREADS + tid) * 16);
          const F2 dgp[2] = {f2(d4.x, d4.y), f2(d4.z, d4.w)};
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            // dL/dGp = -M'^T dZbar - te15 (K dW + db)
            const F2 dg = f2fma(f2add(pr(kdw[nt], r), dbias[nt]), f2(-te15), dgp[r]);
            pg_ = f2fma(f2mul(G[nt][r], f2(lr_row[r])), dbias[nt], pg_);
            pdl[r] = f2fma(dg, G[nt][r], pdl[r]);
            const F2 uu = f2mul(dg, f2(lr_row[r]));  // dL/dG
            const F2 vv = f2mul(uu, f2(-rstd1[r]));
            u[nt][r] = uu;
            v[nt][r] = vv;
            p1[r] = f2add(p1[r], vv);
            p2[r] = f2fma(vv, xh[nt][r], p2[r]);
          }
        }
        pgb = f2hsum(pg_);
        float4 o0, o1;
        xch_rows<SEG, true, 2, false>(&xch[xsel], L, make_float4(f2hsum(p1[0]), f2hsum(p2[0]), f2hsum(pdl[0]), 0.f),
                                      make_float4(f2hsum(p1[1]), f2hsum(p2[1]), f2hsum(pdl[1]), 0.f), o0, o1, fail);
        xsel ^= 1;
        if (fail) {
          if (tid == 0) report_timeout(p.status, 13, s);
          break;
        }
        s1t[0] = o0.x * INV_F; s2t[0] = o0.y * INV_F;
        s1t[1] = o1.x * INV_F; s2t[1] = o1.y * INV_F;
        // (every warp holds these row values; warp 2 writes them, of a pair of heads the first warp of each)
        if ((SEG == 32 ? (warp & 1) == 0 : warp == 2) && t == 0) {
          const size_t o = (SEG == 32 ? (size_t)(2 * stream + hsel) : (size_t)stream) * p.T + (size_t)s * MB;
          st_from_float<T>(p.d_lr, o + g, o0.z);
          if constexpr (MB == CS) st_from_float<T>(p.d_lr, o + g + 8, o1.z);
        }
      }
      // ---- 4. second derivative through LN + L2 gradient -> dZ1, dT; dW^T += dZbar^T Q
      F2 dz1[2][2], dT[2][2];
      {
        F2 pd[2] = {f2(0.f), f2(0.f)}, ps[2] = {f2(0.f), f2(0.f)};
        F2 dxh[2][2];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const F2 x = xh[nt][r], vv = v[nt][r];
            const F2 dgxh = f2fma(x, f2(s2t[r]), f2sub(f2(s1t[r]), vv));
            const F2 dy = f2mul(gam[nt], dgxh);
            dgam[nt] = f2fma(gy[nt][r], dgxh, f2fma(dy, x, dgam[nt]));
            dbet[nt] = f2add(dbet[nt], dy);
            const F2 dx = f2fma(dy, gam[nt], f2fma(gx[nt][r], f2(s2t[r]), f2mul(vv, f2(Bv1[r]))));
            dxh[nt][r] = dx;
            dT[nt][r] = f2neg(dy);
            pd[r] = f2add(pd[r], dx);
            ps[r] = f2fma(f2fma(dx, x, f2mul(u[nt][r], G[nt][r])), f2(-rstd1[r]), ps[r]);
          }
        {
          Pk<NP> adzt[4];
          ldsm_np<NP>(adzt, rr + SM::R_DZ + lane_off_B_nk(lane, nb), PL, true);
          state_update_direct<NP, SEG>(dwt, adzt, pq, lane, khalf);
        }
        float2 a0, a1;
        int f2_ = 0;
        xch_rows2<SEG, false, 2>(&xch[xsel], L, f2hsum(pd[0]), f2hsum(ps[0]), f2hsum(pd[1]), f2hsum(ps[1]), a0, a1, f2_);
        xsel ^= 1;
        const float D[2] = {a0.x * INV_F, a1.x * INV_F}, S[2] = {a0.y * INV_F, a1.y * INV_F};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r)
            dz1[nt][r] = f2fma(f2sub(dxh[nt][r], f2(D[r])), f2(rstd1[r]), f2mul(xh[nt][r], f2(S[r])));
      }
      // ---- 5. dW^T += dZ1^T K, the record (dZ1 as an operand tile, dT), the bias gradient
      {
        Pk<NP> pz[2][2], gt[2][2];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            pz[nt][r] = split_pack<NP>(dz1[nt][r].x, dz1[nt][r].y);
            gt[nt][r] = movm_t_np<NP>(pz[nt][r]);
          }
        const Pk<NP> agt[4] = {gt[0][0], gt[1][0], gt[0][1], gt[1][1]};
        state_update_direct<NP, SEG>(dwt, agt, pk, lane, khalf);
        if (n >= NZ && !mbar_wait_or_stop(b_ztaken + 8 * zb, ((n / NZ) - 1) & 1, stop)) fail = 1;
        stsm_np<NP>(rz + SM::Z_DZ1 + lane_off_A(lane, nb), pz[0][0], pz[0][1], pz[1][0], pz[1][1]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          st_f4(rz + SM::Z_DT + (nt * NTHREADS + tid) * 16, dT[nt][0].x, dT[nt][0].y, dT[nt][1].x, dT[nt][1].y);
        }
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(rz + SM::Z_PS + tid * 4), "f"(pgb) : "memory");
      }
      mbar_arrive_warp(b_zgiven + 8 * zb);
      mbar_arrive_warp(b_empty + 8 * slot);
      {
        const float4 ds = ld_f4(rr + SM::R_SUM + tid * 16);
        const F2 dzsum[2] = {f2(ds.x, ds.y), f2(ds.z, ds.w)};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const F2 cs = f2add(dzsum[nt], f2add(dz1[nt][0], dz1[nt][1]));
          dbias[nt] = f2add(dbias[nt], f2(col_sum(cs.x), col_sum(cs.y)));
        }
      }
      if (rec.w & BR_LAST) {
        // ---- end of the item: LN partials of this (stream, chunk); then either hand the state to the earlier chunk or, for
        // the first chunk of the sequence, write the gradients w.r.t. the initial state
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float a = col_sum(dgam[nt].x), b = col_sum(dgam[nt].y), c = col_sum(dbet[nt].x), d = col_sum(dbet[nt].y);
          if (g == 0) {
            const float4 o = ld_f4(rr + SM::R_LN + (nb / 2 + 4 * nt + t) * 16);
            float* pl = p.part_ln + ((size_t)stream * p.NCH + chunk) * 2 * HD + nb + 8 * nt + 2 * t;
            pl[0] = o.x + a;
            pl[1] = o.y + b;
            pl[HD] = o.z + c;
            pl[HD + 1] = o.w + d;
          }
        }
        if (chunk > 0) {
#pragma unroll
          for (int kt = 0; kt < 8; ++kt)
            reinterpret_cast<float4*>(ho + HD * HD)[kt * NTHREADS + tid] = make_float4(dwt[kt][0], dwt[kt][1], dwt[kt][2], dwt[kt][3]);
          if (g == 0) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) *reinterpret_cast<float2*>(ho + 2 * HD * HD + nb + 8 * nt + 2 * t) = dbias[nt];
          }
          __threadfence();
          if (!group_sync_or<2>(fail) && tid == 0) *reinterpret_cast<volatile int*>(p.sched + 1 + stream) = crank + 1;
        } else {
          const size_t wo = (size_t)stream * HD * HD;
#pragma unroll
          for (int kt = 0; kt < 8; ++kt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int k = 8 * kt + 2 * t + (i & 1), nn = nb + g + 8 * (i >> 1);
              if constexpr (SEG == 64) {
                const int idx = k * HD + nn;
                st_from_float<T>(p.d_w, wo + idx, dwt[kt][i]);
                if (p.part_w != nullptr) p.part_w[(size_t)stream * (HD * HD + HD) + idx] = dwt[kt][i];
              } else if ((kt >> 2) == hsel) {
                // the head's own 32 x 32 block, at the head's place in the caller's [B, H, 32, 32] layout
                const size_t hs = (size_t)(2 * stream + hsel);
                const int idx = (k & 31) * 32 + (nn & 31);
                st_from_float<T>(p.d_w, hs * 32 * 32 + idx, dwt[kt][i]);
                if (p.part_w != nullptr) p.part_w[hs * (32 * 32 + 32) + idx] = dwt[kt][i];
              }
            }
          if (g == 0) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              const float dbi[2] = {dbias[nt].x, dbias[nt].y};
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int c = nb + 8 * nt + 2 * t + e;
                st_from_float<T>(p.d_b, (size_t)stream * HD + c, dbi[e]);  // [B, H, 32] flat = [B, H/2, 64] flat
                if (p.part_w != nullptr) {
                  if constexpr (SEG == 64) p.part_w[(size_t)stream * (HD * HD + HD) + HD * HD + c] = dbi[e];
                  else p.part_w[(size_t)(2 * stream + hsel) * (32 * 32 + 32) + 32 * 32 + (c & 31)] = dbi[e];
                }
              }
            }
          }
        }
      }
      mbar_arrive_warp(b_rtaken + 8 * rb);
    }
  } else {
    // ============================== output: dq, dk, dv, token_eta terms ==============================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    float* const ox = reinterpret_cast<float*>(gbase + SM::OFF_OX);
    int fail = 0;
    for (int n = 0;; ++n) {
      const int slot = n % NST, rb = n % NR, db = n % ND, zb = n % NZ;
      const uint32_t sl = base + slot * SM::SLOT;
      const uint32_t tk = sl + SM::OFF_K, tdo = sl + SM::OFF_DO, pq = sl + SM::OFF_Q + TF::PLANE_OFF, pk = tk + TF::PLANE_OFF,
                     pg = sl + SM::OFF_G + TF::PLANE_OFF;
      const uint32_t rr = base + SM::OFF_R + rb * SM::R_BYTES, rd = base + SM::OFF_D + db * 4 * SM::PLANES,
                     rz = base + SM::OFF_Z + zb * SM::Z_BYTES;
      if (!mbar_wait_or_stop(b_ready + 8 * slot, (n / NST) & 1, stop)) fail = 1;
      const int4 rec = fail ? make_int4(0, 0, 0, 0) : *reinterpret_cast<const int4*>(gbase + slot * SM::SLOT + SM::OFF_REC);
      if (rec.w & BR_END) {
        group_sync_or<3>(1);
        break;
      }
      const int stream = rec.x, s = rec.y;
      if (!mbar_wait_or_stop(b_rgiven + 8 * rb, (n / NR) & 1, stop)) fail = 1;
      // ---- 1. P' = dZbar Gp^T (over the head's own columns), dq = d_out + dZbar W^T
      const uint32_t tDZ = rr + SM::R_DZ, tW = rr + SM::R_W;
      float pp[2][4] = {}, dq[2][4], dk[2][4] = {}, gl[2][4] = {}, xw[2][4] = {};
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const F2 d = ld_io<T, SEG>(tdo, g + 8 * r, nb + 8 * nt + 2 * t);
          dq[nt][2 * r] = d.x;
          dq[nt][2 * r + 1] = d.y;
        }
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        Pk<NP> adz[4], bwt[4];
        ldsm_np<NP>(adz, tDZ + lane_off_A(lane, 16 * ks), PL, false);
        ldsm_np<NP>(bwt, tW + ks * SM::PLANES + lane_off_B_kn(lane, nb), PL, true);
        if (SEG == 64 || (ks >> 1) == hsel) {
          // the A fragments of Gp serve as its B fragments (same 8x8 blocks, other order)
          Pk<NP> ags[4];
          ldsm_np<NP>(ags, pg + lane_off_A(lane, 16 * ks), PL, false);
          const Pk<NP> b0[2] = {ags[0], ags[2]}, b1[2] = {ags[1], ags[3]};
          mma_np2<NP>(pp[0], adz, b0, pp[1], adz, b1);
        }
        const Pk<NP> b0[2] = {bwt[0], bwt[1]}, b1[2] = {bwt[2], bwt[3]};
        mma_np2<NP>(xw[0], adz, b0, xw[1], adz, b1);
      }
      add_scaled(dq, wscale, xw);
      // ---- 2. Gl' = Gp dW^T
      if (!mbar_wait_or_stop(b_dgiven + 8 * db, (n / ND) & 1, stop)) fail = 1;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        Pk<NP> ags[4], bdw[4];
        ldsm_np<NP>(ags, pg + lane_off_A(lane, 16 * ks), PL, false);
        ldsm_np<NP>(bdw, rd + ks * SM::PLANES + lane_off_B_kn(lane, nb), PL, true);
        const Pk<NP> b0[2] = {bdw[0], bdw[1]}, b1[2] = {bdw[2], bdw[3]};
        mma_np2<NP>(gl[0], ags, b0, gl[1], ags, b1);
      }
      mbar_arrive_warp(b_dtaken + 8 * db);
      // ---- 3. dM' = -tril(P');  dA = dM' o te[i];  d te[i] = sum_j dM'[i,j] (1 + Attn[i,j]);  dq += dA K, dk = dA^T Q
      float dte_row[2];
      {
        Pk<NP> ada[4];
        F2 acc[2] = {f2(0.f), f2(0.f)};
#pragma unroll
        for (int jt = 0; jt < 2; ++jt) {
          const float4 a4 = ld_f4(base + SM::OFF_AT + slot * SM::AT_BYTES + (SEG == 32 ? hsel * 1024 : 0) + jt * 512 + lane * 16);
          const F2 at[2] = {f2(a4.x, a4.y), f2(a4.z, a4.w)};
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int i = g + 8 * r, jj = 8 * jt + 2 * t;
            const F2 d = f2((jj <= i) ? -pp[jt][2 * r] : 0.f, (jj + 1 <= i) ? -pp[jt][2 * r + 1] : 0.f);
            acc[r] = f2add(acc[r], f2fma(d, at[r], d));
            const F2 da = f2mul(d, f2(te_row[r]));
            ada[2 * jt + r] = split_pack<NP>(da.x, da.y);
          }
        }
        dte_row[0] = quad_sum(f2hsum(acc[0]));
        dte_row[1] = quad_sum(f2hsum(acc[1]));
        Pk<NP> bkt[4], bqt[4];
        ldsm_np<NP>(bkt, pk + lane_off_io<T, SEG>(lane, nb), PL, true);
        ldsm_np<NP>(bqt, pq + lane_off_io<T, SEG>(lane, nb), PL, true);
        const Pk<NP> adat[4] = {movm_t_np<NP>(ada[0]), movm_t_np<NP>(ada[2]), movm_t_np<NP>(ada[1]), movm_t_np<NP>(ada[3])};
        const Pk<NP> k0[2] = {bkt[0], bkt[1]}, k1[2] = {bkt[2], bkt[3]};
        const Pk<NP> q0[2] = {bqt[0], bqt[1]}, q1[2] = {bqt[2], bqt[3]};
        mma_np2<NP>(dq[0], ada, k0, dq[1], ada, k1);
        mma_np2<NP>(dk[0], adat, q0, dk[1], adat, q1);
      }
      float prt;
      {
        F2 ps[2] = {f2(0.f), f2(0.f)};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const F2 kk = ld_io<T, SEG>(tk, g + 8 * r, nb + 8 * nt + 2 * t);
            const F2 glp = pr(gl[nt], r);
            const F2 dkn = f2fma(glp, f2(-te15), pr(dk[nt], r));
            dk[nt][2 * r] = dkn.x;
            dk[nt][2 * r + 1] = dkn.y;
            ps[r] = f2fma(kk, glp, ps[r]);
          }
        prt = f2hsum(f2add(ps[0], ps[1]));
      }
      mbar_arrive_warp(b_empty + 8 * slot);
      // ---- 4. dk += dZ1 W^T;  dk = -dT + ..., dv = dT
      float xk[2][4] = {};
      if (!mbar_wait_or_stop(b_zgiven + 8 * zb, (n / NZ) & 1, stop)) fail = 1;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        Pk<NP> adz1[4], bwt[4];
        ldsm_np<NP>(adz1, rz + SM::Z_DZ1 + lane_off_A(lane, 16 * ks), PL, false);
        ldsm_np<NP>(bwt, tW + ks * SM::PLANES + lane_off_B_kn(lane, nb), PL, true);
        const Pk<NP> b0[2] = {bwt[0], bwt[1]}, b1[2] = {bwt[2], bwt[3]};
        mma_np2<NP>(xk[0], adz1, b0, xk[1], adz1, b1);
      }
      add_scaled(dk, wscale, xk);
      mbar_arrive_warp(b_rtaken + 8 * rb);
      F2 dT[2][2];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const float4 v = ld_f4(rz + SM::Z_DT + (nt * NTHREADS + tid) * 16);
        dT[nt][0] = f2(v.x, v.y);
        dT[nt][1] = f2(v.z, v.w);
      }
      {
        float pgb;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(pgb) : "r"(rz + SM::Z_PS + tid * 4) : "memory");
        prt = col_sum(quad_sum(prt + pgb));  // over the mini-batch and this warp's columns
      }
      mbar_arrive_warp(b_ztaken + 8 * zb);
      float* const oxb = ox + 4 * (n & 1);
      if (lane == 0) oxb[warp] = prt;
      if (!fail) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int row = g + 8 * r, col = nb + 8 * nt + 2 * t;
            const F2 dkk = f2sub(pr(dk[nt], r), dT[nt][r]);
            if (row < MB) {
              // (float32 pairs of four lanes are whole 32-byte sectors: straight to memory)
              const size_t o = SEG == 64 ? ((size_t)stream * p.T + (size_t)s * MB + row) * 64 + col
                                         : ((size_t)(2 * stream + hsel) * p.T + (size_t)s * MB + row) * 32 + (col & 31);
              *reinterpret_cast<float2*>(static_cast<float*>(p.d_q) + o) = make_float2(dq[nt][2 * r], dq[nt][2 * r + 1]);
              *reinterpret_cast<float2*>(static_cast<float*>(p.d_k) + o) = dkk;
              *reinterpret_cast<float2*>(static_cast<float*>(p.d_v) + o) = dT[nt][r];
            }
          }
      }
      fail = group_sync_or<3>(fail);
      if (fail) {
        if (tid == 0) report_timeout(p.status, 14, s);
        break;
      }
      if ((SEG == 32 ? (warp & 1) == 0 : warp == 3) && t == 0) {
        // per (batch, head) stream of the caller's tensors: the pair's heads are streams 2 * stream and 2 * stream + 1
        const float rt = SEG == 32 ? oxb[2 * hsel] + oxb[2 * hsel + 1] : (oxb[0] + oxb[1]) + (oxb[2] + oxb[3]);
        const size_t o = (SEG == 32 ? (size_t)(2 * stream + hsel) : (size_t)stream) * p.T + (size_t)s * MB;
        if constexpr (MB == CS) {
          p.part_te[o + g] = dte_row[0];
          p.part_te[o + g + 8] = dte_row[1] - (g == 7 ? rt : 0.f);
        } else {
          p.part_te[o + g] = dte_row[0] - (g == 7 ? rt : 0.f);  // the last token of an 8-token mini-batch is row 7
        }
      }
    }
  }
  __syncthreads();
}

template <int SEG, int MB>
static cudaError_t launch_t(const CUtensorMap* m, LinBwdParams& p, int nstreams, cudaStream_t st) {
  using SM = BwdRoleSmem<SEG>;
  auto kfn = ttt_linear_bwd_f32_kernel<SEG, MB>;
  static DeviceValue ready;
  int bytes = 0, sms = 0;
  cudaError_t e = ready.get(0, &bytes, [&](int* n) {
    // the groups' shares of the registers add up to those of the launch (the build fails otherwise; a library built in another
    // way must not wait for registers that do not exist)
    cudaFuncAttributes fa;
    const cudaError_t a = cudaFuncGetAttributes(&fa, kfn);
    if (a != cudaSuccess) return a;
    if (fa.numRegs != 128) return cudaErrorLaunchOutOfResources;
    *n = (int)SM::DYN_BYTES;
    return cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, *n);
  });
  if (e != cudaSuccess || (e = device_sms(&sms)) != cudaSuccess) return e;
  if (nstreams <= sms && p.item_base == 0) {
    // every stream alone on an SM: nothing to balance, so no chunks, no hand-offs of the state and no scheduler to clear
    p.CH = p.NS;
    p.NCH = 1;
    p.sched = nullptr;
  }
  const int nitems = nstreams * p.NCH;
  const int grid = sms < nitems ? sms : nitems;
  if (p.sched != nullptr && (e = cudaMemsetAsync(p.sched, 0, sizeof(int) * (size_t)(1 + nstreams), st)) != cudaSuccess)
    return e;
  kfn<<<grid, BR_THREADS, SM::DYN_BYTES, st>>>(m[0], m[1], m[2], m[3], m[7], p);
  return cudaGetLastError();
}
cudaError_t launch_linear_bwd_f32(int seg, int mb, const CUtensorMap* m, LinBwdParams& p, int nstreams, cudaStream_t st) {
  if (seg == 32) return mb == 8 ? launch_t<32, 8>(m, p, nstreams, st) : launch_t<32, 16>(m, p, nstreams, st);
  return mb == 8 ? launch_t<64, 8>(m, p, nstreams, st) : launch_t<64, 16>(m, p, nstreams, st);
}

}  // namespace ttt
