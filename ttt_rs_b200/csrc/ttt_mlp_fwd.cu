// Fused TTT-MLP forward scan for sm_100a (bf16 I/O): one CTA of two groups of eight warps per (batch, head) stream.
//
// The reference has no fused kernel for the 2-layer inner model; its semantics are the unfused
// `TTTMLP::forward_mini_batch` (rust/core/src/mlp.rs:127-208; PyTorch twin reference/ttt.py:1107-1229), with the
// fused-kernel conventions of the linear path (token_eta read at [0, CS) in every stage).  Per 16-token stage, with
// F = 64, E = 256, Gp = lr o G, M'[i][j] = te[i] (1 + A[i][j]) for j <= i:
//     Z1 = K W1 + b1;  X2 = gelu(Z1);  Z2 = X2 W2 + b2;  G2 = d/dZ2 0.5|LN(Z2) - (V-K)|^2;  G1 = (G2 W2^T) o gelu'(Z1)
//     Zb1 = Q W1 + b1 - M1' G1p,  A1 = Q K^T;   Xb2 = gelu(Zb1);   Zb2 = Xb2 W2 + b2 - M2' G2p,  A2 = Xb2 X2^T
//     out = Q + LN(Zb2);   W1 -= te15 K^T G1p;  b1 -= te15 colsum(G1p);  W2 -= te15 X2^T G2p;  b2 -= te15 colsum(G2p)
//
// What bounds it: the chain W -> Z1 -> X2 -> Z2 -> G2 -> G1 -> W from one stage to the next on one SM (the state and its
// copies fill it), and the instructions of a stage: 16 warps issue them, 4 096 tanh twice, ~1 000 mma.sync.  So:
//  * Only that chain is the first group's work (warps 0..7).  The second group (warps 8..15) forms the stage's output from
//    what the chain publishes in shared memory -- bf16 copies of W1 and W2, X2, G1p, G2p -- about half a stage behind.
//  * Warp w of either group owns hidden features e in [32w, 32w+32) of every 16 x 256 tile, in mma accumulator layout, from Z1
//    to G1p and from Zb1 to Xb2.  Sums over all hidden features (Z2, Zb2) are formed by each warp over its own 32 straight from
//    registers; the eight partial tiles meet in shared memory, where a half-warp adds up a token's row and has the whole row for
//    its LayerNorm: two barriers of the group a stage in the chain, where column owners exchanging row sums needed six.
//  * A2 = Xb2 X2^T meets the same way, two of its rows per warp; each warp then forms a column tile of M2' G2p.
//  * A1 and M1' of the next stage are formed by one warp of the second group in turn while it would wait.
//  * The float32 masters of W1^T[e][k] and W2[e][n] are tensor-memory accumulators of 128 hidden features x 64; both rank-16
//    updates are tcgen05.mma into them (operands: the token tiles, tokens the contraction), and each warp of the chain reads its
//    32 rows back and refreshes their bf16 copies in shared memory, the operand of every product with the state.
// One group of eight warps with the masters in registers: 9.2 k cycles a stage, 48 streams of 31 stages 150 us, forward +
// backward of 192 streams of 128 stages 2 528 us; this form 6.8 k, 115 and 2 284 us.
//
// Scheduling.  One CTA fills an SM, so a launch of one CTA per stream runs in whole
// waves: 192 streams on 148 SMs cost two stream-times.  When the caller passes the backward's workspace (training),
// the kernel is launched persistently instead: blocks take work items (stream, chunk of stages: mlp_chunk_stages), first
// chunks of all streams first, and a chunk hands the state to the next one through the stream's workspace block (which
// is where the final state goes anyway) behind a per-stream counter -- the scheme of the TTT-Linear backward.
#include "ttt_kernels.h"
#include "ttt_common.cuh"
#include "ttt_stage.cuh"

namespace ttt {

constexpr int MLP_GROUP = 256;  // threads of a group
constexpr int MLP_THREADS = 2 * MLP_GROUP;
constexpr int MLP_E = 256;
constexpr int MLP_NST = 3;

struct MlpSmem {
  static constexpr uint32_t TILE = TILE_BF16_BYTES, ET = 4 * TILE;    // [16][64] bf16; [16 tok][256 e] = four of them
  static constexpr uint32_t SLOT = 3 * TILE;                          // q, k, v
  static constexpr uint32_t WC = MLP_E * HD * 2;                      // [256 e][64] bf16, 128-byte rows, swizzled
  static constexpr uint32_t PART = 8 * 4096;                          // float [8 warps][16][64]
  static constexpr uint32_t OFF_W1 = MLP_NST * SLOT;                  // copy of W1^T
  static constexpr uint32_t OFF_W2 = OFF_W1 + WC;                     // two copies of W2 (stage parity)
  static constexpr uint32_t OFF_X2 = OFF_W2 + 2 * WC;                 // two X2, then two G1p
  static constexpr uint32_t OFF_G1 = OFF_X2 + 2 * ET;
  static constexpr uint32_t OFF_G2 = OFF_G1 + 2 * ET;                 // two G2p
  static constexpr uint32_t OFF_PC = OFF_G2 + 2 * TILE;               // partials of Z2
  static constexpr uint32_t OFF_PO = OFF_PC + PART;                   // partials of Zb2
  static constexpr uint32_t OFF_B1 = OFF_PO + PART;                   // float [256]
  static constexpr uint32_t B2 = 8 * HD * 4;                          // b2 / wscale as shares of the eight warps of the chain
  static constexpr uint32_t OFF_B2 = OFF_B1 + MLP_E * 4;              // float [2][8][64] (stage parity)
  static constexpr uint32_t OFF_M1 = OFF_B2 + 2 * B2;                 // two bf16 [16][24]: -M1', then -M2' (stage parity)
  static constexpr uint32_t OFF_A2 = OFF_M1 + 2 * 16 * 24 * 2;        // float [8 warps][3][8][8]: partials of A2 (its lower blocks)
  static constexpr uint32_t OFF_LR = OFF_A2 + 8 * 768;                // MLP_NST x 32 bytes
  // mbarriers: full [MLP_NST], published [2], done [2], state, read, updates of W1, W2; then item, failure flag, tensor-memory base
  static constexpr uint32_t OFF_BAR = OFF_LR + MLP_NST * 32;
  static constexpr uint32_t OFF_WORDS = OFF_BAR + (MLP_NST + 8) * 8;
  static constexpr uint32_t TOTAL = OFF_WORDS + 16;
};
static_assert(MlpSmem::TOTAL <= 227 * 1024, "shared-memory tiles exceed one SM");
static_assert(MlpSmem::OFF_M1 % 16 == 0 && MlpSmem::OFF_LR % 16 == 0 && MlpSmem::OFF_BAR % 8 == 0, "alignment");

// tanh-approximated GELU of a column pair and (DERIV) its derivative times sc.  tanh(x) = 1 - 2 / (1 + e^{2x}) (relative error
// ~1e-6; the hardware tanh.approx is only good to ~5e-4, which shows after a few dozen chained stages).  The two quotients share
// one reciprocal, 1/a = b / (ab): the special-function unit, which a stage's 8 192 tanh keep busy for a thousand cycles, is
// asked three times instead of four.  Exponents stop at 2^60, where tanh is 1, so that the product stays finite.
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <bool DERIV>
__device__ __forceinline__ F2 gelu2(F2 z, F2& deriv, float sc) {
  constexpr float C0 = 0.7978845608028654f, C1 = 0.044715f, L2E2 = 2.f * 1.4426950408889634f;
  const F2 z2 = f2mul(z, z);
  const F2 a = f2mul(z, f2fma(z2, f2(L2E2 * C0 * C1), f2(L2E2 * C0)));
  const F2 d = f2add(f2(ex2_approx(fminf(a.x, 60.f)), ex2_approx(fminf(a.y, 60.f))), f2(1.f));
  const F2 th = f2fma(f2mul(f2(rcp_approx(d.x * d.y)), f2(d.y, d.x)), f2(-2.f), f2(1.f));
  const F2 hz = f2mul(z, f2(0.5f));
  if constexpr (DERIV) {
    // sc (0.5 z (1 - t^2) c0 (1 + 3 c1 z^2) + 0.5 (1 + t))
    const F2 sech2 = f2fma(f2neg(th), th, f2(1.f));
    const F2 poly = f2fma(z2, f2(sc * (3.f * C0 * C1)), f2(sc * C0));
    deriv = f2fma(f2mul(hz, sech2), poly, f2fma(th, f2(0.5f * sc), f2(0.5f * sc)));
  }
  return f2fma(hz, th, hz);
}

namespace {
template <int BAR>
__device__ __forceinline__ void mlp_group_sync() {
  asm volatile("bar.sync %0, %1;" ::"n"(BAR), "n"(MLP_GROUP) : "memory");
}
__device__ __forceinline__ float4 lds_f4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ F2 lds_pair(uint32_t a) {
  F2 v;
  asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_pair(uint32_t a, F2 v) { asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory"); }
__device__ __forceinline__ uint2 lds_u2(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds_word(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_word(uint32_t a, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ F2 bf_pair(uint32_t v) { return make_float2(bf16_lo(v), bf16_hi(v)); }
// four columns of a token's row summed over the eight warps' partial tiles (addresses: see `part_row`)
__device__ __forceinline__ void sum_partials(uint32_t a, F2 (&z)[2]) {
  float4 v[8];
#pragma unroll
  for (int w = 0; w < 8; ++w) v[w] = lds_f4(a + 4096 * w);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    F2 x[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) x[w] = h ? f2(v[w].z, v[w].w) : f2(v[w].x, v[w].y);
    z[h] = f2add(f2add(f2add(x[0], x[1]), f2add(x[2], x[3])), f2add(f2add(x[4], x[5]), f2add(x[6], x[7])));
  }
}
// sums of two values over the sixteen lanes that share a row
__device__ __forceinline__ F2 row_sum2(float a, float b) {
  F2 v = f2(a, b);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = f2add(v, f2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o)));
  return v;
}
}  // namespace

// SAVE: persistent, with the backward's workspace (the tests of a record pointer in the stage loop cost inference 1.5 %)
template <bool SAVE>
__global__ void __launch_bounds__(MLP_THREADS, 1)
    ttt_mlp_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                       const __grid_constant__ CUtensorMap tm_v, const MlpFwdParams p) {
  using T = __nv_bfloat16;
  using SM = MlpSmem;
  constexpr uint32_t TL = TILE_BF16_BYTES;

  extern __shared__ __align__(1024) uint8_t mlp_fwd_smem[];
  const uint32_t base = smem_u32(mlp_fwd_smem);
  if ((base & 1023u) != 0) {  // (the tiles need it; dynamic shared memory starts there when there is no static one)
    if (threadIdx.x == 0) report_timeout(p.status, 20, 0);
    return;
  }
  const uint32_t bar_full = base + SM::OFF_BAR, bar_pub = bar_full + 8 * MLP_NST, bar_done = bar_pub + 16,
                 bar_state = bar_done + 16, bar_read = bar_state + 8, bar_w1 = bar_read + 8, bar_w2 = bar_w1 + 8;
  const uint32_t w_item = base + SM::OFF_WORDS, w_fail = w_item + 4, w_tmem = w_item + 8;

  const bool output_group = __shfl_sync(0xffffffffu, threadIdx.x >> 8, 0) != 0;
  const int tid = threadIdx.x & (MLP_GROUP - 1), lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int NS = p.NS, CH = SAVE ? p.CH : NS, NCH = SAVE ? p.NCH : 1;
  const int nitems = SAVE ? p.nstreams * NCH : (int)gridDim.x;

  if (threadIdx.x < 32) tmem_alloc(w_tmem, 256);
  if (threadIdx.x == MLP_GROUP) {
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
    for (int i = 0; i < MLP_NST; ++i) mbar_init(bar_full + 8 * i, 1);
    for (int i = 0; i < 6; ++i) mbar_init(bar_pub + 8 * i, 8);
    mbar_init(bar_w1, 2);
    mbar_init(bar_w2, 2);
    fence_mbar_init();
    sts_word(w_fail, 0u);
  }
  tmem_fence_before_sync();
  __syncthreads();
  tmem_fence_after_sync();
  // tensor memory: W1^T, W2, each as two accumulators of 128 hidden features (lanes) x 64 columns
  const uint32_t tmem = lds_word(w_tmem);

  const float te15 = ld_as_float<T>(p.token_eta, CS - 1);
  // both states are carried divided by wscale = -te15, so that their rank-16 updates accumulate directly by mma
  const bool w_moves = (te15 != 0.f);
  const float wscale = w_moves ? -te15 : 1.f;

  // A lane's place in what ldmatrix / stmatrix (x4) take: rows lane & 15, the 16-byte chunk lane >> 4 of a 128-byte row.  The
  // chunks of k-step or column pair i: ^ (i << 5); the next chunk's blocks: ^ (1 << 4).
  const uint32_t tl = lane_off_A(lane, 0);
  const uint32_t own = (warp >> 1) * TL + (tl ^ ((warp & 1) << 6));  // this warp's 32 columns of a 16 x 256 tile
  const uint32_t wrow = warp * 32 * 128 + tl;                        // this warp's 32 rows of a copy of W1^T or W2
  // partial sums: a fragment's pairs (rows g, g + 8; column tile nt: ^ (nt << 5)) and a row owner's four columns
  const uint32_t part_frag = warp * 4096 + g * 256 + ((8 * t) ^ ((g & 3) << 5));
  const int row = 2 * warp + (lane >> 4), c4 = 4 * (lane & 15);
  const uint32_t part_row = row * 256 + ((4 * c4) ^ ((row & 3) << 5));
  const uint32_t tile_row = off_bf16(row, c4);

  // Waits.  One that runs out raises the block's failure flag; from then on nobody waits, all warps walk through the rest of
  // the item (every barrier of a group still met) and leave at its end.
  auto wait_for = [&](uint32_t bar, uint32_t parity, uint32_t where, int s) {
    if (mbar_try_wait(bar, parity)) return;
    for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
      if (mbar_try_wait(bar, parity)) return;
      if (lds_word(w_fail) != 0u) return;
    }
    sts_word(w_fail, 1u);
    if (lane == 0) report_timeout(p.status, where, s);
  };

  uint32_t n = 0;  // stages visited by this block so far (ring slot and barrier parities)
  for (int round = 0;; ++round) {
    // ---- next work item: (stream, chunk); one block per stream and a single chunk when not persistent
    int item;
    if constexpr (SAVE) {
      if (threadIdx.x == 0) sts_word(w_item, (uint32_t)atomicAdd(&p.sched[0], 1));
      __syncthreads();
      item = (int)lds_word(w_item);
      __syncthreads();
    } else {
      item = (round == 0) ? (int)blockIdx.x : nitems;
    }
    if (item >= nitems) break;
    const int chunk = SAVE ? item / p.nstreams : 0, stream = SAVE ? item - chunk * p.nstreams : item;
    const int head = stream % p.H, row_base = stream * p.T;
    const int s_lo = chunk * CH, s_hi = min(s_lo + CH, NS) - 1;
    // Optional: the backward's per-stream workspace block (layout in ttt_kernels.h).  The lr-scaled inner gradients of
    // every stage (the bf16 operands of the state updates) and the final state go there, so that the backward can
    // start its reverse walk at once.
    float* const bws = SAVE ? p.bwd_ws + (size_t)stream * p.bwd_ws_stride : nullptr;
    uint8_t* const rec0 = SAVE ? reinterpret_cast<uint8_t*>(bws + 4 * HD * MLP_E + MLP_BWD_HANDOFF_FLOATS) : nullptr;
    if (SAVE && chunk > 0) {
      // wait (bounded) until the previous chunk of this stream has parked its state in the workspace block
      int ok = 1;
      if (threadIdx.x == 0) {
        ok = 0;
        const volatile int* flag = p.sched + 1 + stream;
        for (uint32_t it = 0; it < p.handoff_polls; ++it) {
          if (*flag >= chunk) {
            ok = 1;
            break;
          }
          __nanosleep(100);
        }
        __threadfence();
      }
      if (__syncthreads_or(ok ? 0 : 1)) {
        if (threadIdx.x == 0) report_timeout(p.status, 22, item);
        break;
      }
    }
    const F2 gam[2] = {f2(ld_as_float<T>(p.ln_g, (size_t)head * HD + c4), ld_as_float<T>(p.ln_g, (size_t)head * HD + c4 + 1)),
                       f2(ld_as_float<T>(p.ln_g, (size_t)head * HD + c4 + 2), ld_as_float<T>(p.ln_g, (size_t)head * HD + c4 + 3))};
    const F2 bet[2] = {f2(ld_as_float<T>(p.ln_b, (size_t)head * HD + c4), ld_as_float<T>(p.ln_b, (size_t)head * HD + c4 + 1)),
                       f2(ld_as_float<T>(p.ln_b, (size_t)head * HD + c4 + 2), ld_as_float<T>(p.ln_b, (size_t)head * HD + c4 + 3))};

    if (!output_group) {
      // ============================== chain ==============================
      // warp w reads back lanes 32 (w % 4) .. of accumulator w / 4: the masters' rows e = 32 w + lane
      const uint32_t tm_own = tmem + ((32u * (uint32_t)(warp & 3)) << 16) + 64u * (uint32_t)(warp >> 2);
      const int e_own = 32 * warp + lane, b1_col = 32 * warp + 8 * (g >> 1) + 2 * t + (g & 1);
      // bf16 copy of 32 columns of this warp's rows of a master
      auto put_copy = [&](uint32_t copy, int cc, const float (&v)[8][4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          st_u4(copy + e_own * 128 + (((4 * cc + i) ^ (lane & 7)) << 4), pack_bf16(v[2 * i][0], v[2 * i][1]), pack_bf16(v[2 * i][2], v[2 * i][3]),
                pack_bf16(v[2 * i + 1][0], v[2 * i + 1][1]), pack_bf16(v[2 * i + 1][2], v[2 * i + 1][3]));
      };
      auto refresh = [&](uint32_t copy, int mat) {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float v[8][4];
          tmem_ld_8x4(tm_own + 128 * mat + 32 * cc, v);
          put_copy(copy, cc, v);
        }
      };
      // the rank-16 update of this half's 128 hidden features: one thread of warps 0 and 4
      auto issue_update = [&](int mat, uint32_t a_tile, uint32_t b_tile, uint32_t bar) {
        if ((warp & 3) == 0 && elect_one()) {
          tmem_fence_after_sync();
          if (w_moves) umma_update(tmem + 128 * mat + 16 * warp, a_tile + (warp >> 1) * TL, b_tile, UPD_IDESC);
          umma_commit_to(bar);
        }
        __syncwarp();
      };
      float b1c;  // b1[b1_col]
      {
        const float winv = 1.f / wscale;
        const float4* const parked = reinterpret_cast<const float4*>(bws) + warp * 16 * 32 + lane;  // (order: mlp_master_at)
#pragma unroll
        for (int mat = 0; mat < 2; ++mat)
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            float v[8][4];
            if (SAVE && chunk > 0) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float4 a = __ldcg(parked + mat * (HD * MLP_E / 4) + (8 * cc + i) * 32);
                v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
              }
            } else if (mat == 0) {  // the stream starts from the caller's initial state
#pragma unroll
              for (int i = 0; i < 32; ++i)
                v[i >> 2][i & 3] = ld_as_float<T>(p.w1, (size_t)stream * HD * MLP_E + (size_t)(32 * cc + i) * MLP_E + e_own) * winv;
            } else {
              const uint4* const src = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(p.w2) + ((size_t)stream * HD * MLP_E + (size_t)e_own * HD + 32 * cc) * 2);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint4 a = src[i];
                v[2 * i][0] = bf16_lo(a.x) * winv; v[2 * i][1] = bf16_hi(a.x) * winv; v[2 * i][2] = bf16_lo(a.y) * winv; v[2 * i][3] = bf16_hi(a.y) * winv;
                v[2 * i + 1][0] = bf16_lo(a.z) * winv; v[2 * i + 1][1] = bf16_hi(a.z) * winv; v[2 * i + 1][2] = bf16_lo(a.w) * winv; v[2 * i + 1][3] = bf16_hi(a.w) * winv;
              }
            }
            tmem_st_8x4(tm_own + 128 * mat + 32 * cc, v);
            put_copy(base + (mat == 0 ? SM::OFF_W1 : SM::OFF_W2 + (n & 1) * SM::WC), cc, v);
          }
        const float* const ho = bws + 4 * HD * MLP_E;
        const bool first = !SAVE || chunk == 0;
        b1c = first ? ld_as_float<T>(p.b1, (size_t)stream * MLP_E + b1_col) : __ldcg(ho + MLP_HO_B1 + b1_col);
        sts_word(base + SM::OFF_B1 + 4 * b1_col, __float_as_uint(b1c));
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // b2: the first warp's share
          const int c = lane + 32 * h;
          const float b = first ? ld_as_float<T>(p.b2, (size_t)stream * HD + c) : __ldcg(ho + MLP_HO_B2 + c);
          sts_word(base + SM::OFF_B2 + (n & 1) * SM::B2 + 4 * (warp * HD + c), warp == 0 ? __float_as_uint(b * winv) : 0u);
        }
        tmem_wait_st();
        tmem_fence_before_sync();
        mbar_arrive_warp(bar_state);
      }

      for (int s = s_lo; s <= s_hi; ++s, ++n) {
        const uint32_t slot = n % MLP_NST, par = n & 1;
        const uint32_t tq = base + slot * SM::SLOT, tk = tq + TL, tv = tk + TL;
        const uint32_t w2c = base + SM::OFF_W2 + par * SM::WC, tx2 = base + SM::OFF_X2 + par * SM::ET,
                       tg1 = base + SM::OFF_G1 + par * SM::ET, tg2 = base + SM::OFF_G2 + par * TL;
        uint8_t* const rec = SAVE ? rec0 + (size_t)s * MLP_REC_BYTES : nullptr;  // the backward's record of the stage
        if (SAVE) *reinterpret_cast<float*>(rec + MLP_REC_B1 + 4 * b1_col) = b1c;
        const uint32_t sh = base + SM::OFF_B2 + par * SM::B2 + warp * HD * 4;  // this warp's share of b2
        wait_for(bar_full + 8 * slot, (n / MLP_NST) & 1, 21, s);
        // ---- C1. Z1 = K W1 + b1 (this warp's hidden features), X2 = gelu(Z1), D1 = wscale gelu'(Z1)
        F2 d1[4][2];
        uint32_t x2[4][2];
        {
          float z1[4][4] = {};
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            uint32_t ak[4], b[2][4];
            ldsm_x4(ak, tk + (tl ^ (ks << 5)));
            ldsm_x4(b[0], (base + SM::OFF_W1 + wrow) ^ (ks << 5));
            ldsm_x4(b[1], (base + SM::OFF_W1 + wrow + 16 * 128) ^ (ks << 5));
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_bf16(z1[j], ak[0], ak[1], ak[2], ak[3], b[j >> 1][j & 1], b[j >> 1][2 + (j & 1)]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const F2 b1 = lds_pair(base + SM::OFF_B1 + 4 * (32 * warp + 8 * j + 2 * t));
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const F2 x = gelu2<true>(f2fma(pr(z1[j], r), f2(wscale), b1), d1[j][r], wscale);
              x2[j][r] = pack_bf16(x.x, x.y);
            }
          }
        }
        stsm_x4(tx2 + own, x2[0][0], x2[0][1], x2[1][0], x2[1][1]);
        stsm_x4((tx2 + own) ^ 32u, x2[2][0], x2[2][1], x2[3][0], x2[3][1]);
        // ---- C2. this warp's share of (X2 W2 + b2) / wscale (all 64 columns, its own 32 hidden features)
        {
          float z[8][4];
#pragma unroll
          for (int nt = 0; nt < 8; ++nt) {
            const F2 b = lds_pair(sh + 4 * (8 * nt + 2 * t));
            z[nt][0] = z[nt][2] = b.x;
            z[nt][1] = z[nt][3] = b.y;
          }
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int nt = 0; nt < 8; nt += 2) {
              uint32_t b[4];
              ldsm_x4_t(b, (w2c + wrow + 16 * 128 * c) ^ (nt << 4));
              mma_bf16(z[nt], x2[2 * c][0], x2[2 * c][1], x2[2 * c + 1][0], x2[2 * c + 1][1], b[0], b[1]);
              mma_bf16(z[nt + 1], x2[2 * c][0], x2[2 * c][1], x2[2 * c + 1][0], x2[2 * c + 1][1], b[2], b[3]);
            }
          const uint32_t pf = base + SM::OFF_PC + part_frag;
#pragma unroll
          for (int nt = 0; nt < 8; ++nt) {
            sts_pair(pf ^ (nt << 5), pr(z[nt], 0));
            sts_pair((pf ^ (nt << 5)) + 8 * 256, pr(z[nt], 1));
          }
        }
        F2 btg[2];  // beta - (v - k)
        {
          const uint2 v = lds_u2(tv + tile_row), k = lds_u2(tk + tile_row);
          btg[0] = f2sub(bet[0], f2sub(bf_pair(v.x), bf_pair(k.x)));
          btg[1] = f2sub(bet[1], f2sub(bf_pair(v.y), bf_pair(k.y)));
        }
        const uint32_t lr2 = lds_word(base + SM::OFF_LR + slot * 32 + 4 * warp);  // (rows 2 warp, 2 warp + 1)
        const float lr = lane < 16 ? bf16_lo(lr2) : bf16_hi(lr2);
        mlp_group_sync<1>();  // the partials of Z2
        // ---- C3. LN + L2 gradient of Z2 against V - K, a row per half-warp; G2p = lr o G2 to its operand tile
        F2 gp[2];
        {
          F2 z[2], x[2], gg[2];
          sum_partials(base + SM::OFF_PC + part_row, z);
          z[0] = f2mul(z[0], f2(wscale));
          z[1] = f2mul(z[1], f2(wscale));
          if (SAVE) *reinterpret_cast<float4*>(rec + MLP_REC_Z2 + 4 * (row * HD + c4)) = make_float4(z[0].x, z[0].y, z[1].x, z[1].y);
          const F2 s1 = row_sum2(f2hsum(f2add(z[0], z[1])), f2hsum(f2fma(z[0], z[0], f2mul(z[1], z[1]))));
          const float mean = s1.x * (1.f / HD), rstd = rsqrtf(fmaxf(s1.y * (1.f / HD) - mean * mean, 0.f) + p.eps);
          if (SAVE && (lane & 15) == 0) *reinterpret_cast<float*>(rec + MLP_REC_MEAN + 8 * row) = mean;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            x[h] = f2mul(f2add(z[h], f2(-mean)), f2(rstd));
            gg[h] = f2mul(f2fma(gam[h], x[h], btg[h]), gam[h]);
          }
          const F2 s2 = row_sum2(f2hsum(f2add(gg[0], gg[1])), f2hsum(f2fma(gg[0], x[0], f2mul(gg[1], x[1]))));
          const float A = s2.x * (1.f / HD), Bv = s2.y * (1.f / HD);
#pragma unroll
          for (int h = 0; h < 2; ++h) gp[h] = f2mul(f2fma(x[h], f2(-Bv), f2add(gg[h], f2(-A))), f2(rstd * lr));
          asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(tg2 + tile_row), "r"(pack_bf16(gp[0].x, gp[0].y)), "r"(pack_bf16(gp[1].x, gp[1].y)) : "memory");
        }
        fence_proxy_async_smem();  // (X2 and G2p are read by tcgen05.mma and, SAVE, leave by bulk copies)
        tmem_fence_before_sync();
        mlp_group_sync<1>();  // G2p
        issue_update(1, tx2, tg2, bar_w2);
        // ---- C4. G1p = (G2p W2^T) o gelu'(Z1)
        F2 cs1[4];  // float32 column sums of G1p over rows g, g + 8
        {
          float h[4][4] = {};
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            uint32_t ag[4], b[2][4];
            ldsm_x4(ag, tg2 + (tl ^ (ks << 5)));
            ldsm_x4(b[0], (w2c + wrow) ^ (ks << 5));
            ldsm_x4(b[1], (w2c + wrow + 16 * 128) ^ (ks << 5));
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_bf16(h[j], ag[0], ag[1], ag[2], ag[3], b[j >> 1][j & 1], b[j >> 1][2 + (j & 1)]);
          }
          uint32_t gp[4][2];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const F2 a = f2mul(pr(h[j], 0), d1[j][0]), b = f2mul(pr(h[j], 1), d1[j][1]);
            gp[j][0] = pack_bf16(a.x, a.y);
            gp[j][1] = pack_bf16(b.x, b.y);
            cs1[j] = f2add(a, b);
          }
          stsm_x4(tg1 + own, gp[0][0], gp[0][1], gp[1][0], gp[1][1]);
          stsm_x4((tg1 + own) ^ 32u, gp[2][0], gp[2][1], gp[3][0], gp[3][1]);
        }
        fence_proxy_async_smem();
        mbar_arrive_warp(bar_pub + 8 * par);  // X2, G2p, G1p of the stage
        asm volatile("bar.sync %0, 128;" ::"r"(3 + (warp >> 2)) : "memory");  // G1p of the half's hidden features
        issue_update(0, tg1, tk, bar_w1);
        // ---- C5. under the updates: float32 column sums (like the reference) of G2p and G1p; then the next stage's copies
        const bool more = s < s_hi;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          gp[h] = f2add(gp[h], f2(__shfl_xor_sync(0xffffffffu, gp[h].x, 16), __shfl_xor_sync(0xffffffffu, gp[h].y, 16)));
        {  // lanes of a column pair take one column each
          F2 a[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const F2 send = lane & 16 ? cs1[i] : cs1[2 + i];
            a[i] = f2add(lane & 16 ? cs1[2 + i] : cs1[i], f2(__shfl_xor_sync(0xffffffffu, send.x, 16), __shfl_xor_sync(0xffffffffu, send.y, 16)));
          }
          const F2 send = lane & 8 ? a[0] : a[1];
          const F2 b = f2add(lane & 8 ? a[1] : a[0], f2(__shfl_xor_sync(0xffffffffu, send.x, 8), __shfl_xor_sync(0xffffffffu, send.y, 8)));
          const float c = (lane & 4 ? b.y : b.x) + __shfl_xor_sync(0xffffffffu, lane & 4 ? b.x : b.y, 4);
          b1c = fmaf(c, -te15, b1c);
        }
        if (n > 0) wait_for(bar_done + 8 * (par ^ 1), ((n - 1) >> 1) & 1, 25, s);  // the output group is done with the stage before
        if (lane < 16) {
          const float4 b = lds_f4(sh + 4 * c4);
          const F2 m = f2(w_moves ? 1.f : 0.f);
          const uint32_t to = base + SM::OFF_B2 + (par ^ 1) * SM::B2 + warp * HD * 4 + 4 * c4;
          sts_pair(to, f2fma(gp[0], m, f2(b.x, b.y)));
          sts_pair(to + 8, f2fma(gp[1], m, f2(b.z, b.w)));
        }
        wait_for(bar_w2, n & 1, 23, s);
        tmem_fence_after_sync();
        if (more) {
          refresh(base + SM::OFF_W2 + (par ^ 1) * SM::WC, 1);
          wait_for(bar_read, n & 1, 24, s);  // the output group has read W1 and b1 of this stage
        }
        wait_for(bar_w1, n & 1, 23, s);
        tmem_fence_after_sync();
        if (more) {
          refresh(base + SM::OFF_W1, 0);
          sts_word(base + SM::OFF_B1 + 4 * b1_col, __float_as_uint(b1c));
          mbar_arrive_warp(bar_state);
        }
        // (stage ends)
      }

      // ---- the item's state: float32 masters and biases
      mlp_group_sync<1>();  // (the shares of b2)
      float* const ho = bws + 4 * HD * MLP_E;
      const bool park = SAVE && chunk < NCH - 1, results = !park && !(SAVE && p.walk_only);
#pragma unroll
      for (int mat = 0; mat < 2; ++mat)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float v[8][4];
          tmem_ld_8x4(tm_own + 128 * mat + 32 * cc, v);
          if (SAVE) {  // for the next chunk of this stream, or as the backward takes them up
            float4* const to = reinterpret_cast<float4*>(bws + mat * HD * MLP_E) + warp * 16 * 32 + lane;
#pragma unroll
            for (int i = 0; i < 8; ++i) to[(8 * cc + i) * 32] = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
          }
          if (results && mat == 0) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              st_from_float<T>(p.w1_out, (size_t)stream * HD * MLP_E + (size_t)(32 * cc + i) * MLP_E + e_own, v[i >> 2][i & 3] * wscale);
          } else if (results) {
            uint4* const to = reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.w2_out) + ((size_t)stream * HD * MLP_E + (size_t)e_own * HD + 32 * cc) * 2);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              to[i] = make_uint4(pack_bf16(v[2 * i][0] * wscale, v[2 * i][1] * wscale), pack_bf16(v[2 * i][2] * wscale, v[2 * i][3] * wscale),
                                 pack_bf16(v[2 * i + 1][0] * wscale, v[2 * i + 1][1] * wscale), pack_bf16(v[2 * i + 1][2] * wscale, v[2 * i + 1][3] * wscale));
          }
        }
      if (park) ho[MLP_HO_B1 + b1_col] = b1c;
      if (results) st_from_float<T>(p.b1_out, (size_t)stream * MLP_E + b1_col, b1c);
      if (tid < HD) {
        float b = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) b += __uint_as_float(lds_word(base + SM::OFF_B2 + (n & 1) * SM::B2 + 4 * (w * HD + tid)));
        if (park) ho[MLP_HO_B2 + tid] = b * wscale;
        if (results) st_from_float<T>(p.b2_out, (size_t)stream * HD + tid, b * wscale);
      }
      if (park) {
        __threadfence();
        mlp_group_sync<1>();
        if (tid == 0 && lds_word(w_fail) == 0u) *reinterpret_cast<volatile int*>(p.sched + 1 + stream) = chunk + 1;
      }
      tmem_fence_before_sync();
    } else {
      // ============================== output ==============================
      const float te_row[2] = {ld_as_float<T>(p.token_eta, g), ld_as_float<T>(p.token_eta, g + 8)};
      const float te_two = ld_as_float<T>(p.token_eta, 2 * warp + (lane >> 4));
      // -M1' = -te (1 + tril(Q K^T)) of the n'th stage, as bf16 rows
      auto form_m1 = [&](uint32_t n, int s) {
        const uint32_t slot = n % MLP_NST, tq = base + slot * SM::SLOT, tk = tq + TL;
        wait_for(bar_full + 8 * slot, (n / MLP_NST) & 1, 26, s);
        float at[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t ak[4], aq[4];  // (the blocks of an A fragment are those of a B fragment)
          ldsm_x4(ak, tk + (tl ^ (ks << 5)));
          ldsm_x4(aq, tq + (tl ^ (ks << 5)));
          mma_bf16(at[0], aq[0], aq[1], aq[2], aq[3], ak[0], ak[2]);
          mma_bf16(at[1], aq[0], aq[1], aq[2], aq[3], ak[1], ak[3]);
        }
#pragma unroll
        for (int jt = 0; jt < 2; ++jt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int i = g + 8 * r, jj = 8 * jt + 2 * t;
            const F2 m = f2fma(pr(at[jt], r), f2(-te_row[r]), f2(-te_row[r]));
            sts_word(base + SM::OFF_M1 + (n & 1) * 768 + 2 * (24 * i + jj), pack_bf16(jj <= i ? m.x : 0.f, jj + 1 <= i ? m.y : 0.f));
          }
      };
      // stage s, the n'th of this block, into its ring slot
      auto issue_loads = [&](uint32_t n, int s) {
        const uint32_t slot = n % MLP_NST, bar = bar_full + 8 * slot, tq = base + slot * SM::SLOT;
        mbar_expect_tx(bar, 3 * TL + CS * 2);
        const int r0 = row_base + s * CS;
        tma_load_2d(tq + TL, &tm_k, 0, r0, bar);
        tma_load_2d(tq, &tm_q, 0, r0, bar);
        tma_load_2d(tq + 2 * TL, &tm_v, 0, r0, bar);
        bulk_load_1d(base + SM::OFF_LR + slot * 32, static_cast<const uint8_t*>(p.lr) + (size_t)r0 * 2, CS * 2, bar);
      };
      uint32_t asked = n + (s_lo < s_hi ? 2 : 1);  // stages whose loads have been issued
      if (warp == 2) {
        if (elect_one()) {
          issue_loads(n, s_lo);
          if (s_lo < s_hi) issue_loads(n + 1, s_lo + 1);
        }
        __syncwarp();
      }
      if (warp == 0) form_m1(n, s_lo);
      mlp_group_sync<2>();
      for (int s = s_lo; s <= s_hi; ++s, ++n) {
        const uint32_t slot = n % MLP_NST, par = n & 1, tq = base + slot * SM::SLOT;
        const uint32_t w2c = base + SM::OFF_W2 + par * SM::WC, tx2 = base + SM::OFF_X2 + par * SM::ET,
                       tg1 = base + SM::OFF_G1 + par * SM::ET, tg2 = base + SM::OFF_G2 + par * TL;
        uint8_t* const rec = SAVE ? rec0 + (size_t)s * MLP_REC_BYTES : nullptr;
        // ---- O1. Q W1 + b1 (this warp's hidden features)
        wait_for(bar_full + 8 * slot, (n / MLP_NST) & 1, 26, s);
        wait_for(bar_state, n & 1, 27, s);
        float zq[4][4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t aq[4], b[2][4];
          ldsm_x4(aq, tq + (tl ^ (ks << 5)));
          ldsm_x4(b[0], (base + SM::OFF_W1 + wrow) ^ (ks << 5));
          ldsm_x4(b[1], (base + SM::OFF_W1 + wrow + 16 * 128) ^ (ks << 5));
#pragma unroll
          for (int j = 0; j < 4; ++j) mma_bf16(zq[j], aq[0], aq[1], aq[2], aq[3], b[j >> 1][j & 1], b[j >> 1][2 + (j & 1)]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const F2 b1 = lds_pair(base + SM::OFF_B1 + 4 * (32 * warp + 8 * j + 2 * t));
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const F2 z = f2fma(pr(zq[j], r), f2(wscale), b1);
            zq[j][2 * r] = z.x;
            zq[j][2 * r + 1] = z.y;
          }
        }
        mbar_arrive_warp(bar_read);
        uint32_t am[4];
        ldsm_x4(am, base + SM::OFF_M1 + par * 768 + (lane & 15) * 48 + ((lane >> 4) << 4));
        if (s < s_hi && warp == (int)((n + 1) & 7)) form_m1(n + 1, s + 1);
        // ---- O2. Zb1 = Q W1 + b1 - M1' G1p;  Xb2 = gelu(Zb1)
        wait_for(bar_pub + 8 * par, (n >> 1) & 1, 28, s);
        if (SAVE && warp == 1) {  // the stage's operands to its record
          if (elect_one()) {
            bulk_store_1d(rec + MLP_REC_X2, tx2, SM::ET);
            bulk_store_1d(rec + MLP_REC_G1P, tg1, SM::ET);
            bulk_store_1d(rec + MLP_REC_G2P, tg2, TL);
            bulk_commit();
          }
          __syncwarp();
        }
        uint32_t xb[4][2];
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          uint32_t b[4];
          ldsm_x4_t(b, (tg1 + own) ^ (j << 4));
          mma_bf16(zq[j], am[0], am[1], am[2], am[3], b[0], b[1]);
          mma_bf16(zq[j + 1], am[0], am[1], am[2], am[3], b[2], b[3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            F2 unused;
            const F2 x = gelu2<false>(pr(zq[j], r), unused, 1.f);
            xb[j][r] = pack_bf16(x.x, x.y);
          }
        // ---- O3. this warp's share of A2 = Xb2 X2^T and of (Xb2 W2 + b2) / wscale: its 32 hidden features
        {
          float a2[2][4] = {};
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t b[4];
            ldsm_x4(b, (tx2 + own) ^ (c << 5));
            mma_bf16(a2[0], xb[2 * c][0], xb[2 * c][1], xb[2 * c + 1][0], xb[2 * c + 1][1], b[0], b[2]);
            mma_bf16(a2[1], xb[2 * c][0], xb[2 * c][1], xb[2 * c + 1][0], xb[2 * c + 1][1], b[1], b[3]);
          }
          const uint32_t to = base + SM::OFF_A2 + warp * 768 + g * 32 + 8 * t;
          sts_pair(to, pr(a2[0], 0));
          sts_pair(to + 256, pr(a2[0], 1));
          sts_pair(to + 512, pr(a2[1], 1));
        }
        float z[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          const F2 b = lds_pair(base + SM::OFF_B2 + par * SM::B2 + 4 * (warp * HD + 8 * nt + 2 * t));
          z[nt][0] = z[nt][2] = b.x;
          z[nt][1] = z[nt][3] = b.y;
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int nt = 0; nt < 8; nt += 2) {
            uint32_t b[4];
            ldsm_x4_t(b, (w2c + wrow + 16 * 128 * c) ^ (nt << 4));
            mma_bf16(z[nt], xb[2 * c][0], xb[2 * c][1], xb[2 * c + 1][0], xb[2 * c + 1][1], b[0], b[1]);
            mma_bf16(z[nt + 1], xb[2 * c][0], xb[2 * c][1], xb[2 * c + 1][0], xb[2 * c + 1][1], b[2], b[3]);
          }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) z[nt][i] *= wscale;
        mlp_group_sync<2>();  // the partials of A2; those of the stage before's Zb2 have been read
        {  // -M2' = -te (1 + tril(A2)), two rows per warp
          const int i = 2 * warp + (lane >> 4), j = lane & 15;
          float a = 0.f;
          if (j <= i) {
            const uint32_t at = base + SM::OFF_A2 + (i & 8 ? 256 : 0) + (j & 8 ? 256 : 0) + (i & 7) * 32 + (j & 7) * 4;
#pragma unroll
            for (int w = 0; w < 8; ++w) a += __uint_as_float(lds_word(at + 768 * w));
            a = fmaf(a, -te_two, -te_two);
          }
          const float hi = __shfl_down_sync(0xffffffffu, a, 1);
          if ((lane & 1) == 0) sts_word(base + SM::OFF_M1 + par * 768 + 2 * (24 * i + j), pack_bf16(a, hi));
        }
        // the slot of the stage before, which everyone has left (the chain has published this one), takes the stage after next
        if (warp == 2 && s + 2 <= s_hi && __shfl_sync(0xffffffffu, lds_word(w_fail), 0) == 0u) {
          if (elect_one()) issue_loads(n + 2, s + 2);
          asked = n + 3;
          __syncwarp();
        }
        mlp_group_sync<2>();  // -M2'
        {  // M2' G2p: column tile `warp` goes into this warp's partial
          uint32_t b[4];
          ldsm_x4(am, base + SM::OFF_M1 + par * 768 + (lane & 15) * 48 + ((lane >> 4) << 4));
          ldsm_x4_t(b, tg2 + (tl ^ ((warp & 6) << 4)));
          const uint32_t b0 = warp & 1 ? b[2] : b[0], b1 = warp & 1 ? b[3] : b[1];
#pragma unroll
          for (int nt = 0; nt < 8; ++nt)
            if (nt == warp) mma_bf16(z[nt], am[0], am[1], am[2], am[3], b0, b1);
        }
        const uint32_t pf = base + SM::OFF_PO + part_frag;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          sts_pair(pf ^ (nt << 5), pr(z[nt], 0));
          sts_pair((pf ^ (nt << 5)) + 8 * 256, pr(z[nt], 1));
        }
        const uint2 qv = lds_u2(tq + tile_row);
        mlp_group_sync<2>();  // the partials of Zb2
        // ---- O4. out = Q + LN(Zb2), a row per half-warp
        F2 zb[2], o[2];
        sum_partials(base + SM::OFF_PO + part_row, zb);
        if (SAVE) *reinterpret_cast<float4*>(rec + MLP_REC_ZB2 + 4 * (row * HD + c4)) = make_float4(zb[0].x, zb[0].y, zb[1].x, zb[1].y);
        if (SAVE && warp == 1) {  // the bulk copies have left
          if (elect_one()) bulk_wait_read<0>();
          __syncwarp();
        }
        mbar_arrive_warp(bar_done + 8 * par);
        const F2 s1 = row_sum2(f2hsum(f2add(zb[0], zb[1])), f2hsum(f2fma(zb[0], zb[0], f2mul(zb[1], zb[1]))));
        const float mean = s1.x * (1.f / HD), rstd = rsqrtf(fmaxf(s1.y * (1.f / HD) - mean * mean, 0.f) + p.eps);
        if (SAVE && (lane & 15) == 0) *reinterpret_cast<float*>(rec + MLP_REC_MEAN + 8 * row + 4) = mean;
        if (!(SAVE && p.walk_only)) {
          o[0] = f2add(bf_pair(qv.x), f2fma(gam[0], f2mul(f2add(zb[0], f2(-mean)), f2(rstd)), bet[0]));
          o[1] = f2add(bf_pair(qv.y), f2fma(gam[1], f2mul(f2add(zb[1], f2(-mean)), f2(rstd)), bet[1]));
          *reinterpret_cast<uint2*>(static_cast<uint8_t*>(p.out) + ((size_t)(row_base + s * CS + row) * HD + c4) * 2) =
              make_uint2(pack_bf16(o[0].x, o[0].y), pack_bf16(o[1].x, o[1].y));
        }
      }
      if (warp == 2 && lds_word(w_fail) != 0u) {  // copies that are on their way land before the block leaves
        for (uint32_t i = 1; i <= MLP_NST && i <= asked; ++i) mbar_wait_bounded(bar_full + 8 * ((asked - i) % MLP_NST), ((asked - i) / MLP_NST) & 1);
      }
    }
    __syncthreads();  // the item is left by both groups
    if (lds_word(w_fail) != 0u) break;
  }  // work items
  tmem_fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(lds_word(w_tmem), 256);
  if (SAVE) bulk_wait_all<0>();
}

cudaError_t launch_mlp_fwd(const CUtensorMap* m, const MlpFwdParams& p, int nstreams, cudaStream_t st) {
  const bool save = p.bwd_ws != nullptr;
  auto kfn = save ? ttt_mlp_fwd_kernel<true> : ttt_mlp_fwd_kernel<false>;
  static DeviceValue resident[2];
  int sms = 0, per_sm = 0;
  cudaError_t e = resident[save].get(0, &per_sm, [&](int* n) {
    const cudaError_t a = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MlpSmem::TOTAL);
    return a != cudaSuccess ? a : cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kfn, MLP_THREADS, MlpSmem::TOTAL);
  });
  if (e != cudaSuccess) return e;
  if (!save) {  // no workspace to park state in: one block per stream
    kfn<<<nstreams, MLP_THREADS, MlpSmem::TOTAL, st>>>(m[0], m[1], m[2], p);
    return cudaGetLastError();
  }
  // persistent: as many blocks as are co-resident (they wait on one another's hand-offs), never more than items
  if ((e = device_sms(&sms)) != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  MlpFwdParams pp = p;
  pp.nstreams = nstreams;
  int grid = sms * per_sm;
  if (grid > nstreams) grid = nstreams;
  pp.CH = mlp_chunk_stages(p.NS, nstreams, grid);
  pp.NCH = (p.NS + pp.CH - 1) / pp.CH;
  if ((e = cudaMemsetAsync(pp.sched, 0, sizeof(int) * (size_t)(1 + nstreams), st)) != cudaSuccess) return e;
  void* args[] = {(void*)&m[0], (void*)&m[1], (void*)&m[2], (void*)&pp};
  return cudaLaunchCooperativeKernel((const void*)kfn, dim3(grid), dim3(MLP_THREADS), args, MlpSmem::TOTAL, st);
}
}  // namespace ttt
