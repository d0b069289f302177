// TTT-MLP backward (bf16 I/O, float32 state): one 16-warp CTA per (batch, head) stream.
//
// What it computes: the gradient of the whole-sequence TTT-MLP forward (semantics rust/core/src/mlp.rs:127-208; the
// reference obtains this gradient from Burn autodiff, it has no fused MLP kernel) for loss = <grad_output, output>:
// grad_xq/xk/xv, grad_w1/b1/w2/b2 (per batch element), grad_ttt_lr_eta, and per-stream partials of grad_token_eta and
// of the LayerNorm parameter gradients (summed over streams in a fixed order by ttt_mlp_bwd_reduce_kernel).
//
// How: the stage-by-stage analytic backward (reverse walk over the mini-batches carrying dW1, db1, dW2, db2; GELU and
// LayerNorm second derivatives).  The forward kernel leaves one record per stage (MlpStage: X2, the lr-scaled inner
// gradients G1p and G2p, Z2, Zb2, b1): W1_s = W1_{s+1} + te15 K^T G1p, W2_s = W2_{s+1} + te15 X2^T G2p undo the stage's
// update, and both LayerNorms of the stage are differentiated straight from the saved Z2 and Zb2, with statistics of two passes.
//
// Where things live, and who does what:
//  * The float32 masters of W1^T, W2, dW1^T, dW2 fill the SM's tensor memory, each as [256 hidden][64 features] = two
//    128-lane accumulators of 64 columns.  Undoing the two updates and adding the five rank-16 terms of dW1, dW2 are
//    fourteen tcgen05.mma (M = 128, N = 64, K = 16) that accumulate into them in place; their operands are the token tiles
//    as they are, read MN-major (hidden or features contiguous, tokens the contraction).
//  * After every stage each warp reads its quarter of one matrix back (tcgen05.ld) and refreshes that matrix's bf16 copy
//    in shared memory ([256][64], 128-byte rows, swizzled): the operand of all products that involve the state.
//  * A warp owns 16 hidden features of every 16 x 256 tile, in mma.sync accumulator layout, from Z1 to dZ1: GELU and its
//    derivatives, the small causal matrices (each warp forms Q K^T and dZb2 G2^T for itself, 16 products that would
//    otherwise cost a barrier and a trip through shared memory) and their products with its own columns (operands through
//    movmatrix) never leave its registers.  Only what is contracted over all 256 hidden features is written out.
//  * A warp also owns one token row of the 16 x 64 tiles for the two LayerNorms.
// A stage is six barrier intervals (I1..I6 below).  Before, 25 phases passed every intermediate tile through shared
// memory as bf16, undid the updates through registers and read dW from L2: 43 k cycles a stage; 192 streams of 128 stages
// forward and backward 4.11 ms, now 2.21 ms (2.53 before the forward's two groups).
// What the tensor cores' accumulation does to the masters: undone over 112 / 470 stages they are 7e-6 / 3e-5 (2-norm) off the
// forward's own state there (terms summed from zero and added in registers: W1 4e-6 / 2e-5, W2 6e-6 / 3e-5); the bf16 copies that
// the products read are 1.7e-3 off.  Gradients against float64: 128 stages 0.74 to 1.01 times the errors of the sums in
// registers, 512 stages 0.81 to 0.99 (264 streams).
#include "ttt_kernels.h"
#include "ttt_common.cuh"
#include "ttt_stage.cuh"

namespace ttt {

constexpr int MB_THREADS = 512;
constexpr uint32_t ONES = 0x3f803f80u;  // a pair of bf16 ones
constexpr int MB_E = 256;  // hidden width of the inner MLP (4 * head_dim)
typedef __nv_bfloat16 bf;

// Shared memory: offsets from a 1024-byte aligned base.  Token tiles are [16][64] bf16 with the 128-byte swizzle; the
// 16 x 256 ones are four of those (64 hidden features each).
struct MlpBwdSmem {
  static constexpr uint32_t TL = TILE_BF16_BYTES, ET = 4 * TILE_BF16_BYTES, WM = MB_E * HD * 2;
  static constexpr uint32_t W1 = 0, W2 = W1 + WM, DW1 = W2 + WM, DW2 = DW1 + WM;  // [256 hidden][64] bf16
  static constexpr uint32_t X2 = DW2 + WM;          // two: this stage's and the next one's
  static constexpr uint32_t X2B = X2 + 2 * ET, G1 = X2B + ET, DZ1B = G1 + ET, DH = DZ1B + ET;
  static constexpr uint32_t DZ1 = DH + ET, G1P = DZ1 + ET;
  static constexpr uint32_t PART = DZ1;             // float [4][16][64], I3..I4 only: dZ1 is written in I5, G1p (with the next V) lands after I4
  static constexpr uint32_t IN = G1P + ET;          // two x (q, k, dO)
  static constexpr uint32_t V = IN + 6 * TL, G2P = V + TL, G2 = G2P + TL, DZ2B = G2 + TL, DZ2 = DZ2B + TL;
  static constexpr uint32_t EXD = DZ2 + TL;         // float [16][64]: dk products; in I3..I4 partials of A2
  static constexpr uint32_t EXG = EXD + 4096;       // float [16][64]: -l o gl1; in I3..I4 partials of dM1
  static constexpr uint32_t AD = EXG + 4096;        // float [16][17]: A1[i][j] at [i][j], dM2[i][j] at [j][i + 1]  (j <= i)
  static constexpr uint32_t DET = AD + 16 * 17 * 4; // float [16][17]: dEta o lr; before I4 the row sums of 16 warps [16][16]
  static constexpr uint32_t DA1 = DET + 16 * 17 * 4;  // bf16 [16][24]
  static constexpr uint32_t DB2 = DA1 + 16 * 24 * 2;  // float [64]
  static constexpr uint32_t LR = DB2 + HD * 4;      // float [2][16], then ell = te15 lr [2][16]
  static constexpr uint32_t TE = LR + 4 * CS * 4;   // float [16]
  static constexpr uint32_t M1T = TE + CS * 4;      // bf16 [16][24]: -M1
  static constexpr uint32_t DLP = M1T + 16 * 24 * 2;  // float [16] sum over i of dEta te, then [16] the rest of dell
  static constexpr uint32_t LN = DLP + 2 * CS * 4;  // float [2][64]: LayerNorm weight, bias
  static constexpr uint32_t BAR = LN + 2 * HD * 4; // mbarriers: stage inputs, late inputs, dW products, undone updates; then item, tensor-memory base
  static constexpr uint32_t TOTAL = BAR + 4 * 8 + 8;
};
static_assert(MlpBwdSmem::TOTAL <= 227 * 1024, "shared-memory tiles exceed one SM");
static_assert(MlpBwdSmem::DA1 % 16 == 0 && MlpBwdSmem::M1T % 16 == 0 && MlpBwdSmem::BAR % 8 == 0, "alignment");

__device__ __forceinline__ void mma4(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  mma_bf16(c, a[0], a[1], a[2], a[3], b0, b1);
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts_f(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ float lds_f(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds_u(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ F2 lds_f2(uint32_t a) {
  F2 v;
  asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_f2(uint32_t a, F2 v) { asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory"); }
// loads that stay where they are written (an ordinary one is sunk to its first use, behind the barrier it was to overlap)
__device__ __forceinline__ F2 ldg_now2(const void* p) {
  F2 v;
  asm volatile("ld.global.cg.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ F2 unpack_bf16(uint32_t v) { return make_float2(bf16_lo(v), bf16_hi(v)); }
// sums over the warp of two (four) values: the halves of the warp (quarters) reduce one value each
__device__ __forceinline__ F2 warp_sum2(float a, float b) {
  const bool hi = threadIdx.x & 16;
  float v = (hi ? b : a) + __shfl_xor_sync(0xffffffffu, hi ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const float w = __shfl_xor_sync(0xffffffffu, v, 16);
  return hi ? f2(w, v) : f2(v, w);
}
__device__ __forceinline__ float warp_sum4_spread(float a, float b, float c, float d) {  // lanes 8 i ..: the i-th sum
  const bool hi = threadIdx.x & 16, mid = threadIdx.x & 8;
  const float x = (hi ? c : a) + __shfl_xor_sync(0xffffffffu, hi ? a : c, 16);
  const float y = (hi ? d : b) + __shfl_xor_sync(0xffffffffu, hi ? b : d, 16);
  float v = (mid ? y : x) + __shfl_xor_sync(0xffffffffu, mid ? x : y, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// float [16][64] exchange tile: column groups of 8 permuted by the row, so that the 64-bit accesses of an accumulator
// fragment (4 rows x 4 column pairs per half-warp) fall in distinct banks
__device__ __forceinline__ uint32_t off_x(int row, int col) { return (uint32_t)(row * 256 + ((col ^ ((row & 3) << 3)) << 2)); }

// float [16][16] partial sum of a causal matrix, stored by columns: even columns before odd ones, rows turned by 8 in every
// other pair of them, so that neither the fragments' stores nor a column's load meet in a bank
__device__ __forceinline__ uint32_t off_causal(int j, int i) {
  return (uint32_t)((((j >> 1) + 8 * (j & 1)) * 16 + (i ^ (((j >> 2) & 1) << 3))) << 2);
}

// The thread's place, read anew in every interval of a stage: what follows from it (a dozen addresses) is then formed where
// it is used instead of being kept across the loop, which would push the tiles' values into local memory.
struct Place {
  int tid, warp, lane, g, t;
  __device__ __forceinline__ Place() {
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    warp = tid >> 5;
    lane = tid & 31;
    g = lane >> 2;
    t = lane & 3;
  }
  // ldmatrix address of an A fragment in a token tile; k-step ks: ^ (ks << 5)
  __device__ __forceinline__ uint32_t a_off() const { return lane_off_A(lane, 0); }
  // of a B fragment (both n-tiles) in a [256][64] matrix whose rows are this warp's 16 hidden features; k-step ks: ^ (ks << 5)
  __device__ __forceinline__ uint32_t bn_off() const {
    return (16 * warp + (lane & 7) + ((lane >> 4) << 3)) * 128 + ((((lane >> 3) & 1) ^ (lane & 7)) << 4);
  }
  // ldmatrix / stmatrix address (x4) of this warp's 16 columns of a 16 x 256 tile: blocks (n-tile, row half) in the order of
  // the accumulator registers; read transposed they are the B fragments of a contraction over the tokens
  __device__ __forceinline__ uint32_t e_off() const {
    return (warp >> 2) * TILE_BF16_BYTES + (lane & 15) * 128 + (((2 * (warp & 3) + (lane >> 4)) ^ (lane & 7)) << 4);
  }
  // this warp's share of the masters between work items: matrix warp / 4 (W1, W2, dW1, dW2), lane quarter warp % 4 =
  // hidden features 32 (warp % 4) + lane and, 64 columns on, those + 128
  __device__ __forceinline__ int mi() const { return warp >> 2; }
  __device__ __forceinline__ uint32_t tm(uint32_t tmem) const { return tmem + ((32u * (uint32_t)(warp & 3)) << 16) + 128u * (uint32_t)mi(); }
  __device__ __forceinline__ int rc() const { return 2 * lane; }  // row-wise steps: row = warp, columns rc, rc + 1
};
#define TTT_PLACE \
  const Place P;  \
  [[maybe_unused]] const int tid = P.tid, warp = P.warp, lane = P.lane, g = P.g, t = P.t, rc = P.rc();

__global__ void __launch_bounds__(MB_THREADS, 1)
    ttt_mlp_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                       const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                       const MlpBwdParams p) {
  using SM = MlpBwdSmem;
  typedef __nv_bfloat16 T;
  constexpr uint32_t TL = SM::TL, ET = SM::ET;
  extern __shared__ __align__(1024) uint8_t mlp_bwd_smem[];
  const uint32_t base0 = smem_u32(mlp_bwd_smem);
  const int NS = p.NS;
  const uint32_t barL = base0 + SM::BAR, barG = barL + 8, barD = barL + 16, barU = barL + 24;
  int* const s_item = reinterpret_cast<int*>(mlp_bwd_smem + SM::BAR + 32);
  if ((base0 & 1023u) != 0) {  // (the tiles need it; dynamic shared memory starts there when there is no static one)
    if (threadIdx.x == 0) report_timeout(p.status, 2, 0);
    return;
  }
  // Tensor memory, all 512 columns (shared memory keeps the block alone on its SM).  The warp that allocates frees it at
  // the end of the kernel; every way out of the item loop leads there.
  if (threadIdx.x < 32) tmem_alloc(base0 + SM::BAR + 36, 512);
  if (threadIdx.x == 32) {
    mbar_init(barL, 1);
    mbar_init(barG, 1);
    mbar_init(barD, 1);
    mbar_init(barU, 1);
    fence_mbar_init();
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
    prefetch_tmap(&tm_do);
  }
  tmem_fence_before_sync();
  __syncthreads();
  tmem_fence_after_sync();
  pdl_go();  // (the reduction waits)
  const auto tmem = [&]() { return lds_u(base0 + SM::BAR + 36); };  // (read where it is used, like te15: a register less across the stage loop)
  const auto te15 = [&]() { return lds_f(base0 + SM::TE + 4 * (CS - 1)); };
  // the masters of W1, W2 are carried divided by -te15, so that a stage's update accumulates directly (te15 = 0: they never
  // move)
  if (threadIdx.x < CS) sts_f(base0 + SM::TE + 4 * threadIdx.x, ld_as_float<T>(p.token_eta, threadIdx.x));

  const int nitems = p.nstreams * p.NCH;
  uint32_t nload = 0, nmma = 0;  // stages whose inputs have been asked for / batches of products issued (barrier parities)
  int failed = 0;
  while (true) {
    // Persistent block.  A stream is a chain of NCH work items, its chunks of CH stages from the last to the first.  Items
    // are handed out rank by rank over all streams, so an item only waits for an item with a smaller index, which is
    // done or held by a resident block.  Between items a stream's masters, bias gradients and LayerNorm parameter
    // gradients are in the workspace.
    if (threadIdx.x == 0) *s_item = atomicAdd(&p.sched[0], 1);
    __syncthreads();
    const int item = *s_item;
    __syncthreads();
    if (item >= nitems) break;
    const int rank = item / p.nstreams, stream = item - rank * p.nstreams, head = stream % p.H;
    const int chunk = p.NCH - 1 - rank, s_lo = chunk * p.CH, s_hi = min(s_lo + p.CH, NS) - 1;
    const int row_base = stream * p.T;
    float* const ws = p.workspace + (size_t)stream * p.ws_stride;
    float* const ho = ws + 4 * HD * MB_E;
    const uint8_t* const rec0 = reinterpret_cast<const uint8_t*>(ho + MLP_BWD_HANDOFF_FLOATS);
    if (rank > 0) {
      // wait (bounded) until the previous item of this stream has published its state
      int ok = 1;
      if (threadIdx.x == 0) {
        ok = 0;
        const volatile int* flag = p.sched + 1 + stream;
        for (uint32_t it = 0; it < (1u << 24); ++it) {
          if (*flag >= rank) {
            ok = 1;
            break;
          }
          __nanosleep(100);
        }
        __threadfence();
      }
      if (__syncthreads_or(ok ? 0 : 1)) {
        if (threadIdx.x == 0) report_timeout(p.status, 1, item);
        break;
      }
    }
    // one thread of each of five warps (a copy costs its thread a hundred cycles)
    auto issue_inputs = [&](int s, int buf) {
      const int which = threadIdx.x >> 5;
      if ((threadIdx.x & 31) != 0 || which > 4) return;
      const uint8_t* rec = rec0 + (size_t)s * MLP_REC_BYTES;
      const int r0 = row_base + s * CS;
      const uint32_t in = base0 + SM::IN + buf * 3 * TL;
      if (which == 0) {
        mbar_expect_tx(barL, 4 * TL + ET);
        tma_load_2d(in, &tm_q, 0, r0, barL);
      } else if (which == 1) {
        tma_load_2d(in + TL, &tm_k, 0, r0, barL);
      } else if (which == 2) {
        tma_load_2d(in + 2 * TL, &tm_do, 0, r0, barL);
      } else if (which == 3) {
        bulk_load_1d(base0 + SM::X2 + buf * ET, rec + MLP_REC_X2, ET, barL);
      } else {
        bulk_load_1d(base0 + SM::G2P, rec + MLP_REC_G2P, TL, barL);
      }
    };
    auto issue_late = [&](int s) {  // what is read until I4: V, and G1p where the partial sums of I3 are
      mbar_expect_tx(barG, ET + TL);
      tma_load_2d(base0 + SM::V, &tm_v, 0, row_base + s * CS, barG);
      bulk_load_1d(base0 + SM::G1P, rec0 + (size_t)s * MLP_REC_BYTES + MLP_REC_G1P, ET, barG);
    };
    // the lines of a stage's record that are read late (G1p) or by ordinary loads, asked into L2
    auto prefetch_record = [&](int s) {
      const int tid = threadIdx.x;
      const uint8_t* rec = rec0 + (size_t)s * MLP_REC_BYTES;
      if (tid < 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(rec + MLP_REC_G1P + 128 * tid));
      else if (tid < 64 + (MLP_REC_BYTES - MLP_REC_Z2) / 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(rec + MLP_REC_Z2 + 128 * (tid - 64)));
    };
    // (asked together: an answer takes a hundred cycles)
    auto wait_both = [&](uint32_t a, uint32_t b, uint32_t parity) {
      const uint32_t there = mbar_try_wait(a, parity) & mbar_try_wait(b, parity);
      return there || (mbar_wait_bounded(a, parity) && mbar_wait_bounded(b, parity));
    };
    // what a thread reads of a stage by itself: its pair of Z2 and Zb2 and the row's means, its hidden columns of b1
    F2 zz, zzb, b1v[2], means;
    float ln_row;  // Z2's row, lanes 8 i ..: the two means of its LayerNorm gradient, 1 / std, mean
    auto load_z2 = [&](int s) {
      TTT_PLACE
      zz = ldg_now2(rec0 + (size_t)s * MLP_REC_BYTES + MLP_REC_Z2 + 8 * tid);
    };
    auto load_own = [&](int s) {
      load_z2(s);
      TTT_PLACE
      const uint8_t* rec = rec0 + (size_t)s * MLP_REC_BYTES;
      zzb = ldg_now2(rec + MLP_REC_ZB2 + 8 * tid);
      means = ldg_now2(rec + MLP_REC_MEAN + 8 * warp);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) b1v[nt] = ldg_now2(rec + MLP_REC_B1 + 8 * (8 * warp + 4 * nt + t));
    };
    auto put_rates = [&](int buf, float lr) {  // 16 lanes
      const int lane = threadIdx.x & 31;
      sts_f(base0 + SM::LR + buf * CS * 4 + 4 * lane, lr);
      sts_f(base0 + SM::LR + (2 + buf) * CS * 4 + 4 * lane, te15() * lr);
    };
    // W1_s, W2_s from W1_{s+1}, W2_{s+1} (inputs of stage s in buffer `buf`): one thread
    auto undo_updates = [&](int buf) {
      if (te15() == 0.f) return;
      const uint32_t k = base0 + SM::IN + buf * 3 * TL + TL, tm = tmem();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        umma_update(tm + 64 * h, base0 + SM::G1P + h * 2 * TL, k, UPD_IDESC | UPD_NEGATE);
        umma_update(tm + 128 + 64 * h, base0 + SM::X2 + buf * ET + h * 2 * TL, base0 + SM::G2P, UPD_IDESC | UPD_NEGATE);
      }
    };

    // ---- item begins: masters into tensor memory, gradients carried from the later chunk, the inputs of its last stage
    int s = s_hi;
    uint32_t buf = nload & 1;
    issue_inputs(s, buf);
    if (threadIdx.x == 0) issue_late(s);
    load_own(s);
    if (threadIdx.x < CS) put_rates(buf, ld_as_float<T>(p.lr, row_base + (size_t)s * CS + threadIdx.x));
    const bool fresh = rank == 0;  // the gradients w.r.t. the final state are zero
    F2 db1v[2], dgam = f2(0.f), dbet = f2(0.f);
    {
      TTT_PLACE
      const float4* src = reinterpret_cast<const float4*>(ws + P.mi() * HD * MB_E) + lane;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float v[8][4];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            if (P.mi() < 2 || !fresh) f = __ldcg(src + ((h * 4 + (warp & 3)) * 16 + cc * 8 + j) * 32);
            v[j][0] = f.x; v[j][1] = f.y; v[j][2] = f.z; v[j][3] = f.w;
          }
          tmem_st_8x4(P.tm(tmem()) + 64 * h + 32 * cc, v);
        }
      tmem_wait_st();
      if (tid < 2 * HD) sts_f(base0 + SM::LN + 4 * tid, ld_as_float<T>(tid < HD ? p.ln_g : p.ln_b, (size_t)head * HD + (tid & (HD - 1))));
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
        db1v[nt] = fresh ? f2(0.f) : __ldcg(reinterpret_cast<const float2*>(ho + MLP_HO_DB1) + 8 * warp + 4 * nt + t);
      if (tid < HD) sts_f(base0 + SM::DB2 + 4 * tid, fresh ? 0.f : __ldcg(ho + MLP_HO_DB2 + tid));
    }
    tmem_fence_before_sync();
    __syncthreads();
    // bf16 copy of half a master (128 hidden features; this warp's 32) to its operand matrix
    auto convert = [&](const Place& P, int mat, int half) {
      const float te = te15(), sc = mat < 2 && te != 0.f ? -te : 1.f;
      const uint32_t src = tmem() + ((32u * (uint32_t)(P.warp & 3)) << 16) + 128 * mat + 64 * half;
      const uint32_t dst = base0 + SM::W1 + mat * SM::WM + (128 * half + 32 * (P.warp & 3) + P.lane) * 128;
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        float v[8][4];
        tmem_ld_8x4(src + 32 * cc, v);
        if (mat < 2) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const F2 x = f2mul(pr(v[i], j), f2(sc));
              v[i][2 * j] = x.x;
              v[i][2 * j + 1] = x.y;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) w[j] = pack_bf16(v[2 * i + (j >> 1)][2 * (j & 1)], v[2 * i + (j >> 1)][2 * (j & 1) + 1]);
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + (((4 * cc + i) ^ (P.lane & 7)) << 4)), "r"(w[0]),
                       "r"(w[1]), "r"(w[2]), "r"(w[3])
                       : "memory");
        }
      }
    };
    // What a stage needs before its first barrier and does not take from the stage after it; `b`: its input buffer.
    //  * both LayerNorms, a row per warp: G2 and dZb2 as bf16 pairs.  Variances are sums of squared deviations: with the forward's
    //    E[z^2] - mean^2, rows whose mean is 100 standard deviations had state gradients 3e-2 to 4e-2 off (5e-3 to 7e-3 this way; 1.3 % of the time)
    uint32_t g2_pair, dzb_pair;
    F2 rstds;
    auto row_stats = [&]() {
      const F2 xc = f2add(zz, f2(-means.x)), bc = f2add(zzb, f2(-means.y));
      const F2 var = f2mul(warp_sum2(f2hsum(f2mul(xc, xc)), f2hsum(f2mul(bc, bc))), f2(1.f / HD));
      rstds = f2(rsqrtf(var.x + p.eps), rsqrtf(var.y + p.eps));
    };
    auto rows_of = [&](int b) {
      if (!wait_both(barL, barG, nload & 1)) failed = 1;
      TTT_PLACE
      const uint32_t in = base0 + SM::IN + b * 3 * TL;
      const F2 gam = lds_f2(base0 + SM::LN + 4 * rc), bet = lds_f2(base0 + SM::LN + 4 * (HD + rc));
      const F2 vv = ld_pair<T>(base0 + SM::V, warp, rc), kk = ld_pair<T>(in + TL, warp, rc), dd = ld_pair<T>(in + 2 * TL, warp, rc);
      const F2 xh = f2mul(f2add(zz, f2(-means.x)), f2(rstds.x)), xb = f2mul(f2add(zzb, f2(-means.y)), f2(rstds.y));
      const F2 gxh = f2mul(f2sub(f2fma(gam, xh, bet), f2sub(vv, kk)), gam), tt = f2mul(dd, gam);
      const float m = warp_sum4_spread(f2hsum(gxh), f2hsum(f2mul(gxh, xh)), f2hsum(tt), f2hsum(f2mul(tt, xb))) * (1.f / HD);
      float mi[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) mi[i] = __shfl_sync(0xffffffffu, m, 8 * i);
      const F2 G = f2mul(f2fma(xh, f2(-mi[1]), f2add(gxh, f2(-mi[0]))), f2(rstds.x));
      const F2 dzb = f2mul(f2fma(xb, f2(-mi[3]), f2add(tt, f2(-mi[2]))), f2(rstds.y));
      ln_row = lane < 16 ? m : lane < 24 ? rstds.x : means.x;
      dgam = f2fma(dd, xb, dgam);
      dbet = f2add(dbet, dd);
      g2_pair = pack_bf16(G.x, G.y);
      dzb_pair = pack_bf16(dzb.x, dzb.y);
    };
    //  * (one warp) the learning rates, A1 = Q K^T and -M1 = -eta o (1 + A1)
    auto causal_first = [&](int s, int b) {
      TTT_PLACE
      float lr = 0.f;
      if (lane < CS) lr = ld_as_float<T>(p.lr, row_base + (size_t)s * CS + lane);
      if (!mbar_wait_bounded(barL, nload & 1)) failed = 1;
      const uint32_t q = base0 + SM::IN + b * 3 * TL + P.a_off();
      float at[2][4] = {};
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint32_t ak[4], aq[4];
        ldsm_x4(ak, (q + TL) ^ (ks << 5));
        ldsm_x4(aq, q ^ (ks << 5));
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) mma4(at[nt], aq, ak[nt], ak[nt + 2]);  // (the blocks of an A fragment are those of a B fragment)
      }
      if (lane < CS) put_rates(b, lr);
      __syncwarp();
#pragma unroll
      for (int jt = 0; jt < 2; ++jt)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int i = g + 8 * r, j = 8 * jt + 2 * t;
          const F2 e = f2mul(lds_f2(base0 + SM::LR + 4 * (b * CS + j)), f2(-lds_f(base0 + SM::TE + 4 * i))), m = f2fma(pr(at[jt], r), e, e);
          sts32(base0 + SM::M1T + 2 * (24 * i + j), pack_bf16(j <= i ? m.x : 0.f, j + 1 <= i ? m.y : 0.f));
          if (j <= i) sts_f(base0 + SM::AD + 4 * (17 * i + j), at[jt][2 * r]);
          if (j + 1 <= i) sts_f(base0 + SM::AD + 4 * (17 * i + j + 1), at[jt][2 * r + 1]);
        }
    };
    //  * (warps 8..15) the bf16 copies of dW2 and W2, whose last readers are further back than those of dW1 and W1
    auto second_layer_copies = [&]() {
      TTT_PLACE
      if (!mbar_wait_bounded(warp < 12 ? barD : barU, nmma & 1)) failed = 1;
      tmem_fence_after_sync();
      convert(P, warp < 12 ? 3 : 1, 0);
      convert(P, warp < 12 ? 3 : 1, 1);
    };
    if (threadIdx.x >> 5 == 15 && elect_one()) {
      tmem_fence_after_sync();
      umma_commit_to(barD);
      if (!mbar_wait_bounded(barL, nload & 1) || !mbar_wait_bounded(barG, nload & 1)) failed = 1;
      undo_updates(buf);
      umma_commit_to(barU);
    }
    __syncwarp();
    if (threadIdx.x >> 5 == 8) causal_first(s, buf);
    if (threadIdx.x >= 256) second_layer_copies();
    row_stats();
    rows_of(buf);

    while (true) {
      // (addresses formed anew in every stage: kept across the loop they would push the tiles' values into local memory)
      uint32_t base = base0;
      asm volatile("" : "+r"(base));
      const uint32_t sAD = base + SM::AD, sDET = base + SM::DET, sDB2 = base + SM::DB2, sTE = base + SM::TE, sLN = base + SM::LN;
      const uint32_t tq = base + SM::IN + buf * 3 * TL, tk = tq + TL, tdo = tk + TL, tx2 = base + SM::X2 + buf * ET;
      const uint32_t sLR = base + SM::LR + buf * CS * 4, sELL = sLR + 2 * CS * 4;
      // ---- I1. G2 and dZb2 (their tiles have been read by the products of the stage before), bf16 copies of W1 and dW1
      ++nload;
      if (!wait_both(barD, barU, nmma & 1)) failed = 1;
      ++nmma;
      tmem_fence_after_sync();
      {
        TTT_PLACE
        sts32(base + SM::G2 + off_bf16(warp, rc), g2_pair);
        sts32(base + SM::DZ2B + off_bf16(warp, rc), dzb_pair);
        convert(P, (warp >> 3) * 2, (warp >> 2) & 1);
      }
      tmem_fence_before_sync();
      failed = __syncthreads_or(failed);  // 1
      if (failed) break;
      if (s > s_lo) {
        issue_inputs(s - 1, buf ^ 1);
        prefetch_record(s - 1);
      }

      // ---- I2. From Z1 to dH, this warp's 16 hidden features
      F2 gd1[2][2], dz1a[2][2];  // gelu'(Z1); dG1 o H o gelu''(Z1)
      float dx[2][4];            // dX2 so far: dA2^T X2b - l o gl2
      {
        TTT_PLACE
        const uint32_t a_off = P.a_off(), bn_off = P.bn_off(), e_off = P.e_off();
        float z1[2][4] = {}, zq[2][4] = {}, u1[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t ak[4], aq[4], bw[4], bd[4];
          ldsm_x4(ak, (tk + a_off) ^ (ks << 5));
          ldsm_x4(bw, (base + SM::W1 + bn_off) ^ (ks << 5));
          ldsm_x4(aq, (tq + a_off) ^ (ks << 5));
          ldsm_x4(bd, (base + SM::DW1 + bn_off) ^ (ks << 5));
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma4(z1[nt], ak, bw[2 * nt], bw[2 * nt + 1]);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            mma4(zq[nt], aq, bw[2 * nt], bw[2 * nt + 1]);
            mma4(u1[nt], ak, bd[2 * nt], bd[2 * nt + 1]);  // K dW1
          }
        }
        uint32_t gd2[2][2];  // gelu''(Z1), bf16 pairs
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            F2 d2;
            gelu_pair<2>(f2add(pr(z1[nt], r), b1v[nt]), gd1[nt][r], d2);
            gd2[nt][r] = pack_bf16(d2.x, d2.y);
            zq[nt][2 * r] += b1v[nt].x;
            zq[nt][2 * r + 1] += b1v[nt].y;
            u1[nt][2 * r] += db1v[nt].x;  // K dW1 + db1
            u1[nt][2 * r + 1] += db1v[nt].y;
          }
        float h[2][4] = {}, dzw[2][4] = {}, gl2[2][4] = {}, dm[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t ag[4], az[4], bw[4], bd[4];
          ldsm_x4(ag, (base + SM::G2 + a_off) ^ (ks << 5));
          ldsm_x4(bw, (base + SM::W2 + bn_off) ^ (ks << 5));
          ldsm_x4(az, (base + SM::DZ2B + a_off) ^ (ks << 5));
          ldsm_x4(bd, (base + SM::DW2 + bn_off) ^ (ks << 5));
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            mma4(h[nt], ag, bw[2 * nt], bw[2 * nt + 1]);     // H = G2 W2^T
            mma4(dzw[nt], az, bw[2 * nt], bw[2 * nt + 1]);   // dZb2 W2^T
            mma4(gl2[nt], ag, bd[2 * nt], bd[2 * nt + 1]);   // G2 dW2^T
            mma4(dm[nt], az, ag[nt], ag[nt + 2]);            // dZb2 G2^T = -dM2
          }
        }
        // G1 = H o gelu'(Z1);  Zb1 = Q W1 + b1 - M1 G1;  the row sums of dell that are ready here: G1.(K dW1 + db1) + gl2.X2
        uint32_t own[4], tb[4];  // a tile's own columns: as pairs, and as a B operand (contraction over the tokens)
        {
          uint32_t x2[4];
          ldsm_x4(x2, tx2 + e_off);
          float del[2] = {0.f, 0.f};
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const F2 g1 = f2mul(pr(h[nt], r), gd1[nt][r]);
              own[2 * nt + r] = pack_bf16(g1.x, g1.y);
              del[r] += f2hsum(f2fma(g1, pr(u1[nt], r), f2mul(pr(gl2[nt], r), unpack_bf16(x2[2 * nt + r]))));
            }
          stsm_x4(base + SM::G1 + e_off, own[0], own[1], own[2], own[3]);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            del[r] = quad_sum(del[r]);
            if (t == 0) sts_f(sDET + 4 * (16 * warp + g + 8 * r), del[r]);
          }
        }
        __syncwarp();
        {
          uint32_t am1[4];
          ldsm_x4_t(tb, base + SM::G1 + e_off);
          ldsm_x4(am1, base + SM::M1T + (lane & 15) * 48 + (lane >> 4) * 16);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma4(zq[nt], am1, tb[2 * nt], tb[2 * nt + 1]);
        }
        // dA2 = dM2 o eta, as an A operand;  dZb2 W2^T + dA2 X2;  dX2 = dA2^T X2b - l o gl2 + ..
        uint32_t ad2[4];
#pragma unroll
        for (int jt = 0; jt < 2; ++jt) {
          const F2 lrc = lds_f2(sLR + 4 * (8 * jt + 2 * t));
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int i = g + 8 * r, j = 8 * jt + 2 * t;
            const F2 m = f2mul(pr(dm[jt], r), f2mul(lrc, f2(-lds_f(sTE + 4 * i))));
            ad2[2 * jt + r] = pack_bf16(j <= i ? m.x : 0.f, j + 1 <= i ? m.y : 0.f);
            if (warp == 1) {
              if (j <= i) sts_f(sAD + 4 * (17 * j + i + 1), -dm[jt][2 * r]);
              if (j + 1 <= i) sts_f(sAD + 4 * (17 * (j + 1) + i + 1), -dm[jt][2 * r + 1]);
            }
          }
        }
        ldsm_x4_t(tb, tx2 + e_off);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) mma4(dzw[nt], ad2, tb[2 * nt], tb[2 * nt + 1]);
        const float ell[2] = {lds_f(sELL + 4 * g), lds_f(sELL + 4 * (g + 8))};
        // X2b = gelu(Zb1);  dZ1b = (dZb2 W2^T + dA2 X2) o gelu'(Zb1)
        uint32_t own2[4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            F2 d1, unused;
            const F2 x = gelu_pair<1>(pr(zq[nt], r), d1, unused), d = f2mul(pr(dzw[nt], r), d1);
            own[2 * nt + r] = pack_bf16(x.x, x.y);
            own2[2 * nt + r] = pack_bf16(d.x, d.y);
            dx[nt][2 * r] = -ell[r] * gl2[nt][2 * r];
            dx[nt][2 * r + 1] = -ell[r] * gl2[nt][2 * r + 1];
          }
        stsm_x4(base + SM::X2B + e_off, own[0], own[1], own[2], own[3]);
        stsm_x4(base + SM::DZ1B + e_off, own2[0], own2[1], own2[2], own2[3]);
        __syncwarp();
        {
          const uint32_t ad2t[4] = {movm_t(ad2[0]), movm_t(ad2[2]), movm_t(ad2[1]), movm_t(ad2[3])};
          ldsm_x4_t(tb, base + SM::X2B + e_off);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma4(dx[nt], ad2t, tb[2 * nt], tb[2 * nt + 1]);
        }
        // dG1 = -M1^T dZ1b - l o (K dW1 + db1);  dH = dG1 o gelu'(Z1)
        uint32_t am1t[4];
        ldsm_x4_t(am1t, base + SM::M1T + ((lane & 7) + ((lane >> 4) << 3)) * 48 + ((lane >> 3) & 1) * 16);
        ldsm_x4_t(tb, base + SM::DZ1B + e_off);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          float d[4] = {}, cs[4] = {};
          mma4(d, am1t, tb[2 * nt], tb[2 * nt + 1]);
          mma_bf16(cs, ONES, ONES, ONES, ONES, tb[2 * nt], tb[2 * nt + 1]);  // column sums
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const F2 dg = f2fma(pr(u1[nt], r), f2(-ell[r]), pr(d, r));
            const F2 dh = f2mul(dg, gd1[nt][r]);
            dz1a[nt][r] = f2mul(f2mul(dg, pr(h[nt], r)), unpack_bf16(gd2[nt][r]));
            own[2 * nt + r] = pack_bf16(dh.x, dh.y);
          }
          db1v[nt] = f2add(db1v[nt], f2(cs[0], cs[1]));
        }
        stsm_x4(base + SM::DH + e_off, own[0], own[1], own[2], own[3]);
      }
      __syncthreads();  // 2

      // ---- I3. Contractions over the hidden features that the chain waits for: dH W2 - l o (X2 dW2) (four partial sums), and
      //      the causal matrices A2 = X2b X2^T, dZ1b G1^T (eight warps, a quarter of one of them each)
      float dell_row;
      load_z2(s);  // Z2's LayerNorm once more, for I4
      {
        TTT_PLACE
        const uint32_t a_off = P.a_off();
        const int np = warp & 3, kq = warp >> 2;
        const uint32_t b_off = (64 * kq + (lane & 15)) * 128 + (((2 * np + (lane >> 4)) ^ (lane & 7)) << 4);
        float p1[2][4] = {}, p2[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t ax[4], ah[4], bd[4], bw[4];
          ldsm_x4(ax, (tx2 + kq * TL + a_off) ^ (ks << 5));
          ldsm_x4(ah, (base + SM::DH + kq * TL + a_off) ^ (ks << 5));
          ldsm_x4_t(bd, base + SM::DW2 + b_off + ks * 2048);
          ldsm_x4_t(bw, base + SM::W2 + b_off + ks * 2048);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            mma4(p1[nt], ax, bd[2 * nt], bd[2 * nt + 1]);
            mma4(p2[nt], ah, bw[2 * nt], bw[2 * nt + 1]);
          }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float l = lds_f(sELL + 4 * (g + 8 * r));
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
            sts_f2(base + SM::PART + kq * 4096 + off_x(g + 8 * r, 16 * np + 8 * nt + 2 * t), f2fma(pr(p1[nt], r), f2(-l), pr(p2[nt], r)));
        }
        if (warp < 8) {
          const int q = warp & 3;
          const uint32_t ta = (warp < 4 ? base + SM::X2B : base + SM::DZ1B) + q * TL + a_off;
          const uint32_t tb_ = (warp < 4 ? tx2 : base + SM::G1) + q * TL + a_off;
          float c[2][4] = {};
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            uint32_t a[4], b[4];
            ldsm_x4(a, ta ^ (ks << 5));
            ldsm_x4(b, tb_ ^ (ks << 5));
            mma4(c[0], a, b[0], b[2]);
            mma4(c[1], a, b[1], b[3]);
          }
          const uint32_t dst = (warp < 4 ? base + SM::EXD : base + SM::EXG) + q * 1024;
#pragma unroll
          for (int jt = 0; jt < 2; ++jt)
#pragma unroll
            for (int r = 0; r < 2; ++r) {  // transposed: the reader takes a column of the matrix
              sts_f(dst + off_causal(8 * jt + 2 * t, g + 8 * r), c[jt][2 * r]);
              sts_f(dst + off_causal(8 * jt + 2 * t + 1, g + 8 * r), c[jt][2 * r + 1]);
            }
        }
        dell_row = lane < 16 ? lds_f(sDET + 4 * (16 * lane + warp)) : 0.f;  // row sums of the 16 warps (finished in I4)
      }
      __syncthreads();  // 3

      // ---- I4. Token row j = warp: dG2, the second derivative of the LayerNorm (dZ2, d target), the row's eta gradients
      F2 dT;
      {
        TTT_PLACE
        const uint32_t r_off = off_bf16(warp, rc), x_off = off_x(warp, rc);
        const F2 bet = lds_f2(sLN + 4 * (HD + rc)), vk = f2sub(ld_pair<T>(base + SM::V, warp, rc), ld_pair<T>(tk, warp, rc));
        const float lr_j = lds_f(sLR + 4 * warp), ell_j = lds_f(sELL + 4 * warp);
        const F2 db2v = lds_f2(sDB2 + 4 * rc), gam = lds_f2(sLN + 4 * rc);
        const float rs = __shfl_sync(0xffffffffu, ln_row, 16), sg = __shfl_sync(0xffffffffu, ln_row, 0), sgx = __shfl_sync(0xffffffffu, ln_row, 8);
        const F2 xh = f2mul(f2add(zz, f2(-__shfl_sync(0xffffffffu, ln_row, 24))), f2(rs)), gy = f2sub(f2fma(gam, xh, bet), vk);  // its output minus the target
        const F2 gxh = f2mul(gy, gam), G = f2mul(f2fma(xh, f2(-sgx), f2add(gxh, f2(-sg))), f2(rs));
        F2 dg2 = f2mul(db2v, f2(-ell_j));
#pragma unroll
        for (int kq = 0; kq < 4; ++kq) dg2 = f2add(dg2, lds_f2(base + SM::PART + kq * 4096 + x_off));
        // lane i < 16: column j of the causal matrices
        const uint32_t sM2 = base + SM::EXG + 3 * 1024 + 64 * ((warp >> 1) + 8 * (warp & 1));  // (the row's own partial sums, read by then)
        float m2 = 0.f, dlr = 0.f;
        if (lane < 16) {
          float a2 = 0.f, d1 = 0.f;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            a2 += lds_f(base + SM::EXD + q * 1024 + off_causal(warp, lane));
            d1 -= lds_f(base + SM::EXG + q * 1024 + off_causal(warp, lane));
          }
          const float te_i = lds_f(sTE + 4 * lane);
          float deta = 0.f, da1 = 0.f;
          if (lane >= warp) {
            m2 = te_i * lr_j * (1.f + a2);
            deta = lds_f(sAD + 4 * (17 * warp + lane + 1)) * (1.f + a2) + d1 * (1.f + lds_f(sAD + 4 * (17 * lane + warp)));
            da1 = d1 * te_i * lr_j;
          }
          dlr = deta * te_i;
          __syncwarp(0xffffu);
          sts_f(sM2 + 4 * lane, m2);
          sts_f(sDET + 4 * (17 * lane + warp), deta * lr_j);
          *reinterpret_cast<bf*>(mlp_bwd_smem + SM::DA1 + 2 * (24 * lane + warp)) = __float2bfloat16_rn(da1);
        }
        // dG2 = dH W2 - l o (X2 dW2) - l (x) db2 - M2^T dZb2
        __syncwarp();
#pragma unroll
        for (int i = 0; i < CS; i += 4) {
          float m[4];
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(m[0]), "=f"(m[1]), "=f"(m[2]), "=f"(m[3]) : "r"(sM2 + 4 * i) : "memory");
#pragma unroll
          for (int j = 0; j < 4; ++j) dg2 = f2fma(ld_pair<T>(base + SM::DZ2B, i + j, rc), f2(-m[j]), dg2);
        }
        const F2 vv = f2mul(dg2, f2(-rs));
        const float sums = warp_sum4_spread(f2hsum(vv), dlr, f2hsum(f2mul(vv, xh)), dell_row + f2hsum(f2mul(G, db2v)));
        const float sv = __shfl_sync(0xffffffffu, sums, 0) * (1.f / HD), svx = __shfl_sync(0xffffffffu, sums, 16) * (1.f / HD);
        const F2 dgxh = f2fma(xh, f2(svx), f2fma(dg2, f2(rs), f2(sv))), dy = f2mul(gam, dgxh);
        dgam = f2add(dgam, f2fma(gy, dgxh, f2mul(dy, xh)));
        dbet = f2add(dbet, dy);
        dT = f2neg(dy);
        const F2 dxh = f2fma(dy, gam, f2fma(gxh, f2(svx), f2mul(vv, f2(sgx))));
        const F2 sd = warp_sum2(f2hsum(dxh), f2hsum(f2fma(dxh, xh, f2mul(dg2, G))));
        const F2 dz2 = f2fma(xh, f2(sd.y * (-1.f / HD) * rs), f2mul(f2add(dxh, f2(sd.x * (-1.f / HD))), f2(rs)));
        sts32(base + SM::DZ2 + r_off, pack_bf16(dz2.x, dz2.y));
        if (lane == 8) sts_f(base + SM::DLP + 4 * warp, sums);
        if (lane == 24) sts_f(base + SM::DLP + 4 * (CS + warp), sums);
        fence_proxy_async_smem();  // (G1p lands where the partial sums were)
      }
      __syncthreads();  // 4
      if (s > s_lo) {
        if (threadIdx.x == 0) issue_late(s - 1);
        load_own(s - 1);
      }

      // ---- I5. dX2 += dZ2 W2^T;  dZ1 = dG1 o H o gelu''(Z1) + dX2 o gelu'(Z1)
      {
        TTT_PLACE
        const uint32_t a_off = P.a_off(), bn_off = P.bn_off(), e_off = P.e_off();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t az[4], bw[4];
          ldsm_x4(az, (base + SM::DZ2 + a_off) ^ (ks << 5));
          ldsm_x4(bw, (base + SM::W2 + bn_off) ^ (ks << 5));
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma4(dx[nt], az, bw[2 * nt], bw[2 * nt + 1]);
        }
        uint32_t own[4], tb[4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const F2 d = f2fma(pr(dx[nt], r), gd1[nt][r], dz1a[nt][r]);
            own[2 * nt + r] = pack_bf16(d.x, d.y);
          }
        stsm_x4(base + SM::DZ1 + e_off, own[0], own[1], own[2], own[3]);
        fence_proxy_async_smem();  // every operand tile of the products below has been written by now
        __syncwarp();
        ldsm_x4_t(tb, base + SM::DZ1 + e_off);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          float cs[4] = {};
          mma_bf16(cs, ONES, ONES, ONES, ONES, tb[2 * nt], tb[2 * nt + 1]);
          db1v[nt] = f2add(db1v[nt], f2(cs[0], cs[1]));
        }
      }
      __syncthreads();  // 5

      // ---- I6. dW1 += Q^T dZ1b + K^T dZ1, dW2 += X2^T dZ2 + X2b^T dZb2 + dH^T G2, and W1, W2 one stage back: tcgen05.
      //      Meanwhile, 16 features of a product each: warps 0..3 dq = dZ1b W1^T + dA1 K, 4..7 dk = dZ1 W1^T + dA1^T Q and db2, 8..11
      //      gl1 = G1 dW1^T, then the copy of dW2; 12..15 the eta gradients, the next stage's rates and causal matrix, the copy of W2.
      //      All: the next stage's LayerNorms, warps 12..15 while they would wait for the products.  (dq and dk on the same four
      //      warps, the copies' eight warps with their LayerNorms last, one product's loads at a time: 192 streams of 128 stages 1 670 us,
      //      1 614 this way and with GELU's derivatives from one quotient.)
      const size_t r0 = (size_t)(row_base + s * CS) * HD;
      if (threadIdx.x >> 5 == 15) {
        if (elect_one()) {
          tmem_fence_after_sync();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t d1 = tmem() + 256 + 64 * h, d2 = d1 + 128, o = h * 2 * TL;
            umma_update(d1, base + SM::DZ1B + o, tq, UPD_IDESC);
            umma_update(d1, base + SM::DZ1 + o, tk, UPD_IDESC);
            umma_update(d2, tx2 + o, base + SM::DZ2, UPD_IDESC);
            umma_update(d2, base + SM::X2B + o, base + SM::DZ2B, UPD_IDESC);
            umma_update(d2, base + SM::DH + o, base + SM::G2, UPD_IDESC);
          }
          umma_commit_to(barD);
          if (s > s_lo) {
            if (!mbar_wait_bounded(barL, nload & 1) || !mbar_wait_bounded(barG, nload & 1)) failed = 1;
            undo_updates(buf ^ 1);
          }
          umma_commit_to(barU);
        }
        __syncwarp();
      }
      if (s > s_lo) row_stats();
      if (threadIdx.x < 384) {
        TTT_PLACE
        const int np = warp & 3, what = warp >> 2;  // dq, dk, gl1
        const uint32_t a_off = P.a_off();
        const uint32_t b_off = (lane & 15) * 128 + (((2 * np + (lane >> 4)) ^ (lane & 7)) << 4);  // 16 rows as k, columns 16 np.. as n
        const uint32_t ta = base + (what == 0 ? SM::DZ1B : what == 1 ? SM::DZ1 : SM::G1) + a_off, tb = base + (what < 2 ? SM::W1 : SM::DW1) + b_off;
        float c[2][2][4] = {};
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          uint32_t a[4][4], b[4][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            ldsm_x4_t(b[i], tb + (4 * k4 + i) * 2048);
            ldsm_x4(a[i], (ta + k4 * TL) ^ (i << 5));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) mma4(c[nt][i & 1], a[i], b[i][2 * nt], b[i][2 * nt + 1]);
        }
        if (what < 2) {
          uint32_t d[4], b[4];
          if (what == 0) ldsm_x4(d, base + SM::DA1 + (lane & 15) * 48 + (lane >> 4) * 16);                                  // dA1
          else ldsm_x4_t(d, base + SM::DA1 + ((lane & 7) + ((lane >> 4) << 3)) * 48 + ((lane >> 3) & 1) * 16);  // dA1^T
          ldsm_x4_t(b, (what == 0 ? tk : tq) + b_off);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma4(c[nt][0], d, b[2 * nt], b[2 * nt + 1]);
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const int col = 16 * np + 8 * nt + 2 * t;
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const F2 o = f2add(pr(c[nt][0], r), pr(c[nt][1], r));
            if (what == 0) {
              const F2 q = f2add(o, ld_pair<T>(tdo, g + 8 * r, col));
              static_cast<uint32_t*>(p.d_q)[(r0 + (g + 8 * r) * HD + col) >> 1] = pack_bf16(q.x, q.y);
            } else if (what == 1) {
              sts_f2(base + SM::EXD + off_x(g + 8 * r, col), o);
            } else {
              sts_f2(base + SM::EXG + off_x(g + 8 * r, col), f2mul(o, f2(-lds_f(sELL + 4 * (g + 8 * r)))));
            }
          }
        }
        if (what == 1) {
          uint32_t bz[4], by[4];
          ldsm_x4_t(bz, base + SM::DZ2B + b_off);
          ldsm_x4_t(by, base + SM::DZ2 + b_off);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const int col = 16 * np + 8 * nt + 2 * t;
            float cs[4] = {}, ct[4] = {};
            mma_bf16(cs, ONES, ONES, ONES, ONES, bz[2 * nt], bz[2 * nt + 1]);
            mma_bf16(ct, ONES, ONES, ONES, ONES, by[2 * nt], by[2 * nt + 1]);
            if (g == 0) sts_f2(sDB2 + 4 * col, f2add(lds_f2(sDB2 + 4 * col), f2(cs[0] + ct[0], cs[1] + ct[1])));
          }
        }
      } else {
        if (threadIdx.x >> 5 == 13) {
          // dell[j] = -(gl1[j].K[j] + G1[j].db1 + gl2[j].X2[j] + G2[j].db2)
          const int lane = threadIdx.x & 31;
          float dell = 0.f, dte = 0.f, lr = 0.f;
          if (lane < CS) {
            dell = -lds_f(base + SM::DLP + 4 * (CS + lane));
            lr = lds_f(sLR + 4 * lane);
#pragma unroll
            for (int j = 0; j < CS; ++j) dte += lds_f(sDET + 4 * (17 * lane + j));
            st_from_float<T>(p.d_lr, row_base + (size_t)s * CS + lane, lds_f(base + SM::DLP + 4 * lane) + dell * te15());
          }
          const float sum = warp_sum(dell * lr);
          if (lane < CS) p.part_te[(size_t)row_base + (size_t)s * CS + lane] = lane == CS - 1 ? dte + sum : dte;
        }
        if (s > s_lo) {
          if (threadIdx.x >> 5 == 12) causal_first(s - 1, buf ^ 1);
          rows_of(buf ^ 1);
        }
      }
      if (s > s_lo) {
        if (threadIdx.x >= 256) second_layer_copies();
        if (threadIdx.x < 384) rows_of(buf ^ 1);
      }
      __syncthreads();  // 6
      // ---- outputs of the stage: dk = (products) - l o gl1 - dT, dv = dT
      {
        TTT_PLACE
        const uint32_t x_off = off_x(warp, rc);
        const F2 dk = f2sub(f2add(lds_f2(base + SM::EXD + x_off), lds_f2(base + SM::EXG + x_off)), dT);
        const size_t at = (r0 >> 1) + tid;
        static_cast<uint32_t*>(p.d_k)[at] = pack_bf16(dk.x, dk.y);
        static_cast<uint32_t*>(p.d_v)[at] = pack_bf16(dT.x, dT.y);
      }
      if (s == s_lo) break;
      --s;
      buf ^= 1;
    }
    if (!failed) {
      if (!mbar_wait_bounded(barD, nmma & 1) || !mbar_wait_bounded(barU, nmma & 1)) failed = 1;
      ++nmma;
      tmem_fence_after_sync();
    }
    failed = __syncthreads_or(failed);
    if (failed) {
      if (threadIdx.x == 0) report_timeout(p.status, 3, item);
      break;
    }
    // ---- item ends: LayerNorm parameter gradients over the 16 rows; the masters and gradients go to the workspace for the
    //      stream's next item, or (last item) the state gradients to the caller
    const bool last = rank == p.NCH - 1;
    TTT_PLACE
    {
      sts_f2(base0 + SM::PART + 4 * (128 * warp + rc), dgam);
      sts_f2(base0 + SM::PART + 4 * (128 * warp + HD + rc), dbet);
    }
    if (!last || P.mi() >= 2) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float v[8][4];
          tmem_ld_8x4(P.tm(tmem()) + 64 * h + 32 * cc, v);
          const int e = 128 * h + 32 * (warp & 3) + lane;
          if (!last) {
            float4* dst = reinterpret_cast<float4*>(ws + P.mi() * HD * MB_E) + lane;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              dst[((h * 4 + (warp & 3)) * 16 + cc * 8 + j) * 32] = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
          } else if (P.mi() == 2) {  // dW1^T [e][k] -> grad_w1 [k][e]
#pragma unroll
            for (int j = 0; j < 32; ++j)
              st_from_float<T>(p.d_w1, ((size_t)stream * HD + 32 * cc + j) * MB_E + e, v[j >> 2][j & 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              st_from_float<T>(p.d_w2, ((size_t)stream * MB_E + e) * HD + 32 * cc + j, v[j >> 2][j & 3]);
          }
        }
    }
    if (g == 0) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int e = 16 * warp + 8 * nt + 2 * t;
        if (!last) *reinterpret_cast<float2*>(ho + MLP_HO_DB1 + e) = db1v[nt];
        else {
          st_from_float<T>(p.d_b1, (size_t)stream * MB_E + e, db1v[nt].x);
          st_from_float<T>(p.d_b1, (size_t)stream * MB_E + e + 1, db1v[nt].y);
        }
      }
    }
    tmem_fence_before_sync();
    __syncthreads();
    if (tid < 2 * HD) {
      float sum = fresh ? 0.f : __ldcg(ho + MLP_HO_DG + tid);
#pragma unroll
      for (int w = 0; w < CS; ++w) sum += lds_f(base0 + SM::PART + 4 * (128 * w + tid));
      if (!last) ho[MLP_HO_DG + tid] = sum;
      else p.part_ln[(size_t)stream * 2 * HD + tid] = sum;
    } else if (tid < 3 * HD) {
      const int f = tid - 2 * HD;
      if (!last) ho[MLP_HO_DB2 + f] = lds_f((base0 + SM::DB2) + 4 * f);
      else st_from_float<T>(p.d_b2, (size_t)stream * HD + f, lds_f((base0 + SM::DB2) + 4 * f));
    }
    fence_proxy_async_smem();  // (the next item's G1p lands where the row sums were)
    if (!last) {
      __threadfence();
      __syncthreads();
      if (tid == 0) *reinterpret_cast<volatile int*>(p.sched + 1 + stream) = rank + 1;
    }
  }  // item loop
  if (failed && threadIdx.x == 0)  // copies and products in flight land before the block leaves
    for (int i = 0; i < 4096; ++i)
      if (mbar_try_wait(barL, nload & 1) && mbar_try_wait(barG, nload & 1) && mbar_try_wait(barU, nmma & 1)) break;
  tmem_fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(tmem(), 512);
}

// grad_token_eta[t] = sum over streams, grad_ln_weight / grad_ln_bias [h][f] = sum over the batch; fixed order.  Block =
// 32 consecutive outputs x 8 warps: warp w adds terms w, w + 8, ... (coalesced 128-byte reads), the eight sums are added
// in warp order.  (One thread per output walking all streams took 14.5 us at 192 streams of 2048 tokens.)
__global__ void __launch_bounds__(256) ttt_mlp_bwd_reduce_kernel(const float* part_te, const float* part_ln, int B, int H,
                                                                 int T, int bf16, void* dte, void* dg, void* db) {
  __shared__ float part[8][32];
  pdl_join();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane, n_ln = 2 * H * HD;
  float acc = 0.f;
  if (i < T) {
    for (int st = warp; st < B * H; st += 8) acc += part_te[(size_t)st * T + i];
  } else if (i < T + n_ln) {
    const int j = i - T, which = j / (H * HD), hf = j % (H * HD), h = hf / HD, f = hf % HD;
    for (int b = warp; b < B; b += 8) acc += part_ln[((size_t)(b * H + h) * 2 + which) * HD + f];
  }
  part[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && i < T + n_ln) {
    float sum = part[0][lane];
#pragma unroll
    for (int w = 1; w < 8; ++w) sum += part[w][lane];
    const int j = i - T;
    void* const dst = i < T ? dte : (j < H * HD ? dg : db);
    const size_t at = i < T ? (size_t)i : (size_t)(j % (H * HD));
    if (bf16) st_from_float<bf>(dst, at, sum);
    else st_from_float<float>(dst, at, sum);
  }
}

// floats of workspace per stream: the four float32 masters, the hand-off record, one record per stage
size_t mlp_bwd_ws_stride_floats(int T) {
  return 4 * (size_t)HD * MB_E + MLP_BWD_HANDOFF_FLOATS + (size_t)T / CS * (MLP_REC_BYTES / 4);
}

cudaError_t launch_mlp_bwd(const CUtensorMap* m, const MlpBwdParams& p0, int B, cudaStream_t st) {
  MlpBwdParams p = p0;
  p.nstreams = B * p.H;
  static DeviceValue resident;
  int sms = 0, per_sm = 0;
  cudaError_t e = resident.get(0, &per_sm, [&](int* n) {
    const cudaError_t a = cudaFuncSetAttribute(ttt_mlp_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MlpBwdSmem::TOTAL);
    return a != cudaSuccess ? a : cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, ttt_mlp_bwd_kernel, MB_THREADS, MlpBwdSmem::TOTAL);
  });
  if (e != cudaSuccess || (e = device_sms(&sms)) != cudaSuccess) return e;
  // persistent grid: blocks wait on one another's hand-offs, so all of them must be resident (cooperative launch);
  // more blocks than streams would only wait (a stream's items run one after the other)
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  int grid = sms * per_sm;
  if (grid > p.nstreams) grid = p.nstreams;
  p.CH = mlp_chunk_stages(p.NS, p.nstreams, grid);
  p.NCH = (p.NS + p.CH - 1) / p.CH;
  if ((e = cudaMemsetAsync(p.sched, 0, sizeof(int) * (size_t)(1 + p.nstreams), st)) != cudaSuccess) return e;
  void* args[] = {(void*)&m[0], (void*)&m[1], (void*)&m[2], (void*)&m[3], (void*)&p};
  e = cudaLaunchCooperativeKernel((const void*)ttt_mlp_bwd_kernel, dim3(grid), dim3(MB_THREADS), args, MlpBwdSmem::TOTAL, st);
  if (e != cudaSuccess) return e;
  const int n = p.T + 2 * p.H * HD;
  return launch_dependent(ttt_mlp_bwd_reduce_kernel, (n + 31) / 32, 256, 0, st, (const float*)p.part_te, (const float*)p.part_ln, B, p.H, p.T, (int)p.reduced_bf16,
                          p.d_token_eta, p.d_ln_g, p.d_ln_b);
}

}  // namespace ttt
