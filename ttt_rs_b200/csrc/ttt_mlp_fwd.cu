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
// copies fill it): 6.3 k cycles a stage, 5.0 k with nothing beside it, of them 1.2 k round trips of three dependent tcgen05
// products and their commits, the rest instructions of two warps a scheduler at seven cycles each (the 5.0 k and what follows: of a
// GELU that was 0.15 k cycles a stage shorter).  So:
//  * Only that chain is the first group's work (warps 0..7).  The second group (warps 8..15) forms the stage's output from
//    what the chain publishes in shared and tensor memory, about half a stage behind.
//  * Warp w of either group owns hidden features e in [32w, 32w+32) of every 16 x 256 tile, in mma accumulator layout, from Z1
//    to G1p and from Zb1 to Xb2.  Products of tokens with the state over its 64 columns (Q W1, K W1, G2p W2^T) are tcgen05.mma
//    with hidden features as lanes, two halves of 128.
//  * Sums over all hidden features (Z2, Zb2) are formed by each warp over its own 32 by mma.sync; the eight partial tiles meet
//    in shared memory, where a half-warp adds up a token's row and has the whole row for
//    its LayerNorm: two barriers of the group a stage in the chain, where column owners exchanging row sums needed six.
//  * A2 = Xb2 X2^T meets the same way, two of its rows per warp; each warp then forms a column tile of M2' G2p.
//  * A1 and M1' of the next stage are formed by one warp of the second group in turn.
//  * The float32 masters of W1^T[e][k] and W2[e][n] are tensor-memory accumulators of 128 hidden features x 64; both rank-16
//    updates are tcgen05.mma into them (operands: the token tiles, tokens the contraction).  Each warp of the chain reads its 32
//    rows back and refreshes their bf16 copies: in tensor memory, the A operand of the products with the state, and W2's in
//    shared memory.  (With the copies in shared memory only, a product of 128 x 16 read 4 KB of them at the 128 bytes a cycle that
//    everything else there needs too: 119 against 106 us.)
// 48 streams of 31 stages / forward + backward of 192 streams of 128 stages: one group of eight warps with the masters in
// registers 150 / 2 528 us; two groups, products with the state by mma.sync 115 / 2 284; by tcgen05 106 / 2 243.  Not better: two groups
// of sixteen warps 121 / 2 355; K_next W1_next taken as K_next W1 plus a product with G1p, which takes W1's refresh off the chain, 111 / 2 284.
// Now 108.6 / 2 207 (with the backward's last interval on twelve warps, and a reciprocal for every element of GELU: one that two shared
// was 106.1 / 2 188 and lost the negative tail of the derivatives).
//
// Scheduling.  One CTA fills an SM, so a launch of one CTA per stream runs in whole
// waves: 192 streams on 148 SMs cost two stream-times.  When there is memory to park a stream's state in -- the backward's
// workspace in training (where the final state goes anyway), a scratch buffer of the host path in inference with more
// streams than SMs -- blocks take work items (stream, chunk of stages: mlp_chunk_stages) instead, first
// chunks of all streams first, and a chunk hands the state to the next one through the stream's block of that memory
// behind a per-stream counter -- the scheme of the TTT-Linear backward.  Inference: 192 streams of 128 stages
// 836 -> 591 us, 384 of 64 stages 640 -> 623, 300 of 32 stages 332 -> 296.
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
  static constexpr uint32_t SLOT = 3 * TILE;                          // q, k, v; in odd stages k, q, v
  static constexpr uint32_t WC = MLP_E * HD * 2;                      // [256 e][64] bf16, 128-byte rows, swizzled
  static constexpr uint32_t PART = 8 * 4096;                          // float [8 warps][16][64]
  static constexpr uint32_t OFF_W2 = MLP_NST * SLOT;                  // two copies of W2 (stage parity)
  static constexpr uint32_t OFF_X2 = OFF_W2 + 2 * WC;                 // two X2, then two G1p
  static constexpr uint32_t OFF_G1 = OFF_X2 + 2 * ET;
  static constexpr uint32_t OFF_G2 = OFF_G1 + 2 * ET;                 // two G2p
  static constexpr uint32_t OFF_PC = OFF_G2 + 2 * TILE;               // partials of Z2
  static constexpr uint32_t OFF_PO = OFF_PC + PART;                   // partials of Zb2, and M2' G2p
  static constexpr uint32_t OFF_M1 = OFF_PO + PART + 4096;                   // two [16][16] in tile form (the first columns of a [16][64]): -M1' / wscale
  static constexpr uint32_t OFF_B1 = OFF_M1 + 2 * TILE;               // float [2][256] (stage parity)
  static constexpr uint32_t B2 = 8 * HD * 4;                          // b2 / wscale as shares of the eight warps of the chain
  static constexpr uint32_t OFF_B2 = OFF_B1 + 2 * MLP_E * 4;              // float [2][8][64] (stage parity)
  static constexpr uint32_t OFF_M2 = OFF_B2 + 2 * B2;                 // bf16 [16][24]: -M2'
  static constexpr uint32_t OFF_A2 = OFF_M2 + 16 * 24 * 2;            // float [8 warps][3][8][8]: partials of A2 (its lower blocks)
  static constexpr uint32_t OFF_LR = OFF_A2 + 8 * 768;                // MLP_NST x 32 bytes
  // mbarriers: full [MLP_NST], published [2], done [2], partials read; products: Zb1 [2], Z1, G1, updates of W1, W2; M1'; end;
  // then item, failure flag, tensor-memory base
  static constexpr uint32_t OFF_BAR = OFF_LR + MLP_NST * 32;
  static constexpr uint32_t OFF_WORDS = OFF_BAR + (MLP_NST + 13) * 8;
  static constexpr uint32_t TOTAL = OFF_WORDS + 16;
};
static_assert(MlpSmem::TOTAL <= 227 * 1024, "shared-memory tiles exceed one SM");
static_assert(MlpSmem::OFF_M1 % 1024 == 0 && MlpSmem::OFF_M2 % 16 == 0 && MlpSmem::OFF_LR % 16 == 0 && MlpSmem::OFF_BAR % 8 == 0, "alignment");

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
template <int N>
__device__ __forceinline__ void sum_partials(uint32_t a, F2 (&z)[2]) {
  float4 v[N];
#pragma unroll
  for (int w = 0; w < N; ++w) v[w] = lds_f4(a + 4096 * w);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    F2 x[N];
#pragma unroll
    for (int w = 0; w < N; ++w) x[w] = h ? f2(v[w].z, v[w].w) : f2(v[w].x, v[w].y);
    z[h] = f2add(f2add(f2add(x[0], x[1]), f2add(x[2], x[3])), f2add(f2add(x[4], x[5]), f2add(x[6], x[7])));
    if constexpr (N == 9) z[h] = f2add(z[h], x[8]);
  }
}
// An accumulator of sixteen tokens (columns) for this warp's 32 hidden features (lanes), in mma accumulator layout:
// z[mt][nt][2r + c] is hidden feature 16 mt + 8 r + g, token 8 nt + 2 t + c.
__device__ __forceinline__ void tmem_ld_tokens(uint32_t taddr, float (&z)[2][2][4]) {
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(z[mt][0][0]), "=f"(z[mt][0][1]), "=f"(z[mt][0][2]), "=f"(z[mt][0][3]), "=f"(z[mt][1][0]), "=f"(z[mt][1][1]), "=f"(z[mt][1][2]), "=f"(z[mt][1][3])
                 : "r"(taddr + (16u << 16) * mt));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) asm volatile("" : "+f"(z[i >> 3][(i >> 2) & 1][i & 3]));  // (not used before the wait)
}
__device__ __forceinline__ void tmem_st_16(uint32_t taddr, const uint32_t (&w)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]), "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]),
               "r"(w[15]), "r"(taddr)
               : "memory");
}
// D[128 x N] (float32) += A . B over 16 of the contraction; A bf16 in tensor memory (a pair of the contraction per word), B K-major
__device__ __forceinline__ void umma_bf16_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d), "r"(a),
               "l"(b), "r"(idesc), "r"(accumulate)
               : "memory");
}
__device__ __forceinline__ void stsm_x4_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// A warp's share of X W2 + b2 over its 32 hidden features, all in units of wscale, times sc, to its partial tile: x2f the A
// fragments of X, w2 the warp's rows of the copy, sh its share of b2.  Four column tiles at a time, their loads ahead of the
// products: with all eight accumulators live the registers left serialised every ldmatrix with its products.
__device__ __forceinline__ void share_of_hidden_sum(const uint32_t (&a)[2][4], uint32_t w2, uint32_t sh, uint32_t part, float sc) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t b[4][4];
    float z[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) ldsm_x4_t(b[i], (w2 + 16 * 128 * (i >> 1)) ^ ((4 * h + 2 * (i & 1)) << 4));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const F2 v = lds_pair(sh + 32 * (4 * h + j));
      z[j][0] = z[j][2] = v.x;
      z[j][1] = z[j][3] = v.y;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        mma_bf16(z[j], a[c][0], a[c][1], a[c][2], a[c][3], b[2 * c + (j >> 1)][2 * (j & 1)], b[2 * c + (j >> 1)][2 * (j & 1) + 1]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sts_pair(part ^ ((4 * h + j) << 5), f2mul(pr(z[j], 0), f2(sc)));
      sts_pair((part ^ ((4 * h + j) << 5)) + 8 * 256, f2mul(pr(z[j], 1), f2(sc)));
    }
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

// CHUNKS: work items of several stages; SAVE: into the backward's workspace, with its records (the tests of a record pointer in
// the stage loop cost inference 1.5 %)
template <bool SAVE, bool CHUNKS>
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
                 bar_parts = bar_done + 16, bar_zq = bar_parts + 8, bar_z = bar_zq + 16, bar_h = bar_z + 8,
                 bar_w1 = bar_h + 8, bar_w2 = bar_w1 + 8, bar_m1 = bar_w2 + 8, bar_end = bar_m1 + 8;
  const uint32_t w_item = base + SM::OFF_WORDS, w_fail = w_item + 4, w_tmem = w_item + 8;

  const bool output_group = __shfl_sync(0xffffffffu, threadIdx.x >> 8, 0) != 0;
  const int tid = threadIdx.x & (MLP_GROUP - 1), lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  static_assert(CHUNKS || !SAVE, "the backward's workspace comes with chunks");
  constexpr size_t HANDOFF = (SAVE ? 4 : 2) * HD * MLP_E;  // biases, in floats, behind the masters
  const int NS = p.NS, CH = CHUNKS ? p.CH : NS, NCH = CHUNKS ? p.NCH : 1;
  const int nitems = CHUNKS ? p.nstreams * NCH : (int)gridDim.x;

  if (threadIdx.x < 32) tmem_alloc(w_tmem, 512);
  if (threadIdx.x == MLP_GROUP) {
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
    for (int i = 0; i < MLP_NST; ++i) mbar_init(bar_full + 8 * i, 1);
    for (int i = 0; i < 5; ++i) mbar_init(bar_pub + 8 * i, 8);
    for (int i = 0; i < 6; ++i) mbar_init(bar_zq + 8 * i, 2);  // (a commit for each half of the hidden features)
    mbar_init(bar_m1, 1);
    mbar_init(bar_end, 6);  // (the warps that issue products: three of each half)
    fence_mbar_init();
    sts_word(w_fail, 0u);
  }
  tmem_fence_before_sync();
  __syncthreads();
  tmem_fence_after_sync();
  // Tensor memory, hidden features as lanes, two halves of 128.  Masters W1^T and W2 [half][64 columns]; products with columns of
  // tokens [half][Zb1 of even stages, Z1 (then G1), Zb1 of odd stages]; bf16 copies of W1^T and W2 [half][32 columns].
  const uint32_t tmem = lds_word(w_tmem);
  constexpr uint32_t TM_Z = 256, TM_W1B = 352, TM_W2B = 416;
  const uint32_t tm_lane = (32u * (uint32_t)(warp & 3)) << 16;  // this warp's lanes: hidden features 32 warp .. of half warp / 4
  const int half = warp >> 2;

  const float te15 = ld_as_float<T>(p.token_eta, CS - 1);
  // both states are carried divided by wscale = -te15, so that their rank-16 updates accumulate directly by mma
  const bool w_moves = (te15 != 0.f);
  const float wscale = w_moves ? -te15 : 1.f;

  // A lane's place in what ldmatrix / stmatrix (x4) take: rows lane & 15, the 16-byte chunk lane >> 4 of a 128-byte row.  The
  // chunks of k-step or column pair i: ^ (i << 5); the next chunk's blocks: ^ (1 << 4).
  const uint32_t tl = lane_off_A(lane, 0);
  const uint32_t own = (warp >> 1) * TL + (tl ^ ((warp & 1) << 6));  // this warp's 32 columns of a 16 x 256 tile
  const uint32_t wrow = warp * 32 * 128 + tl;                        // this warp's 32 rows of a copy of W2
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
    if constexpr (CHUNKS) {
      if (threadIdx.x == 0) sts_word(w_item, (uint32_t)atomicAdd(&p.sched[0], 1));
      __syncthreads();
      item = (int)lds_word(w_item);
      __syncthreads();
    } else {
      item = (round == 0) ? (int)blockIdx.x : nitems;
    }
    if (item >= nitems) break;
    const int chunk = CHUNKS ? item / p.nstreams : 0, stream = CHUNKS ? item - chunk * p.nstreams : item;
    const int head = stream % p.H, row_base = stream * p.T;
    const int s_lo = chunk * CH, s_hi = min(s_lo + CH, NS) - 1;
    // The stream's block of the workspace or scratch buffer (layout in ttt_kernels.h).  SAVE: the lr-scaled inner gradients of
    // every stage (the bf16 operands of the state updates) and the final state go there, so that the backward can
    // start its reverse walk at once.
    float* const bws = CHUNKS ? p.bwd_ws + (size_t)stream * p.bwd_ws_stride : nullptr;
    uint8_t* const rec0 = SAVE ? reinterpret_cast<uint8_t*>(bws + HANDOFF + MLP_BWD_HANDOFF_FLOATS) : nullptr;
    if (CHUNKS && chunk > 0) {
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
      const uint32_t tm_own = tmem + tm_lane + 64u * half;
      const int e_own = 32 * warp + lane, b1_col = 32 * warp + 8 * t + g;
      // bf16 copies of 32 columns of this warp's rows of a master: in tensor memory, the A operand of products with the state, and
      // of W2 in shared memory too
      auto put_copy = [&](int mat, uint32_t buf, int cc, const float (&v)[8][4]) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = pack_bf16(v[i >> 1][2 * (i & 1)], v[i >> 1][2 * (i & 1) + 1]);
        tmem_st_16(tmem + tm_lane + (mat == 0 ? TM_W1B : TM_W2B) + 32 * half + 16 * cc, w);
        if (mat == 1) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            st_u4(base + SM::OFF_W2 + buf * SM::WC + e_own * 128 + (((4 * cc + i) ^ (lane & 7)) << 4), w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        }
      };
      auto refresh = [&](int mat, uint32_t buf) {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float v[8][4];
          tmem_ld_8x4(tm_own + 128 * mat + 32 * cc, v);
          put_copy(mat, buf, cc, v);
        }
      };
      // Products of this half's 128 hidden features, issued by one thread of its i-th warp (four of them keep it for 400 cycles).
      auto issue = [&](int i, uint32_t bar, auto&& products) {
        if ((warp & 3) == i) {
          if (elect_one()) {
            tmem_fence_after_sync();
            products();
            umma_commit_to(bar);
          }
          __syncwarp();
        }
      };
      auto half_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(3 + half) : "memory"); };
      // [Q; K] W1 / wscale of the n'th stage
      auto issue_first = [&](uint32_t n, int s) {
        const uint32_t slot = n % MLP_NST;
        if ((warp & 3) == 0) wait_for(bar_full + 8 * slot, (n / MLP_NST) & 1, 21, s);
        issue(0, bar_z, [&]() {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16_ts(tmem + TM_Z + 48 * half + 16 * (n & 1), tmem + TM_W1B + 32 * half + 8 * ks, umma_desc_sw128(base + slot * SM::SLOT + 32 * ks),
                         umma_idesc_bf16(128, 32), ks != 0);
        });
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
            if (CHUNKS && chunk > 0) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float4 a = __ldcg(parked + mat * (HD * MLP_E / 4) + (8 * cc + i) * 32);
                v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
              }
            } else if (mat == 0) {  // the stream starts from the caller's initial state
#pragma unroll
              for (int i = 0; i < 32; ++i)
                v[i >> 2][i & 3] = ld_as_float<T>(p.w1, (size_t)stream * HD * MLP_E + (size_t)(32 * cc + i) * MLP_E + e_own) * winv;
            } else if (SAVE && (reinterpret_cast<uintptr_t>(p.w2) & 15) != 0) {  // (the backward's own walk takes any address)
#pragma unroll
              for (int i = 0; i < 32; ++i)
                v[i >> 2][i & 3] = ld_as_float<T>(p.w2, (size_t)stream * HD * MLP_E + (size_t)e_own * HD + 32 * cc + i) * winv;
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
            put_copy(mat, n & 1, cc, v);
          }
        const float* const ho = bws + HANDOFF;
        const bool first = !CHUNKS || chunk == 0;
        b1c = first ? ld_as_float<T>(p.b1, (size_t)stream * MLP_E + b1_col) : __ldcg(ho + MLP_HO_B1 + b1_col);
        sts_word(base + SM::OFF_B1 + (n & 1) * MLP_E * 4 + 4 * b1_col, __float_as_uint(b1c));
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // b2: at first all of it the first warp's share
          const int c = lane + 32 * h;
          float b = 0.f;
          if (!first) b = __ldcg(ho + MLP_HO_B2 + warp * HD + c);
          else if (warp == 0) b = ld_as_float<T>(p.b2, (size_t)stream * HD + c) * winv;
          sts_word(base + SM::OFF_B2 + (n & 1) * SM::B2 + 4 * (warp * HD + c), __float_as_uint(b));
        }
        tmem_wait_st();
        tmem_fence_before_sync();
        half_sync();
        issue_first(n, s_lo);
      }

      for (int s = s_lo; s <= s_hi; ++s, ++n) {
        const uint32_t slot = n % MLP_NST, par = n & 1;
        const uint32_t tk = base + slot * SM::SLOT + (par ^ 1) * TL, tv = base + slot * SM::SLOT + 2 * TL;
        const uint32_t w2c = base + SM::OFF_W2 + par * SM::WC, tx2 = base + SM::OFF_X2 + par * SM::ET,
                       tg1 = base + SM::OFF_G1 + par * SM::ET, tg2 = base + SM::OFF_G2 + par * TL;
        uint8_t* const rec = SAVE ? rec0 + (size_t)s * MLP_REC_BYTES : nullptr;  // the backward's record of the stage
        if (SAVE) *reinterpret_cast<float*>(rec + MLP_REC_B1 + 4 * b1_col) = b1c;
        const uint32_t sh = base + SM::OFF_B2 + par * SM::B2 + warp * HD * 4;  // this warp's share of b2
        wait_for(bar_full + 8 * slot, (n / MLP_NST) & 1, 21, s);
        wait_for(bar_z, n & 1, 24, s);
        tmem_fence_after_sync();
        // ---- C1. Z1 = K W1 + b1 (this warp's hidden features), X2 = gelu(Z1), D1 = wscale gelu'(Z1)
        F2 d1[4][2];         // [i][nt]: hidden feature 8 i + g, tokens 8 nt + 2 t, + 1
        {
          float z1[2][2][4];
          uint32_t x2[4][2];
          tmem_ld_tokens(tmem + tm_lane + TM_Z + 48 * half + 16, z1);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const F2 b1 = f2(__uint_as_float(lds_word(base + SM::OFF_B1 + par * MLP_E * 4 + 4 * (32 * warp + 8 * i + g))));
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              F2 unused;
              const F2 x = gelu_pair<1>(f2fma(pr(z1[i >> 1][nt], i & 1), f2(wscale), b1), d1[i][nt], unused, wscale);
              x2[i][nt] = pack_bf16(x.x, x.y);
            }
          }
          stsm_x4_t(tx2 + own, x2[0][0], x2[0][1], x2[1][0], x2[1][1]);
          stsm_x4_t((tx2 + own) ^ 32u, x2[2][0], x2[2][1], x2[3][0], x2[3][1]);
        }
        // ---- C2. this warp's share of Z2 = X2 W2 + b2 (all 64 columns, its own 32 hidden features)
        {
          uint32_t a[2][4];
          __syncwarp();
          ldsm_x4(a[0], tx2 + own);
          ldsm_x4(a[1], (tx2 + own) ^ 32u);
          share_of_hidden_sum(a, w2c + wrow, sh + 8 * t, base + SM::OFF_PC + part_frag, wscale);
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
          sum_partials<8>(base + SM::OFF_PC + part_row, z);
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
        issue(0, bar_h, [&]() {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16_ts(tmem + TM_Z + 48 * half + 16, tmem + TM_W2B + 32 * half + 8 * ks, umma_desc_sw128(tg2 + 32 * ks), umma_idesc_bf16(128, 16), ks != 0);
        });
        issue(1, bar_w2, [&]() {
          if (w_moves) umma_update(tmem + 128 + 64 * half, tx2 + half * 2 * TL, tg2, UPD_IDESC);
        });
        // ---- C4. G1p = (G2p W2^T) o gelu'(Z1)
        wait_for(bar_h, n & 1, 24, s);
        tmem_fence_after_sync();
        float cs1[4];  // float32 sums over this thread's tokens
        {
          float h[2][2][4];
          tmem_ld_tokens(tmem + tm_lane + TM_Z + 48 * half + 16, h);
          uint32_t gp[4][2];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const F2 a = f2mul(pr(h[i >> 1][0], i & 1), d1[i][0]), b = f2mul(pr(h[i >> 1][1], i & 1), d1[i][1]);
            gp[i][0] = pack_bf16(a.x, a.y);
            gp[i][1] = pack_bf16(b.x, b.y);
            cs1[i] = f2hsum(f2add(a, b));
          }
          stsm_x4_t(tg1 + own, gp[0][0], gp[0][1], gp[1][0], gp[1][1]);
          stsm_x4_t((tg1 + own) ^ 32u, gp[2][0], gp[2][1], gp[3][0], gp[3][1]);
        }
        fence_proxy_async_smem();
        tmem_fence_before_sync();
        mbar_arrive_warp(bar_pub + 8 * par);  // X2, G2p, G1p of the stage, and the copies and biases that it began with
        half_sync();  // G1p of the half's hidden features
        issue(0, bar_w1, [&]() {
          if (w_moves) umma_update(tmem + 64 * half, tg1 + half * 2 * TL, tk, UPD_IDESC);
        });
        if ((warp & 3) == 2) wait_for(bar_m1, n & 1, 24, s);
        issue(2, bar_zq + 8 * par, [&]() {  // Zb1 = Q W1 - M1' G1p
          umma_bf16(tmem + TM_Z + 48 * half + 32 * par, token_desc(tg1 + half * 2 * TL), umma_desc_sw128(base + SM::OFF_M1 + par * TL), umma_idesc_bf16(128, 16) | (1u << 15), 1u);
        });
        // ---- C5. under the updates: float32 column sums (like the reference) of G2p and G1p; then the next stage's copies
        const bool more = s < s_hi;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          gp[h] = f2add(gp[h], f2(__shfl_xor_sync(0xffffffffu, gp[h].x, 16), __shfl_xor_sync(0xffffffffu, gp[h].y, 16)));
        {  // lanes of a quad take one hidden feature each
          const float a0 = (t & 2 ? cs1[2] : cs1[0]) + __shfl_xor_sync(0xffffffffu, t & 2 ? cs1[0] : cs1[2], 2);
          const float a1 = (t & 2 ? cs1[3] : cs1[1]) + __shfl_xor_sync(0xffffffffu, t & 2 ? cs1[1] : cs1[3], 2);
          const float c = (t & 1 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, t & 1 ? a0 : a1, 1);
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
        if (more) refresh(1, par ^ 1);
        wait_for(bar_w1, n & 1, 23, s);
        tmem_fence_after_sync();
        if (more) {
          refresh(0, 0);
          sts_word(base + SM::OFF_B1 + (par ^ 1) * MLP_E * 4 + 4 * b1_col, __float_as_uint(b1c));
          tmem_wait_st();
          tmem_fence_before_sync();
          half_sync();
          issue_first(n + 1, s + 1);
        }
        // (stage ends)
      }

      // ---- the item's state: float32 masters and biases
      mlp_group_sync<1>();  // (the shares of b2)
      float* const ho = bws + HANDOFF;
      const bool park = CHUNKS && chunk < NCH - 1, results = !park && !(SAVE && p.walk_only);
#pragma unroll
      for (int mat = 0; mat < 2; ++mat)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float v[8][4];
          tmem_ld_8x4(tm_own + 128 * mat + 32 * cc, v);
          if (SAVE || park) {  // for the next chunk of this stream, or as the backward takes them up
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
      // (the shares as they are: a stream's results are the same bits whether it runs in chunks or not)
      if (park) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          ho[MLP_HO_B2 + tid + MLP_GROUP * h] = __uint_as_float(lds_word(base + SM::OFF_B2 + (n & 1) * SM::B2 + 4 * (tid + MLP_GROUP * h)));
      }
      if (results && tid < HD) {
        float b = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) b += __uint_as_float(lds_word(base + SM::OFF_B2 + (n & 1) * SM::B2 + 4 * (w * HD + tid)));
        st_from_float<T>(p.b2_out, (size_t)stream * HD + tid, b * wscale);
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
      const float m1_row[2] = {-te_row[0] / wscale, -te_row[1] / wscale};
      // -M1' / wscale = -te (1 + tril(Q K^T)) / wscale of the n'th stage, the K-major operand of a product over its tokens
      auto form_m1 = [&](uint32_t n, int s) {
        const uint32_t slot = n % MLP_NST, tq = base + slot * SM::SLOT + (n & 1) * TL, tk = base + slot * SM::SLOT + ((n & 1) ^ 1) * TL;
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
            const F2 m = f2fma(pr(at[jt], r), f2(m1_row[r]), f2(m1_row[r]));
            sts_word(base + SM::OFF_M1 + (n & 1) * TL + off_bf16(i, jj), pack_bf16(jj <= i ? m.x : 0.f, jj + 1 <= i ? m.y : 0.f));
          }
        fence_proxy_async_smem();
        mbar_arrive_warp(bar_m1);
      };
      // stage s, the n'th of this block, into its ring slot: four copies by a warp each (a copy costs its thread a hundred cycles)
      auto issue_load = [&](uint32_t n, int s, int which) {
        if (elect_one()) {
          const uint32_t slot = n % MLP_NST, bar = bar_full + 8 * slot, to = base + slot * SM::SLOT;
          const int r0 = row_base + s * CS;
          if (which == 0) {
            mbar_expect_tx(bar, 3 * TL + CS * 2);
            tma_load_2d(to + ((n & 1) ^ 1) * TL, &tm_k, 0, r0, bar);
          } else if (which == 1) {
            tma_load_2d(to + (n & 1) * TL, &tm_q, 0, r0, bar);
          } else if (which == 2) {
            tma_load_2d(to + 2 * TL, &tm_v, 0, r0, bar);
          } else {
            bulk_load_1d(base + SM::OFF_LR + slot * 32, static_cast<const uint8_t*>(p.lr) + (size_t)r0 * 2, CS * 2, bar);
          }
        }
        __syncwarp();
      };
      uint32_t asked = n + (s_lo < s_hi ? 2 : 1);  // stages whose loads have been issued
      if (warp >= 2 && warp < 6) {
        issue_load(n, s_lo, warp - 2);
        if (s_lo < s_hi) issue_load(n + 1, s_lo + 1, warp - 2);
      }
      if (warp == 0) form_m1(n, s_lo);
      for (int s = s_lo; s <= s_hi; ++s, ++n) {
        const uint32_t slot = n % MLP_NST, par = n & 1, tq = base + slot * SM::SLOT + par * TL;
        const uint32_t w2c = base + SM::OFF_W2 + par * SM::WC, tx2 = base + SM::OFF_X2 + par * SM::ET,
                       tg1 = base + SM::OFF_G1 + par * SM::ET, tg2 = base + SM::OFF_G2 + par * TL;
        uint8_t* const rec = SAVE ? rec0 + (size_t)s * MLP_REC_BYTES : nullptr;
        wait_for(bar_full + 8 * slot, (n / MLP_NST) & 1, 26, s);
        // ---- O1. Zb1 = Q W1 + b1 - M1' G1p;  Xb2 = gelu(Zb1)
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
        wait_for(bar_zq + 8 * par, (n >> 1) & 1, 28, s);
        tmem_fence_after_sync();
        uint32_t xb[4][2];  // token 8 nt + g, hidden features 8 i + 2 t, + 1
        {
          float zq[2][2][4];
          tmem_ld_tokens(tmem + tm_lane + TM_Z + 48 * half + 32 * par, zq);
          tmem_fence_before_sync();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const F2 b1 = f2(__uint_as_float(lds_word(base + SM::OFF_B1 + par * MLP_E * 4 + 4 * (32 * warp + 8 * i + g))));
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              F2 unused;
              const F2 x = gelu_pair<0>(f2fma(pr(zq[i >> 1][nt], i & 1), f2(wscale), b1), unused, unused);
              xb[i][nt] = movm_t(pack_bf16(x.x, x.y));
            }
          }
        }
        // ---- O2. this warp's share of A2 = Xb2 X2^T and of (Xb2 W2 + b2) / wscale: its 32 hidden features
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
        if (n > 0) wait_for(bar_parts, (n - 1) & 1, 29, s);  // the partials of the stage before have been read
        {
          const uint32_t a[2][4] = {{xb[0][0], xb[0][1], xb[1][0], xb[1][1]}, {xb[2][0], xb[2][1], xb[3][0], xb[3][1]}};
          share_of_hidden_sum(a, w2c + wrow, base + SM::OFF_B2 + par * SM::B2 + warp * HD * 4 + 8 * t, base + SM::OFF_PO + part_frag, wscale);
        }
        mlp_group_sync<2>();  // the partials of A2
        // the slot of the stage before, which everyone has left (the chain has published this one), takes the stage after next
        if (s + 2 <= s_hi) {
          if (warp >= 2 && warp < 6 && lds_word(w_fail) == 0u) issue_load(n + 2, s + 2, warp - 2);
          asked = n + 3;
        }
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
          if ((lane & 1) == 0) sts_word(base + SM::OFF_M2 + 2 * (24 * i + j), pack_bf16(a, hi));
        }
        mlp_group_sync<2>();  // -M2'
        {  // M2' G2p, a column tile per warp: the ninth partial
          uint32_t am[4], b[4];
          float z[4] = {};
          ldsm_x4(am, base + SM::OFF_M2 + (lane & 15) * 48 + ((lane >> 4) << 4));
          ldsm_x4_t(b, tg2 + (tl ^ ((warp & 6) << 4)));
          mma_bf16(z, am[0], am[1], am[2], am[3], warp & 1 ? b[2] : b[0], warp & 1 ? b[3] : b[1]);
          const uint32_t to = base + SM::OFF_PO + 8 * 4096 + g * 256 + ((32 * warp + 8 * t) ^ ((g & 3) << 5));
          sts_pair(to, pr(z, 0));
          sts_pair(to + 8 * 256, pr(z, 1));
        }
        const uint2 qv = lds_u2(tq + tile_row);
        mlp_group_sync<2>();  // the partials of Zb2
        // ---- O3. out = Q + LN(Zb2), a row per half-warp
        F2 zb[2], o[2];
        sum_partials<9>(base + SM::OFF_PO + part_row, zb);
        mbar_arrive_warp(bar_parts);
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
        if (s < s_hi && warp == (int)((n + 1) & 7)) form_m1(n + 1, s + 1);  // (one warp)
      }
      if (warp == 2 && lds_word(w_fail) != 0u) {  // copies that are on their way land before the block leaves
        for (uint32_t i = 1; i <= MLP_NST && i <= asked; ++i) mbar_wait_bounded(bar_full + 8 * ((asked - i) % MLP_NST), ((asked - i) / MLP_NST) & 1);
      }
    }
    __syncthreads();  // the item is left by both groups
    if (lds_word(w_fail) != 0u) break;
  }  // work items
  if (lds_word(w_fail) != 0u) {  // products that nobody waited for end before tensor memory and the block's memory are given back
    if (!output_group && (warp & 3) < 3) {
      if (elect_one()) umma_commit_to(bar_end);
      __syncwarp();
    }
    if (threadIdx.x < 32) mbar_wait_bounded(bar_end, 0);
  }
  tmem_fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(lds_word(w_tmem), 512);
  if (SAVE) bulk_wait_all<0>();
}

cudaError_t launch_mlp_fwd(const CUtensorMap* m, const MlpFwdParams& p, int nstreams, cudaStream_t st) {
  const bool chunks = p.bwd_ws != nullptr, save = chunks && p.records;
  auto kfn = save ? ttt_mlp_fwd_kernel<true, true> : chunks ? ttt_mlp_fwd_kernel<false, true> : ttt_mlp_fwd_kernel<false, false>;
  static DeviceValue resident[3];
  int sms = 0, per_sm = 0;
  cudaError_t e = resident[save ? 2 : chunks].get(0, &per_sm, [&](int* n) {
    const cudaError_t a = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MlpSmem::TOTAL);
    return a != cudaSuccess ? a : cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kfn, MLP_THREADS, MlpSmem::TOTAL);
  });
  if (e != cudaSuccess) return e;
  if (!chunks) {  // nothing to park state in: one block per stream
    kfn<<<nstreams, MLP_THREADS, MlpSmem::TOTAL, st>>>(m[0], m[1], m[2], p);
    return cudaGetLastError();
  }
  if ((e = device_sms(&sms)) != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  MlpFwdParams pp = p;
  pp.nstreams = nstreams;
  int grid = sms * per_sm;
  if (grid > nstreams) grid = nstreams;
  pp.CH = mlp_chunk_stages(p.NS, nstreams, grid);
  pp.NCH = (p.NS + pp.CH - 1) / pp.CH;
  if ((e = cudaMemsetAsync(pp.sched, 0, sizeof(int) * (size_t)(1 + nstreams), st)) != cudaSuccess) return e;
  if (!save) {  // (an item waits only for one of smaller index, which a block holds that runs or has run)
    kfn<<<grid, MLP_THREADS, MlpSmem::TOTAL, st>>>(m[0], m[1], m[2], pp);
    return cudaGetLastError();
  }
  // as many blocks as are co-resident, never more than streams
  void* args[] = {(void*)&m[0], (void*)&m[1], (void*)&m[2], (void*)&pp};
  return cudaLaunchCooperativeKernel((const void*)kfn, dim3(grid), dim3(MLP_THREADS), args, MlpSmem::TOTAL, st);
}
// Floats per stream, and whether the scheme above gains anything (one CTA per SM): no more streams than SMs, or chunks of less
// than the whole sequence would cost more than the waves they even out, and no scratch is used.
constexpr size_t MLP_PARK_FLOATS = 2 * HD * MLP_E + MLP_BWD_HANDOFF_FLOATS;
size_t mlp_fwd_scratch_floats(int NS, int nstreams) {
  int sms = 0;
  if (device_sms(&sms) != cudaSuccess || nstreams <= sms || mlp_chunk_stages(NS, nstreams, sms) >= NS) return 0;
  return MLP_PARK_FLOATS * (size_t)nstreams + (size_t)((1 + nstreams + 3) & ~3);
}
void mlp_fwd_use_scratch(MlpFwdParams& p, float* scratch, int nstreams) {
  p.bwd_ws = scratch;
  p.bwd_ws_stride = MLP_PARK_FLOATS;
  p.records = 0;
  p.sched = reinterpret_cast<int*>(scratch + MLP_PARK_FLOATS * (size_t)nstreams);
}
}  // namespace ttt
