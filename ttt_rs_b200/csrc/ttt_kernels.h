// Internal interface between the C-ABI layer (ttt_abi.cu) and the kernel translation units.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace ttt {

// A launch parameter that depends on the device (and at most on `key`), computed on first use: the queries behind it
// (function attributes, occupancy) cost a microsecond or more each, and a launch makes several.  `fn(int* value)` is
// idempotent.
struct DeviceValue {
  static constexpr int N = 64;
  std::atomic<uint64_t> slot[N] = {};
  template <class Fn>
  cudaError_t get(uint32_t key, int* value, Fn fn) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t have = dev < N ? slot[dev].load(std::memory_order_acquire) : 0;
    if (have != 0 && (uint32_t)(have >> 32) == key + 1) {
      *value = (int)(uint32_t)have;
      return cudaSuccess;
    }
    if ((e = fn(value)) != cudaSuccess) return e;
    if (dev < N) slot[dev].store(((uint64_t)(key + 1) << 32) | (uint32_t)*value, std::memory_order_release);
    return cudaSuccess;
  }
};
inline cudaError_t device_sms(int* sms) {
  static DeviceValue v;
  return v.get(0, sms, [](int* n) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    return e != cudaSuccess ? e : cudaDeviceGetAttribute(n, cudaDevAttrMultiProcessorCount, dev);
  });
}

struct LinFwdParams {
  const void* w0;         // [B,H,F,F] element type T
  const void* b0;         // [B,H,F]
  const void* token_eta;  // [T], first 16 entries read
  const void* lr;         // [B,H,lr_ld], lr_ld elements per (batch, head): T, or more where the caller pads the rows
  const void* ln_g;       // [H,F]
  const void* ln_b;       // [H,F]
  void* w_out;            // [B,H,F,F]
  void* b_out;            // [B,H,F]
  float* w_ckpt;          // [B*H*(NCK+1), F, F] float32: state before stage c*K for c < NCK, final state at c = NCK
  float4* stats;          // [B*H*T][2]: (mean1, rstd1, A, Bv), (mean2, rstd2, 0, 0) per token
  float* b_stage;         // [B*H*(NS+1), F] float32: bias at the start of every stage, final bias last
  uint32_t* status;       // device uint32[4] or null
  int H, T, NS, K, NCK;   // T: tokens per stream in memory (NS mini-batches of them are walked)
  int lr_ld;
  float eps;
};

struct LinBwdParams {
  const void* w0;
  const void* b0;
  const void* token_eta;
  const void* lr;
  const void* ln_g;
  const void* ln_b;
  const float* w_ckpt;
  const float4* stats;
  const float* b_stage;
  const void* dw_in;  // [B,H,F,F] T: upstream gradient of the returned final weight, or null (zero)
  const void* db_in;  // [B,H,F]   T: upstream gradient of the returned final bias, or null (zero)
  void* d_w;        // [B,H,F,F] element type T (per batch element), nullable
  void* d_b;        // [B,H,F], nullable
  void* d_lr;       // [B,H,T]
  void *d_q, *d_k, *d_v;  // [B,H,T,F]: what the tensor maps of the gradients cover
  int* sched;       // workspace: [0] next work item, [1 + stream] chunks of the stream finished so far (zeroed per launch)
  float* handoff;   // workspace: [B*H][2*F*F + F] W^T, dW^T (register layout) and db handed from chunk to chunk
  int CH, NCH, nstreams;  // stages per chunk, chunks per stream, B*H (the launcher sets CH = NS, NCH = 1, sched = null
                          // where every stream has an SM of its own)
  uint32_t handoff_polls;  // iteration limit of the wait for another chunk's hand-off (each poll sleeps ~100 ns)
  int item_base;           // added to every work-item number (0 in normal use; the wait-limit test starts past the
                           // items that would publish the first hand-offs, so that a wait runs out)
  float* part_ln;   // workspace: [B*H][NCH][2][F] per-(stream, chunk) partial LN gradients (weight, bias)
  float* part_te;   // workspace: [B*H][T] per-stream token_eta gradient terms
  float* part_w;    // workspace: [B*H][F*F + F] float32 dW, db per stream (for the packed reduction)
  uint32_t* status;
  int H, T, NS, K, NCK;
  float eps;
};

struct ReduceParams {
  const float* part_ln;
  float* part_te;  // (with `packed`, row 0 receives the sums)
  const float* part_w;
  void* d_token_eta;  // [T], float32 or bf16
  void* d_ln_g;       // [H,F]
  void* d_ln_b;       // [H,F]
  int out_bf16;       // element type of the three
  float* packed;      // nullable: [H*F*F + 3*H*F + CS] f32
  int B, H, T, NCH;
  int F;   // features per head: 64, or 32 (two heads per 64-wide tile in part_ln)
  int mb;  // tokens per mini-batch (16 or 8): d_token_eta is folded to [mb]
};

struct MlpFwdParams {
  const void* w1;         // [B,H,F,E] bf16, E = 4F
  const void* b1;         // [B,H,E]
  const void* w2;         // [B,H,E,F]
  const void* b2;         // [B,H,F]
  const void* token_eta;  // [T], first 16 entries read
  const void* lr;         // [B,H,T]
  const void* ln_g;       // [H,F]
  const void* ln_b;       // [H,F]
  void* out;              // [B,H,T,F]
  void* w1_out;
  void* b1_out;
  void* w2_out;
  void* b2_out;
  uint32_t* status;
  float* bwd_ws;         // optional: a block per stream to park its state in between work items
  size_t bwd_ws_stride;
  int records;           // it is the backward's workspace: the final state and a record of every stage are left there
  int walk_only;         // only that: no output and no final state for the caller
  int* sched;            // with bwd_ws (null otherwise): [1 + B*H] work-item counter and per-stream count of finished chunks (the
                         // persistent launch; zeroed by the launcher)
  int nstreams, CH, NCH; // set by the launcher: streams, stages per work item, items per stream
  uint32_t handoff_polls;  // iteration limit of the wait for the previous chunk's state
  int H, T, NS;
  float eps;
};
// token_eta of one mini-batch as the layer forms it from its parameters (bf16), written by the kernel that writes the
// learning rates: out[i] = max(idx[i] + learnable[i], 0).  n = 0: not asked for.
struct TokenEtaParams {
  const void *idx, *learnable;
  void* out;
  int n;
};
// Outer-layer steps either side of the inner loop (ttt_layer.cu).
struct LayerProParams {
  const void* q_src;   // projection outputs, rows = tokens (b*T + t), this head-major column block of H*F columns;
  const void* k_src;   // with the shared-QK convolutions q_src is the shared projection and k_src is unused
  const void* v_src;
  long ld_src;         // row stride of the three sources, in elements
  const void* lr_logits;  // [B*T, ld_lr], first H columns used
  long ld_lr;
  const void* lr_bias;    // [H] or null
  const void* conv_q_w;   // [H*F, conv_k] or null (no convolution)
  const void* conv_q_b;   // [H*F]
  const void* conv_k_w;
  const void* conv_k_b;
  int conv_k;
  void* xq;            // [B,H,T,F]
  void* xk;
  void* xv;
  void* lr_out;        // [B,H,lr_ld_out] (lr_ld_out >= T)
  int lr_ld_out;
  int tchunk;          // tokens per warp task, set by the launcher
  TokenEtaParams te;   // (bf16)
  int B, H, T;
  int start_idx, pos_mod, rope_mode;  // rope_mode: 0 none, 1 positions modulo pos_mod, 2 global positions
  float rope_theta, base_lr;
};
struct LayerEpiParams {
  const void* inner_out;  // [B,H,T,F]
  const void* gate;       // [B*T, ld_gate] (first H*F columns) or null
  long ld_gate;
  const void* ln_w;       // [H*F]
  const void* ln_b;
  void* y;                // [B,T,H*F]
  int row_groups;         // set by the launcher: rows of a tile that a CTA's threads work on at once
  int tile_rows;          // set by the launcher: tokens of a tile
  int B, H, T;
  float eps;
};
// Few-token forms of the layer's two sides (ttt_layer_small.cu): up to SMALL_M rows, bf16, head_dim 64 or 32, at most 2048
// features, hidden a multiple of 32.
constexpr int SMALL_M = 32;
// The output side only where it is faster than epilogue + tensor-core GEMM.  Up to 16 rows that is everywhere.  From 17 on
// every CTA normalises (and gates) up to 32 rows for itself and holds them in 64 C bytes of shared memory (from 1700 features
// on one CTA per SM and two waves).  Decode step of a layer, output side few-token / general, us (all general: 31 to 47):
//   features          768               1024              1280              1536              2048
//   17 rows       20.2 / 22.7       22.5 / 24.6       25.8 / 26.7       30.8 / 29.8       47.7 / 33.8
//   24 rows       20.5 / 22.6       23.5 / 24.7       27.5 / 27.7       32.8 / 29.9       50.2 / 34.0
//   32 rows       23.0 / 22.6       26.6 / 25.8       31.7 / 28.8       38.4 / 31.7       59.3 / 35.9
//   24, gated     25.2 / 24.6       30.1 / 26.7       35.8 / 29.5       43.1 / 32.0       72.4 / 41.0
inline bool layer_small_out_rows(int64_t rows, int64_t features, bool gate) {
  return rows <= 16 || (rows <= SMALL_M && !gate && rows * features <= 24576);
}
struct SmallProjParams {
  const void* x;  // [M, ldx], rows b * T + t
  const void* w;  // [N, ldw]: q | k | v | (gate) blocks of H F rows, then H learning-rate rows from lr_col on
  const void* lr_bias;
  void *xq, *xk, *xv, *gate, *lr_out;  // [B,H,T,F] x 3, [M, H F] or null, [B,H,lr_ld]
  long ldx;  // (one-token calls on a slice of a [B, T, C] buffer: T C elements)
  int M, N, K, ldw, H, F, T, lr_col, lr_ld;
  int start_idx, pos_mod, rope_mode;
  float rope_theta, base_lr;
  TokenEtaParams te;
};
struct SmallOutParams {
  const void* inner_out;  // [B,H,T,F]
  const void* gate;       // [M, ld_gate] or null
  const void *ln_w, *ln_b, *w;  // w [H F, ldw]
  void* y;                // [M, H F]
  int M, H, F, T, ldw, ld_gate;
  float eps;
};
cudaError_t launch_layer_small_proj(const SmallProjParams& p, cudaStream_t st);
cudaError_t launch_layer_small_out(const SmallOutParams& p, cudaStream_t st);
struct LayerProBwdParams {
  const void* dxq;  // [B,H,T,F] gradients of the prologue's outputs
  const void* dxk;
  const void* dxv;
  const void* dlr;  // [B,H,T]
  const void* lr;   // [B,H,T] the forward's ttt_lr_eta
  void* dq_dst;     // [B*T, ld_dst] column blocks of the projection-output gradient
  void* dk_dst;
  void* dv_dst;
  long ld_dst;
  void* dlogits_dst;  // [B*T, ld_dlr]: lr_cols columns written (H logit gradients, then zeros)
  long ld_dlr;
  int lr_cols;
  int B, H, T;
  int tchunk;  // set by the launcher
  int start_idx, pos_mod, rope_mode;
  float rope_theta, base_lr;
};
struct LayerEpiBwdParams {
  const void* dy;         // [B*T, H*F] gradient of the epilogue's output
  const void* inner_out;  // [B,H,T,F]
  const void* gate;       // [B*T, ld_gate] or null
  long ld_gate;
  const void* ln_w;
  const void* ln_b;
  void* d_inner;          // [B,H,T,F]
  void* dgate;            // [B*T, ld_dgate] (written when gate != null)
  long ld_dgate;
  float* d_ln_w;          // [H*F] float32
  float* d_ln_b;
  float* partials;        // workspace (float32): [CTAs][2][H*F] partial sums
  int row_groups;         // set by the launcher: rows of a tile that a CTA's threads work on at once
  int tile_rows;          // set by the launcher: tokens of a tile
  int B, H, T;
  float eps;
};
// Shared-QK causal depthwise convolutions as a training step of their own (ttt_layer.cu): q = conv_q(x) + bq,
// k = conv_k(x) + bk over the token axis, four taps aligned to the end (tap j multiplies token t - 3 + j; shorter
// kernels are passed zero-padded at the front), zeros before the start of the sequence.
struct LayerConvParams {
  const void* x;   // [B*T, ld_x] shared projection output, C = H*F columns used
  long ld_x;
  const void* wq;  // [C][4]
  const void* bq;  // [C]
  const void* wk;
  const void* bk;
  void* q;         // [B*T, C] (out)
  void* k;         // [B*T, C] (out)
  int B, T, C;
};
struct LayerConvBwdParams {
  const void* dq;  // [B*T, C]
  const void* dk;
  const void* x;   // as in the forward
  long ld_x;
  const void* wq;
  const void* wk;
  void* dx;        // [B*T, C] (out)
  float* partials; // [B * ceil(T / LAYER_CONV_CHUNK)][10 C] per-chunk parameter-gradient partials
  float* dparams_q;  // [5 C]: d wq as [4][C] (tap-major), then d bq [C]
  float* dparams_k;  // [5 C]
  int B, T, C;
};
constexpr int LAYER_CONV_CHUNK = 64;  // tokens a thread walks
cudaError_t launch_layer_conv(int dtype, const LayerConvParams& p, cudaStream_t st);
cudaError_t launch_layer_conv_bwd(int dtype, const LayerConvBwdParams& p, cudaStream_t st);
cudaError_t launch_layer_prologue(int dtype, int head_dim, const LayerProParams& p, cudaStream_t st);
cudaError_t launch_layer_prologue_bwd(int dtype, int head_dim, const LayerProBwdParams& p, cudaStream_t st);
cudaError_t launch_layer_epilogue_bwd(int dtype, int head_dim, const LayerEpiBwdParams& p, cudaStream_t st);
size_t layer_epilogue_bwd_workspace_bytes(int B, int H, int T, int head_dim);
cudaError_t launch_layer_epilogue(int dtype, int head_dim, const LayerEpiParams& p, cudaStream_t st);

// One mini-batch of R <= 16 tokens per stream (decode step, sequence tail): ttt_linear_partial.cu.
// One mini-batch of R rows per stream; row i of stream s is row s * row_ld + row_off + i of xq, xk, xv, out, and element
// s * lr_ld + row_off + i of lr (a mini-batch of its own: row_ld = lr_ld = R, row_off = 0; the tail of a longer sequence:
// the sequence's pitch and the tail's first token).
struct LinPartialParams {
  const void* xq;  // [B,H,row_ld,F]
  const void* xk;
  const void* xv;
  const void* w0;         // [B,H,F,F]
  const void* b0;         // [B,H,F]
  const void* token_eta;  // [R]
  const void* lr;         // [B,H,lr_ld]
  const void* ln_g;       // [H,F]
  const void* ln_b;
  void* out;              // [B,H,row_ld,F]
  void* w_out;            // may alias w0
  void* b_out;            // may alias b0
  int H, R;
  int row_ld, row_off, lr_ld;
  float eps;
  int state_settled;  // the kernel before this one on the stream does not write the state (see launch_dependent)
};
cudaError_t launch_linear_partial(int dtype, int head_dim, const LinPartialParams& p, int nstreams, cudaStream_t st);

// TTT-MLP backward (ttt_mlp_bwd.cu), bf16 I/O.
struct MlpBwdParams {
  const void* token_eta;
  const void* lr;
  const void* ln_g;
  const void* ln_b;
  void* d_q;  // [B,H,T,F]
  void* d_k;
  void* d_v;
  void* d_w1;
  void* d_b1;
  void* d_w2;
  void* d_b2;
  void* d_lr;
  void* d_token_eta;  // [T], float32 or bf16
  void* d_ln_g;       // [H,F]
  void* d_ln_b;
  int reduced_bf16;   // element type of the three
  float* workspace;   // per stream `ws_stride` floats, filled by the forward
  size_t ws_stride;
  float* part_te;      // [B*H][T]
  float* part_ln;      // [B*H][2][F]
  int* sched;           // [1 + B*H] work-item counter and per-stream count of finished items (zeroed by the launcher)
  uint32_t* status;     // optional 4 words: {TTT_ERR_TIMEOUT, where, block, item} if a hand-off wait ran out
  int H, T, NS;
  int nstreams, CH, NCH;  // set by the launcher: streams, stages per work item, items per stream
  float eps;
};
// Per-stream block of the TTT-MLP backward's workspace: the float32 masters of W1^T, W2, dW1^T, dW2, each [256 hidden][64]
// (order: mlp_master_at; W1 and W2 divided by -token_eta[15], as the kernels carry them, unless that is zero), the hand-off
// record between work items, then one record per stage, written by the forward.
constexpr int MLP_BWD_HANDOFF_FLOATS = 2 * 256 + 4 * 64;
constexpr int MLP_HO_B1 = 0, MLP_HO_B2 = 256;                             // the forward's: b1, eight shares of b2 [8][64]
constexpr int MLP_HO_DB1 = 320, MLP_HO_DB2 = 576, MLP_HO_DG = 640;        // the backward's, once the forward is done; DG: weight, bias [2][64]
static_assert(MLP_HO_B2 + 8 * 64 <= MLP_BWD_HANDOFF_FLOATS && MLP_HO_DG + 2 * 64 <= MLP_BWD_HANDOFF_FLOATS, "hand-off record");
// element (hidden feature e, feature f) of a master, as a float index: 16-byte pieces of 32 consecutive hidden features
// (the lanes of a warp) side by side
__host__ __device__ inline int mlp_master_at(int e, int f) { return ((((e >> 5) * 16 + (f >> 2)) * 32 + (e & 31)) << 2) + (f & 3); }
// A stage's record, in bytes.  X2 [16][256] and G1p [16][256] (four tiles of 64 columns) and G2p [16][64]: bf16, in the
// swizzled form that shared memory holds them in (off_bf16); float32: Z2, Zb2 [16][64], b1 [256] at the start of the stage, and
// per token the means of Z2 and of Zb2
constexpr int MLP_REC_X2 = 0, MLP_REC_G1P = 8192, MLP_REC_G2P = 16384, MLP_REC_Z2 = 18432, MLP_REC_ZB2 = 22528,
              MLP_REC_B1 = 26624, MLP_REC_MEAN = 27648, MLP_REC_BYTES = 27776;
// Stages per work item of the persistent launches: a stream that has a block to itself is one item; otherwise the length
// for which the busiest block has least to do, a hand-over of a stream counted as one stage and a half (the backward: 512 KB
// through L2 against a stage of 4 us)
inline int mlp_chunk_stages(int NS, int nstreams, int blocks) {
  if (nstreams <= blocks) return NS;
  int best = NS;
  long long least = -1;
  for (int ch = 8; ch <= 64; ++ch) {
    const long long nch = (NS + ch - 1) / ch, rounds = (nch * nstreams + blocks - 1) / blocks;
    const long long cost = rounds * (2 * (ch < NS ? ch : NS) + 3);
    if (least < 0 || cost < least) {
      least = cost;
      best = ch;
    }
  }
  return best < NS ? best : NS;
}
size_t mlp_bwd_ws_stride_floats(int T);
// maps: q, k, v, d_out
cudaError_t launch_mlp_bwd(const CUtensorMap* maps, const MlpBwdParams& p, int B, cudaStream_t st);

// bf16 projection GEMM C[M,N] = A[M,K] . B[N,K]^T on tcgen05 (ttt_gemm.cu).  maps: A, B (loads, box 64 x 128), C (store).
// Fused epilogue of the layer's stacked projection (ttt_layer_projections): where the column blocks of the product
// start (multiples of 64; g_col < 0 = no gate) and where their results go.
struct GemmFuse {
  int q_col, k_col, v_col, g_col, lr_col;
  int H, T;                 // heads, tokens per sequence (T % 128 == 0)
  int start_idx, pos_mod, rope_mode;  // rope_mode 0 none, 1 positions (start_idx + t) mod pos_mod, pos_mod <= 16
  int round_proj;  // round the projections to bf16 first, as a product followed by the prologue would (training)
  float rope_theta, base_lr;
  const void* lr_bias;      // [H] bf16 or null
  void* lr_out;             // ttt_lr_eta [B,H,T] bf16
  TokenEtaParams te;
};
struct GemmParams {
  int M, N, K;
  uint32_t* status;  // optional 4 words
  GemmFuse f;        // read by the fused kernel only
};
cudaError_t launch_gemm_bf16_tn(const CUtensorMap* maps, const GemmParams& p, bool fused, bool pair, cudaStream_t st);

// bf16 only.  maps: q, k, v.
cudaError_t launch_mlp_fwd(const CUtensorMap* maps, const MlpFwdParams& p, int nstreams, cudaStream_t st);
// scratch of an inference call (current device), 0: none is used
size_t mlp_fwd_scratch_floats(int NS, int nstreams);
void mlp_fwd_use_scratch(MlpFwdParams& p, float* scratch, int nstreams);

// dtype: 0 = float32, 1 = bfloat16.  seg: features per head, 64 or 32 (two heads per tile).  mb: tokens per
// mini-batch, 16 or 8 (the tile maps then have boxes of 8 rows).
// maps: q, k, v, out, gp (saved lr-scaled LN gradient, [B*H*T, 64] of T)
cudaError_t launch_linear_fwd(int dtype, int seg, int mb, const CUtensorMap* maps, const LinFwdParams& p, int nstreams,
                              cudaStream_t st);
// the form for streams that have an SM each (ttt_linear_fwd_roles.cu), chosen by launch_linear_fwd
cudaError_t launch_linear_fwd_roles(int dtype, int seg, int mb, const CUtensorMap* maps, const LinFwdParams& p, int nstreams,
                                    cudaStream_t st);
// maps: q, k, v, d_out, d_q, d_k, d_v, gp
cudaError_t launch_linear_bwd(int dtype, int seg, int mb, const CUtensorMap* maps, LinBwdParams& p, int nstreams,
                              cudaStream_t st);
cudaError_t launch_linear_bwd_f32(int seg, int mb, const CUtensorMap* maps, LinBwdParams& p, int nstreams, cudaStream_t st);
cudaError_t launch_linear_bwd_reduce(const ReduceParams& p, cudaStream_t st);

}  // namespace ttt
