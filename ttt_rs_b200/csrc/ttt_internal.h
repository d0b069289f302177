// Entry points of libttt_b200.so for this package's own native host path (ttt_host.cpp); not part of the C ABI.
#pragma once

#include <stddef.h>

#include "../../include/ttt_b200.h"

extern "C" {

// ttt_linear_backward_state_grads with the three reduced gradients (token_eta, LayerNorm weight and bias) written in
// `reduced_dtype` (TTT_F32 / TTT_BF16), rounded once from the float32 sums.
int ttt_internal_linear_backward(const ttt_dims* d, const void* xq, const void* xk, const void* xv, const void* weight,
                                 const void* bias, const void* token_eta, const void* ttt_lr_eta, const void* ln_weight,
                                 const void* ln_bias, const void* weight_ckpt, const void* bias_ckpt,
                                 const void* grad_output, const void* grad_weight_out, const void* grad_bias_out,
                                 void* grad_xq, void* grad_xk, void* grad_xv, void* grad_weight, void* grad_bias,
                                 void* grad_ttt_lr_eta, void* grad_token_eta, void* grad_ln_weight, void* grad_ln_bias,
                                 int reduced_dtype, float* outer_grad_packed, void* workspace, size_t workspace_bytes,
                                 void* status, void* stream);

// ttt_mlp_backward, likewise
int ttt_internal_mlp_backward(const ttt_dims* d, const void* xq, const void* xk, const void* xv, const void* w1,
                              const void* b1, const void* w2, const void* b2, const void* token_eta,
                              const void* ttt_lr_eta, const void* ln_weight, const void* ln_bias,
                              const void* grad_output, void* grad_xq, void* grad_xk, void* grad_xv, void* grad_w1,
                              void* grad_b1, void* grad_w2, void* grad_b2, void* grad_ttt_lr_eta, void* grad_token_eta,
                              void* grad_ln_weight, void* grad_ln_bias, int reduced_dtype, void* workspace,
                              size_t workspace_bytes, int workspace_from_forward, void* status, void* stream);

// ttt_mlp_forward without a backward to follow.  scratch (16-byte aligned; null: none): memory to park streams' states in,
// with which more streams than SMs need not run in whole waves; bytes 0: not used for these dims on the current device.
size_t ttt_internal_mlp_infer_scratch_bytes(const ttt_dims* d);
int ttt_internal_mlp_infer(const ttt_dims* d, const void* xq, const void* xk, const void* xv, const void* w1, const void* b1,
                           const void* w2, const void* b2, const void* token_eta, const void* ttt_lr_eta,
                           const void* ln_weight, const void* ln_bias, void* output, void* w1_out, void* b1_out, void* w2_out,
                           void* b2_out, void* scratch, size_t scratch_bytes, void* status, void* stream);

// Inference forward over the first `d->seq_len` tokens (whole mini-batches) of sequences whose rows are `seq_pitch` tokens
// apart in xq, xk, xv, output and `lr_pitch` elements apart in ttt_lr_eta; token_eta: the first mini-batch's.
int ttt_internal_linear_infer(const ttt_dims* d, int seq_pitch, int lr_pitch, const void* xq, const void* xk,
                              const void* xv, const void* weight, const void* bias, const void* token_eta,
                              const void* ttt_lr_eta, const void* ln_weight, const void* ln_bias, void* output,
                              void* weight_out, void* bias_out, void* status, void* stream);
// ttt_linear_forward_partial on tokens [first, first + d->seq_len) of such sequences.  state_settled: the launch before
// this one on the stream was ttt_internal_layer_small_proj (the state may be read before that has finished).
int ttt_internal_linear_tail(const ttt_dims* d, int seq_pitch, int first, int lr_pitch, int state_settled, const void* xq, const void* xk,
                             const void* xv, const void* weight, const void* bias, const void* token_eta,
                             const void* ttt_lr_eta, const void* ln_weight, const void* ln_bias, void* output,
                             void* weight_out, void* bias_out, void* stream);
// ttt_layer_prologue with rows of lr_pitch elements in ttt_lr_eta.  token_idx, learnable_token_idx (bf16, d->mini_batch each,
// or null): token_eta_out [16] gets max(token_idx + learnable_token_idx, 0), up to 16 of them, in this and the next two.
int ttt_internal_layer_prologue(const ttt_dims* d, const void* q_src, const void* k_src, const void* v_src,
                                int64_t src_ld, const void* lr_logits, int64_t lr_ld, const void* lr_bias,
                                const void* conv_q_weight, const void* conv_q_bias, const void* conv_k_weight,
                                const void* conv_k_bias, int conv_kernel, int start_idx, int rope_mode,
                                float rope_theta, float base_lr, const void* token_idx, const void* learnable_token_idx,
                                void* token_eta_out, void* xq, void* xk, void* xv, void* ttt_lr_eta, int lr_pitch,
                                void* stream);
// ttt_layer_projections; round_proj: the projections are rounded to bf16 before the rotation and the learning-rate gate, as
// they are when a product and ttt_layer_prologue compute them one after the other (training).
int ttt_internal_layer_projections(const ttt_dims* d, const void* x, int64_t x_ld, int64_t hidden, const void* weights,
                                   int64_t w_ld, int64_t w_rows, int64_t q_col, int64_t k_col, int64_t v_col, int64_t g_col,
                                   int64_t lr_col, const void* lr_bias, int start_idx, int rope_mode, float rope_theta,
                                   float base_lr, int round_proj, const void* token_idx, const void* learnable_token_idx,
                                   void* token_eta_out, void* xq, void* xk, void* xv, void* gate,
                                   void* ttt_lr_eta, void* status, void* stream);
// Few-token forms (bf16): projections with the prologue, and post norm (+ gate) with the output projection; 0 from
// _fits and _out_fits: not for this shape.  weights: q | k | v | (gate) blocks of heads * head_dim rows, learning-rate rows from lr_col.
int ttt_internal_layer_small_fits(const ttt_dims* d);
int ttt_internal_layer_small_out_fits(const ttt_dims* d, int gate);
int ttt_internal_layer_small_proj(const ttt_dims* d, const void* x, int64_t x_ld, const void* weights, int64_t w_ld,
                                  int w_rows, int lr_col, const void* lr_bias, int start_idx, int rope_mode,
                                  float rope_theta, float base_lr, const void* token_idx,
                                  const void* learnable_token_idx, void* token_eta_out, void* xq, void* xk, void* xv,
                                  void* gate, void* ttt_lr_eta, int lr_pitch, void* stream);
int ttt_internal_layer_small_out(const ttt_dims* d, const void* inner_out, const void* gate, int gate_ld,
                                 const void* post_norm_weight, const void* post_norm_bias, float eps, const void* o_proj,
                                 int64_t o_ld, void* y, void* stream);

}  // extern "C"
