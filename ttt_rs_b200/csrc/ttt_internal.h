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

}  // extern "C"
