/* fused.h - layer calls with the element-wise work of an encoder block folded in, for block.c.  CUDA tensors
 * only; each equals the public call followed by the separate operation, with one rounding less. */
#ifndef BOAT_FUSED_H
#define BOAT_FUSED_H

#include "../core/boat_internal.h"
#include <boat/layers.h>
#include <boat/layers/attention.h>
#include <boat/layers/norm.h>

/* GELU(dense(input)); *pre_activation gets the dense output (a new tensor). */
boat_tensor_t* boat_dense_forward_gelu(boat_dense_layer_t* l, const boat_tensor_t* input, boat_tensor_t** pre_activation);
/* dense(input) + residual (same shape and dtype as the result). */
boat_tensor_t* boat_dense_forward_add(boat_dense_layer_t* l, const boat_tensor_t* input, const boat_tensor_t* residual);
/* Backward of dense(GELU(pre_activation)) to pre_activation. */
boat_tensor_t* boat_dense_backward_gelu(boat_dense_layer_t* l, const boat_tensor_t* grad_output, const boat_tensor_t* pre_activation);
/* attention(x, x, x) + residual. */
boat_tensor_t* boat_attention_forward_add(boat_attention_t* a, const boat_tensor_t* x, const boat_tensor_t* residual);
/* Gradient of x, which was query, key and value of the last forward; NULL on failure. */
boat_tensor_t* boat_attention_backward_self(boat_attention_t* a, const boat_tensor_t* grad_output);
/* LayerNorm backward + residual. */
boat_tensor_t* boat_layernorm_backward_add(boat_layernorm_t* n, const boat_tensor_t* grad_output, const boat_tensor_t* residual);

#endif
