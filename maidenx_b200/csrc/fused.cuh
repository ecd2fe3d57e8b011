// Passes of the training step that do more than one exported mx_* call (instantiated for bf16 and f16 in fused.cu).
#pragma once
#include "common.cuh"

namespace mx {

// mx_mse_loss_grad_<T>, and the rounded sum of the gradient it writes in *grad_sum.  arrived: a zeroed device word, left zeroed.
template <class T>
void mse_loss_grad_sum(size_t n, const T* pred, const T* target, T* grad, float* loss, T* grad_sum, uint32_t* arrived, const char* where);
// mx_gelu_backward_<T>, and the rounded sum of the gradient it writes in *grad_sum.
template <class T>
void gelu_backward_sum(size_t n, const T* dy, const T* u, T* du, T* grad_sum, uint32_t* arrived, const char* where);
// mx_sgd_update_<T> of a layer's weights and of its one-element bias in one launch.
template <class T>
void sgd_update_layer(size_t n, float* w32, const T* grad, T* w16, float* b32, const T* grad_b, T* b16, float lr, float grad_scale, const char* where);

}  // namespace mx
