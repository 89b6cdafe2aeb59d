// Launcher of the tensor-memory backward kernel of the plain MLP, shared between mlp_backward_tc.cu and mlp.cu, which selects it.
#pragma once

#include "common.cuh"

// input, output, layers; hidden width 64
#define NB_MLP_TC_SHAPES(X) \
    X(32, 16, 2)            \
    X(32, 8, 3)             \
    X(32, 8, 2)             \
    X(32, 16, 3)            \
    X(64, 64, 2)            \
    X(64, 64, 4)

namespace nb {
inline bool mlp_backward_tc_supported(const nb_mlp_desc* d) {
#define X(K0, OUT, NL) \
    if (d->input_dim == K0 && d->hidden_dim == 64 && d->output_dim == OUT && d->num_layers == NL) return true;
    NB_MLP_TC_SHAPES(X)
#undef X
    return false;
}
int launch_mlp_backward_tc(const nb_mlp_desc* d, const void* dL, const void* W, const void* act0, const void* acts, int64_t n, float* dW, float* db,
                           void* dX, cudaStream_t st);
}  // namespace nb
