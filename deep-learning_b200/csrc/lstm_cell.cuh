// The squashing functions of an LSTM block, shared by the kernels that run one time
// step (lstm.cu) and the ones that walk over all of them (lstm_walk.cu).
#pragma once

#include "common.cuh"

namespace dlb {

__device__ __forceinline__ float sigmoid_ref(float x) { return 1.f / (1.f + expf(-x)); }
// The reference's tanh: 2 / (1 + exp(-2 x)) - 1 (v1/ops/activations/functions.hpp L:44).
__device__ __forceinline__ float tanh_ref(float x) { return 2.f / (1.f + expf(-2.f * x)) - 1.f; }

}  // namespace dlb
