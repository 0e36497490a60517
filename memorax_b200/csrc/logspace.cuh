// Arithmetic of the log-space recurrences (MinGRU).
#pragma once

#include <cuda_runtime.h>

namespace mxk {

// MXK_LOGSPACE_FAST (default): exp / log through the special-function unit's approximations (ex2, lg2: relative
// error about 2^-22) instead of the full-precision library sequences, which are most of these kernels'
// instructions.  Measured against the fp64 oracle on the fused MinGRU path (8 x 256 x 256, inputs of a few units):
// x 8e-8, y 3e-7, cotangents 4e-7 / 6e-7 of each tensor's max-abs, against 8e-8, 2e-7, 2e-7 / 3e-7 with the library
// functions (-DMXK_LOGSPACE_FAST=0) -- both far inside the 1e-5 / 1e-4 the tests allow -- and 0.72 against 0.91 ms
// for the 256 x 256 x 1024 forward + backward.
#ifndef MXK_LOGSPACE_FAST
#define MXK_LOGSPACE_FAST 1
#endif
__device__ __forceinline__ float exp_ls(float x) { return MXK_LOGSPACE_FAST ? __expf(x) : expf(x); }
__device__ __forceinline__ float log_ls(float x) { return MXK_LOGSPACE_FAST ? __logf(x) : logf(x); }
// log(1 + e) for e in [0, 1]
__device__ __forceinline__ float log1p_ls(float e) { return MXK_LOGSPACE_FAST ? __logf(1.f + e) : log1pf(e); }

__device__ __forceinline__ float log_add_exp(float p, float q) {
  const float hi = fmaxf(p, q), lo = fminf(p, q);
  if (hi == -INFINITY) return -INFINITY;
  return hi + log1p_ls(exp_ls(lo - hi));
}

// MinGRU's gate math (min_gru.py:52-61), fused into the scan when the kernels are handed the Dense layers'
// pre-activations instead of the elements:
//   log_state = -softplus(-z) + log g(h~),  decay = -softplus(z),  g(h) = h >= 0 ? h + 0.5 : sigmoid(h).
__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.f) + log1p_ls(exp_ls(-fabsf(x))); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + exp_ls(-x)); }
__device__ __forceinline__ float log_g(float h) { return h >= 0.f ? log_ls(h + 0.5f) : -softplus_f(-h); }
__device__ __forceinline__ float dlog_g(float h) { return h >= 0.f ? 1.f / (h + 0.5f) : sigmoid_f(-h); }

}  // namespace mxk
