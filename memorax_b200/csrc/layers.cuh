// Kernels of whole layers around the scans (host-side interface): what a cell does besides its recurrence and the
// large matrix products.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mxk.h"

namespace mxk {
namespace layers {

// ---- complex-diagonal layer (LRU), lru.cu -------------------------------------------------------------------
struct LruWeights {
  const float *nu_log, *theta_log, *gamma_log;   // (N)
  const float *b_re, *b_im;                      // (N, F)
  const float *c_re, *c_im;                      // (F, N)
  const float* d;                                // (F)
};
// One time step of `B` sequences: h (B, N) complex, y (B, F); h0 / a0 / done / a_last may be null.
int lru_step(const LruWeights& w, const float* x, const float* h0, const float* a0, const uint8_t* done, float* h,
             float* a_last, float* y, int B, int F, int N, cudaStream_t stream);

// Sum over the rows of gy * x, (rows, F) each, left as `*blocks` partial rows of F in `partial` (lru_skip_blocks rows).
int skip_grad_blocks(long long rows);
int skip_grad(const float* gy, const float* x, float* partial, long long rows, int F, cudaStream_t stream);

// Gradients of the parameters from those of the real projection matrices (partial products of split contractions) and
// of lambda (torch's complex convention).
struct LruGrads {
  const float* in_partial;    // [in_splits][2N][F]
  const float* out_partial;   // [out_splits][F][2N]
  const float* skip_partial;  // [skip_blocks][F]
  const float* lambda;        // (N) complex, and its cotangent
  const float* g_lambda;
  int in_splits, out_splits, skip_blocks;
  float *g_nu, *g_theta, *g_gamma, *g_b_re, *g_b_im, *g_c_re, *g_c_im, *g_d;
};
int lru_param_grads(const LruWeights& w, const LruGrads& g, int F, int N, cudaStream_t stream);

// RTRL: sensitivities after a segment of T steps from those before it.  h (B, T, N) holds the states, h0 (B, N) the one
// the segment started from, u (B, T, F) the inputs; each sensitivity (B, N) or (B, N, F) complex, in and out.
struct LruSensitivities {
  const float *nu, *theta, *gamma, *b_re, *b_im;
  float *nu_out, *theta_out, *gamma_out, *b_re_out, *b_im_out;
};
int lru_sensitivities(const LruWeights& w, const float* lambda, const float* h, const float* h0, const float* u,
                      const uint8_t* done, const LruSensitivities& s, int B, int T, int F, int N, cudaStream_t stream);

// ---- MinGRU, mingru.cu -----------------------------------------------------------------------------------------
// z and h_tilde are (B, T, D) with rows of both (and of their cotangents) `ld` floats apart; the rest is dense.
// With `h_kink` (= h_tilde, writable) elements too close to zero for their sign to be sure are replaced by the product
// dense_in (B, T, F) dense_w (D, F)^T in plain float32 order.
int mingru_fwd(const float* z, const float* h_tilde, float* h_kink, const float* dense_in, const float* dense_w, int F,
               long long ld, const float* x0, const float* a0, const uint8_t* done,
               float* x, float* y, float* a_last, int B, int T, int D, cudaStream_t stream);
// y: the read-out exp(x), or null
int mingru_bwd(const float* z, const float* h_tilde, long long ld, const float* x, const float* y, const float* x0, const uint8_t* done,
               const float* gx, const float* gy, const float* gx_last, float* gz, float* gh, float* gx0, int B, int T, int D,
               cudaStream_t stream);
// One time step of the layer: the two Dense layers w_z, w_h (D, F), the gates and the recurrence.
int mingru_step(const float* in, const float* w_z, const float* w_h, const float* x0, const float* a0, const uint8_t* done,
                float* x, float* y, float* a_last, int B, int F, int D, cudaStream_t stream);

}  // namespace layers
}  // namespace mxk
