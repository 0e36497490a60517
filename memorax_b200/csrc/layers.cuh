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

// Sum over the rows of gy * x (x null: of gy), (rows, F) each, left as `*blocks` partial rows of F in `partial` (lru_skip_blocks rows).
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
// out: the two-norms of the rows of a, then of those of b, each row F long.
int row_norms(const float* a, long long rows_a, const float* b, long long rows_b, int F, float* out, cudaStream_t stream);
// The elements of h_tilde whose sign is not sure are replaced by the product in (B, T, F) w (D, F)^T in plain float32 order.
struct NearKink {
  float* h = nullptr;             // = h_tilde, writable; null: they stay as they are
  const float *in = nullptr, *w = nullptr, *norms = nullptr;   // norms: row_norms of in and w
  int F = 0;
};
// z and h_tilde are (B, T, D) with rows of both (and of their cotangents) `ld` floats apart; the rest is dense.
// states (or null): the log states; with `forms` (mingru_forms bytes) each block leaves a turn's as it had them, linear or log,
// for the backward pass, and says which.  y: the read-out; x_last, a_last: the next carry.  Each may be null.
size_t mingru_forms(int B, int T, int D);
int mingru_fwd(const float* z, const float* h_tilde, const NearKink& kink, long long ld, const float* x0, const float* a0,
               const uint8_t* done, float* states, uint8_t* forms, float* y, float* x_last, float* a_last, int B, int T, int D,
               cudaStream_t stream);
int mingru_bwd(const float* z, const float* h_tilde, long long ld, const float* states, const uint8_t* forms, const float* x0, const uint8_t* done,
               const float* gx, const float* gy, const float* gx_last, float* gz, float* gh, float* gx0, int B, int T, int D,
               cudaStream_t stream);
// One time step of the layer: the two Dense layers w_z, w_h (D, F), the gates and the recurrence.
int mingru_step(const float* in, const float* w_z, const float* w_h, const float* x0, const float* a0, const uint8_t* done,
                float* x, float* y, float* a_last, int B, int F, int D, cudaStream_t stream);

// ---- sums over the rows of several float matrices (rows, cols) in one launch, in a fixed order ---------------------
struct ColumnSum {
  const float* src;
  int rows, cols;
  float* dst;
  void* dst16 = nullptr;   // given: the sums leave in bf16, here
};
int column_sums(const ColumnSum* jobs, int count, cudaStream_t stream);   // at most four

// ---- Mamba with heads of 16 x 16 states and four convolution taps, mamba.cu -----------------------------------------
// `proj` (B, T, ld): what the Dense layers make of the inputs, columns hidden (16 H) | gate (16 H) | B (16 H) | C (16 H) |
// dt (H); channels of the convolution: hidden | B | C.
struct MambaParams {
  const float *a_log, *d, *dt_bias;   // (H)
  const float *conv_w, *conv_b;       // (48 H, 4), (48 H)
  const float* norm_w;                // (16 H)
  float eps;
};
// Convolution, gates, scan and C h + D x: y_pre (B, T, 16 H); h0 / a0 / done / states may be null.  states: the state each
// stretch of 64 steps starts from, for the backward pass (mamba_state_floats).
size_t mamba_state_floats(int B, int T, int H);
int mamba_scan_fwd(const MambaParams& w, const float* proj, long long ld, const float* h0, const float* a0, const uint8_t* done,
                   float* y_pre, float* h_last, float* a_last, float* states, int B, int T, int H, cudaStream_t stream);
// z = RMSNorm(y_pre) silu(gate)
int mamba_gate_fwd(const MambaParams& w, const float* proj, long long ld, const float* y_pre, float* z, long long tokens, int H,
                   cudaStream_t stream);
// gz -> gy_pre and the gate columns of gproj, for at most kMambaGradHeads heads (each warp keeps a row of sums in shared memory); norm_partial: mamba_gate_blocks rows of 16 H
constexpr int kMambaGradHeads = 454;
int mamba_gate_blocks(long long tokens);
int mamba_gate_bwd(const MambaParams& w, const float* proj, long long ld, const float* y_pre, const float* gz, float* gy_pre,
                   float* gproj, float* norm_partial, long long tokens, int H, cudaStream_t stream);
// gy_pre -> the other columns of gproj; partial (B, mamba_partial_floats(H)): conv_w | conv_b | a_log | dt_bias | d
int mamba_partial_floats(int H);
int mamba_scan_bwd(const MambaParams& w, const float* proj, long long ld, const uint8_t* done, const float* states,
                   const float* gy_pre, const float* gh_last, float* gproj, float* gh0,
                   float* partial, int B, int T, int H, cudaStream_t stream);

// ---- attention-style layers in bf16, attn_layers.cu --------------------------------------------------------------------
constexpr int kMaxWeights = 5;
struct WeightRows {                 // bf16 matrices (rows[i], K) on top of each other
  const void* ptr[kMaxWeights];
  int rows[kMaxWeights];
  int count;
};
// dst (padded, K): the stacked rows, then zeros
int stack_rows(const WeightRows& w, void* dst, int padded, int K, cudaStream_t stream);
// c (M, ldc) = x (M, K) w^T (+ bias (N) or null) for few rows; K a multiple of 32, columns past the stacked rows untouched
// `bias` belongs to the columns from bias_from on.
int small_product(const void* x, const WeightRows& w, const void* bias, int bias_from, void* c, long long ldc, int M, int K, cudaStream_t stream);
// One step of linear attention with its RMSNorm: qkv (B, ld) holds q | k | v of H heads of d (32 or 64); y (B, H d) bf16.
int linattn_step(const void* qkv, long long ld, const float* s0, const float* z0, const uint8_t* done, const void* norm_w,
                 float norm_eps, float eps, void* y, float* s_last, float* z_last, int B, int H, int d, cudaStream_t stream);
// One step of the gated delta rule with the normalisation of q and k, the gates and the RMSNorm: qkvg (B, ld) holds
// q | k | v | beta logits (H) | decay logits (H); d 64 or 128.
int gdelta_step(const void* qkvg, long long ld, const float* s0, const uint8_t* done, const void* norm_w,
                float norm_eps, void* y, float* s_last, int B, int H, int d, cudaStream_t stream);
// The same normalisation and gates over whole segments: q, k (tokens, H d) bf16, alpha, beta (tokens, H).
int delta_inputs(const void* qkvg, long long ld, void* q, void* k, float* alpha, float* beta,
                 long long tokens, int H, int d, cudaStream_t stream);
// dq, dk, dalpha, dbeta -> the q, k and gate columns of g (tokens, ld) (and zeros from `used` to ld);
// partial: delta_gate_blocks rows of 2 H (the gates' bias gradient).
int delta_gate_blocks(long long tokens);
int delta_inputs_bwd(const void* qkvg, long long ld, const void* dq, const void* dk, const float* dalpha,
                     const float* dbeta, void* g, float* partial, long long tokens, int H, int d, cudaStream_t stream);

// ---- mLSTM in bf16, mlstm_layer.cu: what is elementwise around its products and its chunk kernels ------------------
// u (tokens, hid) = silu(conv(x)), x the first `hid` columns of up (tokens, ld); weights (hid, 4), bias (hid)
int mlstm_conv_fwd(const void* up, long long ld, const void* conv_w, const void* conv_b, void* u, int B, int T, int hid,
                   cudaStream_t stream);
// The weights as the layer's products take them, one launch: qk_w (H, 2d, d) = q over k of each head, gate_w (2H, 3 H d) and
// gate_b (2H) = input gate over forget gate.
int mlstm_weights(const void* q, const void* k, const void* i_w, const void* f_w, const void* i_b, const void* f_b, void* qk_w, void* gate_w,
                  void* gate_b, int H, int d, cudaStream_t stream);
// logits (tokens, 2H) -> log_i, log_f = log sigmoid (tokens, H); k_scaled = k scale, k a slice with pitch ld
// between steps and hp between heads
int mlstm_gates_fwd(const void* logits, const void* k, long long ld, int hp, float scale,
                    float* log_i, float* log_f, void* k_scaled, long long tokens, int H, int d, cudaStream_t stream);
// g = (LayerNorm_head(h) (1 + norm_w) + skip u) silu(z), z a slice with pitch ld
int mlstm_out_fwd(const void* h, const void* u, const void* z, long long ld, const void* norm_w, const void* skip, void* g,
                  long long tokens, int H, int d, cudaStream_t stream);
// gg -> gh, gz (slice with pitch ld_gz), gu (the skip's share); partial: mlstm_out_blocks rows of norm_w | skip (2 hid)
int mlstm_out_blocks(long long tokens, int hid);
int mlstm_out_bwd(const void* gg, const void* h, const void* u, const void* z, long long ld, const void* norm_w, const void* skip,
                  void* gh, void* gz, long long ld_gz, void* gu, float* partial, long long tokens, int H, int d, cudaStream_t stream);
// gk (slice with pitches ld, hp) = gk_scaled scale; glogits (tokens, 2H); partial: mlstm_gate_blocks rows of 2 H (bias gradients)
int mlstm_gate_blocks(long long tokens);
int mlstm_gates_bwd(const void* logits, const float* glog_i, const float* glog_f, const void* gk_scaled,
                    float scale, void* gk, long long ld, int hp, void* glogits, float* partial, long long tokens, int H, int d,
                    cudaStream_t stream);
// gu -> the first `hid` columns of gup (through SiLU and the convolution, + gx); partial: mlstm_conv_blocks rows of
// conv_w (hid, 4) | conv_b (hid)
int mlstm_conv_blocks(int B, int T, int hid);
int mlstm_conv_bwd(const void* up, long long ld, const void* conv_w, const void* conv_b, const void* gu, const void* gx, void* gup,
                   float* partial, int B, int T, int hid, cudaStream_t stream);

}  // namespace layers
}  // namespace mxk
