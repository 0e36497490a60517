// The LRU layer: projections, scan and read-out as one call, and its backward pass as one autograd node.
#include "common.h"

#include "../gemm32.cuh"
#include "../layers.cuh"

namespace mxk_host {
namespace {

using mxk::gemm32::Form;
using mxk::gemm32::LambdaJob;
using mxk::gemm32::Weight;
using mxk::gemm32::WeightJob;
using mxk::layers::LruWeights;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int kParams = 8;   // nu_log, theta_log, gamma_log, B_real, B_imag, C_real, C_imag, D

LruWeights weights_of(const variable_list& p) {
  return {ptr(p[0]), ptr(p[1]), ptr(p[2]), ptr(p[3]), ptr(p[4]), ptr(p[5]), ptr(p[6]), ptr(p[7])};
}
Weight input_rows(const LruWeights& w, int F) {   // [2N][F]
  Weight r;
  r.form = Form::kComplexRows;
  r.ptr[0] = w.b_re; r.ptr[1] = w.b_im;
  r.count = 2;
  r.ld = F;
  r.log_scale = w.gamma_log;
  return r;
}
Weight output_cols(const LruWeights& w, int N) {   // [F][2N]
  Weight r;
  r.form = Form::kComplexCols;
  r.ptr[0] = w.c_re; r.ptr[1] = w.c_im;
  r.count = 2;
  r.ld = N;
  return r;
}

struct Result {
  Tensor h, a_last, y, lambda;   // h: every state (B, T, N)
};

Result forward(const Tensor& x, const variable_list& params, const Tensor& h0, const Tensor& a0, const Tensor& done, bool keep_lambda = false) {
  const int B = x.size(0), T = x.size(1), F = x.size(2), N = params[0].size(0);
  const auto s = stream();
  const LruWeights w = weights_of(params);
  Result r;
  r.h = empty_like_of(x, {B, T, N}, at::kComplexFloat);
  r.a_last = empty_like_of(x, {B, 1, N}, at::kComplexFloat);
  r.y = empty_like_of(x, x.sizes(), at::kFloat);
  if (T == 1 && !keep_lambda) {   // acting: two launches, no intermediate but the state
    check("lru_step", mxk::layers::lru_step(w, ptr(x), ptr(h0), ptr(a0), bytes(done), ptr(r.h), ptr(r.a_last), ptr(r.y), B, F, N, s));
    return r;
  }
  const int M = B * T;
  namespace g = mxk::gemm32;
  Arena mem;
  const size_t img_in = mem.take(g::image_bytes(M, 2 * N, F)), img_out = mem.take(g::image_bytes(M, F, 2 * N));
  const size_t ws_bytes = std::max(g::workspace_bytes(M, 2 * N, F), g::workspace_bytes(M, F, 2 * N)), ws = mem.take(ws_bytes);
  mem.alloc(x);
  int* const status = status_ptr(x);
  WeightJob jobs[2];
  jobs[0] = {input_rows(w, F), false, 2 * N, F, g::tile_width(M, 2 * N, F), mem.at<void>(img_in)};
  jobs[1] = {output_cols(w, N), false, F, 2 * N, g::tile_width(M, F, 2 * N), mem.at<void>(img_out)};
  r.lambda = empty_like_of(x, {N}, at::kComplexFloat);
  check("split_weights", g::split_weights(jobs, 2, LambdaJob{w.nu_log, w.theta_log, ptr(r.lambda), N}, s));
  // the projected inputs become the states in place: every element is read before the scan writes it
  check("run_weights", g::run_weights(ptr(x), F, mem.at<void>(img_in), ptr(r.h), 2 * N, M, 2 * N, F, {}, mem.at(ws), ws_bytes, status, s));
  check("mxk_linrec_c64_fwd", mxk_linrec_c64_fwd(ptr(r.lambda), 1, ptr(r.h), ptr(h0), ptr(a0), bytes(done), ptr(r.h), ptr(r.a_last), B, T, N, s));
  g::Epilogue skip;
  skip.add = ptr(x);
  skip.ld_add = F;
  skip.add_scale = w.d;
  check("run_weights", g::run_weights(ptr(r.h), 2 * N, mem.at<void>(img_out), ptr(r.y), F, M, F, 2 * N, skip, mem.at(ws), ws_bytes, status, s));
  return r;
}

struct LruLayer : torch::autograd::Function<LruLayer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& nu, const Tensor& theta, const Tensor& gamma,
                               const Tensor& b_re, const Tensor& b_im, const Tensor& c_re, const Tensor& c_im, const Tensor& d,
                               const OptTensor& h0_in, const OptTensor& a0_in, const OptTensor& done_in) {
    const Tensor h0 = h0_in.value_or(Tensor()), a0 = a0_in.value_or(Tensor()), done = done_in.value_or(Tensor());
    const variable_list params{nu, theta, gamma, b_re, b_im, c_re, c_im, d};
    Result r = mxk_host::forward(x, params, h0, a0, done);
    ctx->set_materialize_grads(false);
    variable_list saved{x, nu, theta, gamma, b_re, b_im, c_re, c_im, d, h0, done, r.h, r.lambda};
    ctx->save_for_backward(std::move(saved));
    Tensor last = last_state(r.h).clone();   // (an output may not share memory with what the backward pass reads)
    ctx->mark_non_differentiable({r.a_last});
    return {last, r.a_last, r.y};
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& gout) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &h0 = saved[9], &done = saved[10], &h = saved[11];
    Tensor lambda = saved[12];
    const c10::cuda::CUDAGuard guard(x.device());
    const variable_list params(saved.begin() + 1, saved.begin() + 1 + kParams);
    const int B = x.size(0), T = x.size(1), F = x.size(2), N = params[0].size(0), M = B * T;
    const auto s = stream();
    namespace g = mxk::gemm32;
    const LruWeights w = weights_of(params);
    bool need_params = false;
    for (int i = 1; i <= kParams; ++i) need_params |= ctx->needs_input_grad(i);
    const bool need_x = ctx->needs_input_grad(0), need_h0 = h0.defined() && ctx->needs_input_grad(9);
    const Tensor gh_last = gout[0].defined() ? dense(gout[0]) : Tensor();
    const Tensor gy = gout[2].defined() ? dense(gout[2]) : at::zeros_like(x);

    Tensor gx = empty_like_of(x, x.sizes(), at::kFloat);
    Tensor gh0 = need_h0 ? empty_like_of(x, {B, 1, N}, at::kComplexFloat) : Tensor();
    Tensor gz = empty_like_of(x, {B, T, N}, at::kComplexFloat);   // cotangent of the states, then of the projected inputs
    Arena mem;
    const size_t img_out = mem.take(g::image_bytes(M, 2 * N, F)), img_in = mem.take(g::image_bytes(M, F, 2 * N));
    const size_t ws_bytes = std::max(g::workspace_bytes(M, 2 * N, F), g::workspace_bytes(M, F, 2 * N)), ws = mem.take(ws_bytes);
    const size_t lam = mem.take(8 * N), glam = mem.take(8 * N);
    const size_t scan_bytes = mxk_linrec_bwd_workspace_bytes(1, 1, B, T, N), scan = mem.take(scan_bytes);
    const size_t in_bytes = std::max(g::workspace_bytes(2 * N, F, M), sizeof(float) * 2 * N * F), in = mem.take(in_bytes);
    const size_t out_bytes = std::max(g::workspace_bytes(F, 2 * N, M), sizeof(float) * 2 * N * F), out = mem.take(out_bytes);
    const int skip_blocks = mxk::layers::skip_grad_blocks(M);
    const size_t skip = mem.take(sizeof(float) * skip_blocks * F);
    mem.alloc(x);
    int* const status = status_ptr(x);
    float* const lambda_p = lambda.defined() ? ptr(lambda) : mem.at(lam);

    WeightJob jobs[2];
    jobs[0] = {output_cols(w, N), true, 2 * N, F, g::tile_width(M, 2 * N, F), mem.at<void>(img_out)};
    jobs[1] = {input_rows(w, F), true, F, 2 * N, g::tile_width(M, F, 2 * N), mem.at<void>(img_in)};
    check("split_weights", g::split_weights(jobs, 2, lambda.defined() ? LambdaJob{} : LambdaJob{w.nu_log, w.theta_log, lambda_p, N}, s));
    check("run_weights", g::run_weights(ptr(gy), F, mem.at<void>(img_out), ptr(gz), 2 * N, M, 2 * N, F, {}, mem.at(ws), ws_bytes, status, s));
    check("mxk_linrec_c64_bwd", mxk_linrec_c64_bwd(lambda_p, 1, ptr(h), ptr(h0), bytes(done), ptr(gz), ptr(gh_last), ptr(gz), need_params ? mem.at(glam) : nullptr,
                                                   ptr(gh0), mem.at<void>(scan), scan_bytes, B, T, N, 1, s));
    if (need_x) {
      g::Epilogue ep;
      ep.add = ptr(gy);
      ep.ld_add = F;
      ep.add_scale = w.d;
      check("run_weights", g::run_weights(ptr(gz), 2 * N, mem.at<void>(img_in), ptr(gx), F, M, F, 2 * N, ep, mem.at(ws), ws_bytes, status, s));
    }
    variable_list grads(12);
    if (need_params) {
      mxk::layers::LruGrads gr{};
      check("run_outer", g::run_outer(ptr(gz), 2 * N, ptr(x), F, mem.at(in), F, 2 * N, F, M, mem.at(in), in_bytes, &gr.in_splits, status, s));
      check("run_outer", g::run_outer(ptr(gy), F, ptr(h), 2 * N, mem.at(out), 2 * N, F, 2 * N, M, mem.at(out), out_bytes, &gr.out_splits, status, s));
      check("skip_grad", mxk::layers::skip_grad(ptr(gy), ptr(x), mem.at(skip), M, F, s));
      for (int i = 0; i < kParams; ++i) grads[1 + i] = empty_like_of(x, params[i].sizes(), at::kFloat);
      gr.in_partial = mem.at(in);
      gr.out_partial = mem.at(out);
      gr.skip_partial = mem.at(skip);
      gr.skip_blocks = skip_blocks;
      gr.lambda = lambda_p;
      gr.g_lambda = mem.at(glam);
      float** const dst[kParams] = {&gr.g_nu, &gr.g_theta, &gr.g_gamma, &gr.g_b_re, &gr.g_b_im, &gr.g_c_re, &gr.g_c_im, &gr.g_d};
      for (int i = 0; i < kParams; ++i) *dst[i] = ptr(grads[1 + i]);
      check("lru_param_grads", mxk::layers::lru_param_grads(w, gr, F, N, s));
    }
    if (need_x) grads[0] = gx;
    grads[9] = gh0;
    return grads;
  }
};

// Whether a call is one for the native layer; what is not (another dtype, tensors elsewhere, a lower precision asked for)
// the caller composes from its parts.
bool native(const Tensor& x, const variable_list& params) {
  if (!x.is_cuda() || x.dim() != 3 || x.numel() == 0 || !x.is_floating_point() || x.scalar_type() == at::kDouble ||
      (x.size(1) > 1 && tf32_products()) || at::autocast::is_autocast_enabled(at::kCUDA) ||
      x.size(0) * x.size(1) > 0x7fffffff || params.size() != kParams || params[3].dim() != 2)
    return false;
  const int64_t N = params[3].size(0), F = x.size(2);
  for (int i : {0, 1, 2})
    if (!shaped(params[i], {N})) return false;
  for (int i : {3, 4})
    if (!shaped(params[i], {N, F}) || !shaped(params[i + 2], {F, N})) return false;
  if (!shaped(params[7], {F})) return false;
  for (const Tensor& p : params)
    if (p.scalar_type() != at::kFloat || p.device() != x.device() || !p.is_contiguous()) return false;
  return true;
}
bool wants_grad(const Tensor& x, const variable_list& params, const Tensor& h0) {
  if (!at::GradMode::is_enabled()) return false;
  bool grad = x.requires_grad() || (h0.defined() && h0.requires_grad());
  for (const Tensor& p : params) grad |= p.requires_grad();
  return grad;
}

// -> (last state (B,1,N), decay leaf (B,1,N), y (B,T,F)), or None
pybind11::object lru_layer(const Tensor& x_in, const variable_list& params, const OptTensor& h0_in, const OptTensor& a0_in,
                           const OptTensor& done_in) {
  if (!native(x_in, params) || followed(x_in, params, h0_in, a0_in)) return pybind11::none();
  const c10::cuda::CUDAGuard guard(x_in.device());
  const Tensor x = dense(x_in.scalar_type() == at::kFloat ? x_in : x_in.to(at::kFloat));
  const Tensor h0 = carry_leaf(h0_in, x.size(0) * params[0].size(0), at::kComplexFloat, "h0"), a0 = carry_leaf(a0_in, x.size(0) * params[0].size(0), at::kComplexFloat, "a0"), done = done_bytes(done_in, x.size(0) * x.size(1));
  if (wants_grad(x, params, h0)) {
    const variable_list out = LruLayer::apply(x, params[0], params[1], params[2], params[3], params[4], params[5], params[6],
                                              params[7], opt(h0), opt(a0), opt(done));
    return pybind11::cast(std::make_tuple(out[0], out[1], out[2]));
  }
  const Result r = forward(x, params, h0, a0, done);
  return pybind11::cast(std::make_tuple(last_state(r.h), r.a_last, r.y));
}

// One RTRL segment without gradients: -> (last state, decay leaf, y, sensitivities of B_imag, B_real, gamma_log, nu_log,
// theta_log), or None
pybind11::object lru_rtrl(const Tensor& x_in, const variable_list& params, const OptTensor& h0_in, const OptTensor& a0_in,
                          const OptTensor& done_in, const variable_list& sens_in) {
  if (!native(x_in, params) || sens_in.size() != 5 || x_in.size(0) > 65535 || followed(x_in, params, h0_in, a0_in) || followed(x_in, sens_in)) return pybind11::none();
  const int B = x_in.size(0), T = x_in.size(1), F = x_in.size(2), N = params[0].size(0);
  const c10::cuda::CUDAGuard guard(x_in.device());
  const Tensor x = dense(x_in.scalar_type() == at::kFloat ? x_in : x_in.to(at::kFloat));
  const Tensor h0 = carry_leaf(h0_in, x.size(0) * params[0].size(0), at::kComplexFloat, "h0"), a0 = carry_leaf(a0_in, x.size(0) * params[0].size(0), at::kComplexFloat, "a0"), done = done_bytes(done_in, x.size(0) * x.size(1));
  bool grad = wants_grad(x, params, h0);
  variable_list sens, out;
  for (int i = 0; i < 5; ++i) {
    const Tensor& t = sens_in[i];
    grad |= at::GradMode::is_enabled() && t.requires_grad();
    if (!t.is_cuda() || (i < 2 ? t.sizes() != at::IntArrayRef({B, 1, N, F}) : t.sizes() != at::IntArrayRef({B, 1, N}))) return pybind11::none();
    sens.push_back(dev(t, at::kComplexFloat, "sensitivity"));
    out.push_back(at::empty_like(sens.back()));
  }
  if (grad) return pybind11::none();
  const Result r = forward(x, params, h0, a0, done, true);
  mxk::layers::LruSensitivities s{ptr(sens[3]), ptr(sens[4]), ptr(sens[2]), ptr(sens[1]), ptr(sens[0]),
                                  ptr(out[3]), ptr(out[4]), ptr(out[2]), ptr(out[1]), ptr(out[0])};
  check("lru_sensitivities", mxk::layers::lru_sensitivities(weights_of(params), ptr(r.lambda), ptr(r.h), ptr(h0), ptr(x), bytes(done), s, B, T, F, N, stream()));
  return pybind11::cast(std::make_tuple(last_state(r.h), r.a_last, r.y, out));
}

}  // namespace

void bind_lru(pybind11::module_& m) {
  m.def("lru_layer", &lru_layer);
  m.def("lru_rtrl", &lru_rtrl);
}

}  // namespace mxk_host
