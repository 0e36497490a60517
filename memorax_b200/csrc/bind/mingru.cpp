// The MinGRU layer: both Dense layers as one product, scan with gate math and read-out, and its backward pass as one node.
#include "common.h"

#include "../gemm32.cuh"
#include "../layers.cuh"

namespace mxk_host {
namespace {

namespace g = mxk::gemm32;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// the two weights on top of each other, (2D, F)
g::Weight stacked(const Tensor& w_z, const Tensor& w_h) {
  const int D = w_z.size(0);
  g::Weight w;
  w.ptr[0] = ptr(w_z); w.ptr[1] = ptr(w_h);
  w.row_end[0] = D; w.row_end[1] = 2 * D;
  w.count = 2;
  w.ld = w_z.size(1);
  return w;
}

struct Result {
  Tensor y, x_last, a_last;
  Tensor zh, states, forms;   // for the backward pass; zh: both pre-activations, (B, T, 2D)
};

Result forward(const Tensor& in, const Tensor& w_z, const Tensor& w_h, const Tensor& x0, const Tensor& a0, const Tensor& done,
               bool keep) {
  const int B = in.size(0), T = in.size(1), F = in.size(2), D = w_z.size(0), M = B * T;
  Result r;
  r.y = empty_like_of(in, {B, T, D}, at::kFloat);
  r.x_last = empty_like_of(in, {B, 1, D}, at::kFloat);
  r.a_last = empty_like_of(in, {B, 1, D}, at::kFloat);
  if (T == 1 && !keep) {
    check("mingru_step", mxk::layers::mingru_step(ptr(in), ptr(w_z), ptr(w_h), ptr(x0), ptr(a0), bytes(done), ptr(r.x_last), ptr(r.y), ptr(r.a_last), B, F, D, stream()));
    return r;
  }
  r.zh = empty_like_of(in, {B, T, 2 * D}, at::kFloat);
  Arena mem;
  const size_t image = mem.take(g::image_bytes(M, 2 * D, F)), ws_bytes = g::workspace_bytes(M, 2 * D, F), ws = mem.take(ws_bytes);
  const size_t norms = keep ? mem.take(sizeof(float) * (static_cast<size_t>(M) + D)) : 0;
  mem.alloc(in);
  mxk::layers::NearKink kink;
  if (keep) {   // (only gradients tell the two sides of the kink apart)
    r.states = empty_like_of(in, {B, T, D}, at::kFloat);
    r.forms = scratch(in, mxk::layers::mingru_forms(B, T, D));
    kink = {ptr(r.zh) + D, ptr(in), ptr(w_h), mem.at(norms), F};
    check("row_norms", mxk::layers::row_norms(ptr(in), M, ptr(w_h), D, F, mem.at(norms), stream()));
  }
  const g::WeightJob job{stacked(w_z, w_h), false, 2 * D, F, g::tile_width(M, 2 * D, F), mem.at<void>(image)};
  check("split_weights", g::split_weights(&job, 1, {}, stream()));
  check("run_weights", g::run_weights(ptr(in), F, job.image, ptr(r.zh), 2 * D, M, 2 * D, F, {}, mem.at(ws), ws_bytes, status_ptr(in), stream()));
  check("mingru_fwd", mxk::layers::mingru_fwd(ptr(r.zh), ptr(r.zh) + D, kink, 2 * D, ptr(x0), ptr(a0), bytes(done), ptr(r.states), ptr<uint8_t>(r.forms), ptr(r.y),
                                              ptr(r.x_last), ptr(r.a_last), B, T, D, stream()));
  return r;
}

struct MinGruLayer : torch::autograd::Function<MinGruLayer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& in, const Tensor& w_z, const Tensor& w_h, const OptTensor& x0_in,
                               const OptTensor& a0_in, const OptTensor& done_in) {
    const Tensor x0 = x0_in.value_or(Tensor()), a0 = a0_in.value_or(Tensor()), done = done_in.value_or(Tensor());
    Result r = mxk_host::forward(in, w_z, w_h, x0, a0, done, true);
    ctx->set_materialize_grads(false);
    // (not the read-out, which the caller may change in place)
    ctx->save_for_backward({in, w_z, w_h, x0, done, r.zh, r.states, r.forms});
    ctx->mark_non_differentiable({r.a_last});
    return {r.x_last, r.a_last, r.y};
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& gout) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &in = saved[0], &w_z = saved[1], &w_h = saved[2], &x0 = saved[3], &done = saved[4], &zh = saved[5], &states = saved[6];
    const c10::cuda::CUDAGuard guard(in.device());
    const int B = in.size(0), T = in.size(1), F = in.size(2), D = w_z.size(0), M = B * T;
    const bool need_in = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1) || ctx->needs_input_grad(2);
    const bool need_x0 = x0.defined() && ctx->needs_input_grad(3);
    const Tensor gx_last = gout[0].defined() ? dense(gout[0]) : Tensor();
    const Tensor gy = gout[2].defined() ? dense(gout[2]) : empty_like_of(in, {B, T, D}, at::kFloat).zero_();
    variable_list grads(6);
    if (need_x0) grads[3] = empty_like_of(in, {B, 1, D}, at::kFloat);
    if (need_in) grads[0] = empty_like_of(in, in.sizes(), at::kFloat);
    const Tensor gw = need_w ? empty_like_of(in, {2 * D, F}, at::kFloat) : Tensor();
    Arena mem;
    const size_t gzh = mem.take(sizeof(float) * 2 * D * M), image = mem.take(g::image_bytes(M, F, 2 * D));
    const size_t ws_bytes = std::max(g::workspace_bytes(M, F, 2 * D), g::workspace_bytes(2 * D, F, M)), ws = mem.take(ws_bytes);
    mem.alloc(in);
    check("mingru_bwd", mxk::layers::mingru_bwd(ptr(zh), ptr(zh) + D, 2 * D, ptr(states), bytes(saved[7]), ptr(x0), bytes(done), nullptr, ptr(gy), ptr(gx_last), mem.at(gzh),
                                                mem.at(gzh) + D, need_x0 ? ptr(grads[3]) : nullptr, B, T, D, stream()));
    if (need_in) {
      const g::WeightJob job{stacked(w_z, w_h), true, F, 2 * D, g::tile_width(M, F, 2 * D), mem.at<void>(image)};
      check("split_weights", g::split_weights(&job, 1, {}, stream()));
      check("run_weights", g::run_weights(mem.at(gzh), 2 * D, job.image, ptr(grads[0]), F, M, F, 2 * D, {}, mem.at(ws), ws_bytes, status_ptr(in), stream()));
    }
    if (need_w) {
      check("run_outer", g::run_outer(mem.at(gzh), 2 * D, ptr(in), F, ptr(gw), F, 2 * D, F, M, mem.at(ws), ws_bytes, nullptr, status_ptr(in), stream()));
      grads[1] = piece(gw, 0, {D, F});
      grads[2] = piece(gw, static_cast<int64_t>(D) * F, {D, F});
    }
    return grads;
  }
};

// -> (last log state (B,1,D), decay leaf (B,1,D), y (B,T,D)), or None where the caller has to compose the layer
pybind11::object mingru_layer(const Tensor& in_, const Tensor& w_z, const Tensor& w_h, const OptTensor& x0_in, const OptTensor& a0_in,
                              const OptTensor& done_in) {
  const auto fits = [&](const Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kFloat && t.device() == in_.device(); };
  if (!fits(in_) || !fits(w_z) || !fits(w_h) || in_.dim() != 3 || in_.numel() == 0 || w_z.dim() != 2 || w_z.sizes() != w_h.sizes() ||
      !w_z.is_contiguous() || !w_h.is_contiguous() || in_.size(2) != w_z.size(1) || in_.size(0) * in_.size(1) > 0x7fffffff ||
      (in_.size(1) > 1 && tf32_products()) || at::autocast::is_autocast_enabled(at::kCUDA) ||
      followed(in_, {w_z, w_h}, x0_in, a0_in))
    return pybind11::none();
  const c10::cuda::CUDAGuard guard(in_.device());
  const Tensor in = dense(in_), x0 = carry_leaf(x0_in, in.size(0) * w_z.size(0), at::kFloat, "x0"), a0 = carry_leaf(a0_in, in.size(0) * w_z.size(0), at::kFloat, "a0"), done = done_bytes(done_in, in.size(0) * in.size(1));
  if (at::GradMode::is_enabled() && (in.requires_grad() || w_z.requires_grad() || w_h.requires_grad() || (x0.defined() && x0.requires_grad()))) {
    const variable_list out = MinGruLayer::apply(in, w_z, w_h, opt(x0), opt(a0), opt(done));
    return pybind11::cast(std::make_tuple(out[0], out[1], out[2]));
  }
  const Result r = forward(in, w_z, w_h, x0, a0, done, false);
  return pybind11::cast(std::make_tuple(r.x_last, r.a_last, r.y));
}

}  // namespace

void bind_mingru(pybind11::module_& m) { m.def("mingru_layer", &mingru_layer); }

}  // namespace mxk_host
