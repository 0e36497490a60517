// The Mamba layer: one product for the four Dense layers on the inputs, the fused scan, norm and gate, the output product;
// its backward pass is one autograd node.
#include "common.h"

#include "../gemm32.cuh"
#include "../layers.cuh"

namespace mxk_host {
namespace {

namespace g = mxk::gemm32;
namespace l = mxk::layers;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// parameters in the order the caller passes them
enum { kALog, kD, kDtBias, kIn, kB, kC, kDt, kConvW, kConvB, kNormW, kOutW, kOutB, kParams };

l::MambaParams scan_params(const variable_list& p, double eps) {
  return {ptr(p[kALog]), ptr(p[kD]), ptr(p[kDtBias]), ptr(p[kConvW]), ptr(p[kConvB]), ptr(p[kNormW]), static_cast<float>(eps)};
}
// input projection, B, C and dt on top of each other: (65 H, F)
g::Weight stacked(const variable_list& p, int H) {
  g::Weight w;
  const int src[4] = {kIn, kB, kC, kDt}, rows[4] = {32 * H, 16 * H, 16 * H, H};
  int end = 0;
  for (int i = 0; i < 4; ++i) {
    w.ptr[i] = ptr(p[src[i]]);
    w.row_end[i] = end += rows[i];
  }
  w.count = 4;
  w.ld = p[kIn].size(1);
  return w;
}
// rows padded to a multiple of 8 floats: 32-byte accesses in the products
int proj_ld(int H) { return (65 * H + 7) / 8 * 8; }

struct Result {
  Tensor h_last, a_last, y, proj, y_pre, z, states;
};

Result forward(const Tensor& x, const variable_list& p, const Tensor& h0, const Tensor& a0, const Tensor& done, double eps, bool keep) {
  const int B = x.size(0), T = x.size(1), F = x.size(2), H = p[kALog].size(0), hid = 16 * H, out = p[kOutW].size(0), M = B * T, ld = proj_ld(H);
  const auto s = stream();
  const l::MambaParams w = scan_params(p, eps);
  Result r;
  r.h_last = empty_like_of(x, {B, 1, H, 16, 16}, at::kFloat);
  r.a_last = empty_like_of(x, {B, 1, H, 1, 1}, at::kFloat);
  r.y = empty_like_of(x, {B, T, out}, at::kFloat);
  r.proj = empty_like_of(x, {B, T, ld}, at::kFloat);
  r.y_pre = empty_like_of(x, {B, T, hid}, at::kFloat);
  r.z = empty_like_of(x, {B, T, hid}, at::kFloat);
  if (keep) r.states = empty_like_of(x, {static_cast<int64_t>(l::mamba_state_floats(B, T, H))}, at::kFloat);
  Arena mem;
  const size_t img_in = mem.take(g::image_bytes(M, 65 * H, F)), img_out = mem.take(g::image_bytes(M, out, hid));
  const size_t ws_bytes = std::max(g::workspace_bytes(M, 65 * H, F), g::workspace_bytes(M, out, hid)), ws = mem.take(ws_bytes);
  mem.alloc(x);
  int* const status = status_ptr(x);
  const g::WeightJob jobs[2] = {{stacked(p, H), false, 65 * H, F, g::tile_width(M, 65 * H, F), mem.at<void>(img_in)},
                                {g::weight_of(ptr(p[kOutW]), hid), false, out, hid, g::tile_width(M, out, hid), mem.at<void>(img_out)}};
  check("split_weights", g::split_weights(jobs, 2, {}, s));
  check("run_weights", g::run_weights(ptr(x), F, mem.at<void>(img_in), ptr(r.proj), ld, M, 65 * H, F, {}, mem.at(ws), ws_bytes, status, s));
  check("mamba_scan_fwd", l::mamba_scan_fwd(w, ptr(r.proj), ld, ptr(h0), ptr(a0), bytes(done), ptr(r.y_pre), ptr(r.h_last), ptr(r.a_last), ptr(r.states), B, T, H, s));
  check("mamba_gate_fwd", l::mamba_gate_fwd(w, ptr(r.proj), ld, ptr(r.y_pre), ptr(r.z), M, H, s));
  g::Epilogue ep;
  ep.bias = ptr(p[kOutB]);
  check("run_weights", g::run_weights(ptr(r.z), hid, mem.at<void>(img_out), ptr(r.y), out, M, out, hid, ep, mem.at(ws), ws_bytes, status, s));
  return r;
}

struct MambaLayer : torch::autograd::Function<MambaLayer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& p0, const Tensor& p1, const Tensor& p2, const Tensor& p3,
                               const Tensor& p4, const Tensor& p5, const Tensor& p6, const Tensor& p7, const Tensor& p8, const Tensor& p9,
                               const Tensor& p10, const Tensor& p11, const OptTensor& h0_in, const OptTensor& a0_in, const OptTensor& done_in, double eps) {
    const variable_list p{p0, p1, p2, p3, p4, p5, p6, p7, p8, p9, p10, p11};
    const Tensor h0 = h0_in.value_or(Tensor()), done = done_in.value_or(Tensor());
    Result r = mxk_host::forward(x, p, h0, a0_in.value_or(Tensor()), done, eps, true);
    ctx->set_materialize_grads(false);
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["h0"] = h0.defined();
    variable_list saved{x};
    saved.insert(saved.end(), p.begin(), p.end());
    for (const Tensor& t : {done, r.proj, r.y_pre, r.z, r.states}) saved.push_back(t);
    ctx->save_for_backward(std::move(saved));
    ctx->mark_non_differentiable({r.a_last});
    return {r.h_last, r.a_last, r.y};
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& gout) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor& x = saved[0];
    const variable_list p(saved.begin() + 1, saved.begin() + 1 + kParams);
    const Tensor &done = saved[13], &proj = saved[14], &y_pre = saved[15], &z = saved[16], &states = saved[17];
    const c10::cuda::CUDAGuard guard(x.device());
    const int B = x.size(0), T = x.size(1), F = x.size(2), H = p[kALog].size(0), hid = 16 * H, out = p[kOutW].size(0), M = B * T, ld = proj_ld(H);
    const auto s = stream();
    const l::MambaParams w = scan_params(p, ctx->saved_data["eps"].toDouble());
    const bool need_x = ctx->needs_input_grad(0), need_h0 = ctx->saved_data["h0"].toBool() && ctx->needs_input_grad(13);
    const Tensor gh_last = gout[0].defined() ? dense(gout[0]) : Tensor();
    const Tensor gy = gout[2].defined() ? dense(gout[2]) : empty_like_of(x, {B, T, out}, at::kFloat).zero_();
    variable_list grads(17);
    if (need_x) grads[0] = empty_like_of(x, x.sizes(), at::kFloat);
    if (need_h0) grads[13] = empty_like_of(x, {B, 1, H, 16, 16}, at::kFloat);
    const Tensor gw_in = empty_like_of(x, {65 * H, F}, at::kFloat), gw_out = empty_like_of(x, {out, hid}, at::kFloat);
    const int scan_cols = l::mamba_partial_floats(H), gate_rows = l::mamba_gate_blocks(M), bias_rows = l::skip_grad_blocks(M);
    const Tensor small = empty_like_of(x, {scan_cols + hid + out}, at::kFloat);
    Arena mem;
    const size_t gz = mem.take(sizeof(float) * M * hid), gyp = mem.take(sizeof(float) * M * hid), gproj = mem.take(sizeof(float) * M * ld);
    const size_t img_in = mem.take(g::image_bytes(M, F, 65 * H)), img_out = mem.take(g::image_bytes(M, hid, out));
    size_t ws_bytes = std::max(g::workspace_bytes(M, F, 65 * H), g::workspace_bytes(M, hid, out));
    ws_bytes = std::max({ws_bytes, g::workspace_bytes(65 * H, F, M), g::workspace_bytes(out, hid, M)});
    const size_t ws = mem.take(ws_bytes);
    const size_t scan_part = mem.take(sizeof(float) * B * scan_cols), gate_part = mem.take(sizeof(float) * gate_rows * hid), bias_part = mem.take(sizeof(float) * bias_rows * out);
    mem.alloc(x);
    int* const status = status_ptr(x);
    const g::WeightJob jobs[2] = {{g::weight_of(ptr(p[kOutW]), hid), true, hid, out, g::tile_width(M, hid, out), mem.at<void>(img_out)},
                                  {stacked(p, H), true, F, 65 * H, g::tile_width(M, F, 65 * H), mem.at<void>(img_in)}};
    check("split_weights", g::split_weights(jobs, need_x ? 2 : 1, {}, s));
    check("run_weights", g::run_weights(ptr(gy), out, mem.at<void>(img_out), mem.at(gz), hid, M, hid, out, {}, mem.at(ws), ws_bytes, status, s));
    check("run_outer", g::run_outer(ptr(gy), out, ptr(z), hid, ptr(gw_out), hid, out, hid, M, mem.at(ws), ws_bytes, nullptr, status, s));
    check("skip_grad", l::skip_grad(ptr(gy), nullptr, mem.at(bias_part), M, out, s));
    check("mamba_gate_bwd", l::mamba_gate_bwd(w, ptr(proj), ld, ptr(y_pre), mem.at(gz), mem.at(gyp), mem.at(gproj), mem.at(gate_part), M, H, s));
    check("mamba_scan_bwd", l::mamba_scan_bwd(w, ptr(proj), ld, bytes(done), ptr(states), mem.at(gyp), ptr(gh_last), mem.at(gproj),
                                              need_h0 ? ptr(grads[13]) : nullptr, mem.at(scan_part), B, T, H, s));
    const l::ColumnSum sums[3] = {{mem.at(scan_part), B, scan_cols, ptr(small)}, {mem.at(gate_part), gate_rows, hid, ptr(small) + scan_cols},
                                  {mem.at(bias_part), bias_rows, out, ptr(small) + scan_cols + hid}};
    check("column_sums", l::column_sums(sums, 3, s));
    if (need_x) check("run_weights", g::run_weights(mem.at(gproj), ld, mem.at<void>(img_in), ptr(grads[0]), F, M, F, 65 * H, {}, mem.at(ws), ws_bytes, status, s));
    check("run_outer", g::run_outer(mem.at(gproj), ld, ptr(x), F, ptr(gw_in), F, 65 * H, F, M, mem.at(ws), ws_bytes, nullptr, status, s));
    const int channels = 48 * H;
    grads[1 + kConvW] = piece(small, 0, {channels, 1, 4});
    grads[1 + kConvB] = piece(small, 4 * channels, {channels});
    grads[1 + kALog] = piece(small, 5 * channels, {H});
    grads[1 + kDtBias] = piece(small, 5 * channels + H, {H});
    grads[1 + kD] = piece(small, 5 * channels + 2 * H, {H});
    grads[1 + kNormW] = piece(small, scan_cols, {hid});
    grads[1 + kOutB] = piece(small, scan_cols + hid, {out});
    grads[1 + kOutW] = gw_out;
    grads[1 + kIn] = piece(gw_in, 0, {2 * hid, F});
    grads[1 + kB] = piece(gw_in, 2ll * hid * F, {hid, F});
    grads[1 + kC] = piece(gw_in, 3ll * hid * F, {hid, F});
    grads[1 + kDt] = piece(gw_in, 4ll * hid * F, {H, F});
    return grads;
  }
};

// -> (last state (B,1,H,16,16), decay leaf (B,1,H,1,1), y (B,T,F)), or None where the caller has to compose the layer
pybind11::object mamba_layer(const Tensor& x_in, const variable_list& p, const OptTensor& h0_in, const OptTensor& a0_in, const OptTensor& done_in, double eps) {
  if (!x_in.is_cuda() || x_in.scalar_type() != at::kFloat || x_in.dim() != 3 || x_in.numel() == 0 || x_in.size(0) * x_in.size(1) > 0x7fffffff ||
      tf32_products() || at::autocast::is_autocast_enabled(at::kCUDA) || p.size() != kParams ||
      followed(x_in, p, h0_in, a0_in))
    return pybind11::none();
  for (const Tensor& t : p)
    if (t.scalar_type() != at::kFloat || t.device() != x_in.device() || !t.is_contiguous()) return pybind11::none();
  if (p[kALog].dim() != 1 || p[kOutW].dim() != 2) return pybind11::none();
  const int64_t H = p[kALog].size(0), F = x_in.size(2), out_dim = p[kOutW].size(0);
  if (!shaped(p[kD], {H}) || !shaped(p[kDtBias], {H}) || !shaped(p[kIn], {32 * H, F}) || !shaped(p[kB], {16 * H, F}) || !shaped(p[kC], {16 * H, F}) ||
      !shaped(p[kDt], {H, F}) || !shaped(p[kConvW], {48 * H, 1, 4}) || !shaped(p[kConvB], {48 * H}) || !shaped(p[kNormW], {16 * H}) ||
      !shaped(p[kOutW], {out_dim, 16 * H}) || !shaped(p[kOutB], {out_dim}) || x_in.size(0) * H > 0x7fffffff)
    return pybind11::none();
  const c10::cuda::CUDAGuard guard(x_in.device());
  const Tensor x = dense(x_in), h0 = carry_leaf(h0_in, x.size(0) * H * 256, at::kFloat, "h0"), a0 = carry_leaf(a0_in, x.size(0) * H, at::kFloat, "a0"), done = done_bytes(done_in, x.size(0) * x.size(1));
  bool grad = x.requires_grad() || (h0.defined() && h0.requires_grad());
  for (const Tensor& t : p) grad |= t.requires_grad();
  if (at::GradMode::is_enabled() && grad) {
    if (H > l::kMambaGradHeads) return pybind11::none();
    const variable_list out = MambaLayer::apply(x, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8], p[9], p[10], p[11], opt(h0), opt(a0), opt(done), eps);
    return pybind11::cast(std::make_tuple(out[0], out[1], out[2]));
  }
  const Result r = forward(x, p, h0, a0, done, eps, false);
  return pybind11::cast(std::make_tuple(r.h_last, r.a_last, r.y));
}

}  // namespace

void bind_mamba(pybind11::module_& m) { m.def("mamba_layer", &mamba_layer); }

}  // namespace mxk_host
