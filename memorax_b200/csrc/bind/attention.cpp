// The linear-attention and gated-delta-rule layers in bf16: the Dense layers on the inputs as one product, the chunked
// kernels on slices of its result, RMSNorm and output projection; the backward pass as one autograd node.  One step of a
// few sequences (acting) takes three launches.
#include "product.h"

#include "../attention.cuh"
#include "../layers.cuh"

namespace mxk_host {
namespace {

namespace l = mxk::layers;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int kFewRows = 256;   // up to here small_product beats the 128-row tiles of a library product (and its host cost)

struct Shape {
  int B, T, F, H, d, hid, M, out;
  int64_t ld;                   // columns of the joint projection, padded to 16 bytes
};

l::WeightRows rows_of(const variable_list& w, size_t count) {
  l::WeightRows r{};
  r.count = static_cast<int>(count);
  for (size_t i = 0; i < count; ++i) {
    r.ptr[i] = w[i].data_ptr();
    r.rows[i] = static_cast<int>(w[i].size(0));
  }
  return r;
}

// x (M, F) -> (M, ld), columns past the weights zero; `stacked` keeps the joint weight for the backward pass
// `bias`: of the columns behind q | k | v, added before they are rounded
Tensor project(const Tensor& x, const variable_list& w, size_t count, const Shape& s, Tensor* stacked, const Tensor& bias = Tensor()) {
  const Tensor proj = empty_like_of(x, {s.M, s.ld}, at::kBFloat16);
  if (!stacked && s.M <= kFewRows && s.F % 32 == 0 && aligned16(x)) {
    check("small_product", l::small_product(x.data_ptr(), rows_of(w, count), ptr<void>(bias), static_cast<int>(3 * s.hid), proj.data_ptr(), s.ld, s.M, s.F, stream()));
    return proj;
  }
  const Tensor joint = empty_like_of(x, {s.ld, s.F}, at::kBFloat16);
  check("stack_rows", l::stack_rows(rows_of(w, count), joint.data_ptr(), s.ld, s.F, stream()));
  // tiles fit q | k | v; the few columns behind them would cost a tile column (65536 x 3088 x 512 in the library: 198 us
  // against 160 for 3072 and 17 for 16)
  const Tensor rows = matrix(x, s.M, s.F);
  const int64_t main = 3 * s.hid, rest = bias.defined() ? bias.size(0) : 0;
  product_into(rows, transposed(matrix(joint, main, s.F)), matrix(proj, s.M, main, s.ld));
  if (rest) product_into(rows, transposed(matrix(joint, rest, s.F, 0, main * s.F)), matrix(proj, s.M, rest, s.ld, main), bias);
  if (stacked) *stacked = joint;
  return proj;
}

Tensor output(const Tensor& n, const Tensor& w, const Tensor& bias, const Shape& s, bool few) {
  if (few && s.M <= kFewRows && s.hid % 32 == 0) {
    const Tensor y = empty_like_of(n, {s.B, s.T, s.out}, at::kBFloat16);
    check("small_product", l::small_product(n.data_ptr(), rows_of({w}, 1), bias.data_ptr(), 0, y.data_ptr(), s.out, s.M, s.hid, stream()));
    return y;
  }
  const Tensor y = empty_like_of(n, {s.B, s.T, s.out}, at::kBFloat16);
  product_into(n, transposed(w), matrix(y, s.M, s.out), bias);
  return y;
}

// What follows the mixer: RMSNorm and output projection, and their gradients
struct Tail {
  Tensor n, rstd;
};
Tail norm_forward(const Tensor& o, const Tensor& norm_w, double norm_eps, const Shape& s) {
  Tail t{empty_like_of(o, o.sizes(), at::kBFloat16), empty_like_of(o, {s.M}, at::kFloat)};
  check("mxk_norm_bf16_fwd", mxk_norm_bf16_fwd(o.data_ptr(), norm_w.data_ptr(), nullptr, t.n.data_ptr(), nullptr, ptr(t.rstd), s.M, s.hid,
                                               norm_eps, 1, stream()));
  return t;
}
struct TailGrads {
  Tensor go, norm_w, out_w, out_b;
};
TailGrads tail_backward(const Tensor& gy, const Tensor& o, const Tensor& n, const Tensor& rstd, const Tensor& norm_w, const Tensor& out_w, const Shape& s) {
  TailGrads g;
  const Tensor gn = product(gy, out_w);
  g.out_w = product(transposed(gy), n);
  g.out_b = empty_like_of(gy, {s.out}, at::kBFloat16);
  const size_t sum_bytes = mxk_colsum_workspace_bytes(s.M, s.out), norm_bytes = mxk_norm_bwd_workspace_bytes(s.M, s.hid);
  const Tensor ws = scratch(gy, std::max(sum_bytes, norm_bytes));
  check("mxk_colsum_bf16", mxk_colsum_bf16(gy.data_ptr(), g.out_b.data_ptr(), ws.data_ptr(), sum_bytes, s.M, s.out, stream()));
  g.go = empty_like_of(o, o.sizes(), at::kBFloat16);
  const Tensor gw = empty_like_of(gy, {s.hid}, at::kFloat);
  check("mxk_norm_bf16_bwd", mxk_norm_bf16_bwd(o.data_ptr(), norm_w.data_ptr(), nullptr, ptr(rstd), gn.data_ptr(), g.go.data_ptr(), ptr(gw), nullptr,
                                               ws.data_ptr(), norm_bytes, s.M, s.hid, 1, stream()));
  g.norm_w = gw.to(at::kBFloat16);
  return g;
}

bool all_bf16(const Tensor& x, const variable_list& p) {
  if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() != 3 || x.numel() == 0 || x.size(0) * x.size(1) > 0x7fffffff ||
      at::autocast::is_autocast_enabled(at::kCUDA))
    return false;
  for (const Tensor& t : p)
    if (t.scalar_type() != at::kBFloat16 || t.device() != x.device() || !t.is_contiguous() || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15)) return false;
  return true;
}
bool wants_grad(const Tensor& x, const variable_list& p, std::initializer_list<Tensor> carry) {
  if (!at::GradMode::is_enabled()) return false;
  bool grad = x.requires_grad();
  for (const Tensor& t : p) grad |= t.requires_grad();
  for (const Tensor& t : carry) grad |= t.defined() && t.requires_grad();
  return grad;
}
const uint8_t* cols_of(const Tensor& t, int64_t column) { return static_cast<const uint8_t*>(t.data_ptr()) + 2 * column; }
uint8_t* cols_out(const Tensor& t, int64_t column) { return static_cast<uint8_t*>(t.data_ptr()) + 2 * column; }

// ------------------------------------------------------------------------------------------------ linear attention
enum { kQ, kK, kV, kNorm, kOutW, kOutB, kLinParams };

struct LinAttnLayer : torch::autograd::Function<LinAttnLayer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wq, const Tensor& wk, const Tensor& wv, const Tensor& norm_w,
                               const Tensor& out_w, const Tensor& out_b, const OptTensor& s0_in, const OptTensor& z0_in, const OptTensor& done_in,
                               int64_t heads, double eps, double norm_eps);
  static variable_list backward(AutogradContext* ctx, const variable_list& gout);
};

Shape shape_of(const Tensor& x, int64_t heads, int64_t hid, int64_t out, int64_t extra) {
  Shape s;
  s.B = x.size(0); s.T = x.size(1); s.F = x.size(2);
  s.H = heads; s.hid = hid; s.d = hid / heads;
  s.M = s.B * s.T;
  s.out = out;
  s.ld = (3 * hid + extra + 7) / 8 * 8;
  return s;
}

struct LinResult {
  Tensor s_last, z_last, y, proj, joint, states, o;
  Tail tail;
};
LinResult linattn_forward(const Tensor& x, const variable_list& p, const Tensor& s0, const Tensor& z0, const Tensor& done, const Shape& s, double eps,
                          double norm_eps, bool keep) {
  LinResult r;
  r.s_last = empty_like_of(x, {s.B, 1, s.H, s.d, s.d}, at::kFloat);
  r.z_last = empty_like_of(x, {s.B, 1, s.H, s.d}, at::kFloat);
  r.proj = project(x, p, 3, s, keep ? &r.joint : nullptr);
  // (the chunk kernels take a state from any address)
  if (s.T == 1 && !keep && (s.d == 64 || s.d == 32) && s.hid <= 2048 && aligned16(s0)) {
    const Tensor n = empty_like_of(x, {s.M, s.hid}, at::kBFloat16);
    check("linattn_step", l::linattn_step(r.proj.data_ptr(), s.ld, ptr(s0), ptr(z0), bytes(done), p[kNorm].data_ptr(), norm_eps, eps, n.data_ptr(),
                                          ptr(r.s_last), ptr(r.z_last), s.B, s.H, s.d, stream()));
    r.y = output(n, p[kOutW], p[kOutB], s, true);
    return r;
  }
  r.o = empty_like_of(x, {s.M, s.hid}, at::kBFloat16);
  if (keep) r.states = scratch(x, mxk_linattn_chunk_states_bytes(s.B, s.T, s.H, s.d));
  check("mxk_linattn_bf16_fwd", mxk::linattn::forward(cols_of(r.proj, 0), cols_of(r.proj, s.hid), cols_of(r.proj, 2 * s.hid), s.ld, ptr(s0), ptr(z0), bytes(done),
                                                      r.o.data_ptr(), ptr(r.s_last), ptr(r.z_last), ptr<void>(r.states), status_ptr(x), s.B, s.T, s.H, s.d,
                                                      eps, 1, stream()));
  r.tail = norm_forward(r.o, p[kNorm], norm_eps, s);
  r.y = output(r.tail.n, p[kOutW], p[kOutB], s, !keep);
  return r;
}

variable_list LinAttnLayer::forward(AutogradContext* ctx, const Tensor& x, const Tensor& wq, const Tensor& wk, const Tensor& wv, const Tensor& norm_w,
                                    const Tensor& out_w, const Tensor& out_b, const OptTensor& s0_in, const OptTensor& z0_in, const OptTensor& done_in,
                                    int64_t heads, double eps, double norm_eps) {
  const variable_list p{wq, wk, wv, norm_w, out_w, out_b};
  const Tensor s0 = s0_in.value_or(Tensor()), z0 = z0_in.value_or(Tensor()), done = done_in.value_or(Tensor());
  const Shape s = shape_of(x, heads, wq.size(0), out_w.size(0), 0);
  LinResult r = linattn_forward(x, p, s0, z0, done, s, eps, norm_eps, true);
  ctx->set_materialize_grads(false);
  ctx->saved_data["heads"] = heads;
  ctx->saved_data["eps"] = eps;
  ctx->saved_data["s0"] = s0.defined();
  ctx->saved_data["z0"] = z0.defined();
  ctx->save_for_backward({x, norm_w, out_w, done, r.proj, r.joint, r.states, r.o, r.tail.n, r.tail.rstd});
  return {r.s_last, r.z_last, r.y};
}

variable_list LinAttnLayer::backward(AutogradContext* ctx, const variable_list& gout) {
  const variable_list saved = ctx->get_saved_variables();
  const Tensor &x = saved[0], &norm_w = saved[1], &out_w = saved[2], &done = saved[3], &proj = saved[4], &joint = saved[5], &states = saved[6], &o = saved[7];
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t hid = out_w.size(1);
  const Shape s = shape_of(x, ctx->saved_data["heads"].toInt(), hid, out_w.size(0), 0);
  const Tensor gy = matrix(gout[2].defined() ? dense(gout[2]) : empty_like_of(x, {s.M, s.out}, at::kBFloat16).zero_(), s.M, s.out);
  const Tensor gs = gout[0].defined() ? dense(gout[0]) : Tensor(), gz = gout[1].defined() ? dense(gout[1]) : Tensor();
  const bool has_s = ctx->saved_data["s0"].toBool(), has_z = ctx->saved_data["z0"].toBool();
  const bool need_s = (has_s && ctx->needs_input_grad(7)) || (has_z && ctx->needs_input_grad(has_s ? 8 : 7));
  const TailGrads t = tail_backward(gy, o, saved[8], saved[9], norm_w, out_w, s);
  const Tensor gproj = empty_like_of(x, proj.sizes(), at::kBFloat16);
  const Tensor gs0 = need_s ? empty_like_of(x, {s.B, 1, s.H, s.d, s.d}, at::kFloat) : Tensor(), gz0 = need_s ? empty_like_of(x, {s.B, 1, s.H, s.d}, at::kFloat) : Tensor();
  check("mxk_linattn_bf16_bwd", mxk::linattn::backward(cols_of(proj, 0), cols_of(proj, hid), cols_of(proj, 2 * hid), s.ld, t.go.data_ptr(), states.data_ptr(), bytes(done),
                                                       ptr(gs), ptr(gz), cols_out(gproj, 0), cols_out(gproj, hid), cols_out(gproj, 2 * hid), s.ld, ptr(gs0), ptr(gz0),
                                                       status_ptr(x), s.B, s.T, s.H, s.d, ctx->saved_data["eps"].toDouble(), 1, stream()));
  variable_list grads(13);
  if (ctx->needs_input_grad(0)) {
    grads[0] = empty_like_of(x, x.sizes(), at::kBFloat16);
    product_into(gproj, joint, matrix(grads[0], s.M, s.F));
  }
  const Tensor gw = product(transposed(gproj), matrix(x, s.M, s.F));
  for (int i = 0; i < 3; ++i) grads[1 + i] = piece(gw, i * hid * s.F, {hid, s.F});
  grads[4] = t.norm_w;
  grads[5] = t.out_w;
  grads[6] = t.out_b;
  if (has_s) grads[7] = gs0;
  if (has_z) grads[8] = gz0;
  return grads;
}

// -> (s_last (B,1,H,d,d), z_last (B,1,H,d), y (B,T,F)), or None where the caller has to compose the layer
pybind11::object linattn_layer(const Tensor& x_in, const variable_list& p, const OptTensor& s0_in, const OptTensor& z0_in, const OptTensor& done_in,
                               int64_t heads, double eps, double norm_eps) {
  if (!all_bf16(x_in, p) || p.size() != kLinParams || followed(x_in, p, s0_in, z0_in)) return pybind11::none();
  if (p[kQ].dim() != 2 || p[kOutW].dim() != 2 || heads < 1) return pybind11::none();
  const int64_t hid = p[kQ].size(0), F = x_in.size(2), d = hid / heads, out_dim = p[kOutW].size(0);
  if (d * heads != hid || d % 8 || d < 8 || d > 64 || hid > 1024 || F % 8 || out_dim % 8 || x_in.size(0) * heads > 0x7fffffff) return pybind11::none();
  if (!shaped(p[kQ], {hid, F}) || !shaped(p[kK], {hid, F}) || !shaped(p[kV], {hid, F}) || !shaped(p[kNorm], {hid}) || !shaped(p[kOutW], {out_dim, hid}) ||
      !shaped(p[kOutB], {out_dim}))
    return pybind11::none();
  const c10::cuda::CUDAGuard guard(x_in.device());
  const Tensor x = dense(x_in), s0 = carry_leaf(s0_in, x.size(0) * hid * d, at::kFloat, "s0"), z0 = carry_leaf(z0_in, x.size(0) * hid, at::kFloat, "z0"), done = done_bytes(done_in, x.size(0) * x.size(1));
  if (wants_grad(x, p, {s0, z0})) {
    const variable_list out = LinAttnLayer::apply(x, p[0], p[1], p[2], p[3], p[4], p[5], opt(s0), opt(z0), opt(done), heads, eps, norm_eps);
    return pybind11::cast(std::make_tuple(out[0], out[1], out[2]));
  }
  const LinResult r = linattn_forward(x, p, s0, z0, done, shape_of(x, heads, hid, p[kOutW].size(0), 0), eps, norm_eps, false);
  return pybind11::cast(std::make_tuple(r.s_last, r.z_last, r.y));
}

// ------------------------------------------------------------------------------------------------ gated delta rule
enum { kDq, kDk, kDv, kGateW, kGateB, kDNorm, kDOutW, kDOutB, kDeltaParams };

struct DeltaResult {
  Tensor s_last, y, proj, joint, q, k, alpha, beta, states, ws, o;
  Tail tail;
};
DeltaResult delta_forward(const Tensor& x, const variable_list& p, const Tensor& s0, const Tensor& done, const Shape& s, double norm_eps, bool keep) {
  DeltaResult r;
  r.s_last = empty_like_of(x, {s.B, 1, s.H, s.d, s.d}, at::kFloat);
  r.proj = project(x, p, 4, s, keep ? &r.joint : nullptr, p[kGateB]);
  // (the chunk kernels report a state that is not aligned)
  if (s.T == 1 && !keep && s.hid <= 2048 && aligned16(s0)) {
    const Tensor n = empty_like_of(x, {s.M, s.hid}, at::kBFloat16);
    check("gdelta_step", l::gdelta_step(r.proj.data_ptr(), s.ld, ptr(s0), bytes(done), p[kDNorm].data_ptr(), norm_eps, n.data_ptr(),
                                        ptr(r.s_last), s.B, s.H, s.d, stream()));
    r.y = output(n, p[kDOutW], p[kDOutB], s, true);
    return r;
  }
  r.q = empty_like_of(x, {s.M, s.hid}, at::kBFloat16);
  r.k = empty_like_of(x, {s.M, s.hid}, at::kBFloat16);
  r.alpha = empty_like_of(x, {s.M, s.H}, at::kFloat);
  r.beta = empty_like_of(x, {s.M, s.H}, at::kFloat);
  r.o = empty_like_of(x, {s.M, s.hid}, at::kBFloat16);
  if (keep) r.states = scratch(x, mxk_gdelta_chunk_states_bytes(s.B, s.T, s.H, s.d));
  const size_t ws_bytes = mxk_gdelta_workspace_bytes(s.B, s.T, s.H, s.d);
  r.ws = scratch(x, ws_bytes);
  check("delta_inputs", l::delta_inputs(r.proj.data_ptr(), s.ld, r.q.data_ptr(), r.k.data_ptr(), ptr(r.alpha), ptr(r.beta), s.M, s.H, s.d, stream()));
  check("mxk_gdelta_bf16_fwd", mxk::gdelta::forward(r.q.data_ptr(), r.k.data_ptr(), cols_of(r.proj, 2 * s.hid), s.ld, ptr(r.alpha), ptr(r.beta), ptr(s0), bytes(done),
                                                    r.o.data_ptr(), ptr(r.s_last), ptr<void>(r.states), r.ws.data_ptr(), ws_bytes, status_ptr(x), s.B, s.T, s.H,
                                                    s.d, stream()));
  r.tail = norm_forward(r.o, p[kDNorm], norm_eps, s);
  r.y = output(r.tail.n, p[kDOutW], p[kDOutB], s, !keep);
  return r;
}

struct DeltaLayer : torch::autograd::Function<DeltaLayer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wq, const Tensor& wk, const Tensor& wv, const Tensor& gate_w,
                               const Tensor& gate_b, const Tensor& norm_w, const Tensor& out_w, const Tensor& out_b, const OptTensor& s0_in,
                               const OptTensor& done_in, int64_t heads, double norm_eps) {
    const variable_list p{wq, wk, wv, gate_w, gate_b, norm_w, out_w, out_b};
    const Tensor s0 = s0_in.value_or(Tensor()), done = done_in.value_or(Tensor());
    const Shape s = shape_of(x, heads, wq.size(0), out_w.size(0), 2 * heads);
    DeltaResult r = delta_forward(x, p, s0, done, s, norm_eps, true);
    ctx->set_materialize_grads(false);
    ctx->saved_data["heads"] = heads;
    ctx->saved_data["s0"] = s0.defined();
    ctx->save_for_backward({x, norm_w, out_w, done, r.proj, r.joint, r.q, r.k, r.alpha, r.beta, r.states, r.ws, r.o, r.tail.n, r.tail.rstd});
    return {r.s_last, r.y};
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& gout) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &norm_w = saved[1], &out_w = saved[2], &done = saved[3], &proj = saved[4], &joint = saved[5];
    const Tensor &q = saved[6], &k = saved[7], &alpha = saved[8], &beta = saved[9], &states = saved[10], &ws = saved[11], &o = saved[12];
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t hid = out_w.size(1);
    const Shape s = shape_of(x, ctx->saved_data["heads"].toInt(), hid, out_w.size(0), 2 * ctx->saved_data["heads"].toInt());
    const Tensor gy = matrix(gout[1].defined() ? dense(gout[1]) : empty_like_of(x, {s.M, s.out}, at::kBFloat16).zero_(), s.M, s.out);
    const Tensor gs = gout[0].defined() ? dense(gout[0]) : Tensor();
    const bool need_s0 = ctx->saved_data["s0"].toBool() && ctx->needs_input_grad(9);
    const TailGrads t = tail_backward(gy, o, saved[13], saved[14], norm_w, out_w, s);
    const Tensor gproj = empty_like_of(x, proj.sizes(), at::kBFloat16), gq = empty_like_of(x, q.sizes(), at::kBFloat16), gk = empty_like_of(x, k.sizes(), at::kBFloat16);
    const Tensor ga = empty_like_of(x, alpha.sizes(), at::kFloat), gb = empty_like_of(x, beta.sizes(), at::kFloat);
    variable_list grads(13);
    if (need_s0) grads[9] = empty_like_of(x, {s.B, 1, s.H, s.d, s.d}, at::kFloat);
    check("mxk_gdelta_bf16_bwd", mxk::gdelta::backward(q.data_ptr(), k.data_ptr(), cols_of(proj, 2 * hid), ptr(alpha), ptr(beta), t.go.data_ptr(), states.data_ptr(), ws.data_ptr(),
                                                       bytes(done), ptr(gs), gq.data_ptr(), gk.data_ptr(), cols_out(gproj, 2 * hid), s.ld, ptr(ga), ptr(gb),
                                                       need_s0 ? ptr(grads[9]) : nullptr, status_ptr(x), s.B, s.T, s.H, s.d, stream()));
    const int rows = l::delta_gate_blocks(s.M);
    const Tensor part = empty_like_of(x, {rows, 2 * s.H}, at::kFloat);
    check("delta_inputs_bwd", l::delta_inputs_bwd(proj.data_ptr(), s.ld, gq.data_ptr(), gk.data_ptr(), ptr(ga), ptr(gb), gproj.data_ptr(), ptr(part), s.M, s.H,
                                                  s.d, stream()));
    grads[5] = empty_like_of(x, {2 * s.H}, at::kBFloat16);
    const l::ColumnSum sum{ptr(part), rows, 2 * s.H, nullptr, grads[5].data_ptr()};
    check("column_sums", l::column_sums(&sum, 1, stream()));
    if (ctx->needs_input_grad(0)) {
      grads[0] = empty_like_of(x, x.sizes(), at::kBFloat16);
      product_into(gproj, joint, matrix(grads[0], s.M, s.F));
    }
    const Tensor rows_in = matrix(x, s.M, s.F), gw = product(transposed(matrix(gproj, s.M, 3 * hid, s.ld)), rows_in);
    for (int i = 0; i < 3; ++i) grads[1 + i] = piece(gw, i * hid * s.F, {hid, s.F});
    grads[4] = product(transposed(matrix(gproj, s.M, 2 * s.H, s.ld, 3 * hid)), rows_in);
    grads[6] = t.norm_w;
    grads[7] = t.out_w;
    grads[8] = t.out_b;
    return grads;
  }
};

// -> (s_last (B,1,H,d,d), y (B,T,F)), or None
pybind11::object deltanet_layer(const Tensor& x_in, const variable_list& p, const OptTensor& s0_in, const OptTensor& done_in, int64_t heads, double norm_eps) {
  if (!all_bf16(x_in, p) || p.size() != kDeltaParams || followed(x_in, p, s0_in)) return pybind11::none();
  if (p[kDq].dim() != 2 || p[kDOutW].dim() != 2 || heads < 1) return pybind11::none();
  const int64_t hid = p[kDq].size(0), F = x_in.size(2), d = hid / heads, out_dim = p[kDOutW].size(0);
  if (d * heads != hid || (d != 64 && d != 128) || hid > 1024 || heads > 64 || F % 8 || out_dim % 8 || x_in.size(0) * heads > 0x7fffffff) return pybind11::none();
  if (!shaped(p[kDq], {hid, F}) || !shaped(p[kDk], {hid, F}) || !shaped(p[kDv], {hid, F}) || !shaped(p[kGateW], {2 * heads, F}) || !shaped(p[kGateB], {2 * heads}) ||
      !shaped(p[kDNorm], {hid}) || !shaped(p[kDOutW], {out_dim, hid}) || !shaped(p[kDOutB], {out_dim}))
    return pybind11::none();
  const c10::cuda::CUDAGuard guard(x_in.device());
  const Tensor x = dense(x_in), s0 = carry_leaf(s0_in, x.size(0) * hid * d, at::kFloat, "s0"), done = done_bytes(done_in, x.size(0) * x.size(1));
  if (wants_grad(x, p, {s0})) {
    const variable_list out = DeltaLayer::apply(x, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], opt(s0), opt(done), heads, norm_eps);
    return pybind11::cast(std::make_tuple(out[0], out[1]));
  }
  const DeltaResult r = delta_forward(x, p, s0, done, shape_of(x, heads, hid, p[kDOutW].size(0), 2 * heads), norm_eps, false);
  return pybind11::cast(std::make_tuple(r.s_last, r.y));
}

}  // namespace

void bind_attention(pybind11::module_& m) {
  m.def("linattn_layer", &linattn_layer);
  m.def("deltanet_layer", &deltanet_layer);
}

}  // namespace mxk_host
