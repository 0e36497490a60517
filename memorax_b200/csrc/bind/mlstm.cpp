// The mLSTM layer on the tensor cores (bf16): its products on slices of joint buffers, everything else fused; the backward pass as one autograd node.
#include "product.h"

#include <cmath>

#include "../attention.cuh"
#include "../layers.cuh"

namespace mxk_host {
namespace {

namespace l = mxk::layers;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

enum { kUp, kConvW, kConvB, kQ, kK, kV, kIW, kIB, kFW, kFB, kSkip, kNorm, kOut, kParams };

struct Shape {
  int B, T, F, H, d, hid, M;
  float scale() const { return 1.f / std::sqrt(static_cast<float>(d)); }
};
Shape shape_of(const Tensor& x, const variable_list& p) {
  Shape s;
  s.B = x.size(0); s.T = x.size(1); s.F = x.size(2);
  s.H = p[kQ].size(0); s.d = p[kQ].size(1);
  s.hid = s.H * s.d;
  s.M = s.B * s.T;
  return s;
}
// (H, a, b) -> (H, b, a)
Tensor swapped(const Tensor& t) { return view_of(t, 0, {t.size(0), t.size(2), t.size(1)}, {t.stride(0), t.stride(2), t.stride(1)}); }
// columns [at, at + hid) of a (M, n) buffer as per-head matrices (H, M, d)
Tensor heads(const Tensor& t, int at, const Shape& s) { return view_of(t, at, {s.H, s.M, s.d}, {s.d, t.size(1), 1}); }
// parts [first, first + count) of q | k | v of every head, out of a buffer (M, H, 3, d): (H, M, count d).  With the head
// outermost this is the order the gates' weights are in, and q and k are one product.
Tensor parts(const Tensor& t, int first, int count, const Shape& s) {
  return view_of(t, first * s.d, {s.H, s.M, count * s.d}, {3 * s.d, t.size(1), 1});
}
// Buffers of one allocation: places in a bf16 tensor, on 512-byte boundaries (a layer of this many short launches waits for the host,
// where a tensor of its own for each took 1 us to make and as much again to keep for the backward pass).
struct Places {
  int64_t used = 0;
  int64_t take(int64_t elements) {
    const int64_t at = used;
    used += (elements + 255) / 256 * 256;
    return at;
  }
  int64_t take_floats(int64_t n) { return take(2 * n); }
  int64_t take_bytes(int64_t n) { return take((n + 1) / 2); }
};
void* column(const Tensor& t, int64_t c) { return static_cast<uint8_t*>(t.data_ptr()) + 2 * c; }
float* floats(const Tensor& t, int64_t at) { return static_cast<float*>(column(t, at)); }

// What the forward pass leaves for the backward pass.
struct Kept {
  int64_t up, u, qkv, qk_w, gates, logits, log_i, log_f, ks, h, g, m_steps, states, size;
  Kept(const Shape& s, bool keep) {
    Places at;
    up = at.take(2ll * s.M * s.hid);
    u = at.take(1ll * s.M * s.hid);
    qkv = at.take(3ll * s.M * s.hid);
    qk_w = at.take(2ll * s.hid * s.d);
    gates = at.take(6ll * s.H * s.hid + 2 * s.H);
    logits = at.take(2ll * s.M * s.H);
    log_i = at.take_floats(1ll * s.M * s.H);
    log_f = at.take_floats(1ll * s.M * s.H);
    ks = at.take(1ll * s.M * s.hid);
    h = at.take(1ll * s.M * s.hid);
    g = at.take(1ll * s.M * s.hid);
    m_steps = keep ? at.take_floats(1ll * s.M * s.H) : 0;
    states = keep ? at.take_bytes(mxk_mlstm_bf16_chunk_states_bytes(s.B, s.T, s.H, s.d)) : 0;
    size = at.used;
  }
};

struct Result {
  Tensor y, c_last, n_last, m_last, f_last, kept;
};

Result forward(const Tensor& x, const variable_list& p, const Tensor& c0, const Tensor& n0, const Tensor& m0, const Tensor& f0, const Tensor& done,
               const Shape& s, double eps, bool keep) {
  Result r;
  const auto bf = at::kBFloat16;
  const auto st = stream();
  r.c_last = empty_like_of(x, {s.B, 1, s.H, s.d, s.d}, at::kFloat);
  r.n_last = empty_like_of(x, {s.B, 1, s.H, s.d, 1}, at::kFloat);
  r.m_last = empty_like_of(x, {s.B, 1, s.H, 1, 1}, at::kFloat);
  r.f_last = empty_like_of(x, {s.B, 1, s.H, 1, 1}, at::kFloat);
  const Kept at(s, keep);
  const Tensor& all = r.kept = empty_like_of(x, {at.size}, bf);
  const Tensor up = matrix(all, s.M, 2 * s.hid, 0, at.up), u = matrix(all, s.M, s.hid, 0, at.u), qkv = matrix(all, s.M, 3 * s.hid, 0, at.qkv),
               g = matrix(all, s.M, s.hid, 0, at.g), qk_w = piece(all, at.qk_w, {s.H, 2 * s.d, s.d}), logits = matrix(all, s.M, 2 * s.H, 0, at.logits);
  const int64_t gate_w_size = 6ll * s.H * s.hid;
  const Tensor gate_w = matrix(all, 2 * s.H, 3 * s.hid, 0, at.gates), gate_b = piece(all, at.gates + gate_w_size, {2 * s.H});
  float *const log_i = floats(all, at.log_i), *const log_f = floats(all, at.log_f);
  void *const ks = column(all, at.ks), *const h = column(all, at.h);
  product_into(matrix(x, s.M, s.F), transposed(p[kUp]), up);
  check("mlstm_conv_fwd", l::mlstm_conv_fwd(up.data_ptr(), 2 * s.hid, p[kConvW].data_ptr(), p[kConvB].data_ptr(), u.data_ptr(), s.B, s.T, s.hid, st));
  check("mlstm_weights", l::mlstm_weights(p[kQ].data_ptr(), p[kK].data_ptr(), p[kIW].data_ptr(), p[kFW].data_ptr(), p[kIB].data_ptr(), p[kFB].data_ptr(),
                                          qk_w.data_ptr(), gate_w.data_ptr(), gate_b.data_ptr(), s.H, s.d, st));
  products_into({{heads(u, 0, s), swapped(qk_w), parts(qkv, 0, 2, s)}, {heads(up, 0, s), swapped(p[kV]), parts(qkv, 2, 1, s)}});
  product_into(qkv, transposed(gate_w), logits, gate_b);
  check("mlstm_gates_fwd", l::mlstm_gates_fwd(logits.data_ptr(), column(qkv, s.d), 3 * s.hid, 3 * s.d, s.scale(), log_i, log_f, ks, s.M, s.H, s.d, st));
  check("mxk_mlstm_bf16_fwd", mxk::mlstm_tc::forward(qkv.data_ptr(), ks, column(qkv, 2 * s.d), 3 * s.hid, 3 * s.d, log_i, log_f, ptr(c0), ptr(n0),
                                                     ptr(m0), ptr(f0), bytes(done), h, ptr(r.c_last), ptr(r.n_last), ptr(r.m_last), ptr(r.f_last),
                                                     keep ? floats(all, at.m_steps) : nullptr, keep ? column(all, at.states) : nullptr, status_ptr(x), s.B, s.T, s.H, s.d, eps, st));
  check("mlstm_out_fwd", l::mlstm_out_fwd(h, u.data_ptr(), column(up, s.hid), 2 * s.hid, p[kNorm].data_ptr(), p[kSkip].data_ptr(), g.data_ptr(), s.M,
                                          s.H, s.d, st));
  r.y = empty_like_of(x, {s.B, s.T, p[kOut].size(0)}, bf);
  product_into(g, transposed(p[kOut]), matrix(r.y, s.M, p[kOut].size(0)));
  return r;
}

struct MlstmLayer : torch::autograd::Function<MlstmLayer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, at::TensorList params, const OptTensor& c0_in, const OptTensor& n0_in, const OptTensor& m0_in,
                               const OptTensor& f0_in, const OptTensor& done_in, double eps) {
    const variable_list p(params.begin(), params.end());
    const Tensor c0 = c0_in.value_or(Tensor()), n0 = n0_in.value_or(Tensor()), m0 = m0_in.value_or(Tensor()), done = done_in.value_or(Tensor());
    const Shape s = shape_of(x, p);
    Result r = mxk_host::forward(x, p, c0, n0, m0, f0_in.value_or(Tensor()), done, s, eps, true);
    ctx->set_materialize_grads(false);
    ctx->saved_data["eps"] = eps;
    variable_list saved{x};
    saved.insert(saved.end(), p.begin(), p.end());
    for (const Tensor& t : {c0, n0, m0, done, r.kept, r.c_last, r.n_last}) saved.push_back(t);
    ctx->save_for_backward(std::move(saved));
    ctx->mark_non_differentiable({r.f_last});
    return {r.c_last, r.n_last, r.m_last, r.f_last, r.y};
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& gout) {
    const variable_list v = ctx->get_saved_variables();
    const Tensor& x = v[0];
    const variable_list p(v.begin() + 1, v.begin() + 1 + kParams);
    const Tensor *t = &v[1 + kParams];
    const Tensor &c0 = t[0], &n0 = t[1], &m0 = t[2], &done = t[3], &all = t[4], &c_last = t[5], &n_last = t[6];
    const c10::cuda::CUDAGuard guard(x.device());
    const Shape s = shape_of(x, p);
    const auto bf = at::kBFloat16;
    const auto st = stream();
    const int64_t out = p[kOut].size(0);
    const Kept at_kept(s, true);
    const auto rows = [&](const Tensor& in, int64_t at, int64_t cols) { return matrix(in, s.M, cols, 0, at); };
    const Tensor up = rows(all, at_kept.up, 2 * s.hid), u = rows(all, at_kept.u, s.hid), qkv = rows(all, at_kept.qkv, 3 * s.hid), g = rows(all, at_kept.g, s.hid),
                 qk_w = piece(all, at_kept.qk_w, {s.H, 2 * s.d, s.d}), gate_w = matrix(all, 2 * s.H, 3 * s.hid, 0, at_kept.gates);
    float *const log_i = floats(all, at_kept.log_i), *const log_f = floats(all, at_kept.log_f);
    void *const ks = column(all, at_kept.ks), *const h = column(all, at_kept.h), *const logits = column(all, at_kept.logits);
    const auto given = [&](int i) { return gout[i].defined() ? dense(gout[i]) : Tensor(); };
    const Tensor gc = given(0), gn = given(1), gm = given(2);
    const Tensor gy = matrix(gout[4].defined() ? dense(gout[4]) : empty_like_of(x, {s.M, out}, bf).zero_(), s.M, out);
    // inputs of the node: x, the parameters, then what there is of the carry
    variable_list grads(1 + kParams + 6);
    const int first = 1 + kParams;
    const bool need_state = c0.defined() || n0.defined() || m0.defined();
    Tensor gc0, gn0, gm0;
    if (need_state) {
      gc0 = empty_like_of(x, {s.B, 1, s.H, s.d, s.d}, at::kFloat);
      gn0 = empty_like_of(x, {s.B, 1, s.H, s.d, 1}, at::kFloat);
      gm0 = empty_like_of(x, {s.B, 1, s.H, 1, 1}, at::kFloat);
    }
    const int out_rows = l::mlstm_out_blocks(s.M, s.hid), gate_rows = l::mlstm_gate_blocks(s.M), conv_rows = l::mlstm_conv_blocks(s.B, s.T, s.hid);
    const int cols[3] = {2 * s.hid, 2 * s.H, 5 * s.hid};
    const int64_t wide = static_cast<int64_t>(s.M) * s.hid, heads_all = static_cast<int64_t>(s.M) * s.H;
    Places place;
    const int64_t at_gg = place.take(wide), at_gh = place.take(wide), at_gu = place.take(wide), at_gks = place.take(wide), at_gx = place.take(wide), at_gup = place.take(2 * wide),
                  at_gqkv = place.take(3 * wide), at_glogits = place.take(2 * heads_all), at_gli = place.take_floats(heads_all), at_glf = place.take_floats(heads_all),
                  at_part = place.take_floats(static_cast<int64_t>(out_rows) * cols[0] + gate_rows * cols[1] + static_cast<int64_t>(conv_rows) * cols[2]);
    const Tensor temp = empty_like_of(x, {place.used}, bf);
    const Tensor gg = rows(temp, at_gg, s.hid), gu = rows(temp, at_gu, s.hid), gx = rows(temp, at_gx, s.hid), gup = rows(temp, at_gup, 2 * s.hid),
                 gqkv = rows(temp, at_gqkv, 3 * s.hid), glogits = rows(temp, at_glogits, 2 * s.H);
    void *const gh = column(temp, at_gh), *const gks = column(temp, at_gks);
    float *const gli = floats(temp, at_gli), *const glf = floats(temp, at_glf);
    float* const part_out = floats(temp, at_part);
    float* const part_gate = part_out + static_cast<size_t>(out_rows) * cols[0];
    float* const part_conv = part_gate + static_cast<size_t>(gate_rows) * cols[1];
    product_into(gy, p[kOut], gg);
    check("mlstm_out_bwd", l::mlstm_out_bwd(gg.data_ptr(), h, u.data_ptr(), column(up, s.hid), 2 * s.hid, p[kNorm].data_ptr(), p[kSkip].data_ptr(), gh,
                                            column(gup, s.hid), 2 * s.hid, gu.data_ptr(), part_out, s.M, s.H, s.d, st));
    check("mxk_mlstm_bf16_bwd", mxk::mlstm_tc::backward(qkv.data_ptr(), ks, column(qkv, 2 * s.d), 3 * s.hid, 3 * s.d, log_i, log_f, ptr(c0), ptr(n0), ptr(m0),
                                                        bytes(done), gh, ptr(c_last), ptr(n_last), floats(all, at_kept.m_steps), column(all, at_kept.states), ptr(gc), ptr(gn), ptr(gm),
                                                        gqkv.data_ptr(), gks, column(gqkv, 2 * s.d), 3 * s.hid, 3 * s.d, gli, glf, ptr(gc0), ptr(gn0), ptr(gm0),
                                                        status_ptr(x), s.B, s.T, s.H, s.d, ctx->saved_data["eps"].toDouble(), st));
    check("mlstm_gates_bwd", l::mlstm_gates_bwd(logits, gli, glf, gks, s.scale(), column(gqkv, s.d), 3 * s.hid, 3 * s.d,
                                                glogits.data_ptr(), part_gate, s.M, s.H, s.d, st));
    product_into(glogits, gate_w, gqkv, Tensor(), true);
    const Tensor gqk = parts(gqkv, 0, 2, s), gvalue = parts(gqkv, 2, 1, s);
    products_into({{gqk, qk_w, heads(gu, 0, s), true}, {gvalue, p[kV], heads(gx, 0, s)}});
    check("mlstm_conv_bwd", l::mlstm_conv_bwd(up.data_ptr(), 2 * s.hid, p[kConvW].data_ptr(), p[kConvB].data_ptr(), gu.data_ptr(), gx.data_ptr(), gup.data_ptr(), part_conv, s.B,
                                              s.T, s.hid, st));
    const Tensor small = empty_like_of(x, {cols[0] + cols[1] + cols[2]}, bf);
    const l::ColumnSum jobs[3] = {{part_out, out_rows, cols[0], nullptr, small.data_ptr()}, {part_gate, gate_rows, cols[1], nullptr, column(small, cols[0])},
                                  {part_conv, conv_rows, cols[2], nullptr, column(small, cols[0] + cols[1])}};
    check("column_sums", l::column_sums(jobs, 3, st));
    int64_t at = 0;
    const auto give = [&](int i, int64_t n) {
      grads[1 + i] = piece(small, at, p[i].sizes());
      at += n;
    };
    give(kNorm, s.hid);
    give(kSkip, s.hid);
    give(kIB, s.H);
    give(kFB, s.H);
    give(kConvW, 4 * s.hid);
    give(kConvB, s.hid);
    const Tensor ggate = empty_like_of(x, {2 * s.H, 3 * s.hid}, bf), gqk_w = empty_like_of(x, {s.H, 2 * s.d, s.d}, bf);
    for (int i : {kOut, kV, kUp}) grads[1 + i] = empty_like_of(x, p[i].sizes(), bf);
    products_into({{transposed(gup), matrix(x, s.M, s.F), grads[1 + kUp]},
                   {transposed(gy), g, grads[1 + kOut]},
                   {transposed(glogits), qkv, ggate},
                   {swapped(gqk), heads(u, 0, s), gqk_w},
                   {swapped(gvalue), heads(up, 0, s), grads[1 + kV]}});
    grads[1 + kIW] = piece(ggate, 0, {s.H, 3 * s.hid});
    grads[1 + kFW] = piece(ggate, 3ll * s.hid * s.H, {s.H, 3 * s.hid});
    grads[1 + kQ] = view_of(gqk_w, 0, {s.H, s.d, s.d}, {2 * s.d * s.d, s.d, 1});
    grads[1 + kK] = view_of(gqk_w, s.d * s.d, {s.H, s.d, s.d}, {2 * s.d * s.d, s.d, 1});
    if (ctx->needs_input_grad(0)) {
      grads[0] = empty_like_of(x, x.sizes(), bf);
      product_into(gup, p[kUp], matrix(grads[0], s.M, s.F));
    }
    if (c0.defined()) grads[first] = gc0;
    if (n0.defined()) grads[first + 1] = gn0;
    if (m0.defined()) grads[first + 2] = gm0;
    return grads;
  }
};

// -> (c (B,1,H,d,d), f (B,1,H,1,1), n (B,1,H,d,1), m (B,1,H,1,1), y (B,T,F)), or None where the caller has to compose the layer
pybind11::object mlstm_layer(const Tensor& x_in, const variable_list& p, const OptTensor& c_in, const OptTensor& f_in, const OptTensor& n_in, const OptTensor& m_in,
                             const OptTensor& done_in, double eps) {
  if (!x_in.is_cuda() || x_in.scalar_type() != at::kBFloat16 || x_in.dim() != 3 || x_in.numel() == 0 || p.size() != kParams ||
      x_in.size(0) * x_in.size(1) > 0x7fffffff || at::autocast::is_autocast_enabled(at::kCUDA) || followed(x_in, p, c_in, f_in, n_in, m_in))
    return pybind11::none();
  for (const Tensor& t : p)
    if (t.scalar_type() != at::kBFloat16 || t.device() != x_in.device() || !t.is_contiguous() || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15)) return pybind11::none();
  if (p[kQ].dim() != 3 || p[kOut].dim() != 2) return pybind11::none();
  const int64_t H = p[kQ].size(0), d = p[kQ].size(1), hid = H * d, F = x_in.size(2), out_dim = p[kOut].size(0);
  if ((d != 16 && d != 32 && d != 64) || H > 64 || hid > 2048 || 256 % (hid / 8 > 0 ? hid / 8 : 1) || x_in.size(0) * H > 0x7fffffff) return pybind11::none();
  if (!shaped(p[kUp], {2 * hid, F}) || !shaped(p[kConvW], {hid, 1, 4}) || !shaped(p[kConvB], {hid}) || !shaped(p[kQ], {H, d, d}) || !shaped(p[kK], {H, d, d}) ||
      !shaped(p[kV], {H, d, d}) || !shaped(p[kIW], {H, 3 * hid}) || !shaped(p[kIB], {H}) || !shaped(p[kFW], {H, 3 * hid}) || !shaped(p[kFB], {H}) ||
      !shaped(p[kSkip], {hid}) || !shaped(p[kNorm], {H, d}) || !shaped(p[kOut], {out_dim, hid}))
    return pybind11::none();
  const c10::cuda::CUDAGuard guard(x_in.device());
  const int64_t B = x_in.size(0);
  const Tensor x = dense(x_in), done = done_bytes(done_in, x.size(0) * x.size(1));
  const Tensor c0 = carry_leaf(c_in, B * hid * d, at::kFloat, "c0"), f0 = carry_leaf(f_in, B * H, at::kFloat, "f0"), n0 = carry_leaf(n_in, B * hid, at::kFloat, "n0"),
               m0 = carry_leaf(m_in, B * H, at::kFloat, "m0");
  bool grad = x.requires_grad();
  for (const Tensor& t : p) grad |= t.requires_grad();
  for (const Tensor& t : {c0, n0, m0}) grad |= t.defined() && t.requires_grad();
  Tensor c, f, n, m, y;
  if (at::GradMode::is_enabled() && grad) {
    const bool all = c0.defined() && n0.defined() && m0.defined(), none = !c0.defined() && !n0.defined() && !m0.defined();
    if (!all && !none) return pybind11::none();
    const variable_list out = MlstmLayer::apply(x, at::TensorList(p), opt(c0), opt(n0), opt(m0), opt(f0), opt(done), eps);
    c = out[0]; n = out[1]; m = out[2]; f = out[3]; y = out[4];
  } else {
    const Result r = forward(x, p, c0, n0, m0, f0, done, shape_of(x, p), eps, false);
    c = r.c_last; n = r.n_last; m = r.m_last; f = r.f_last; y = r.y;
  }
  return pybind11::cast(std::make_tuple(c, f, n, m, y));
}

}  // namespace

void bind_mlstm(pybind11::module_& m) { m.def("mlstm_layer", &mlstm_layer); }

}  // namespace mxk_host
