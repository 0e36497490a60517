// Dense layers in float32 on the tensor cores (gemm32.cuh), with their gradients.
#include "product.h"

#include "../gemm32.cuh"

namespace mxk_host {
namespace {

namespace g = mxk::gemm32;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// c (M, N) = a (M, K) w^T, w stored (N, K) or, transposed, (K, N)
void product32(const Tensor& a, const Tensor& w, bool transposed, const float* bias, const Tensor& c, int M, int N, int K) {
  Arena mem;
  const size_t image = mem.take(g::image_bytes(M, N, K)), ws_bytes = g::workspace_bytes(M, N, K), ws = mem.take(ws_bytes);
  mem.alloc(a);
  g::WeightJob job;
  job.w = g::weight_of(ptr(w), w.size(1));
  job.transposed = transposed;
  job.N = N; job.K = K;
  job.bn = g::tile_width(M, N, K);
  job.image = mem.at<void>(image);
  check("split_weights", g::split_weights(&job, 1, {}, stream()));
  g::Epilogue ep;
  ep.bias = bias;
  check("run_weights", g::run_weights(ptr(a), K, job.image, ptr(c), N, M, N, K, ep, mem.at(ws), ws_bytes, status_ptr(a), stream()));
}

struct Linear32 : torch::autograd::Function<Linear32> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& bias) {
    const int K = x.size(-1), N = w.size(0), M = x.numel() / K;
    auto sizes = x.sizes().vec();
    sizes.back() = N;
    const Tensor y = empty_like_of(x, sizes, at::kFloat);
    product32(x, w, false, bias ? ptr(*bias) : nullptr, y, M, N, K);
    ctx->saved_data["bias"] = bias.has_value();
    ctx->save_for_backward({x, w});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& gout) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], gy = dense(gout[0]);
    const c10::cuda::CUDAGuard guard(x.device());
    const int K = x.size(-1), N = w.size(0), M = x.numel() / K;
    variable_list grads(3);
    if (ctx->needs_input_grad(0)) {
      grads[0] = empty_like_of(x, x.sizes(), at::kFloat);
      product32(gy, w, true, nullptr, grads[0], M, K, N);
    }
    if (ctx->needs_input_grad(1)) {
      grads[1] = empty_like_of(w, w.sizes(), at::kFloat);
      const size_t ws_bytes = g::workspace_bytes(N, K, M);
      const Tensor ws = scratch(x, ws_bytes);
      check("run_outer", g::run_outer(ptr(gy), N, ptr(x), K, ptr(grads[1]), K, N, K, M, ptr(ws), ws_bytes, nullptr, status_ptr(x), stream()));
    }
    if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2)) grads[2] = gy.reshape({M, N}).sum(0);
    return grads;
  }
};

Tensor linear_f32(const Tensor& x, const Tensor& w, const OptTensor& bias) {
  const auto fits = [&](const Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kFloat && t.device() == x.device(); };
  if (!fits(x) || !fits(w) || (bias && !fits(*bias)) || w.dim() != 2 || x.size(-1) != w.size(1) || x.numel() == 0 || w.numel() == 0 ||
      x.numel() / x.size(-1) > 0x7fffffff || tf32_products() || at::autocast::is_autocast_enabled(at::kCUDA) || followed(x, {w}, bias))
    return at::linear(x, w, bias);
  const c10::cuda::CUDAGuard guard(x.device());
  return Linear32::apply(dense(x), dense(w), bias ? OptTensor(dense(*bias)) : std::nullopt);
}

// a (.., M, K) b (.., K, N) (+ bias) (+ c) in bf16 through this repository's kernel
Tensor product_bf16(const Tensor& a, const Tensor& b, const OptTensor& bias, const OptTensor& c) {
  const c10::cuda::CUDAGuard guard(a.device());
  if (!c) return product(a, b, bias.value_or(Tensor()));
  product_into(a, b, *c, bias.value_or(Tensor()), true);
  return *c;
}

// c[i] = a[i] b[i], in one launch where the kernel takes them all
void products_bf16(const std::vector<Tensor>& a, const std::vector<Tensor>& b, const std::vector<Tensor>& c) {
  const c10::cuda::CUDAGuard guard(a.at(0).device());
  std::vector<Product> products;
  for (size_t i = 0; i < a.size(); ++i) products.push_back({a[i], b.at(i), c.at(i)});
  products_into(products);
}

}  // namespace

void bind_linear(pybind11::module_& m) {
  m.def("product_bf16", &product_bf16, pybind11::arg("a"), pybind11::arg("b"), pybind11::arg("bias") = pybind11::none(), pybind11::arg("c") = pybind11::none());
  m.def("products_bf16", &products_bf16);
  m.def("linear_f32", &linear_f32, pybind11::arg("x"), pybind11::arg("w"), pybind11::arg("bias") = pybind11::none()); }

}  // namespace mxk_host
