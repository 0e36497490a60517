// bf16 products of the native layers: this repository's kernel (gemm16.cuh) where a library call's host time counts, the
// library where the product is large.
#pragma once

#include "common.h"

#include "../gemm16.cuh"

namespace mxk_host {

// 2 M N K above which a product is the library's.  On the GPU its two-SM tiles are the faster form at nearly every size
// (by 1.1 to 1.6, up to 3.4 for weight gradients); below the line a pass waits for the host, which a library call holds up for
// longer.
// Passes with gradients, with the line at 4e9 | 8e9 | 2e10, in microseconds: linear attention (4 heads of 64), 8192 x 512: 185 | 160 | 159;
// 16384 x 512: 199 | 185 | 169; 32768 x 512: 266 | 266 | 274; 65536 x 512: 447 | 448 | 470.  Delta rule, 8192 x 512, 4 heads of 128:
// 252 | 245 | 251; 32768 x 256, 4 heads of 64: 329 | 333 | 343.  mLSTM, 6016 x 256: 237 | 239 | 237; 16384 x 512: 840 | 835 | 840;
// 65536 x 256: 1338 | 1404 | 1408; 65536 x 512: 2621 | 2613 | 2733.
constexpr double kLibraryFlops = 8e9;
// The same for the gradient of a weight, whose long contraction the kernel splits over all SMs (GPU time alone, own | library in
// microseconds): 256 x 256 over 65536 tokens 14 | 25, 768 x 256 over 32768 18 | 20, 512 x 512 over 32768 22 | 27, 1024 x 512 over 16384
// 22 | 23, 128 x 1024 over 65536 32 | 32; beyond, 768 x 256 over 65536 37 | 32, 1024 x 512 over 32768 46 | 33.
constexpr double kLibraryFlopsGradient = 1.75e10;
// 2 M N K above which a product that is no gradient has a launch of its own: the tiles of a joint one are 64 columns wide, which costs more
// than a launch from here on (together | apart in microseconds, two products into the rows of the mLSTM layer's heads, forward and backward, with
// the larger one's operations: 4e8 8.7 | 10.4 and 7.4 | 9.4, 8e8 14.7 | 13.1 and 11.9 | 11.2, 1e9 19.3 | 15.6 and 13.5 | 13.2, 4.3e9 68 | 45 and
// 47 | 37).  Gradients of weights are split over the SMs anyway: together at all sizes that are the kernel's (the layer's five, 6000 tokens of
// 256 features 16 | 41, 16384 of 512 77 | 87, 65536 of 256 110 | 119).
constexpr double kGroupFlops = 6e8;

// A product over the last two dimensions as the kernel's job; `fits`: whether it is one for the kernel.
struct AsJob {
  mxk::gemm16::Job job;
  bool a_rows, b_rows, fits;
  double flops;
};
inline AsJob as_job(const Tensor& a, const Tensor& b, const Tensor& c, const Tensor& bias, bool accumulate) {
  namespace g = mxk::gemm16;
  const int n = static_cast<int>(c.dim()), r = n - 2, q = n - 1;
  const int64_t batch = n == 3 ? c.size(0) : 1, M = c.size(r), N = c.size(q), K = a.size(q);
  const auto rows_of = [&](const Tensor& t, bool& by_rows, bool k_is_col) {
    // stored row-major along whichever index is contiguous
    const bool row_major = t.stride(q) == 1;
    by_rows = row_major != k_is_col;
    return g::Matrix{t.data_ptr(), row_major ? t.stride(r) : t.stride(q), n == 3 ? t.stride(0) : 0};
  };
  AsJob j;
  const g::Matrix ma = rows_of(a, j.a_rows, true), mb = rows_of(b, j.b_rows, false);
  const auto fits = [&](const Tensor& t, const g::Matrix& m) {
    return (t.stride(r) == 1 || t.stride(q) == 1) && m.ld % 8 == 0 && m.batch_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(m.ptr) & 15) == 0;
  };
  j.flops = 2.0 * batch * M * N * K;
  j.fits = j.flops <= (j.a_rows && j.b_rows ? kLibraryFlopsGradient : kLibraryFlops) && fits(a, ma) && fits(b, mb) && c.stride(q) == 1;
  j.job = {ma, mb, bias.defined() ? bias.data_ptr() : nullptr, c.data_ptr(), c.stride(r), n == 3 ? c.stride(0) : 0, accumulate,
           static_cast<int>(batch), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K)};
  return j;
}

// c = a b (+ bias) (+ c when `accumulate`) over the last two dimensions; a (M, K), b (K, N), c (M, N), or the same with a
// leading batch dimension: any views whose rows or columns are contiguous.
inline void product_into(const Tensor& a, const Tensor& b, const Tensor& c, const Tensor& bias = Tensor(), bool accumulate = false) {
  namespace g = mxk::gemm16;
  const int n = static_cast<int>(c.dim());
  if (const AsJob j = as_job(a, b, c, bias, accumulate); j.fits) {
    const size_t bytes = g::workspace_bytes(j.job.batch, j.job.M, j.job.N, j.job.K);
    const Tensor ws = bytes ? scratch(c, bytes) : Tensor();
    check("gemm16", g::run(j.job, j.a_rows, j.b_rows, ptr<void>(ws), bytes, status_ptr(c), stream()));
    return;
  }
  Tensor out = c;
  if (n == 3) {
    if (accumulate) at::baddbmm_out(out, c, a, b);
    else at::bmm_out(out, a, b);
  } else if (accumulate) {
    at::addmm_out(out, c, a, b);
  } else if (bias.defined()) {
    at::addmm_out(out, bias, a, b);
  } else {
    at::mm_out(out, a, b);
  }
}
// Products that do not depend on one another: one launch where all of them are the kernel's, stored alike, and short or gradients.
struct Product {
  Tensor a, b, c;
  bool accumulate = false;
};
inline void products_into(const std::vector<Product>& products) {
  namespace g = mxk::gemm16;
  g::Job jobs[g::kMaxGroup];
  int count = 0;
  bool a_rows = false, b_rows = false, together = products.size() <= g::kMaxGroup;
  for (const Product& p : products) {
    if (!together) break;
    const AsJob j = as_job(p.a, p.b, p.c, Tensor(), p.accumulate);
    together = j.fits && (j.flops <= kGroupFlops || (j.a_rows && j.b_rows)) && (count == 0 || (j.a_rows == a_rows && j.b_rows == b_rows));
    a_rows = j.a_rows;
    b_rows = j.b_rows;
    jobs[count++] = j.job;
  }
  if (!together) {
    for (const Product& p : products) product_into(p.a, p.b, p.c, Tensor(), p.accumulate);
    return;
  }
  const size_t bytes = g::group_workspace_bytes(jobs, count);
  const Tensor& like = products.front().c;
  const Tensor ws = bytes ? scratch(like, bytes) : Tensor();
  check("gemm16 group", g::run_group(jobs, count, a_rows, b_rows, ptr<void>(ws), bytes, status_ptr(like), stream()));
}
inline Tensor product(const Tensor& a, const Tensor& b, const Tensor& bias = Tensor()) {
  auto sizes = a.sizes().vec();
  sizes.back() = b.size(-1);
  const Tensor c = empty_like_of(a, sizes, at::kBFloat16);
  product_into(a, b, c, bias);
  return c;
}

}  // namespace mxk_host
