// The bare diagonal recurrences.
#include "common.h"

namespace mxk_host {
namespace {

std::tuple<Tensor, OptTensor> linrec_fwd(const Tensor& a_in, const Tensor& b_in, const OptTensor& h0_in, const OptTensor& a0_in,
                                         const OptTensor& done_in, bool want_decay) {
  const bool cplx = b_in.is_complex();
  const auto dt = cplx ? at::kComplexFloat : at::kFloat;
  const Tensor b = dev(b_in, dt, "b"), a = dev(a_in, dt, "a"), h0 = dev(h0_in, dt, "h0"), a0 = dev(a0_in, dt, "a0");
  const c10::cuda::CUDAGuard guard(b.device());
  TORCH_CHECK_VALUE(b.dim() == 3, "b must be (B, T, D)");
  const Tensor done = done_bytes(done_in, b.size(0) * b.size(1));
  const int64_t bsz = b.size(0), steps = b.size(1), dim = b.size(2);
  const bool tinv = a.dim() == 1;
  if (tinv ? a.size(0) != dim : a.sizes() != b.sizes()) assertion("a must be (D,) or of b's shape");
  const Tensor h = empty_like_of(b, b.sizes(), dt);
  const Tensor a_last = want_decay ? empty_like_of(b, {bsz, dim}, dt) : Tensor();
  const auto fn = cplx ? mxk_linrec_c64_fwd : mxk_linrec_f32_fwd;
  check(cplx ? "mxk_linrec_c64_fwd" : "mxk_linrec_f32_fwd",
        fn(ptr(a), tinv, ptr(b), ptr(h0), ptr(a0), bytes(done), ptr(h), ptr(a_last), bsz, steps, dim, stream()));
  return {h, want_decay ? OptTensor(a_last) : std::nullopt};
}

}  // namespace

void bind_linrec(pybind11::module_& m) { m.def("linrec_fwd", &linrec_fwd); }

}  // namespace mxk_host
