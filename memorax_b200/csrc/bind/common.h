// What the native host code shares: tensor checks, streams, statuses, workspaces.
#pragma once

#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <optional>

#include "mxk.h"

namespace mxk_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

inline cudaStream_t stream() { return at::cuda::getCurrentCUDAStream().stream(); }

template <typename T = float>
inline T* ptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }
// A trace would hold a native call's results as constants, and forward-mode tangents end at one: such calls are composed, and
// the autograd functions they are composed of refuse them.
inline bool followed(const Tensor& t) { return t.defined() && t._fw_grad(0).defined(); }
inline bool followed(const OptTensor& t) { return t && followed(*t); }
template <typename... T>
inline bool followed(const Tensor& x, at::ArrayRef<Tensor> params, const T&... carry) {
  if (torch::jit::tracer::isTracing()) return true;
  if (!torch::autograd::ForwardADLevel::try_get_by_idx(0)) return false;   // (nobody has tangents)
  if (followed(x) || (followed(carry) || ...)) return true;
  for (const Tensor& p : params)
    if (followed(p)) return true;
  return false;
}
// Float32 products in TF32 were asked for, by either of torch's settings (its query of the older one raises where only the
// newer one was used).
inline bool tf32_products() {
  return at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL) == at::Float32Precision::TF32;
}
// What kernels with 16-byte accesses ask of a tensor that a caller brings (one cut out of a larger buffer may start anywhere).
inline bool aligned16(const Tensor& t) { return !t.defined() || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
inline const uint8_t* bytes(const Tensor& t) { return t.defined() ? static_cast<const uint8_t*>(t.data_ptr()) : nullptr; }

// The per-device word that a kernel whose bounded wait gave up sets to 1.
Tensor status_word(c10::Device device);
inline int* status_ptr(const Tensor& like) { return ptr<int>(status_word(like.device())); }

// Raises memorax_b200._lib.MxkError (RuntimeError where the interpreter is not held, as in the backward pass).
void check(const char* fn, int status);
[[noreturn]] void assertion(const char* text);

// an autograd node takes what may be missing as an optional
inline OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

// Dense memory that holds the values themselves: a conjugated (negated) view is a bit on the same memory, contiguous or not.
inline Tensor dense(const Tensor& t) { return (t.is_conj() || t.is_neg() ? t.resolve_conj().resolve_neg() : t).contiguous(); }
inline Tensor dev(const OptTensor& t, at::ScalarType dtype, const char* name) {
  if (!t || !t->defined()) return Tensor();
  TORCH_CHECK_VALUE(t->is_cuda(), name, " must be a CUDA tensor (memorax_b200 has no CPU path)");
  return dense(t->scalar_type() == dtype ? *t : t->to(dtype));
}
// (B,T) flags of any dtype -> bytes
inline Tensor done_bytes(const OptTensor& done, int64_t steps) {
  if (!done || !done->defined()) return Tensor();
  TORCH_CHECK_VALUE(done->is_cuda(), "done must be a CUDA tensor");
  TORCH_CHECK_VALUE(done->numel() == steps, "done has ", done->numel(), " flags for ", steps, " steps");
  if (done->scalar_type() == at::kBool || done->scalar_type() == at::kByte) return done->contiguous();
  return done->ne(0).contiguous();
}
// Allocations and views of buffers that no graph tracks, without a trip through the dispatcher (1-2 us each, and a layer
// has tens of them).
inline Tensor empty_like_of(const Tensor& t, at::IntArrayRef sizes, at::ScalarType dtype) {
  return Tensor(at::detail::empty_cuda(sizes, dtype, t.device(), std::nullopt));
}
inline Tensor scratch(const Tensor& t, size_t n) { return empty_like_of(t, {static_cast<int64_t>(n ? n : 1)}, at::kByte); }
inline Tensor view_of(const Tensor& t, int64_t offset, at::IntArrayRef sizes, at::IntArrayRef strides) {
  Tensor v = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(t.storage()), t.key_set(), t.dtype());
  v.unsafeGetTensorImpl()->set_storage_offset(t.storage_offset() + offset);
  v.unsafeGetTensorImpl()->set_sizes_and_strides(sizes, strides);
  return v;
}
// (rows, cols) at an element offset, and the same transposed
inline Tensor matrix(const Tensor& t, int64_t rows, int64_t cols, int64_t ld = 0, int64_t offset = 0) {
  return view_of(t, offset, {rows, cols}, {ld ? ld : cols, 1});
}
inline Tensor transposed(const Tensor& t) { return view_of(t, 0, {t.size(1), t.size(0)}, {t.stride(1), t.stride(0)}); }
// contiguous, `sizes` at an element offset
inline Tensor piece(const Tensor& t, int64_t offset, at::IntArrayRef sizes) {
  c10::SmallVector<int64_t, 6> strides(sizes.size(), 1);
  for (int i = static_cast<int>(sizes.size()) - 2; i >= 0; --i) strides[i] = strides[i + 1] * sizes[i + 1];
  return view_of(t, offset, sizes, strides);
}
// A leaf of the carry with its singleton time axis kept: (B, 1, ...) and (B, ...) are the same memory.
inline Tensor carry_leaf(const OptTensor& t, int64_t numel, at::ScalarType dtype, const char* name) {
  if (!t || !t->defined()) return Tensor();
  const Tensor leaf = dev(t->dim() > 1 && t->size(1) != 1 ? t->narrow(1, 0, 1) : *t, dtype, name);
  TORCH_CHECK_VALUE(leaf.numel() == numel, name, " of the carry has ", leaf.numel(), " elements, expected ", numel);
  return leaf;
}
// the last step of contiguous states (B, T, N)
inline Tensor last_state(const Tensor& h) {
  const int64_t B = h.size(0), T = h.size(1), N = h.size(2);
  return view_of(h, (T - 1) * N, {B, 1, N}, {T * N, N, 1});
}
inline bool shaped(const Tensor& t, at::IntArrayRef sizes) { return t.sizes() == sizes; }
inline size_t align_up(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

// One allocation cut into 256-byte aligned pieces.
struct Arena {
  size_t used = 0;
  uint8_t* base = nullptr;
  Tensor buf;
  size_t take(size_t n) { const size_t at = used; used += align_up(n); return at; }
  void alloc(const Tensor& like) { buf = scratch(like, used); base = ptr<uint8_t>(buf); }
  template <typename T = float> T* at(size_t off) const { return reinterpret_cast<T*>(base + off); }
};

void bind_attention(pybind11::module_& m);
void bind_linrec(pybind11::module_& m);
void bind_linear(pybind11::module_& m);
void bind_lru(pybind11::module_& m);
void bind_mamba(pybind11::module_& m);
void bind_mingru(pybind11::module_& m);
void bind_mlstm(pybind11::module_& m);
void bind_modules(pybind11::module_& m);

}  // namespace mxk_host
