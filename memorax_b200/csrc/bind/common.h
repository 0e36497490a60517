// What the native host code shares: tensor checks, streams, statuses, workspaces.
#pragma once

#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <optional>

#include "mxk.h"

namespace mxk_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

inline cudaStream_t stream() { return at::cuda::getCurrentCUDAStream().stream(); }

template <typename T = float>
inline T* ptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }
inline const uint8_t* bytes(const Tensor& t) { return t.defined() ? static_cast<const uint8_t*>(t.data_ptr()) : nullptr; }

// The per-device word that a kernel whose bounded wait gave up sets to 1.
Tensor status_word(c10::Device device);
inline int* status_ptr(const Tensor& like) { return ptr<int>(status_word(like.device())); }

// Raises memorax_b200._lib.MxkError (RuntimeError where the interpreter is not held, as in the backward pass).
void check(const char* fn, int status);
[[noreturn]] void assertion(const char* text);

// an autograd node takes what may be missing as an optional
inline OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

inline Tensor dev(const OptTensor& t, at::ScalarType dtype, const char* name) {
  if (!t || !t->defined()) return Tensor();
  TORCH_CHECK_VALUE(t->is_cuda(), name, " must be a CUDA tensor (memorax_b200 has no CPU path)");
  return (t->scalar_type() == dtype ? *t : t->to(dtype)).contiguous();
}
// (B,T) flags of any dtype -> bytes
inline Tensor done_bytes(const OptTensor& done) {
  if (!done || !done->defined()) return Tensor();
  TORCH_CHECK_VALUE(done->is_cuda(), "done must be a CUDA tensor");
  if (done->scalar_type() == at::kBool || done->scalar_type() == at::kByte) return done->contiguous();
  return done->ne(0).contiguous();
}
inline Tensor empty_like_of(const Tensor& t, at::IntArrayRef sizes, at::ScalarType dtype) {
  return at::empty(sizes, t.options().dtype(dtype).requires_grad(false));
}
inline Tensor scratch(const Tensor& t, size_t n) {
  return at::empty({static_cast<int64_t>(n ? n : 1)}, t.options().dtype(at::kByte).requires_grad(false));
}
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

}  // namespace mxk_host
