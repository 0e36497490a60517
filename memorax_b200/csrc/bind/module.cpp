// memorax_b200._C: the host side of the hot calls in native code (allocation, checks, launches, autograd nodes).
#include "common.h"

#include <mutex>

namespace mxk_host {

Tensor status_word(c10::Device device) {
  static std::mutex mutex;
  static auto* words = new std::array<Tensor, 64>();   // never destroyed: the driver may be gone by then
  const int index = device.has_index() ? device.index() : c10::cuda::current_device();
  std::lock_guard<std::mutex> lock(mutex);
  Tensor& word = words->at(index);
  if (!word.defined()) word = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, index));
  return word;
}

void check(const char* fn, int status) {
  if (status == 0) return;
  if (PyGILState_Check()) pybind11::module_::import("memorax_b200._lib").attr("check")(fn, status);
  TORCH_CHECK(false, fn, " failed with status ", status, ": ", mxk_status_string(status));
}

void assertion(const char* text) {
  PyErr_SetString(PyExc_AssertionError, text);
  throw pybind11::error_already_set();
}

}  // namespace mxk_host

PYBIND11_MODULE(_C, m) {
  using namespace mxk_host;
  m.def("status_word", [](const std::string& device) { return status_word(c10::Device(device)); });
  bind_attention(m);
  bind_linrec(m);
  bind_linear(m);
  bind_lru(m);
  bind_mamba(m);
  bind_mingru(m);
  bind_mlstm(m);
  bind_modules(m);
}
