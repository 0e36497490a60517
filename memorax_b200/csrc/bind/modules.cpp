// What nn.Module holds for the native layers: parameters, and whether a module's call is its class's forward and nothing else.
// Dictionary lookups in place of attribute lookups through nn.Module, which take as long as an acting step's launches
// (parameters of a linear-attention cell: 1.9 us in Python).
#include "common.h"

namespace mxk_host {
namespace {

namespace py = pybind11;

// interned once, for the life of the process
PyObject* name_of(const char* text) { return PyUnicode_InternFromString(text); }

py::object own_dict(PyObject* module) {
  PyObject* const dict = PyObject_GenericGetDict(module, nullptr);
  if (!dict) throw py::error_already_set();
  return py::reinterpret_steal<py::object>(dict);
}
// borrowed; null where there is none
PyObject* entry(PyObject* dict, PyObject* key) {
  PyObject* const value = PyDict_Check(dict) ? PyDict_GetItemWithError(dict, key) : nullptr;
  if (!value && PyErr_Occurred()) throw py::error_already_set();
  return value == Py_None ? nullptr : value;
}

bool any_global_hook() {
  static PyObject* const fn = py::object(py::module_::import("torch.nn.modules.module").attr("_has_any_global_hook")).release().ptr();
  const py::object hooks = py::reinterpret_steal<py::object>(PyObject_CallNoArgs(fn));
  const int some = hooks ? PyObject_IsTrue(hooks.ptr()) : -1;
  if (some < 0) throw py::error_already_set();
  return some != 0;
}
bool has_hooks(PyObject* dict) {
  static PyObject* const names[] = {name_of("_forward_hooks"), name_of("_forward_pre_hooks"), name_of("_backward_hooks"), name_of("_backward_pre_hooks")};
  for (PyObject* name : names)
    if (PyObject* const hooks = entry(dict, name)) {
      const int some = PyObject_IsTrue(hooks);
      if (some < 0) throw py::error_already_set();
      if (some) return true;
    }
  return false;
}
// The module's dictionary, or an empty object where it is not exactly a `kind` without hooks and without a forward of its own
// (weight norm and pruning are hooks too).
py::object plain_dict(PyObject* module, PyObject* kind) {
  static PyObject* const forward = name_of("forward");
  if (reinterpret_cast<PyObject*>(Py_TYPE(module)) != kind) return {};
  py::object dict = own_dict(module);
  return has_hooks(dict.ptr()) || entry(dict.ptr(), forward) ? py::object() : dict;
}

// Whether calling `module` runs kind.forward and nothing else; only such a module may be called through its parts.
bool plain(py::handle module, py::handle kind) { return plain_dict(module.ptr(), kind.ptr()) && !any_global_hook(); }

// The parameters that the native layer of a `kind` takes, or None where the layer has to be composed: the cell or one of its
// submodules is not plain, or has other parameters than these.  spec names them in order: (submodule or None for the cell's
// own, its class, names).
py::object native_params(py::handle cell, py::handle kind, const py::tuple& spec) {
  static PyObject* const modules = name_of("_modules");
  static PyObject* const parameters = name_of("_parameters");
  const py::object own = plain_dict(cell.ptr(), kind.ptr());
  if (!own || any_global_hook()) return py::none();
  py::list out;
  for (const py::handle item : spec) {
    PyObject *const sub = PyTuple_GetItem(item.ptr(), 0), *const sub_kind = PyTuple_GetItem(item.ptr(), 1), *const names = PyTuple_GetItem(item.ptr(), 2);
    if (!sub || !sub_kind || !names || !PyTuple_Check(names)) throw py::value_error("spec: (submodule, class, names)");
    py::object dict = own;
    if (sub != Py_None) {
      PyObject* const subs = entry(own.ptr(), modules);
      PyObject* const module = subs ? entry(subs, sub) : nullptr;
      if (!module || !(dict = plain_dict(module, sub_kind))) return py::none();
    }
    PyObject* const params = entry(dict.ptr(), parameters);
    if (!params) return py::none();
    if (sub != Py_None) {   // (such as a bias that the cell was not built with)
      PyObject *name, *param;
      for (Py_ssize_t at = 0; PyDict_Next(params, &at, &name, &param);) {
        const int known = param == Py_None ? 1 : PySequence_Contains(names, name);
        if (known < 0) throw py::error_already_set();
        if (!known) return py::none();
      }
    }
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(names); ++i) {
      PyObject* const param = entry(params, PyTuple_GET_ITEM(names, i));
      if (!param) return py::none();
      out.append(py::reinterpret_borrow<py::object>(param));
    }
  }
  return std::move(out);
}

}  // namespace

void bind_modules(py::module_& m) {
  m.def("plain", &plain);
  m.def("native_params", &native_params);
}

}  // namespace mxk_host
