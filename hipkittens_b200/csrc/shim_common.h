// Pieces shared by the pybind11 shims: the duck-typed tensor view that mirrors
// include/pyutils/pyutils.cuh:14-47 (class name "Tensor", contiguous, not on the CPU, ndim <= 4, data_ptr();
// no libtorch is linked) with the reference's RuntimeError texts, and the error-code translation.
#pragma once

#include <pybind11/pybind11.h>

#include <array>
#include <cstdint>
#include <stdexcept>
#include <string>

#include "../../include/hk_attn.h"

namespace hk_shim {

namespace py = pybind11;

struct TensorView {
  uint64_t ptr = 0;
  std::array<int, 4> shape{1, 1, 1, 1};  // left-padded with 1s, like make_gl's (b, d, r, c)
  int device = 0;
  std::string dtype;
};

// A call looks at five to nine tensors, and reading one through generic attribute look-ups (device and dtype as Python
// objects turned into strings) took about 1.5 us. torch's own class is recognised by identity and asked through interned
// names for what needs no intermediate objects; anything else, and any such tensor that is not on a CUDA device, goes
// the general way below.
struct TorchNames {
  PyObject *is_cuda, *is_contiguous, *get_device, *shape, *data_ptr, *dtype;
  TorchNames()
      : is_cuda(PyUnicode_InternFromString("is_cuda")),
        is_contiguous(PyUnicode_InternFromString("is_contiguous")),
        get_device(PyUnicode_InternFromString("get_device")),
        shape(PyUnicode_InternFromString("shape")),
        data_ptr(PyUnicode_InternFromString("data_ptr")),
        dtype(PyUnicode_InternFromString("dtype")) {}
};

inline bool is_torch_tensor(PyObject* o) {  // exactly torch.Tensor, whose class object lives as long as the module
  static PyTypeObject* cls = nullptr;
  if (!cls) {
    py::dict modules = py::module_::import("sys").attr("modules");
    if (!modules.contains("torch")) return false;
    py::object torch = modules["torch"];
    if (!py::hasattr(torch, "Tensor")) return false;
    cls = reinterpret_cast<PyTypeObject*>(py::object(torch.attr("Tensor")).release().ptr());
  }
  return Py_TYPE(o) == cls;
}

inline py::object attr_of(PyObject* o, PyObject* name) {
  PyObject* r = PyObject_GetAttr(o, name);
  if (!r) throw py::error_already_set();
  return py::reinterpret_steal<py::object>(r);
}
inline py::object call_of(PyObject* o, PyObject* name) {
  PyObject* r = PyObject_CallMethodNoArgs(o, name);
  if (!r) throw py::error_already_set();
  return py::reinterpret_steal<py::object>(r);
}

inline bool torch_view(PyObject* o, TensorView& t) {
  static const TorchNames* names = new TorchNames();
  if (!is_torch_tensor(o) || attr_of(o, names->is_cuda).ptr() != Py_True) return false;
  if (call_of(o, names->is_contiguous).ptr() != Py_True) throw std::runtime_error("Tensor must be contiguous");
  const py::object shape = attr_of(o, names->shape);
  const Py_ssize_t dims = PyTuple_Size(shape.ptr());
  if (dims < 0) throw py::error_already_set();
  if (dims > 4) throw std::runtime_error("Expected Tensor.ndim <= 4");
  for (Py_ssize_t i = 0; i < dims; ++i)
    t.shape[4 - dims + i] = py::handle(PyTuple_GET_ITEM(shape.ptr(), i)).cast<int>();
  t.ptr = call_of(o, names->data_ptr).cast<uint64_t>();
  t.device = call_of(o, names->get_device).cast<int>();
  const py::object dtype = attr_of(o, names->dtype);
  static PyObject *bf16 = nullptr, *fp32 = nullptr;  // torch's dtype objects are never freed
  if (dtype.ptr() == bf16) t.dtype = "torch.bfloat16";
  else if (dtype.ptr() == fp32) t.dtype = "torch.float32";
  else {
    t.dtype = py::str(dtype).cast<std::string>();
    if (t.dtype == "torch.bfloat16") bf16 = dtype.ptr();
    if (t.dtype == "torch.float32") fp32 = dtype.ptr();
  }
  return true;
}

inline TensorView view_of(const py::object& obj) {
  {
    TensorView t;
    if (torch_view(obj.ptr(), t)) return t;
  }
  if (py::hasattr(obj, "__class__") && obj.attr("__class__").attr("__name__").cast<std::string>() == "Tensor") {
    if (!obj.attr("is_contiguous")().cast<bool>()) throw std::runtime_error("Tensor must be contiguous");
    if (obj.attr("device").attr("type").cast<std::string>() == "cpu")
      throw std::runtime_error("Tensor must be on CUDA device");
    TensorView t;
    auto shape = obj.attr("shape").cast<py::tuple>();
    const size_t dims = shape.size();
    if (dims > 4) throw std::runtime_error("Expected Tensor.ndim <= 4");
    for (size_t i = 0; i < dims; ++i) t.shape[4 - dims + i] = shape[i].cast<int>();
    t.ptr = obj.attr("data_ptr")().cast<uint64_t>();
    py::object idx = obj.attr("device").attr("index");
    t.device = idx.is_none() ? -1 : idx.cast<int>();
    t.dtype = py::str(obj.attr("dtype")).cast<std::string>();
    return t;
  }
  throw std::runtime_error("Expected a torch.Tensor");
}

inline void require(bool cond, const std::string& msg) {
  if (!cond) throw std::runtime_error(msg);
}

inline void raise_for(int rc, const char* what) {
  if (rc == HK_OK) return;
  std::string msg = std::string(what) + ": " + hk_strerror(rc);
  if (rc == HK_ECUDA || rc == HK_EUNSUPPORTED) {
    const char* detail = hk_last_cuda_error();
    if (detail && detail[0]) msg += std::string(" (") + detail + ")";
  }
  throw std::runtime_error(msg);
}

}  // namespace hk_shim
