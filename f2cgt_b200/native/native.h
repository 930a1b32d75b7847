// Helpers of the CPython module `_native`: argument unpacking, the argument checks of ops.py, error translation.
// The module is the torch side of the library's C ABI for the calls whose host time counts; it adds no computation.
#pragma once
#include <Python.h>

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/f2cgt_b200.h"

namespace f2c_native {

struct PythonError {};  // a Python exception is already set

extern PyObject* g_error_class;  // f2cgt_b200._lib.F2CError

[[noreturn]] inline void fail(PyObject* type, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  PyErr_FormatV(type, fmt, ap);
  va_end(ap);
  throw PythonError{};
}

inline void check_status(int rc) {
  if (rc == F2C_OK) return;
  static const char* names[] = {"ok", "invalid argument", "unsupported", "CUDA error", "size limit"};
  fail(g_error_class ? g_error_class : PyExc_RuntimeError, "f2cgt_b200: %s: %s", rc > 0 && rc < 5 ? names[rc] : "error", f2c_last_error());
}

inline int dtype_tag(at::ScalarType t) {
  switch (t) {
    case at::kByte: return F2C_U8;
    case at::kChar: return F2C_I8;
    case at::kShort: return F2C_I16;
    case at::kInt: return F2C_I32;
    case at::kLong: return F2C_I64;
    case at::kHalf: return F2C_F16;
    case at::kFloat: return F2C_F32;
    case at::kDouble: return F2C_F64;
    default: return -1;
  }
}
constexpr unsigned bit(int tag) { return 1u << tag; }
constexpr unsigned kCodes = bit(F2C_U8) | bit(F2C_I8) | bit(F2C_I16), kIndex = bit(F2C_I32) | bit(F2C_I64), kF32 = bit(F2C_F32);

// a contiguous CUDA tensor of one of `allowed` dtypes
inline const at::Tensor& tensor(PyObject* o, const char* name, unsigned allowed) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "%s must be a torch.Tensor", name);
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda()) fail(PyExc_RuntimeError, "%s must be a CUDA tensor", name);
  if (!t.is_contiguous()) fail(PyExc_RuntimeError, "%s must be contiguous", name);
  const int tag = dtype_tag(t.scalar_type());
  if (tag < 0 || !(allowed & bit(tag))) fail(PyExc_RuntimeError, "%s has unsupported dtype %s", name, c10::toString(t.scalar_type()));
  return t;
}

inline int64_t integer(PyObject* o) {
  if (PyLong_Check(o)) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PythonError{};
    return v;
  }
  PyObject* i = PyNumber_Index(o);  // numpy integers and the like
  if (i == nullptr) throw PythonError{};
  const long long v = PyLong_AsLongLong(i);
  Py_DECREF(i);
  if (v == -1 && PyErr_Occurred()) throw PythonError{};
  return v;
}

inline double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PythonError{};
  return v;
}

inline cudaStream_t stream_of(const at::Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

inline at::Tensor empty(at::IntArrayRef size, at::ScalarType dtype, const at::Device& device) {
  return at::detail::empty_cuda(size, dtype, device, c10::nullopt);
}

// Runs `body`, which returns a new reference, and turns what it throws into a Python exception.
template <typename F>
inline PyObject* guarded(F&& body) {
  try {
    return body();
  } catch (const PythonError&) {
  } catch (python_error& e) {  // out of a Python hook that torch called
    e.restore();
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// Runs `body` without the interpreter lock: an allocation may wait for the device, a launch for a place in its stream's queue, and
// other Python threads (a loader's, a server's) go on meanwhile.  `body` may throw; it touches no Python object.
template <typename F>
inline auto unlocked(F&& body) {
  struct Released {
    PyThreadState* state = PyEval_SaveThread();
    ~Released() { PyEval_RestoreThread(state); }
  } released;
  return body();
}


extern PyMethodDef g_sage_methods[], g_loader_methods[];  // sage.cpp, loader.cpp

void arguments(const char* name, Py_ssize_t got, Py_ssize_t want);

}  // namespace f2c_native
