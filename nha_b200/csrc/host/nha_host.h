// Shared pieces of the host module: argument access, errors, allocation.
//
// The operators' host side lives in C++ because the calls it makes are shorter than the Python that used to make them:
// a decode step is 4-20 us on the GPU, and checking arguments, allocating the output and crossing into the library
// through ctypes took 45 us per call.
#pragma once

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <stdlib.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <initializer_list>
#include <string>

#include "../../../include/nha_b200.h"

namespace nha_host {

using at::Tensor;

extern PyObject* library_error;      // nha_b200._lib.NHALibraryError, set when the module is loaded

// Raises a Python exception from any thread (the backward runs on autograd's threads, without the GIL).
[[noreturn]] inline void raise(PyObject* type, const std::string& msg) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(type, msg.c_str());
  python_error e;
  e.persist();
  throw e;
}
inline void require(bool ok, const char* msg) {
  if (C10_UNLIKELY(!ok)) raise(PyExc_AssertionError, msg);
}
inline void check(int status, const char* what) {
  if (C10_LIKELY(status == NHA_OK)) return;
  std::string m = std::string(what) + ": " + nha_status_string(status);
  const char* detail = nha_last_cuda_error();
  if (status == NHA_ERR_LAUNCH && detail && detail[0]) m += std::string(" [") + detail + "]";
  raise(library_error, m);
}

// Every kernel reads raw pointers of one device: a tensor of another device (or of the host) is refused here, before a launch.
inline void same_device(const Tensor& like, std::initializer_list<const Tensor*> rest, const char* what) {
  if (C10_UNLIKELY(!like.is_cuda())) raise(PyExc_AssertionError, std::string(what) + " runs on the CUDA library only (there is no CPU path)");
  for (const Tensor* t : rest)
    if (C10_UNLIKELY(t->defined() && t->device() != like.device()))
      raise(PyExc_AssertionError, std::string(what) + ": the tensors must be on one device, got " + like.device().str() + " and " + t->device().str());
}

// NHA_B200_CHECK=1: the operators read the kernels' device error word after every call (not under stream capture)
inline bool check_device_words() {
  const char* e = getenv("NHA_B200_CHECK");
  if (!e || e[0] != '1' || e[1]) return false;
  return c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None;
}

inline void* stream_of(const Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

inline Tensor empty(at::IntArrayRef size, at::ScalarType dt, const Tensor& like) {
  return at::detail::empty_cuda(size, dt, like.device(), std::nullopt);
}
inline Tensor empty_same(const Tensor& t) { return empty(t.sizes(), t.scalar_type(), t); }
inline Tensor zeros(at::IntArrayRef size, at::ScalarType dt, const Tensor& like) { return empty(size, dt, like).zero_(); }

// contiguous bf16 copies are made only when the tensor is something else
inline Tensor bf16c(const Tensor& x) {
  if (C10_LIKELY(x.scalar_type() == at::kBFloat16 && x.is_contiguous())) return x;
  return x.to(at::kBFloat16).contiguous();
}
inline Tensor typed(const Tensor& x, at::ScalarType dt) {
  if (C10_LIKELY(x.scalar_type() == dt && x.is_contiguous())) return x;
  return x.to(dt).contiguous();
}
// The kernels load and copy 16 bytes at a time: a contiguous view that starts elsewhere is copied.
inline bool on_16_bytes(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
inline Tensor on_16(Tensor t) {
  if (C10_LIKELY(on_16_bytes(t))) return t;
  return t.clone();
}
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

inline const Tensor& tensor(PyObject* o, const char* name) {
  if (C10_UNLIKELY(!THPVariable_Check(o))) raise(PyExc_TypeError, std::string(name) + " must be a tensor");
  return THPVariable_Unpack(o);
}
inline Tensor tensor_or_none(PyObject* o, const char* name) { return o == Py_None ? Tensor() : tensor(o, name); }
inline long integer(PyObject* o) {
  const long v = PyLong_Check(o) ? PyLong_AsLong(o) : (PyNumber_Check(o) ? [&] {
    PyObject* n = PyNumber_Long(o);
    if (!n) throw python_error();
    const long r = PyLong_AsLong(n);
    Py_DECREF(n);
    return r;
  }() : (raise(PyExc_TypeError, "an integer is required"), 0L));
  if (C10_UNLIKELY(v == -1 && PyErr_Occurred())) throw python_error();
  return v;
}
inline double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (C10_UNLIKELY(v == -1.0 && PyErr_Occurred())) throw python_error();
  return v;
}
inline bool truth(PyObject* o) { return o == Py_True || (o != Py_False && PyObject_IsTrue(o) == 1); }
inline PyObject* none() { Py_RETURN_NONE; }
inline PyObject* wrap(const Tensor& t) { return t.defined() ? THPVariable_Wrap(t) : none(); }
// a tuple or list of the given values (references are stolen)
inline PyObject* tuple(std::initializer_list<PyObject*> v) {
  PyObject* t = PyTuple_New((Py_ssize_t)v.size());
  Py_ssize_t i = 0;
  for (PyObject* x : v) PyTuple_SET_ITEM(t, i++, x);
  return t;
}
// (a, b) of an `initial_state` argument: undefined tensors for None and for (None, None)
inline void state_pair(PyObject* o, Tensor& a, Tensor& b) {
  if (o == Py_None) return;
  PyObject* f = PySequence_Fast(o, "initial_state must be a pair of tensors");
  if (!f) throw python_error();
  struct Held { PyObject* p; ~Held() { Py_DECREF(p); } } held{f};
  if (PySequence_Fast_GET_SIZE(f) != 2) raise(PyExc_ValueError, "initial_state must be a pair of tensors");
  a = tensor_or_none(PySequence_Fast_GET_ITEM(f, 0), "initial_state[0]");
  b = tensor_or_none(PySequence_Fast_GET_ITEM(f, 1), "initial_state[1]");
  if (C10_UNLIKELY(a.defined() != b.defined())) raise(PyExc_TypeError, "initial_state must be a pair of tensors");
}

#define NHA_METHOD(name_) PyObject* name_(PyObject*, PyObject* const* args, Py_ssize_t nargs)
#define NHA_BEGIN(n_)                                                                   \
  HANDLE_TH_ERRORS                                                                      \
  if (nargs != (n_)) nha_host::raise(PyExc_TypeError, "wrong number of arguments");
#define NHA_END END_HANDLE_TH_ERRORS

NHA_METHOD(decode);
NHA_METHOD(decode_logits);
NHA_METHOD(decode_ring);
NHA_METHOD(decode_workspace_for);
NHA_METHOD(chunk_nha);
NHA_METHOD(prefill);
NHA_METHOD(slot_gates);
NHA_METHOD(rotary_pair);
NHA_METHOD(feature_maps);
NHA_METHOD(silu_rms_norm);
NHA_METHOD(gsa_aux_loss);

// Zero-initialised scratch of the split decode kernels, one per (device, stream, B * H): the kernels leave their counters
// at zero, so later calls on the same stream use it again (the layout depends on B * H).  A bounded number is kept.
Tensor decode_workspace(const Tensor& like, int B, int HQ, int H, int V, int W);

}  // namespace nha_host
