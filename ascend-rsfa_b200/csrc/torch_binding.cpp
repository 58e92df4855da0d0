// The ordinary attention() call from PyTorch in native code: check the tensors, allocate the result, find the
// current stream, call rsfa_fwd.  The same steps in Python (flash_attention_forward.py, _forward) take 10 us of
// the host's time per call, three times what the launch itself takes, which is what a call of a few heads or
// of a short sequence costs its caller; here they take about 1.5 us.
//
// forward() answers only for the ordinary case and returns None for everything else - tensors to copy first,
// empty ones, another device than the current one, subclasses, dispatch or function modes, transforms,
// tracing, argument types other than the plain ones, anything to refuse - and the Python code decides then.
// So nothing is accepted, refused or seen by a mode differently than without this file.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/rsfa.h"

namespace {

// rsfa_fwd of the library that the Python side has loaded (bind() hands its address over).
using FwdFn = decltype(&rsfa_fwd);
FwdFn g_fwd = nullptr;

bool plain_mode() {
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerBackMode) &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Functionalize) &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Tracer) &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::VmapMode);
}

// A dense CUDA tensor that rsfa_fwd can take as it is: unit innermost stride, the others multiples of eight
// elements, a 16-byte aligned base.
bool plain_tensor(PyObject* obj) {
  if (!THPVariable_CheckExact(obj)) return false;
  const at::Tensor& t = THPVariable_Unpack(obj);
  const c10::DispatchKeySet wrapped({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                     c10::DispatchKey::Batched, c10::DispatchKey::Functionalize, c10::DispatchKey::Negative,
                                     c10::DispatchKey::Conjugate, c10::DispatchKey::ZeroTensor, c10::DispatchKey::Python});
  if (!t.defined() || t.key_set().has_any(wrapped) || t.layout() != c10::kStrided || !t.is_cuda() || t.dim() != 4 ||
      !t.has_storage())
    return false;
  if (t.scalar_type() != at::kHalf && t.scalar_type() != at::kBFloat16) return false;
  const int64_t D = t.size(3);
  if (t.stride(3) != 1 || (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) != 0) return false;
  for (int i = 0; i < 3; ++i)
    if (t.size(i) > 1 && (t.stride(i) % 8 != 0 || t.stride(i) < D)) return false;
  return true;
}

bool plain_int(PyObject* obj, int* out) {
  if (!PyLong_CheckExact(obj)) return false;
  int overflow = 0;
  const long long v = PyLong_AsLongLongAndOverflow(obj, &overflow);
  if (overflow != 0 || v < INT32_MIN || v > INT32_MAX) return false;
  *out = static_cast<int>(v);
  return true;
}

// forward(q, k, v, causal, sm_scale, block_m, block_n, want_lse) -> (o, lse or None), an error code of
// rsfa_fwd (int), or None where this is not the ordinary case.
PyObject* forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int block_m = 0, block_n = 0;
  if (g_fwd == nullptr || n != 8 || !plain_mode() || !plain_tensor(args[0]) || !plain_tensor(args[1]) ||
      !plain_tensor(args[2]) || !PyBool_Check(args[3]) || !PyFloat_CheckExact(args[4]) || !plain_int(args[5], &block_m) ||
      !plain_int(args[6], &block_n) || !PyBool_Check(args[7]))
    Py_RETURN_NONE;
  const at::Tensor& q = THPVariable_Unpack(args[0]);
  const at::Tensor& k = THPVariable_Unpack(args[1]);
  const at::Tensor& v = THPVariable_Unpack(args[2]);
  const int64_t D = q.size(3);
  if (!(D == 16 || D == 32 || D == 64 || D == 128 || D == 256) || q.sizes() != k.sizes() || q.sizes() != v.sizes() ||
      q.numel() == 0 || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type() ||
      k.device() != q.device() || v.device() != q.device() || q.device().index() != c10::cuda::current_device() ||
      q.size(0) > INT32_MAX || q.size(1) > INT32_MAX || q.size(2) > INT32_MAX)
    Py_RETURN_NONE;

  at::Tensor o = at::empty_like(q);
  bool fits = o.stride(3) == 1;
  for (int i = 0; i < 3; ++i) fits = fits && (o.size(i) == 1 || o.stride(i) % 8 == 0);
  if (!fits) o = at::empty(q.sizes(), q.options());
  at::Tensor lse;
  if (args[7] == Py_True) lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));

  int64_t strides[16];
  const at::Tensor* all[4] = {&q, &k, &v, &o};
  for (int t = 0; t < 4; ++t)
    for (int i = 0; i < 4; ++i) strides[4 * t + i] = all[t]->stride(i);
  const void* qp = q.const_data_ptr();
  const void* kp = k.const_data_ptr();
  const void* vp = v.const_data_ptr();
  void* op = o.mutable_data_ptr();
  float* lp = lse.defined() ? static_cast<float*>(lse.mutable_data_ptr()) : nullptr;
  void* stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  const float scale = static_cast<float>(PyFloat_AS_DOUBLE(args[4]));
  const int dtype = q.scalar_type() == at::kBFloat16 ? RSFA_DTYPE_BF16 : RSFA_DTYPE_F16;
  const int B = static_cast<int>(q.size(0)), H = static_cast<int>(q.size(1)), S = static_cast<int>(q.size(2));
  const int causal = args[3] == Py_True ? 1 : 0;
  int rc = 0;
  Py_BEGIN_ALLOW_THREADS   // as ctypes does: a launch can block while the device's queue is full
  rc = g_fwd(qp, kp, vp, op, lp, B, H, S, static_cast<int>(D), strides, causal, scale, block_m, block_n, dtype, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) return PyLong_FromLong(rc);
  PyObject* po = THPVariable_Wrap(std::move(o));
  if (po == nullptr) return nullptr;
  PyObject* pl = Py_None;
  if (lse.defined()) {
    pl = THPVariable_Wrap(std::move(lse));
    if (pl == nullptr) {
      Py_DECREF(po);
      return nullptr;
    }
  } else {
    Py_INCREF(pl);
  }
  PyObject* pair = PyTuple_New(2);
  if (pair == nullptr) {
    Py_DECREF(po);
    Py_DECREF(pl);
    return nullptr;
  }
  PyTuple_SET_ITEM(pair, 0, po);
  PyTuple_SET_ITEM(pair, 1, pl);
  return pair;
  END_HANDLE_TH_ERRORS
}

// bind(address of rsfa_fwd)
PyObject* bind(PyObject*, PyObject* arg) {
  void* p = PyLong_AsVoidPtr(arg);
  if (p == nullptr && PyErr_Occurred()) return nullptr;
  g_fwd = reinterpret_cast<FwdFn>(p);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(forward)), METH_FASTCALL, nullptr},
    {"bind", bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_rsfa_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__rsfa_torch() {
  PyObject* m = PyModule_Create(&module);
  // the torch whose tensor layout this file was compiled for: the Python side uses it with no other
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", RSFA_TORCH_VERSION) != 0) Py_CLEAR(m);
  return m;
}
