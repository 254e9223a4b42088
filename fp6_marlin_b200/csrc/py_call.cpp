// The Python call path of mul / mul_fused: reads the tensors' metadata, checks it and calls the C ABI (include/fp6m.h).
//
// A decode step is a chain of GEMMs of a few microseconds each, so the host time of a call counts: through Python
// attributes and ctypes a call took 11 us, of which the launch itself is about two.  This module handles the calls whose
// arguments are plain CUDA tensors that pass every check; for anything else - subclasses, wrappers of function
// transforms, wrong sizes or types - it answers "not handled" and the caller takes its general path, which raises or
// computes as before.  It holds no state but the addresses of the scratch buffers registered by the caller (one per device and
// stream); the caller never frees a registered buffer, also not one that a larger one replaces: a call may have read its
// address here and not have launched yet.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <unordered_map>

#include "../../include/fp6m.h"

namespace {

// (the types of the C ABI's own declarations: the addresses come as numbers, see bind)
using MulFn = decltype(&fp6m_mul);
using MulFusedFn = decltype(&fp6m_mul_fused);
using ScratchFn = decltype(&fp6m_mul_scratch_bytes);

MulFn g_mul = nullptr;
MulFusedFn g_mul_fused = nullptr;
ScratchFn g_scratch_bytes = nullptr;

constexpr long kNotHandled = -1;

// What the caller registered (all access under the interpreter lock).
struct Scratch {
  void* ptr;
  size_t bytes;
};
struct StreamKey {
  int dev;
  void* stream;
  bool operator==(const StreamKey& o) const { return dev == o.dev && stream == o.stream; }
};
struct StreamKeyHash {
  size_t operator()(const StreamKey& k) const { return std::hash<void*>()(k.stream) * 31 + (size_t)k.dev; }
};
std::unordered_map<StreamKey, Scratch, StreamKeyHash>& scratches() {
  static auto* m = new std::unordered_map<StreamKey, Scratch, StreamKeyHash>();
  return *m;
}
struct Device {
  int* status = nullptr;
  int sms = 0;
};
Device g_devices[64];

// A tensor whose memory may be handed to a kernel directly: a plain torch.Tensor / Parameter, strided, contiguous and on a
// CUDA device, none of torch's wrappers.
const at::Tensor* plain_cuda(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined()) return nullptr;
  // the keys every strided CUDA tensor may have; wrappers, conjugate views and the like have others
  static const c10::DispatchKeySet kPlain = c10::DispatchKeySet(c10::DispatchKey::CUDA) |
                                            c10::getAutogradRelatedKeySetFromBackend(c10::BackendComponent::CUDABit) |
                                            c10::getAutocastRelatedKeySetFromBackend(c10::BackendComponent::CUDABit);
  if ((t.key_set().raw_repr() & ~kPlain.raw_repr()) != 0 || !t.is_cuda() || !t.is_contiguous()) return nullptr;
  return &t;
}

bool as_int(PyObject* o, int* out) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  const long v = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow || v < INT32_MIN || v > INT32_MAX) return false;
  *out = (int)v;
  return true;
}

// mul(A, B, C, s, workspace, quant_cols, thread_k, thread_n, sms, max_par, group_size, epilogue, residual) -> the C ABI's
// status, or -1: not handled.
PyObject* mul_impl(PyObject* const* args) {
  const at::Tensor* A = plain_cuda(args[0]);
  const at::Tensor* B = plain_cuda(args[1]);
  const at::Tensor* C = plain_cuda(args[2]);
  const at::Tensor* s = plain_cuda(args[3]);
  const at::Tensor* ws = plain_cuda(args[4]);
  int quant_cols, thread_k, thread_n, sms, max_par, group_size, epilogue;
  if (!A || !B || !C || !s || !ws || !as_int(args[5], &quant_cols) || !as_int(args[6], &thread_k) || !as_int(args[7], &thread_n) ||
      !as_int(args[8], &sms) || !as_int(args[9], &max_par) || !as_int(args[10], &group_size) || !as_int(args[11], &epilogue))
    return PyLong_FromLong(kNotHandled);
  if (A->dim() != 2 || C->dim() != 2) return PyLong_FromLong(kNotHandled);
  const int64_t M = A->size(0), K = A->size(1), N = C->size(1) * (epilogue == FP6M_EPILOGUE_SILU_MUL ? 2 : 1);
  if (M <= 0 || K <= 0 || N <= 0 || M > INT32_MAX || K > INT32_MAX || N > INT32_MAX || C->size(0) != M || max_par < 1) return PyLong_FromLong(kNotHandled);
  if (ws->numel() < N / 128 * max_par) return PyLong_FromLong(kNotHandled);
  if (A->scalar_type() != at::kHalf || C->scalar_type() != at::kHalf || s->scalar_type() != at::kHalf) return PyLong_FromLong(kNotHandled);
  const void* residual = nullptr;
  if (epilogue == FP6M_EPILOGUE_RESIDUAL) {
    const at::Tensor* r = plain_cuda(args[12]);
    if (!r || r->scalar_type() != at::kHalf || r->dim() != 2 || r->size(0) != M || r->size(1) != N) return PyLong_FromLong(kNotHandled);
    residual = r->data_ptr();
  }
  const int dev = A->device().index();
  if (dev < 0 || dev >= 64 || !g_devices[dev].status) return PyLong_FromLong(kNotHandled);
  void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  const auto it = scratches().find({dev, stream});
  if (it == scratches().end()) return PyLong_FromLong(kNotHandled);
  if (it->second.bytes < g_scratch_bytes((int)M, (int)N, (int)K, quant_cols, g_devices[dev].sms)) return PyLong_FromLong(kNotHandled);
  const void *a = A->data_ptr(), *w = B->data_ptr(), *sc = s->data_ptr();
  void *c = C->data_ptr(), *wsp = ws->data_ptr();
  const size_t ws_bytes = (size_t)ws->numel() * ws->element_size();
  const Scratch scratch = it->second;
  int* status = g_devices[dev].status;
  int rc;
  Py_BEGIN_ALLOW_THREADS        // a launch waits while the GPU's queue is full
  if (epilogue)
    rc = g_mul_fused(a, w, c, sc, (int)M, (int)N, (int)K, wsp, ws_bytes, scratch.ptr, scratch.bytes, dev, stream, thread_k, thread_n, sms, max_par,
                     quant_cols, group_size, FP6M_LAYOUT_B200, status, epilogue, residual);
  else
    rc = g_mul(a, w, c, sc, (int)M, (int)N, (int)K, wsp, ws_bytes, scratch.ptr, scratch.bytes, dev, stream, thread_k, thread_n, sms, max_par,
               quant_cols, group_size, FP6M_LAYOUT_B200, status);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

PyObject* py_mul(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 13) {
    PyErr_SetString(PyExc_TypeError, "mul: 13 arguments");
    return nullptr;
  }
  try {
    return mul_impl(args);
  } catch (const std::exception& e) {          // (torch's accessors report errors as exceptions)
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// bind(mul, mul_fused, scratch_bytes): addresses of the C ABI's functions
PyObject* py_bind(PyObject*, PyObject* args) {
  unsigned long long a, b, c;
  if (!PyArg_ParseTuple(args, "KKK", &a, &b, &c)) return nullptr;
  g_mul = reinterpret_cast<MulFn>(a);
  g_mul_fused = reinterpret_cast<MulFusedFn>(b);
  g_scratch_bytes = reinterpret_cast<ScratchFn>(c);
  Py_RETURN_NONE;
}

// set_device(dev, address of the status word, multiprocessors)
PyObject* py_set_device(PyObject*, PyObject* args) {
  int dev, sms;
  unsigned long long status;
  if (!PyArg_ParseTuple(args, "iKi", &dev, &status, &sms)) return nullptr;
  if (dev >= 0 && dev < 64) {
    g_devices[dev].status = reinterpret_cast<int*>(status);
    g_devices[dev].sms = sms;
  }
  Py_RETURN_NONE;
}

// set_scratch(dev, stream, address, bytes); the caller keeps the memory for the life of the process
PyObject* py_set_scratch(PyObject*, PyObject* args) {
  int dev;
  unsigned long long stream, ptr, bytes;
  if (!PyArg_ParseTuple(args, "iKKK", &dev, &stream, &ptr, &bytes)) return nullptr;
  try {
    scratches()[{dev, reinterpret_cast<void*>(stream)}] = {reinterpret_cast<void*>(ptr), (size_t)bytes};
  } catch (const std::bad_alloc&) {
    return PyErr_NoMemory();
  }
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"mul", (PyCFunction)(void (*)(void))py_mul, METH_FASTCALL, "GEMM on plain CUDA tensors: C ABI status, or -1 when the call is not handled here"},
    {"bind", py_bind, METH_VARARGS, "addresses of the C ABI's functions"},
    {"set_device", py_set_device, METH_VARARGS, "status word and number of multiprocessors of a device"},
    {"set_scratch", py_set_scratch, METH_VARARGS, "split-K scratch of a device's stream"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_call", "host call path of mul and mul_fused", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__call(void) {
  PyObject* module = PyModule_Create(&kModule);
  // the importer compares it with the torch it has: torch's accessors are inlined here
  if (module && PyModule_AddStringConstant(module, "torch_version", FP6M_TORCH_VERSION) != 0) Py_CLEAR(module);
  return module;
}
