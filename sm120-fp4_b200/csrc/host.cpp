// Host side of the quantiser calls that are host time for the most part (16 x 2048 bf16: 2.4 us on the GPU, 11.5 us from Python, of which three allocations
// 4.8, the ctypes call 1.1 and the launch 2.5; 5.7 us this way): argument checks, allocations and the library call in one call into native code. Each function takes plain CUDA
// tensors on the current device only and returns None for whatever it does not take - the caller's general path, with its checks and errors, is then
// the one that runs -, the error code of the library as an int, or the outputs.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

using OwnScale = int (*)(const void*, int, int, int, int, void*, void*, void*, int, void*, long long, void*);
using Quantize = int (*)(const void*, int, const int*, int, int, const void*, int, void*, void*, int, void*);
OwnScale own_scale = nullptr;
Quantize quantize = nullptr;
long long one_cluster = 0;   // values of a matrix up to which own_scale needs no workspace

// Nothing that would see the torch calls of the general path: function and dispatch modes, functorch transforms, functionalisation.
bool plain_call() {
  using c10::DispatchKey;
  return !at::impl::torch_function_mode_enabled() && !c10::impl::tls_is_dispatch_key_included(DispatchKey::Python) &&
         !c10::impl::tls_is_dispatch_key_included(DispatchKey::PythonTLSSnapshot) &&
         !c10::impl::tls_is_dispatch_key_included(DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !c10::impl::tls_is_dispatch_key_included(DispatchKey::FuncTorchDynamicLayerBackMode) &&
         !c10::impl::tls_is_dispatch_key_included(DispatchKey::Functionalize);
}

bool plain_tensor(const at::Tensor& t) {
  using c10::DispatchKey;
  const c10::DispatchKeySet k = t.key_set();
  return t.is_cuda() && t.layout() == at::kStrided && !k.has(DispatchKey::Python) && !k.has(DispatchKey::FuncTorchBatched) && !k.has(DispatchKey::FuncTorchGradWrapper) &&
         !k.has(DispatchKey::Functionalize) && !k.has(DispatchKey::Negative);
}

// a matrix the kernels take as it is: bf16 or fp32, whole blocks of 16, contiguous, on the current device
bool plain_matrix(const at::Tensor& x) {
  return plain_tensor(x) && x.dim() == 2 && (x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kFloat) && x.size(0) > 0 && x.size(1) > 0 && x.size(1) % 16 == 0 &&
         x.is_contiguous() && x.get_device() == c10::cuda::current_device();
}

at::Tensor bytes(int64_t rows, int64_t cols, const at::Tensor& like) { return at::empty({rows, cols}, at::TensorOptions().dtype(at::kByte).device(like.device())); }

// Python runs on meanwhile, as under torch's own calls: an allocation may wait for the device, and the device for a callback that wants the interpreter.
struct Released {
  PyThreadState* state = PyEval_SaveThread();
  ~Released() { PyEval_RestoreThread(state); }
};

PyObject* outputs(int rc, const at::Tensor& packed, const at::Tensor& sf, PyObject* scale) {   // takes over the reference to scale
  if (rc) {
    Py_XDECREF(scale);
    return PyLong_FromLong(rc);
  }
  PyObject *p = THPVariable_Wrap(packed), *s = THPVariable_Wrap(sf), *t = p && s && scale ? PyTuple_New(3) : nullptr;
  if (!t) {
    Py_XDECREF(p), Py_XDECREF(s), Py_XDECREF(scale);
    return nullptr;
  }
  PyTuple_SET_ITEM(t, 0, p), PyTuple_SET_ITEM(t, 1, s), PyTuple_SET_ITEM(t, 2, scale);
  return t;
}

// bind(address of b200moe_quantize_nvfp4_own_scale, of b200moe_quantize_nvfp4, one_cluster)
PyObject* py_bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "bind takes two addresses and a size");
    return nullptr;
  }
  void *a = PyLong_AsVoidPtr(args[0]), *b = PyLong_AsVoidPtr(args[1]);
  const long long c = PyLong_AsLongLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  own_scale = (OwnScale)a, quantize = (Quantize)b, one_cluster = c;
  Py_RETURN_NONE;
}

// quantize_own_scale(x): one matrix small enough to need no workspace, its own global scale, row-major block scales
PyObject* py_quantize_own_scale(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 1 || !own_scale || !THPVariable_CheckExact(args[0]) || !plain_call()) Py_RETURN_NONE;
  const at::Tensor x = THPVariable_Unpack(args[0]);
  if (!plain_matrix(x) || x.numel() > one_cluster) Py_RETURN_NONE;
  const int64_t rows = x.size(0), k = x.size(1);
  at::Tensor packed, sf, gs;
  int rc;
  {
    Released released;
    packed = bytes(rows, k / 2, x), sf = bytes(rows, k / 16, x), gs = at::empty({1}, at::TensorOptions().dtype(at::kFloat).device(x.device()));
    rc = own_scale(x.data_ptr(), x.scalar_type() == at::kFloat, 1, (int)rows, (int)k, gs.data_ptr(), packed.data_ptr(), sf.data_ptr(), 0, nullptr, 0,
                   (void*)c10::cuda::getCurrentCUDAStream().stream());
  }
  return outputs(rc, packed, sf, THPVariable_Wrap(gs));
  END_HANDLE_TH_ERRORS
}

// quantize_128x4(x, global_scale): block scales in the 128x4 swizzle
PyObject* py_quantize_128x4(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !quantize || !THPVariable_CheckExact(args[0]) || !THPVariable_CheckExact(args[1]) || !plain_call()) Py_RETURN_NONE;
  const at::Tensor x = THPVariable_Unpack(args[0]), gs = THPVariable_Unpack(args[1]);
  if (!plain_matrix(x) || !plain_tensor(gs) || gs.scalar_type() != at::kFloat || gs.dim() != 1 || gs.size(0) != 1 || gs.device() != x.device()) Py_RETURN_NONE;
  const int64_t rows = x.size(0), k = x.size(1);
  if (rows > 0x7fffffff - 128 || k > 0x7fffffff) Py_RETURN_NONE;
  at::Tensor packed, sf;
  int rc;
  {
    Released released;
    packed = bytes(rows, k / 2, x), sf = bytes((rows + 127) / 128 * 128, (k / 16 + 3) / 4 * 4, x);
    rc = quantize(x.data_ptr(), x.scalar_type() == at::kFloat, nullptr, (int)rows, (int)k, gs.data_ptr(), 0, packed.data_ptr(), sf.data_ptr(), 1,
                  (void*)c10::cuda::getCurrentCUDAStream().stream());
  }
  Py_INCREF(args[1]);
  return outputs(rc, packed, sf, args[1]);
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"bind", (PyCFunction)(void (*)(void))py_bind, METH_FASTCALL, nullptr},
                         {"quantize_own_scale", (PyCFunction)(void (*)(void))py_quantize_own_scale, METH_FASTCALL, nullptr},
                         {"quantize_128x4", (PyCFunction)(void (*)(void))py_quantize_128x4, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {   // (nothing of torch: the caller compares the version before anything else)
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "torch_version", B200_TORCH_VERSION)) Py_CLEAR(m);
  return m;
}
