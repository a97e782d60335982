// The host side of a repeated matmul_q40 or linear_q40 call: checks, the output tensor and the launch in one native call.
//
// Through Python's attributes and ctypes a call of matmul_q40 takes 10.7 us of the host and one of linear_q40 13.7, where a kernel of one
// row takes 5.5 (4096 x 4096); here they take 3.7 and 4.1.  Nothing is decided here that kernels.py does not decide: a call that is not the plain repeated one (another
// stream, a written or replaced weight, other types, sizes or devices, a subclass of tensor) is handed back as None, and goes
// the way of a first call, which also words the errors.
#include <Python.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ops/empty.h>

namespace {

using MatmulTiled = int (*)(const void*, void*, int64_t, const void*, int64_t, int, int, int, int, void*, int, void*);
using GemmNk = int (*)(const void*, int64_t, const void*, const void*, void*, int64_t, int, int, int, int, void*, size_t, void*);
MatmulTiled matmul_tiled = nullptr;
GemmNk gemm_nk = nullptr;

const at::Tensor* tensor(PyObject* o) {
  return THPVariable_CheckExact(o) || Py_TYPE(o) == reinterpret_cast<PyTypeObject*>(ParameterClass) ? &THPVariable_Unpack(o) : nullptr;
}
bool on(const at::Tensor& t, int dev) { return t.is_cuda() && t.get_device() == dev; }
// The two whole numbers of a tuple
bool two(PyObject* t, int64_t& a, int64_t& b) {
  if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 2 || !PyLong_Check(PyTuple_GET_ITEM(t, 0)) || !PyLong_Check(PyTuple_GET_ITEM(t, 1))) return false;
  a = PyLong_AsLongLong(PyTuple_GET_ITEM(t, 0));
  b = PyLong_AsLongLong(PyTuple_GET_ITEM(t, 1));
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
int64_t version(const at::Tensor& t) { return t.is_inference() ? -1 : (int64_t)t._version(); }
// kernels._workspaces[("gemm", device, stream)] or an undefined tensor
at::Tensor workspace(PyObject* dict, int dev, PyObject* stream) {
  static PyObject* kind = PyUnicode_InternFromString("gemm");
  PyObject* key = Py_BuildValue("(OiO)", kind, dev, stream);
  if (!key) {
    PyErr_Clear();
    return {};
  }
  PyObject* t = PyDict_GetItem(dict, key);
  Py_DECREF(key);
  return t && THPVariable_Check(t) ? THPVariable_Unpack(t) : at::Tensor();
}
// Other Python threads run meanwhile: an allocation may wait for the device, a launch for room in its queue (behind a host function that
// needs the interpreter, say).  What is used in there is owned here
struct WithoutInterpreter {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutInterpreter() { PyEval_RestoreThread(state); }
};
at::Tensor output(int64_t rows, int64_t cols, int dev) {
  return at::empty({rows, cols}, at::TensorOptions().dtype(at::kHalf).device(at::kCUDA, (c10::DeviceIndex)dev));
}

// matmul(a, b_w, b_s, b_shape, entry of kernels._relayout_cache, kernels._cluster_sizes, kernels._workspaces) -> C or None
PyObject* matmul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7 || !matmul_tiled) Py_RETURN_NONE;
  const at::Tensor *a = tensor(args[0]), *w = tensor(args[1]), *s = tensor(args[2]);
  PyObject* e = args[4];
  if (!a || !w || !s || !a->is_cuda() || !PyTuple_Check(e) || PyTuple_GET_SIZE(e) != 8) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  if (!on(*a, dev) || !on(*w, dev) || !on(*s, dev)) Py_RETURN_NONE;
  int64_t K, N, k2, n2, vw, vs, pw, ps;
  // the copy is of these tensors, as they are
  if (PyWeakref_GetObject(PyTuple_GET_ITEM(e, 0)) != args[1] || PyWeakref_GetObject(PyTuple_GET_ITEM(e, 1)) != args[2] ||
      !two(PyTuple_GET_ITEM(e, 2), vw, vs) || !two(PyTuple_GET_ITEM(e, 3), K, N) || !two(args[3], k2, n2) || k2 != K || n2 != N ||
      !two(PyTuple_GET_ITEM(e, 4), pw, ps) || vw != version(*w) || vs != version(*s) || pw != (int64_t)(uintptr_t)w->data_ptr() ||
      ps != (int64_t)(uintptr_t)s->data_ptr() || !THPVariable_Check(PyTuple_GET_ITEM(e, 5)))
    Py_RETURN_NONE;
  if (a->scalar_type() != at::kHalf || s->scalar_type() != at::kHalf || a->dim() != 2 || a->size(1) != K || !a->is_contiguous() ||
      !w->is_contiguous() || !s->is_contiguous() || w->numel() * 2 != K * N || s->numel() * 64 != K * N)
    Py_RETURN_NONE;
  const int64_t M = a->size(0);
  if (M < 1 || M > INT32_MAX || (uintptr_t)a->data_ptr() % 16 || (M <= 16 ? K % 16 != 0 || K < 64 : K % 64 != 0)) Py_RETURN_NONE;
  const auto stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  PyObject* st = PyLong_FromVoidPtr(stream);
  if (!st) return nullptr;
  const int known = PySet_Contains(PyTuple_GET_ITEM(e, 7), st);
  const at::Tensor page = known == 1 && M > 8 ? workspace(args[6], dev, st) : at::Tensor();
  Py_DECREF(st);
  if (known != 1) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  int cluster = 16;
  PyObject* d = PyLong_FromLong(dev);
  PyObject* sizes = d ? PyDict_GetItem(args[5], d) : nullptr;
  Py_XDECREF(d);
  if (sizes && PyTuple_Check(sizes) && PyTuple_GET_SIZE(sizes)) cluster = (int)PyLong_AsLong(PyTuple_GET_ITEM(sizes, 0));
  else if (M <= 8) Py_RETURN_NONE;
  if (M > 8 && !page.defined()) Py_RETURN_NONE;
  const at::Tensor copy = THPVariable_Unpack(PyTuple_GET_ITEM(e, 5)), x = *a;
  at::Tensor c;
  int rc;
  {
    WithoutInterpreter w;
    c = output(M, N, dev);
    rc = matmul_tiled(copy.data_ptr(), c.data_ptr(), N, x.data_ptr(), K, (int)M, (int)N, (int)K, cluster,
                      page.defined() ? (char*)page.data_ptr() + 4092 : nullptr, 1, stream);
  }
  if (rc != 0) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(c));
  END_HANDLE_TH_ERRORS
}

// linear(x, w_q, w_s, w_shape, group, kernels._workspaces) -> y or None
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !gemm_nk) Py_RETURN_NONE;
  const at::Tensor *x = tensor(args[0]), *w = tensor(args[1]), *s = tensor(args[2]);
  if (!x || !w || !s || !x->is_cuda() || !PyLong_Check(args[4])) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  int64_t N, K;
  if (!on(*x, dev) || !on(*w, dev) || !on(*s, dev) || !two(args[3], N, K) || x->dim() != 2 || x->size(1) != K || K < 1 || N < 1 ||
      K > INT32_MAX || N > INT32_MAX || x->scalar_type() != at::kHalf || !x->is_contiguous() || !w->is_contiguous() || !s->is_contiguous())
    Py_RETURN_NONE;
  const int64_t M = x->size(0);
  if (M < 1 || M > INT32_MAX || (M > 32 && (uintptr_t)x->data_ptr() % 16 == 8)) Py_RETURN_NONE;      // those are copied first
  const auto stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  PyObject* st = PyLong_FromVoidPtr(stream);
  if (!st) return nullptr;
  const at::Tensor ws = workspace(args[5], dev, st);
  Py_DECREF(st);
  if (!ws.defined() || ws.numel() > 64 << 20) Py_RETURN_NONE;        // a large one is noted where a capture uses it
  const int group = (int)PyLong_AsLong(args[4]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const at::Tensor in = *x, codes = *w, scales = *s;
  at::Tensor y;
  int rc;
  {
    WithoutInterpreter w;
    y = output(M, N, dev);
    rc = gemm_nk(in.data_ptr(), K, codes.data_ptr(), scales.data_ptr(), y.data_ptr(), N, (int)M, (int)N, (int)K, group, ws.data_ptr(), (size_t)ws.numel(), stream);
  }
  if (rc != 0) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// init(address of q40_matmul_tiled, address of q40_gemm_nk)
PyObject* init(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n == 2) {
    matmul_tiled = (MatmulTiled)PyLong_AsVoidPtr(args[0]);
    gemm_nk = (GemmNk)PyLong_AsVoidPtr(args[1]);
  }
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"matmul", (PyCFunction)(void*)matmul, METH_FASTCALL, nullptr},
                         {"linear", (PyCFunction)(void*)linear, METH_FASTCALL, nullptr},
                         {"init", (PyCFunction)(void*)init, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_calls(void) { return PyModule_Create(&module); }
