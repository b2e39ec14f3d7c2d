// The per-call side of DeviceWeights.gemv / .gemm (device.py) as a Python extension: the checks of the ordinary case, the
// addresses and the current stream straight from torch's C++ objects, then the C entry point.  In Python with ctypes that is
// 2 us a call beside the launch's own 2, more than a small matvec takes on the GPU.
//
// Whatever is not the ordinary case (no plain contiguous f32 CUDA tensor, too short, arguments that are no sizes) is answered
// with None: the caller then goes the way through Python, which knows the errors.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/core/DispatchKeySet.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

// qk_gemv_dev and qk_gemm_dev of the library that the package has loaded (bind)
int (*gemv_dev)(void *ctx, const void *w, const float *x, float *y, void *stream) = nullptr;
int (*gemm_dev)(void *ctx, const void *w, const float *x, float *y, size_t m, size_t ldy, void *stream) = nullptr;

// The address of a tensor with at least n elements, or null: not the ordinary case.
float *floats(PyObject *o, size_t n) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor &t = THPVariable_Unpack(o);
  using K = c10::DispatchKey;
  constexpr c10::DispatchKeySet wrapped({K::Python, K::PythonTLSSnapshot, K::FuncTorchBatched, K::FuncTorchGradWrapper, K::Functionalize, K::Conjugate, K::Negative});
  if (!t.defined() || !t.is_cuda() || t.layout() != c10::kStrided || t.key_set().has_any(wrapped) || t.scalar_type() != c10::kFloat ||
      !t.is_contiguous() || (size_t)t.numel() < n)
    return nullptr;
  return static_cast<float *>(t.data_ptr());
}

// A size, or false with the error cleared.
bool size(PyObject *o, size_t *v) {
  const Py_ssize_t s = PyLong_Check(o) ? PyLong_AsSsize_t(o) : -1;
  if (s < 0) {
    PyErr_Clear();
    return false;
  }
  *v = (size_t)s;
  return true;
}

bool address(PyObject *o, void **p) {
  *p = PyLong_Check(o) ? PyLong_AsVoidPtr(o) : nullptr;
  if (PyErr_Occurred()) PyErr_Clear();
  return *p != nullptr;
}

bool stream_of(PyObject *o, void **s) {
  if (o == Py_None) {
    *s = c10::cuda::getCurrentCUDAStream().stream();
    return true;
  }
  PyObject *h = PyObject_GetAttrString(o, "cuda_stream");
  if (h && PyLong_Check(h)) *s = PyLong_AsVoidPtr(h);
  const bool ok = h && PyLong_Check(h) && !PyErr_Occurred();
  Py_XDECREF(h);
  PyErr_Clear();
  return ok;
}

// gemv(ctx, weights, cols, rows, x, y, stream) -> status or None
PyObject *gemv(PyObject *, PyObject *const *a, Py_ssize_t n) {
  try {
    void *ctx, *w, *s;
    size_t cols, rows;
    float *x, *y;
    if (n == 7 && gemv_dev && address(a[0], &ctx) && address(a[1], &w) && size(a[2], &cols) && size(a[3], &rows) &&
        (x = floats(a[4], cols)) && (y = floats(a[5], rows)) && stream_of(a[6], &s)) {
      int st;
      Py_BEGIN_ALLOW_THREADS st = gemv_dev(ctx, w, x, y, s);
      Py_END_ALLOW_THREADS return PyLong_FromLong(st);
    }
  } catch (...) {
  }
  Py_RETURN_NONE;
}

// gemm(ctx, weights, cols, rows, x, y, m, ldy, column, stream) -> status or None
PyObject *gemm(PyObject *, PyObject *const *a, Py_ssize_t n) {
  try {
    void *ctx, *w, *s;
    size_t cols, rows, m, ldy, col;
    float *x, *y;
    if (n == 10 && gemm_dev && address(a[0], &ctx) && address(a[1], &w) && size(a[2], &cols) && size(a[3], &rows) && size(a[6], &m) &&
        size(a[7], &ldy) && size(a[8], &col) && m > 0 && m < (1ull << 31) && cols < (1ull << 31) && rows < (1ull << 31) &&
        ldy < (1ull << 31) && col < (1ull << 31) && (x = floats(a[4], m * cols)) && (y = floats(a[5], (m - 1) * ldy + col + rows)) &&
        stream_of(a[9], &s)) {
      int st;
      Py_BEGIN_ALLOW_THREADS st = gemm_dev(ctx, w, x, y + col, m, ldy, s);
      Py_END_ALLOW_THREADS return PyLong_FromLong(st);
    }
  } catch (...) {
  }
  Py_RETURN_NONE;
}

// bind(address of qk_gemv_dev, address of qk_gemm_dev)
PyObject *bind(PyObject *, PyObject *const *a, Py_ssize_t n) {
  void *v, *m;
  if (n != 2 || !address(a[0], &v) || !address(a[1], &m)) {
    PyErr_SetString(PyExc_ValueError, "two addresses");
    return nullptr;
  }
  gemv_dev = reinterpret_cast<decltype(gemv_dev)>(v), gemm_dev = reinterpret_cast<decltype(gemm_dev)>(m);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"gemv", (PyCFunction)(void (*)(void))gemv, METH_FASTCALL, nullptr},
                         {"gemm", (PyCFunction)(void (*)(void))gemm, METH_FASTCALL, nullptr},
                         {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_qk_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// The accessors of at::Tensor are inlined, so their offsets are those of the torch that this was compiled with, and a file left
// over from another one can still be loaded: the importer compares both.
PyMODINIT_FUNC PyInit__qk_torch() {
  PyObject *m = PyModule_Create(&module);
  if (m && (PyModule_AddStringConstant(m, "torch_version", QK_TORCH_VERSION) < 0 || PyModule_AddIntConstant(m, "python_version", PY_VERSION_HEX >> 16) < 0)) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
