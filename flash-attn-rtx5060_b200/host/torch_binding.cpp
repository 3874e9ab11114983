// Native part of the Python entry points: argument checks, output allocation and the call of the C ABI for torch tensors,
// as one function of the CPython API, and a caller of flash_forward_noalloc for plain numbers. Nothing is linked or kept
// here: bind() makes both for the library whose entry points it is given, the one that the package has loaded, whatever
// other copies of it the process holds. A small call is bound by
// the host: with ctypes and the checks in Python attention_forward took 9.2 us a call (2.1 of them in the library and
// the driver, 1.5 ctypes, 1.3 the output tensor) where the kernel takes 7.2 (B1 H4 N512 d64).
//
// Every function here answers NotImplemented, or passes its arguments on, where it does not know them, and the Python
// code of the package then does what it always did: errors, tensor subclasses, active torch function or dispatch modes,
// a device other than the current one, the kernels that only tests select.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include "../../include/flash_forward_b200.h"

namespace {

PyObject* not_here() {
  Py_INCREF(Py_NotImplemented);
  return Py_NotImplemented;
}

bool plain_int(PyObject* o) { return PyLong_Check(o); }
// As ctypes does with an int for a C int: the low bits.
int low_int(PyObject* o) { return static_cast<int>(PyLong_AsUnsignedLongMask(o)); }
bool plain_number(PyObject* o) { return PyFloat_Check(o) || PyLong_Check(o); }

// What bind() was given; the `self` of the functions that it returns, as a capsule.
struct Library {
  decltype(&flash_forward) plain;
  decltype(&flash_forward_alibi) alibi;
  decltype(&flash_forward_lse) lse;
  decltype(&flash_forward_dropout) dropout;
  decltype(&flash_forward_noalloc) noalloc;
  PyObject* ctypes_noalloc;  // takes the calls of noalloc() with anything but plain numbers
};
const Library& library(PyObject* self) { return *static_cast<Library*>(PyCapsule_GetPointer(self, nullptr)); }

// forward(q, k, v, causal, window_left, window_right, softmax_scale, out, alibi_slopes, return_lse, dropout_p, seed):
// the result of attention_forward, an int (status code of a call that failed) or NotImplemented.
PyObject* forward(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 12) return not_here();
  PyObject *py_out = a[7], *py_slopes = a[8];
  for (int i = 0; i < 3; ++i)
    if (!THPVariable_CheckExact(a[i])) return not_here();
  if (py_out != Py_None && !THPVariable_CheckExact(py_out)) return not_here();
  if (py_slopes != Py_None && !THPVariable_CheckExact(py_slopes)) return not_here();
  if (!PyBool_Check(a[3]) || !PyBool_Check(a[9]) || !plain_int(a[4]) || !plain_int(a[5]) || !plain_number(a[6]) ||
      !plain_number(a[10]) || !plain_int(a[11]))
    return not_here();
  if (at::impl::torch_function_mode_enabled() || c10::impl::dispatch_mode_enabled()) return not_here();

  const at::Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
  if (!q.is_cuda() || q.dim() != 4) return not_here();
  const auto device = q.get_device();
  // what the kernel may be given the address of
  auto fits = [&](const at::Tensor& t, at::ScalarType type) {
    return t.is_cuda() && t.get_device() == device && t.scalar_type() == type && t.is_contiguous();
  };
  if (!fits(q, at::kHalf) || !fits(k, at::kHalf) || !fits(v, at::kHalf)) return not_here();
  if (k.sizes() != q.sizes() || v.sizes() != q.sizes()) return not_here();
  if (py_out != Py_None && (!fits(THPVariable_Unpack(py_out), at::kHalf) || THPVariable_Unpack(py_out).numel() < q.numel()))
    return not_here();
  const bool causal = a[3] == Py_True, want_lse = a[9] == Py_True;
  const float scale = static_cast<float>(PyFloat_AsDouble(a[6]));
  const double dropout = PyFloat_AsDouble(a[10]);  // (positive, though 0 as a float, it still asks for the dropout call)
  if (PyErr_Occurred()) {  // an int beyond the range of a double
    PyErr_Clear();
    return not_here();
  }
  if (dropout > 0.0 && want_lse) return not_here();
  const auto B = q.size(0), H = q.size(1), N = q.size(2), D = q.size(3);
  const float* slopes = nullptr;
  if (py_slopes != Py_None) {
    const at::Tensor& t = THPVariable_Unpack(py_slopes);
    if (!fits(t, at::kFloat) || t.numel() != H) return not_here();
    slopes = static_cast<const float*>(t.data_ptr());
  }
  if (device != c10::cuda::current_device()) return not_here();

  const at::Tensor out = py_out == Py_None ? at::empty_like(q) : THPVariable_Unpack(py_out);
  at::Tensor lse;
  if (want_lse) lse = at::empty({B, H, N}, q.options().dtype(at::kFloat));
  const void *pq = q.data_ptr(), *pk = k.data_ptr(), *pv = v.data_ptr();
  void* po = out.data_ptr();
  float* pl = want_lse ? static_cast<float*>(lse.data_ptr()) : nullptr;
  void* stream = c10::cuda::getCurrentCUDAStream(device).stream();
  const int b = static_cast<int>(B), h = static_cast<int>(H), s = static_cast<int>(N), d = static_cast<int>(D);
  const int wl = low_int(a[4]), wr = low_int(a[5]);
  const unsigned long long seed = PyLong_AsUnsignedLongLongMask(a[11]);
  const Library& lib = library(self);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  if (dropout > 0.0)
    rc = lib.dropout(pq, pk, pv, po, b, h, s, d, scale, causal, wl, wr, slopes, static_cast<float>(dropout), seed, stream);
  else if (want_lse) rc = lib.lse(pq, pk, pv, po, pl, b, h, s, d, scale, causal, wl, wr, slopes, stream);
  else if (slopes) rc = lib.alibi(pq, pk, pv, po, b, h, s, d, scale, causal, wl, wr, slopes, stream);
  else rc = lib.plain(pq, pk, pv, po, b, h, s, d, scale, causal, wl, wr, stream);
  Py_END_ALLOW_THREADS
  if (rc != FA_OK) return PyLong_FromLong(rc);
  PyObject* py_result = py_out;
  if (py_out == Py_None) py_result = THPVariable_Wrap(out);
  else Py_INCREF(py_out);
  if (!want_lse || !py_result) return py_result;
  PyObject* py_lse = THPVariable_Wrap(lse);
  PyObject* pair = py_lse ? PyTuple_Pack(2, py_result, py_lse) : nullptr;
  Py_DECREF(py_result);
  Py_XDECREF(py_lse);
  return pair;
  END_HANDLE_TH_ERRORS
}

bool address(PyObject* o, void** p) {
  if (o == Py_None) {
    *p = nullptr;
    return true;
  }
  if (!PyLong_CheckExact(o)) return false;
  *p = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(o));
  return true;
}

// flash_forward_noalloc for pointers given as ints or None and numbers
PyObject* noalloc(PyObject* self, PyObject* const* a, Py_ssize_t n, PyObject* names) {
  void *q, *k, *v, *o, *stream;
  bool known = n == 15 && (names == nullptr || PyTuple_GET_SIZE(names) == 0) && address(a[0], &q) && address(a[1], &k) &&
               address(a[2], &v) && address(a[3], &o) && address(a[12], &stream) && plain_number(a[8]);
  constexpr int ints[] = {4, 5, 6, 7, 9, 10, 11, 13, 14};
  for (int i : ints) known = known && plain_int(a[i]);
  float scale = 0.f;
  if (known) {
    scale = static_cast<float>(PyFloat_AsDouble(a[8]));
    if (PyErr_Occurred()) {
      PyErr_Clear();
      known = false;
    }
  }
  const Library& lib = library(self);
  if (!known) return PyObject_Vectorcall(lib.ctypes_noalloc, a, n, names);
  const int x[] = {low_int(a[4]), low_int(a[5]), low_int(a[6]), low_int(a[7]), low_int(a[9]), low_int(a[10]), low_int(a[11]),
                   low_int(a[13]), low_int(a[14])};
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.noalloc(q, k, v, o, x[0], x[1], x[2], x[3], scale, x[4], x[5], x[6], stream, x[7], x[8]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

PyMethodDef forward_def = {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward)), METH_FASTCALL, nullptr};
PyMethodDef noalloc_def = {"flash_forward_noalloc", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(noalloc)),
                           METH_FASTCALL | METH_KEYWORDS, nullptr};

void drop_library(PyObject* capsule) {
  Library* lib = static_cast<Library*>(PyCapsule_GetPointer(capsule, nullptr));
  Py_DECREF(lib->ctypes_noalloc);
  delete lib;
}

// bind(addresses of flash_forward, flash_forward_alibi, flash_forward_lse, flash_forward_dropout, flash_forward_noalloc as
// ints, the ctypes function of the last): (forward, noalloc)
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long plain, alibi, lse, dropout, noalloc_address;
  PyObject* fn;
  if (!PyArg_ParseTuple(args, "KKKKKO", &plain, &alibi, &lse, &dropout, &noalloc_address, &fn)) return nullptr;
  Library* lib = new Library{reinterpret_cast<decltype(Library::plain)>(plain), reinterpret_cast<decltype(Library::alibi)>(alibi),
                             reinterpret_cast<decltype(Library::lse)>(lse), reinterpret_cast<decltype(Library::dropout)>(dropout),
                             reinterpret_cast<decltype(Library::noalloc)>(noalloc_address), fn};
  PyObject* capsule = PyCapsule_New(lib, nullptr, drop_library);
  if (!capsule) {
    delete lib;
    return nullptr;
  }
  Py_INCREF(fn);
  PyObject* pair = Py_BuildValue("(NN)", PyCFunction_New(&forward_def, capsule), PyCFunction_New(&noalloc_def, capsule));
  Py_DECREF(capsule);
  return pair;
}

PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

#define FA_STRING_OF(x) #x
#define FA_STRING(x) FA_STRING_OF(x)

PyMODINIT_FUNC PyInit__torch_binding(void) {
  PyObject* m = PyModule_Create(&module);
  // the torch whose object layouts are compiled in
  if (m && PyModule_AddStringConstant(m, "torch_version", FA_STRING(FA_TORCH_VERSION)) < 0) Py_CLEAR(m);
  return m;
}
