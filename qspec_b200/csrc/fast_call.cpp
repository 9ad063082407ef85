// The linear layers' call path in native code: checks and one C call, for a product of a few microseconds that a Python path of ten would hide.
// Takes exactly the calls that the Python functions in ops.py take without an error; everything else (another type or layout, sizes that do not
// match, an empty batch, a workspace that is missing or too small) it leaves to them: returns None, nothing launched.
// 4 tokens, 4096 x 4096, W4A4, through nn.Linear4bit in a row of calls: 11.1 -> 6.3 us (the kernel 2.7).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

#include "../../include/qspec_b200.h"

namespace {

typedef decltype(&qspec_gemm_w4a4) Int4Fn;                    // (of qspec_gemm_w4a8, too)
typedef decltype(&qspec_gemm_w4a16) Fp16Fn;
static_assert(std::is_same<Int4Fn, decltype(&qspec_gemm_w4a8)>::value, "one call for both");

PyTypeObject* parameter_type = nullptr;

// A plain CUDA tensor, contiguous; subclasses with behaviour of their own are the Python path's business.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o) && Py_TYPE(o) != parameter_type) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() ? &t : nullptr;
}
bool is_int4(const at::Tensor& t) { return t.scalar_type() == at::kChar || t.scalar_type() == at::kByte; }

// linear(address, kind, x, x_scale, weight, weight_scale, bias, out, workspaces, key): kind 0 W4A4, 1 W4A16, 2 W4A8; workspaces is the table of
// ops.py, key its kind. Returns the status of the call, or None.
PyObject* linear_(PyObject* const* a, Py_ssize_t n) {
  if (n != 10) {
    PyErr_SetString(PyExc_TypeError, "linear takes 10 arguments");
    return nullptr;
  }
  void* fn = PyLong_AsVoidPtr(a[0]);
  const long kind = PyLong_AsLong(a[1]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor *x = plain(a[2]), *w = plain(a[4]), *ws = plain(a[5]), *out = plain(a[7]);
  if (!fn || !x || !w || !ws || !out) Py_RETURN_NONE;
  const at::Tensor *xs = nullptr, *bias = nullptr;
  const auto type = out->scalar_type();
  if (type != at::kHalf && type != at::kBFloat16) Py_RETURN_NONE;
  if (kind == 1) {
    if (x->scalar_type() != type) Py_RETURN_NONE;
  } else {
    xs = plain(a[3]);
    if (!xs || xs->scalar_type() != type || !is_int4(*x) || (kind == 2 && x->scalar_type() != at::kChar)) Py_RETURN_NONE;
  }
  if (a[6] != Py_None) {
    bias = plain(a[6]);
    if (!bias || bias->scalar_type() != type) Py_RETURN_NONE;
  }
  if (!is_int4(*w) || ws->scalar_type() != type || w->dim() != 2 || x->dim() < 1) Py_RETURN_NONE;
  const int64_t N = w->size(0), K = 2 * w->size(1), cols = kind == 0 ? K / 2 : K;
  if (N <= 0 || K <= 0 || x->size(-1) != cols) Py_RETURN_NONE;
  const int64_t M = x->numel() / cols;
  if (M <= 0 || M > INT32_MAX || N > INT32_MAX || K > INT32_MAX || (xs && xs->numel() != M) || ws->numel() != N || out->numel() != M * N ||
      (bias && bias->numel() != N))
    Py_RETURN_NONE;
  PyObject* index = PyLong_FromLong(x->get_device());
  if (!index) return nullptr;
  PyObject* key = PyTuple_Pack(2, a[9], index);
  Py_DECREF(index);
  if (!key) return nullptr;
  PyObject* space = PyDict_GetItemWithError(a[8], key);      // borrowed
  Py_DECREF(key);
  if (!space) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const at::Tensor* room = plain(space);
  if (!room) Py_RETURN_NONE;
  void* stream = c10::cuda::getCurrentCUDAStream().stream();
  const void* b = bias ? bias->const_data_ptr() : nullptr;
  const int dtype = type == at::kBFloat16 ? 1 : 0;
  const void *xp = x->const_data_ptr(), *sp = xs ? xs->const_data_ptr() : nullptr, *wp = w->const_data_ptr(), *wsp = ws->const_data_ptr();
  void *op = out->mutable_data_ptr(), *rp = room->mutable_data_ptr();
  const size_t bytes = (size_t)room->nbytes();
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = kind == 1 ? ((Fp16Fn)fn)(xp, (const int8_t*)wp, wsp, b, op, (int)M, (int)N, (int)K, dtype, rp, bytes, stream)
                     : ((Int4Fn)fn)((const int8_t*)xp, sp, (const int8_t*)wp, wsp, b, op, (int)M, (int)N, (int)K, dtype, rp, bytes, stream);
  Py_END_ALLOW_THREADS
  if (status == QSPEC_ERR_WORKSPACE) Py_RETURN_NONE;
  return PyLong_FromLong(status);
}

// Tensors without memory of their own (inside a functional transform) throw when asked for it: the Python path's business.
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    return linear_(a, n);
  } catch (const std::exception&) {
    Py_RETURN_NONE;
  }
}

PyMethodDef methods[] = {{"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fast() {
  PyObject* nn = PyImport_ImportModule("torch.nn");
  if (!nn) return nullptr;
  PyObject* type = PyObject_GetAttrString(nn, "Parameter");
  Py_DECREF(nn);
  if (!type) return nullptr;
  parameter_type = (PyTypeObject*)type;                       // kept for the life of the process
  return PyModule_Create(&module);
}
