// The device-tensor operator calls of the Python layer, natively: reads the operands of torch tensors, keeps parsed
// option text, takes torch's current stream and calls the C ABI.
//
// A small operator is bound by what the host does per call.  The same steps through Python attribute calls and ctypes
// (five operands x four attributes, option parsing, a stream object) took 11 us a call against 2.8 us of GPU time for
// a 4096 x 4096 SpMV.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <unordered_map>

#include "../../../include/sparsewave_b200.h"

namespace {

PyObject *g_error = nullptr;         // SparseWaveError(status, message)
PyTypeObject *g_options = nullptr;   // ctypes SwbOptions

struct Failed {};  // a Python exception is set

[[noreturn]] void raise_status(int status, const char *message) {
  PyObject *e = PyObject_CallFunction(g_error, "is", status, message ? message : "");
  if (e) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  }
  throw Failed();
}

[[noreturn]] void raise_type(const char *name, const char *what) {
  PyErr_Format(PyExc_TypeError, "%s %s", name, what);
  throw Failed();
}

// Parsed option texts.  The GIL guards the table; a program uses a handful of texts, and the table starts over at 256.
const swb_options &parsed(const char *text, Py_ssize_t length) {
  static std::unordered_map<std::string, swb_options> table;
  std::string key(text, (size_t)length);
  auto it = table.find(key);
  if (it != table.end()) return it->second;
  swb_options o;
  swb_options_default(&o);
  const int st = swb_options_parse(nullptr, &o, key.c_str());
  if (st != SWB_OK) raise_status(st, swb_last_error(nullptr));
  if (table.size() >= 256) table.clear();
  return table.emplace(std::move(key), o).first->second;
}

// A copy: the caller's block may change and the table may move while the GIL is released.
swb_options options_of(PyObject *obj) {
  if (PyUnicode_Check(obj)) {
    Py_ssize_t n = 0;
    const char *s = PyUnicode_AsUTF8AndSize(obj, &n);
    if (!s) throw Failed();
    return parsed(s, n);
  }
  if (Py_TYPE(obj) == g_options || PyType_IsSubtype(Py_TYPE(obj), g_options)) {
    Py_buffer view;
    if (PyObject_GetBuffer(obj, &view, PyBUF_SIMPLE) != 0) throw Failed();
    swb_options o;
    const bool fits = view.len == (Py_ssize_t)sizeof o;
    if (fits) memcpy(&o, view.buf, sizeof o);
    PyBuffer_Release(&view);
    if (fits) return o;
  }
  const int truth = PyObject_IsTrue(obj);
  if (truth < 0) throw Failed();
  if (!truth) return parsed("", 0);  // None and other empty values: the defaults
  PyErr_SetString(PyExc_TypeError, "options must be a string in the reference's spelling or an SwbOptions");
  throw Failed();
}

const at::Tensor &tensor(PyObject *obj, const char *name) {
  if (!THPVariable_Check(obj)) raise_type(name, "must be a CUDA tensor");
  return THPVariable_Unpack(obj);
}

void *device_pointer(const at::Tensor &t, at::ScalarType dtype, const char *name) {
  if (!t.is_cuda()) raise_type(name, "must be a CUDA tensor");
  if (t.scalar_type() != dtype) {
    PyErr_Format(PyExc_TypeError, "%s must have dtype %S, got %S", name, (PyObject *)torch::getTHPDtype(dtype),
                 (PyObject *)torch::getTHPDtype(t.scalar_type()));
    throw Failed();
  }
  if (!t.is_contiguous()) raise_type(name, "must be contiguous");
  return t.data_ptr();
}

void *device_pointer(PyObject *obj, at::ScalarType dtype, const char *name) {
  return device_pointer(tensor(obj, name), dtype, name);
}

int64_t integer(PyObject *obj) {
  const long long v = PyLong_AsLongLong(obj);
  if (v == -1 && PyErr_Occurred()) throw Failed();
  return v;
}

swb_context *context_of(PyObject *obj) {
  if (obj == Py_None) return nullptr;  // a closed context: the library refuses it
  void *p = PyLong_AsVoidPtr(obj);
  if (!p && PyErr_Occurred()) throw Failed();
  return static_cast<swb_context *>(p);
}

void *stream_of(PyObject *device) {
  return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)integer(device)).stream();
}

at::Tensor output(PyObject *given, at::IntArrayRef sizes, at::ScalarType dtype, const at::Tensor &like) {
  if (given != Py_None) return at::Tensor();
  return at::empty(sizes, at::TensorOptions().dtype(dtype).device(like.device()));
}

// Runs `call` without the GIL, turns its status into an exception, returns the output object.
template <typename Call>
PyObject *finish(swb_context *ctx, PyObject *given, at::Tensor &fresh, Call call) {
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = call();
  Py_END_ALLOW_THREADS
  if (st != SWB_OK) raise_status(st, swb_last_error(ctx));
  if (given != Py_None) {
    Py_INCREF(given);
    return given;
  }
  return THPVariable_Wrap(std::move(fresh));
}

template <typename Body>
PyObject *guarded(Py_ssize_t have, Py_ssize_t want, Body body) {
  if (have != want) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, have);
    return nullptr;
  }
  try {
    return body();
  } catch (const Failed &) {
    return nullptr;
  } catch (const std::exception &e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

void require_rank(const at::Tensor &t, int64_t rank, const char *name) {
  if (t.dim() < rank) {
    PyErr_Format(PyExc_IndexError, "%s must have %d dimensions", name, (int)rank);
    throw Failed();
  }
}

// spmv(ctx, device, options, row_ptr, col_idx, val, x, y | None, rows | None)
PyObject *spmv(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return guarded(n, 9, [&]() -> PyObject * {
    swb_context *ctx = context_of(a[0]);
    const swb_options o = options_of(a[2]);
    const at::Tensor &rp = tensor(a[3], "row_ptr"), &val = tensor(a[5], "val"), &x = tensor(a[6], "x");
    const int64_t rows = a[8] == Py_None ? rp.numel() - 1 : integer(a[8]), cols = x.numel(), nnz = val.numel();
    auto *p_rp = (const int32_t *)device_pointer(rp, at::kInt, "row_ptr");
    auto *p_ci = (const int32_t *)device_pointer(a[4], at::kInt, "col_idx");
    auto *p_v = (const float *)device_pointer(val, at::kFloat, "val");
    auto *p_x = (const float *)device_pointer(x, at::kFloat, "x");
    at::Tensor fresh = output(a[7], {rows}, at::kFloat, x);
    auto *p_y = (float *)(fresh.defined() ? fresh.data_ptr() : device_pointer(a[7], at::kFloat, "y"));
    void *s = stream_of(a[1]);
    return finish(ctx, a[7], fresh, [&] { return swb_spmv(ctx, &o, rows, cols, nnz, p_rp, p_ci, p_v, p_x, p_y, s); });
  });
}

// coo_spmv(ctx, device, options, rows, row_idx, col_idx, val, x, y | None)
PyObject *coo_spmv(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return guarded(n, 9, [&]() -> PyObject * {
    swb_context *ctx = context_of(a[0]);
    const swb_options o = options_of(a[2]);
    const int64_t rows = integer(a[3]);
    const at::Tensor &val = tensor(a[6], "val"), &x = tensor(a[7], "x");
    const int64_t cols = x.numel(), nnz = val.numel();
    auto *p_ri = (const int32_t *)device_pointer(a[4], at::kInt, "row_idx");
    auto *p_ci = (const int32_t *)device_pointer(a[5], at::kInt, "col_idx");
    auto *p_v = (const float *)device_pointer(val, at::kFloat, "val");
    auto *p_x = (const float *)device_pointer(x, at::kFloat, "x");
    at::Tensor fresh = output(a[8], {rows}, at::kFloat, x);
    auto *p_y = (float *)(fresh.defined() ? fresh.data_ptr() : device_pointer(a[8], at::kFloat, "y"));
    void *s = stream_of(a[1]);
    return finish(ctx, a[8], fresh,
                  [&] { return swb_coo_spmv(ctx, &o, rows, cols, nnz, p_ri, p_ci, p_v, p_x, p_y, s); });
  });
}

// spmm(ctx, device, options, row_ptr, col_idx, val, B, C | None, rows | None)
PyObject *spmm(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return guarded(n, 9, [&]() -> PyObject * {
    swb_context *ctx = context_of(a[0]);
    const swb_options o = options_of(a[2]);
    const at::Tensor &rp = tensor(a[3], "row_ptr"), &val = tensor(a[5], "val"), &B = tensor(a[6], "B");
    require_rank(B, 2, "B");
    const int64_t rows = a[8] == Py_None ? rp.numel() - 1 : integer(a[8]), cols = B.size(0), rhs = B.size(1),
                  nnz = val.numel();
    auto *p_rp = (const int32_t *)device_pointer(rp, at::kInt, "row_ptr");
    auto *p_ci = (const int32_t *)device_pointer(a[4], at::kInt, "col_idx");
    auto *p_v = (const float *)device_pointer(val, at::kFloat, "val");
    auto *p_B = (const float *)device_pointer(B, at::kFloat, "B");
    at::Tensor fresh = output(a[7], {rows, rhs}, at::kFloat, B);
    auto *p_C = (float *)(fresh.defined() ? fresh.data_ptr() : device_pointer(a[7], at::kFloat, "C"));
    void *s = stream_of(a[1]);
    return finish(ctx, a[7], fresh,
                  [&] { return swb_spmm(ctx, &o, rows, cols, nnz, rhs, p_rp, p_ci, p_v, p_B, p_C, s); });
  });
}

// bsr_spmm(ctx, device, options, block_row_ptr, block_col_idx, block_values, B, block_size, C | None)
PyObject *bsr_spmm(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return guarded(n, 9, [&]() -> PyObject * {
    swb_context *ctx = context_of(a[0]);
    const swb_options o = options_of(a[2]);
    const at::Tensor &brp = tensor(a[3], "block_row_ptr"), &bci = tensor(a[4], "block_col_idx"),
                     &bv = tensor(a[5], "block_values"), &B = tensor(a[6], "B");
    require_rank(B, 2, "B");
    const int64_t bs = integer(a[7]), rows = (brp.numel() - 1) * bs, cols = B.size(0), rhs = B.size(1),
                  nnzb = bci.numel();
    const at::ScalarType dt = bv.scalar_type();
    if (dt != at::kFloat && dt != at::kBFloat16) raise_type("block_values", "must be float32 or bfloat16");
    if (bv.numel() != nnzb * bs * bs) {
      const std::string message =
          "block values size must equal the number of blocks times block_size squared, but got " +
          std::to_string(bv.numel()) + " and " + std::to_string(nnzb) + " blocks";
      raise_status(SWB_ERR_INVALID_SHAPE, message.c_str());
    }
    auto *p_rp = (const int32_t *)device_pointer(brp, at::kInt, "block_row_ptr");
    auto *p_ci = (const int32_t *)device_pointer(bci, at::kInt, "block_col_idx");
    void *p_v = device_pointer(bv, dt, "block_values"), *p_B = device_pointer(B, dt, "B");
    at::Tensor fresh = output(a[8], {rows, rhs}, dt, B);
    void *p_C = fresh.defined() ? fresh.data_ptr() : device_pointer(a[8], dt, "C");
    void *s = stream_of(a[1]);
    return finish(ctx, a[8], fresh, [&] {
      return dt == at::kFloat ? swb_bsr_spmm_f32(ctx, &o, rows, cols, nnzb, bs, rhs, p_rp, p_ci, (const float *)p_v,
                                                 (const float *)p_B, (float *)p_C, s)
                              : swb_bsr_spmm_bf16(ctx, &o, rows, cols, nnzb, bs, rhs, p_rp, p_ci, (const uint16_t *)p_v,
                                                  (const uint16_t *)p_B, (uint16_t *)p_C, s);
    });
  });
}

// bind(SparseWaveError, SwbOptions): the Python types that the calls above raise and accept
PyObject *bind(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return guarded(n, 2, [&]() -> PyObject * {
    if (!PyType_Check(a[0]) || !PyType_Check(a[1])) raise_type("bind", "needs two types");
    Py_INCREF(a[0]);
    Py_INCREF(a[1]);
    g_error = a[0];
    g_options = (PyTypeObject *)a[1];
    Py_RETURN_NONE;
  });
}

#define SWB_FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {SWB_FAST(spmv), SWB_FAST(coo_spmv), SWB_FAST(spmm), SWB_FAST(bsr_spmm), SWB_FAST(bind),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "swb_torch", "Device-tensor operator calls over the C ABI.", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_swb_torch(void) { return PyModule_Create(&g_module); }
