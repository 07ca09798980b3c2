// Host path of the per-batch operators as a CPython extension.
//
// A masked GEMM of a small batch takes 4 us on a B200; through ctypes the same call spent 11 us in the
// interpreter (attribute reads, argument checks, six argument conversions, a device guard and a stream
// query in Python).  Here the checks read the tensors' C++ objects directly and the C ABI is called without
// conversions: 3 us a call with the launch.  The functions mirror their Python callers in layer.py and masks.py,
// which keep the rarely used forms (peer buffers, the CUDA-core twin) for themselves.
#include <Python.h>

#define NPY_NO_DEPRECATED_API NPY_1_7_API_VERSION
#include <numpy/arrayobject.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <vector>

#include "../../include/tilesparse.h"

namespace {

PyObject* g_error_type = nullptr;   // TileSparseError(code, message)

// The interpreter's lock is given back while the library works, as ctypes does: a call may build a schedule, or wait for
// room in the launch queue behind work that needs the interpreter.
template <typename F>
int unlocked(F&& f) {
  pybind11::gil_scoped_release nogil;
  return f();
}

struct Layer {
  ts_layer_t* h;
  int64_t K, N;
  at::ScalarType dtype;
  int device;
  bool all_columns;                 // every column of W is kept by some tile
};

PyObject* fail_value(const char* msg) {
  PyErr_SetString(PyExc_ValueError, msg);
  return nullptr;
}

PyObject* fail_code(int code) {
  char buf[1024];
  ts_last_error(buf, sizeof(buf));
  PyObject* e = g_error_type ? PyObject_CallFunction(g_error_type, "is", code, buf) : nullptr;
  if (e) {
    PyErr_SetObject(g_error_type, e);
    Py_DECREF(e);
  } else if (!PyErr_Occurred()) {
    PyErr_SetString(PyExc_RuntimeError, buf);
  }
  return nullptr;
}

Layer* layer_of(PyObject* capsule) { return static_cast<Layer*>(PyCapsule_GetPointer(capsule, "ts_layer")); }

bool on_device(const at::Tensor& t, int device) { return t.is_cuda() && t.get_device() == device; }

void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream(); }

at::Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType dtype, int device) {
  return at::detail::empty_cuda(sizes, dtype, c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device)), std::nullopt);
}

// A new [N, M] output.  Rows of columns no tile keeps must read as zero; the GEMM writes all the others, so
// only a beta that reads the output needs the whole buffer cleared.
int new_output(const Layer& l, int64_t M, bool read_back, void* stream, at::Tensor* out) {
  *out = new_tensor({l.N, M}, l.dtype, l.device);
  if (read_back) {
    out->zero_();
  } else if (!l.all_columns && M > 0) {
    return unlocked([&] { return ts_layer_zero_pruned(l.h, static_cast<int>(M), out->data_ptr(), M, stream); });
  }
  return TS_OK;
}

// layer_desc(handle, K, N, is_bf16, device, all_columns) -> capsule
PyObject* py_layer_desc(PyObject*, PyObject* args) {
  unsigned long long h;
  long long K, N;
  int bf16, device, all;
  if (!PyArg_ParseTuple(args, "KLLiii", &h, &K, &N, &bf16, &device, &all)) return nullptr;
  Layer* l = new Layer{reinterpret_cast<ts_layer_t*>(h), K, N, bf16 ? at::kBFloat16 : at::kHalf, device, all != 0};
  return PyCapsule_New(l, "ts_layer", [](PyObject* c) { delete static_cast<Layer*>(PyCapsule_GetPointer(c, "ts_layer")); });
}

bool read_float(PyObject* o, float* out) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) return false;
  *out = static_cast<float>(v);
  return true;
}

// masked_gemm(layer, At, out | None, alpha, beta, bias | None, act[, kept bits]) -> out; with the mask's bits (uint8 [N,
// K / 8]) ts_layer_mask_nonfinite follows
PyObject* py_masked_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7 && n != 8) return fail_value("masked_gemm takes 7 or 8 arguments");
  if (a[0] == Py_None) return fail_code(ts_masked_gemm_ex(nullptr, 0, nullptr, 0, nullptr, 0, nullptr, nullptr));   // a closed layer
  Layer* l = layer_of(a[0]);
  if (!l) return nullptr;
  if (!THPVariable_Check(a[1])) return fail_value("At must be a tensor");
  const at::Tensor& At = THPVariable_Unpack(a[1]);
  if (At.dim() != 2 || At.size(0) != l->K || At.scalar_type() != l->dtype || !on_device(At, l->device)) {
    return fail_value("At must be a [K, M] tensor of the layer's dtype on the layer's device");
  }
  const int64_t M = At.size(1);
  if (At.stride(1) != 1) return fail_value("At must have M contiguous");
  ts_epilogue_t ep = {};
  if (!read_float(a[3], &ep.alpha) || !read_float(a[4], &ep.beta)) return nullptr;
  ep.activation = static_cast<int>(PyLong_AsLong(a[6]));
  if (a[5] != Py_None) {
    if (!THPVariable_Check(a[5])) return fail_value("bias must be a tensor");
    const at::Tensor& b = THPVariable_Unpack(a[5]);
    if (b.scalar_type() != at::kFloat || b.numel() != l->N || !on_device(b, l->device) || !b.is_contiguous()) {
      return fail_value("bias must be a contiguous fp32 [N] tensor on the layer's device");
    }
    ep.bias_dev = static_cast<const float*>(b.data_ptr());
  }
  c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(l->device)));
  void* stream = stream_of(l->device);
  at::Tensor fresh;
  const at::Tensor* out = &fresh;
  if (a[2] == Py_None) {
    const int rc = new_output(*l, M, ep.beta != 0.0f, stream, &fresh);
    if (rc != TS_OK) return fail_code(rc);
  } else {
    if (!THPVariable_Check(a[2])) return fail_value("out must be a tensor");
    out = &THPVariable_Unpack(a[2]);
    if (out->dim() != 2 || out->size(0) != l->N || out->size(1) != M || out->scalar_type() != l->dtype ||
        out->stride(1) != 1 || !on_device(*out, l->device)) {
      return fail_value("out must be an [N, M] tensor of the layer's dtype with M contiguous");
    }
  }
  const uint8_t* bits = nullptr;
  int64_t bits_ld = 0;
  if (n == 8) {
    if (!THPVariable_Check(a[7])) return fail_value("the mask's bits must be a tensor");
    bits = static_cast<const uint8_t*>(THPVariable_Unpack(a[7]).data_ptr());
    bits_ld = THPVariable_Unpack(a[7]).stride(0);
  }
  const int rc = unlocked([&] {
    const int r = ts_masked_gemm_ex(l->h, static_cast<int>(M), At.data_ptr(), At.stride(0), out->data_ptr(), out->stride(0), &ep, stream);
    if (r != TS_OK || !bits) return r;
    return ts_layer_mask_nonfinite(l->h, static_cast<int>(M), At.data_ptr(), At.stride(0), out->data_ptr(), out->stride(0), ep.alpha, bits,
                                   bits_ld, stream);
  });
  if (rc != TS_OK) return fail_code(rc);
  if (out == &fresh) return THPVariable_Wrap(std::move(fresh));
  Py_INCREF(a[2]);
  return a[2];
  END_HANDLE_TH_ERRORS
}

// The transpose of a 16-bit matrix with contiguous rows, or TS_* / a ValueError already set (*out undefined).
bool transpose(const at::Tensor& x, void* stream, at::Tensor* out) {
  if (x.dim() != 2 || x.element_size() != 2 || x.stride(1) != 1 || !x.is_cuda()) {
    fail_value("transpose16 takes a 2-D 16-bit CUDA tensor with contiguous rows");
    return false;
  }
  *out = new_tensor({x.size(1), x.size(0)}, x.scalar_type(), x.get_device());
  const int rc = unlocked([&] {
    return ts_transpose16(x.data_ptr(), x.stride(0), out->data_ptr(), out->stride(0), static_cast<int>(x.size(0)),
                          static_cast<int>(x.size(1)), stream);
  });
  if (rc != TS_OK) fail_code(rc);
  return rc == TS_OK;
}

// transpose16(x) -> its transpose
PyObject* py_transpose16(PyObject*, PyObject* arg) {
  HANDLE_TH_ERRORS
  if (!THPVariable_Check(arg)) return fail_value("transpose16 takes a tensor");
  const at::Tensor& x = THPVariable_Unpack(arg);
  if (!x.is_cuda()) return fail_value("transpose16 takes a 2-D 16-bit CUDA tensor with contiguous rows");
  c10::cuda::OptionalCUDAGuard guard(x.device());
  at::Tensor out;
  if (!transpose(x, stream_of(x.get_device()), &out)) return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// linear(layer, A [M, K], transpose_out) -> C [M, N], or Ct [N, M]
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3) return fail_value("linear takes 3 arguments");
  if (a[0] == Py_None) return fail_code(ts_masked_gemm_ex(nullptr, 0, nullptr, 0, nullptr, 0, nullptr, nullptr));   // a closed layer
  Layer* l = layer_of(a[0]);
  if (!l) return nullptr;
  if (!THPVariable_Check(a[1])) return fail_value("A must be a tensor");
  const at::Tensor& A = THPVariable_Unpack(a[1]);
  if (A.dim() != 2 || A.size(1) != l->K || A.scalar_type() != l->dtype || !on_device(A, l->device)) {
    return fail_value("A must be an [M, K] tensor of the layer's dtype on the layer's device");
  }
  const int64_t M = A.size(0);
  c10::cuda::OptionalCUDAGuard guard(A.device());
  void* stream = stream_of(l->device);
  at::Tensor At, out;
  if (!transpose(A, stream, &At)) return nullptr;
  ts_epilogue_t ep = {};
  ep.alpha = 1.0f;
  int rows = 0, rc = TS_OK;
  if (a[2] == Py_True) rc = ts_layer_row_output(l->h, static_cast<int>(M), &rows);
  if (rc != TS_OK) return fail_code(rc);
  if (rows) {
    out = new_tensor({M, l->N}, l->dtype, l->device);
    rc = unlocked([&] { return ts_masked_gemm_rows(l->h, static_cast<int>(M), At.data_ptr(), At.stride(0), out.data_ptr(), l->N, &ep, stream); });
    if (rc != TS_OK) return fail_code(rc);
    return THPVariable_Wrap(std::move(out));
  }
  rc = new_output(*l, M, false, stream, &out);
  if (rc == TS_OK) {
    rc = unlocked([&] { return ts_masked_gemm_ex(l->h, static_cast<int>(M), At.data_ptr(), At.stride(0), out.data_ptr(), M, &ep, stream); });
  }
  if (rc != TS_OK) return fail_code(rc);
  if (a[2] == Py_True) {
    at::Tensor C;
    if (!transpose(out, stream, &C)) return nullptr;
    return THPVariable_Wrap(std::move(C));
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyObject* int_array(int n, int32_t** data) {
  npy_intp dims[1] = {n};
  PyObject* a = PyArray_SimpleNew(1, dims, NPY_INT32);
  *data = a ? static_cast<int32_t*>(PyArray_DATA(reinterpret_cast<PyArrayObject*>(a))) : nullptr;
  return a;
}

// build_mask(mode, scores, G, sparsity, sparsity_is_f64, g1percent, want_residual, device)
//   -> (masks, residuals | None, [(bounds, tile_k_ptr, kept_k, tile_n_ptr, kept_n)], thresholds),
// or None when a score is not a float32 matrix with contiguous rows on that device (the caller converts).
PyObject* py_build_mask(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  int mode, G, is_f64, want_residual, device;
  double sparsity, g1;
  PyObject* list;
  if (!PyArg_ParseTuple(args, "iO!ididii", &mode, &PyList_Type, &list, &G, &sparsity, &is_f64, &g1, &want_residual, &device)) return nullptr;
  const Py_ssize_t n = PyList_GET_SIZE(list);
  std::vector<const void*> scores(n);
  std::vector<int> K(n), N(n);
  std::vector<int64_t> ld(n), ld_mask(n);
  for (Py_ssize_t l = 0; l < n; ++l) {
    PyObject* o = PyList_GET_ITEM(list, l);
    if (!THPVariable_Check(o)) Py_RETURN_NONE;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (t.dim() != 2 || t.scalar_type() != at::kFloat || !on_device(t, device)) Py_RETURN_NONE;
    scores[l] = t.data_ptr();
    K[l] = static_cast<int>(t.size(0));
    N[l] = static_cast<int>(t.size(1));
    ld[l] = t.stride(0);
    if (t.stride(1) != 1) {
      // a dimension of one element has any stride, and contiguous() leaves such a tensor as it is
      if (t.numel() > 0 && (N[l] != 1 || (ld[l] < 1 && K[l] > 1))) Py_RETURN_NONE;
      ld[l] = std::max<int64_t>(ld[l], N[l]);
    }
  }
  c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device)));
  void* stream = stream_of(device);
  std::vector<at::Tensor> masks, resid;
  std::vector<uint8_t*> mask_ptr(n), resid_ptr(n, nullptr);
  for (Py_ssize_t l = 0; l < n; ++l) {
    masks.push_back(new_tensor({K[l], N[l]}, at::kBool, device));   // the kernels write 0 / 1 bytes
    mask_ptr[l] = static_cast<uint8_t*>(masks[l].data_ptr());
    ld_mask[l] = N[l];
    if (want_residual) {
      resid.push_back(new_tensor({K[l], N[l]}, at::kBool, device));
      resid[l].zero_();
      resid_ptr[l] = static_cast<uint8_t*>(resid[l].data_ptr());
    }
  }
  ts_mask_result_t* res = nullptr;
  const int rc = unlocked([&] {
    return ts_build_tw_mask(mode, static_cast<int>(n), scores.data(), K.data(), N.data(), ld.data(), G, sparsity, is_f64, g1,
                            mask_ptr.data(), ld_mask.data(), want_residual ? resid_ptr.data() : nullptr, &res, stream);
  });
  if (rc != TS_OK) return fail_code(rc);
  PyObject *py_masks = PyList_New(n), *py_tiles = PyList_New(n), *py_resid = nullptr;
  if (want_residual) {
    py_resid = PyList_New(n);
  } else {
    py_resid = Py_None;
    Py_INCREF(Py_None);
  }
  bool ok = py_masks && py_tiles && py_resid;
  for (Py_ssize_t l = 0; ok && l < n; ++l) {
    int nt = 0, nk = 0, nn = 0;
    ts_mask_result_layer(res, static_cast<int>(l), &nt, &nk, &nn);
    int32_t *b, *kp, *kk, *np, *nc;
    PyObject* arrays[5] = {int_array(nt + 1, &b), int_array(nt + 1, &kp), int_array(nk, &kk), int_array(nt + 1, &np), int_array(nn, &nc)};
    for (PyObject* a : arrays) ok = ok && a;
    PyObject* tuple = ok ? PyTuple_New(5) : nullptr;
    ok = ok && tuple;
    if (!ok) {
      for (PyObject* a : arrays) Py_XDECREF(a);
      break;
    }
    ts_mask_result_copy(res, static_cast<int>(l), b, kp, kk, np, nc);
    for (int i = 0; i < 5; ++i) PyTuple_SET_ITEM(tuple, i, arrays[i]);
    PyList_SET_ITEM(py_tiles, l, tuple);
    PyList_SET_ITEM(py_masks, l, THPVariable_Wrap(masks[l]));
    if (want_residual) PyList_SET_ITEM(py_resid, l, THPVariable_Wrap(resid[l]));
  }
  double thr[3];
  ts_mask_result_thresholds(res, thr);
  ts_mask_result_destroy(res);
  if (!ok) {
    Py_XDECREF(py_masks);
    Py_XDECREF(py_tiles);
    Py_XDECREF(py_resid);
    return nullptr;
  }
  return Py_BuildValue("(NNN(ddd))", py_masks, py_resid, py_tiles, thr[0], thr[1], thr[2]);
  END_HANDLE_TH_ERRORS
}

PyObject* py_bind(PyObject*, PyObject* type) {
  Py_XDECREF(g_error_type);
  Py_INCREF(type);
  g_error_type = type;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"bind", py_bind, METH_O, "Sets the exception type raised for C-ABI errors."},
    {"layer_desc", py_layer_desc, METH_VARARGS, "Capsule describing a layer to the functions below."},
    {"masked_gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_masked_gemm)), METH_FASTCALL, "TWLayer.masked_gemm"},
    {"build_mask", py_build_mask, METH_VARARGS, "masks.build_mask on float32 CUDA scores"},
    {"transpose16", py_transpose16, METH_O, "layer.transpose16"},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_linear)), METH_FASTCALL, "layer.masked_linear"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_tsfast", "Host path of the per-batch operators.", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tsfast() {
  import_array();
  return PyModule_Create(&kModule);
}
