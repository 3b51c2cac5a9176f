// The package's Python entry points in native code: argument conversion from torch tensors, result
// allocation and the call into librelax_b200.so.
//
// Why: built from ctypes objects, one call cost 15 to 20 us of host time - as much as, or more than, the
// kernels of a decode step take - so an eager caller was bound by the interpreter.  Here tensors
// become DLTensor views on the stack, the result comes from the caching allocator directly, and a
// call is one C function (the semantics - what is accepted, which checks fail with which message -
// are those of the global functions in librelax_b200.so, which are called as before).
//
// The library's entry points are reached through the addresses the Python side resolved (init), so
// that there is one loaded copy of it, wherever it was loaded from.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/Context.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/relax_b200_packed.h"

namespace {

// ------------------------------------------------------------------ the library
struct Lib {
  decltype(&rb200_last_error) last_error;
  decltype(&rb200_set_stream) set_stream;
  decltype(&RB200FuncCall) func_call;
  decltype(&RB200FuncGetGlobal) func_get_global;
  decltype(&rb200_encode_ft) encode_ft;
  decltype(&rb200_moe_route) moe_route;
  decltype(&rb200_moe_route_workspace_bytes) moe_route_workspace_bytes;
  decltype(&rb200_moe_gather) moe_gather;
  decltype(&rb200_moe_combine) moe_combine;
} lib;
PyObject* error_class = nullptr;

PyObject* fail_library() {
  PyErr_SetString(error_class, lib.last_error());
  return nullptr;
}

// A registered function by name, looked up once.
struct Global {
  const char* name;
  RB200FunctionHandle handle = nullptr;
  explicit Global(const char* n) : name(n) {}
  RB200FunctionHandle get() {
    if (!handle && (lib.func_get_global(name, &handle) != 0 || !handle))
      PyErr_Format(PyExc_ValueError, "Cannot find global function %s", name);
    return handle;
  }
};

// ------------------------------------------------------------------ one call's arguments
constexpr int kMaxArgs = 16;

bool dl_type(c10::ScalarType t, DLDataType* out) {
  switch (t) {
    case c10::ScalarType::Half: *out = {kDLFloat, 16, 1}; return true;
    case c10::ScalarType::Float: *out = {kDLFloat, 32, 1}; return true;
    case c10::ScalarType::Char: *out = {kDLInt, 8, 1}; return true;
    case c10::ScalarType::Byte: *out = {kDLUInt, 8, 1}; return true;
    case c10::ScalarType::Int: *out = {kDLInt, 32, 1}; return true;
    case c10::ScalarType::Long: *out = {kDLInt, 64, 1}; return true;
    case c10::ScalarType::BFloat16: *out = {kDLBfloat, 16, 1}; return true;
    case c10::ScalarType::UInt32: *out = {kDLUInt, 32, 1}; return true;
    default: return false;
  }
}

bool any_device() {
  static const bool have = c10::cuda::device_count() > 0;
  return have;
}

// The library's stream on this thread becomes torch's current stream of the device the tensors are on (and
// stays it until the next call), and that device current for the lifetime of the object.
struct OnStream {
  c10::cuda::OptionalCUDAGuard guard;
  explicit OnStream(int device) {
    if (device < 0 && !any_device()) return;
    if (device >= 0) guard.set_index(static_cast<c10::DeviceIndex>(device));
    lib.set_stream(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream());
  }
};

struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

struct Frame {
  RB200Value v[kMaxArgs];
  int tc[kMaxArgs];
  DLTensor dl[kMaxArgs];
  int n = 0;
  int device = -1;  // index of the first CUDA tensor's device

  void null() {
    v[n].v_handle = nullptr;
    tc[n++] = RB200_ARG_NULL;
  }
  void integer(int64_t x) {
    v[n].v_int64 = x;
    tc[n++] = RB200_ARG_INT;
  }
  void real(double x) {
    v[n].v_float64 = x;
    tc[n++] = RB200_ARG_FLOAT;
  }
  void str(const char* s) {
    v[n].v_str = s;
    tc[n++] = RB200_ARG_STR;
  }
  bool tensor(const at::Tensor& t) {
    DLTensor& d = dl[n];
    if (!dl_type(t.scalar_type(), &d.dtype)) {
      PyErr_Format(PyExc_KeyError, "unsupported tensor dtype %s", c10::toString(t.scalar_type()));
      return false;
    }
    d.data = t.data_ptr();
    const bool cuda = t.is_cuda();
    d.device.device_type = cuda ? kDLCUDA : kDLCPU;
    d.device.device_id = cuda ? t.get_device() : 0;
    if (cuda && device < 0) device = d.device.device_id;
    d.ndim = static_cast<int32_t>(t.dim());
    d.shape = const_cast<int64_t*>(t.sizes().data());
    d.strides = t.is_contiguous() ? nullptr : const_cast<int64_t*>(t.strides().data());
    d.byte_offset = 0;
    v[n].v_handle = &d;
    tc[n++] = RB200_ARG_DLTENSOR;
    return true;
  }
  // any argument a global function takes
  bool object(PyObject* o) {
    if (n >= kMaxArgs) {
      PyErr_SetString(PyExc_TypeError, "too many PackedFunc arguments");
      return false;
    }
    if (o == Py_None) {
      null();
    } else if (THPVariable_Check(o)) {
      return tensor(THPVariable_Unpack(o));
    } else if (PyLong_Check(o)) {  // bool too
      const long long x = PyLong_AsLongLong(o);
      if (x == -1 && PyErr_Occurred()) return false;
      integer(x);
    } else if (PyFloat_Check(o)) {
      real(PyFloat_AS_DOUBLE(o));
    } else if (PyUnicode_Check(o)) {
      const char* s = PyUnicode_AsUTF8(o);
      if (!s) return false;
      str(s);
    } else {
      PyErr_Format(PyExc_TypeError, "unsupported PackedFunc argument %R", reinterpret_cast<PyObject*>(Py_TYPE(o)));
      return false;
    }
    return true;
  }
  bool call(RB200FunctionHandle f, RB200Value* ret, int* ret_tc) {
    if (!f) return false;
    int rc;
    {
      NoGil other_threads_run;  // a call may wait for the device (host tensors, act-order set-up)
      OnStream on(device);
      rc = lib.func_call(f, v, tc, n, ret, ret_tc);
    }
    if (rc != 0) fail_library();
    return rc == 0;
  }
  bool call(RB200FunctionHandle f) {
    RB200Value ret;
    int ret_tc = RB200_ARG_NULL;
    return call(f, &ret, &ret_tc);
  }
};

const at::Tensor* as_tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a tensor, got %R", what, reinterpret_cast<PyObject*>(Py_TYPE(o)));
    return nullptr;
  }
  return &THPVariable_Unpack(o);
}
// what int() takes: a group size may come as the quotient k / groups
bool as_int(PyObject* o, int64_t* out) {
  if (!PyLong_Check(o)) {
    PyObject* i = PyNumber_Long(o);
    if (!i) return false;
    *out = PyLong_AsLongLong(i);
    Py_DECREF(i);
  } else {
    *out = PyLong_AsLongLong(o);
  }
  return !(*out == -1 && PyErr_Occurred());
}
bool as_real(PyObject* o, double* out) {
  *out = PyFloat_AsDouble(o);
  return !(*out == -1.0 && PyErr_Occurred());
}

at::Tensor empty_on(c10::IntArrayRef sizes, c10::ScalarType dtype, const at::Tensor& like) {
  // (under deterministic algorithms torch.empty may fill its result: rows of no expert are then NaN)
  if (like.is_cuda() && !at::globalContext().deterministicAlgorithms())
    return at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt);
  return at::empty(sizes, at::TensorOptions().dtype(dtype).device(like.device()));
}
// x's leading extents followed by n
at::Tensor empty_rows(const at::Tensor& x, int64_t n) {
  c10::SmallVector<int64_t, 6> sizes(x.sizes().begin(), x.sizes().end());
  if (sizes.empty()) sizes.push_back(n);
  sizes.back() = n;
  return empty_on(sizes, c10::ScalarType::Half, x);
}
// the caller's `out`, or a new tensor
struct Out {
  at::Tensor t;
  PyObject* given = nullptr;
  bool take(PyObject* o) {
    if (o == Py_None) return true;
    const at::Tensor* p = as_tensor(o, "out");
    if (!p) return false;
    t = *p;
    given = o;
    return true;
  }
  PyObject* give() { return given ? (Py_INCREF(given), given) : THPVariable_Wrap(std::move(t)); }
};

#define NEED_ARGS(N)                                                                          \
  if (nargs != (N)) {                                                                         \
    PyErr_Format(PyExc_TypeError, "%s expects %d arguments, got %zd", __func__, (N), nargs);  \
    return nullptr;                                                                           \
  }
// C++ exceptions become the Python ones that torch itself raises (torch.OutOfMemoryError among them)
#define GUARD_BEGIN HANDLE_TH_ERRORS
#define GUARD_END END_HANDLE_TH_ERRORS

RB200FunctionHandle as_handle(PyObject* o) { return PyLong_AsVoidPtr(o); }

PyObject* result(const RB200Value& ret, int tc) {
  if (tc == (int)RB200_ARG_HANDLE) {
    if (!ret.v_handle) Py_RETURN_NONE;
    return PyLong_FromVoidPtr(ret.v_handle);
  }
  if (tc == (int)RB200_ARG_INT) return PyLong_FromLongLong(ret.v_int64);
  Py_RETURN_NONE;
}

// call(handle, *args)
PyObject* call(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  if (nargs < 1) return PyErr_SetString(PyExc_TypeError, "call expects a function handle"), nullptr;
  RB200FunctionHandle f = as_handle(a[0]);
  if (!f && PyErr_Occurred()) return nullptr;
  Frame fr;
  for (Py_ssize_t i = 1; i < nargs; ++i)
    if (!fr.object(a[i])) return nullptr;
  RB200Value ret;
  int tc = RB200_ARG_NULL;
  if (!fr.call(f, &ret, &tc)) return nullptr;
  return result(ret, tc);
  GUARD_END
}

// check(*args): raises for what no global function takes
PyObject* check(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  Frame fr;
  for (Py_ssize_t i = 0; i < nargs; ++i)
    if (!fr.object(a[i])) return nullptr;
  Py_RETURN_NONE;
  GUARD_END
}

// call_like(handle, tensor, *args): destination-passing function whose result is a new tensor like the first
PyObject* call_like(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  if (nargs < 2) return PyErr_SetString(PyExc_TypeError, "call_like expects a handle and a tensor"), nullptr;
  RB200FunctionHandle f = as_handle(a[0]);
  if (!f && PyErr_Occurred()) return nullptr;
  const at::Tensor* w = as_tensor(a[1], "argument 0");
  if (!w) return nullptr;
  at::Tensor out = w->is_cuda() && w->is_contiguous() ? empty_on(w->sizes(), w->scalar_type(), *w) : at::empty_like(*w);
  Frame fr;
  for (Py_ssize_t i = 1; i < nargs; ++i)
    if (!fr.object(a[i])) return nullptr;
  if (fr.n >= kMaxArgs) return PyErr_SetString(PyExc_TypeError, "too many PackedFunc arguments"), nullptr;
  if (!fr.tensor(out) || !fr.call(f)) return nullptr;
  return THPVariable_Wrap(std::move(out));
  GUARD_END
}

bool is_swiglu(PyObject* o) { return PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, "swiglu") == 0; }

// gemm_ft(x, w_pre, scales, weight_bits, bias, residual, activation, binary_op, unary_op, group_size, out)
PyObject* gemm_ft(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(11);
  static Global int4("cutlass.ft_gemm_fp16_int4"), int8("cutlass.ft_gemm_fp16_int8");
  const at::Tensor *x = as_tensor(a[0], "x"), *w = x ? as_tensor(a[1], "w_pre") : nullptr;
  int64_t bits, group;
  Out out;
  if (!w || !as_int(a[3], &bits) || !as_int(a[9], &group) || !out.take(a[10])) return nullptr;
  if (x->dim() < 1 || w->dim() < 1) return PyErr_SetString(PyExc_IndexError, "x and w_pre need a dimension"), nullptr;
  const int64_t k = x->size(-1), n = w->size(-1) * (bits == 4 ? 2 : 1), m = k ? x->numel() / k : 0;
  if (!out.given) out.t = empty_rows(*x, is_swiglu(a[6]) ? n / 2 : n);
  int64_t bias_stride = 0;
  if (a[4] != Py_None) {
    const at::Tensor* b = as_tensor(a[4], "bias");
    if (!b) return nullptr;
    if (b->numel() == m * n && m > 1) bias_stride = n;
  }
  Frame f;
  if (!f.tensor(*x) || !f.tensor(*w) || !f.object(a[2]) || !f.object(a[4]) || !f.object(a[5]) || !f.object(a[6]) ||
      !f.object(a[7]) || !f.object(a[8]))
    return nullptr;
  f.integer(m);
  f.integer(n);
  f.integer(k);
  f.integer(group > 0 ? group : k);
  f.integer(bias_stride);
  if (!f.tensor(out.t) || !f.call((bits == 4 ? int4 : int8).get())) return nullptr;
  return out.give();
  GUARD_END
}

// gemm_q4(x, w_pre, scales, zeros, bias, residual, activation, binary_op, unary_op, group_size, zero_const, out)
PyObject* gemm_q4(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(12);
  static Global fn("relax_b200.gemm_fp16_q4f16");
  const at::Tensor *x = as_tensor(a[0], "x"), *w = x ? as_tensor(a[1], "w_pre") : nullptr;
  int64_t group;
  double zero_const;
  Out out;
  if (!w || !as_int(a[9], &group) || !as_real(a[10], &zero_const) || !out.take(a[11])) return nullptr;
  if (x->dim() < 1 || w->dim() < 1) return PyErr_SetString(PyExc_IndexError, "x and w_pre need a dimension"), nullptr;
  if (!out.given) out.t = empty_rows(*x, w->size(0) / (is_swiglu(a[6]) ? 2 : 1));
  Frame f;
  if (!f.tensor(*x) || !f.tensor(*w)) return nullptr;
  for (int i = 2; i < 9; ++i)
    if (!f.object(a[i])) return nullptr;
  f.integer(group);
  f.real(zero_const);
  if (!f.tensor(out.t) || !f.call(fn.get())) return nullptr;
  return out.give();
  GUARD_END
}

bool gather_into(const at::Tensor& x, PyObject* perm, at::Tensor* out) {
  static Global fn("relax_b200.gather_columns");
  const at::Tensor xc = x.contiguous();
  *out = x.is_cuda() ? empty_on(x.sizes(), x.scalar_type(), x) : at::empty_like(xc);
  Frame f;
  return f.tensor(xc) && f.object(perm) && f.tensor(*out) && f.call(fn.get());
}

// gather_columns(x, perm)
PyObject* gather_columns(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(2);
  const at::Tensor* x = as_tensor(a[0], "x");
  at::Tensor out;
  if (!x || !gather_into(*x, a[1], &out)) return nullptr;
  return THPVariable_Wrap(std::move(out));
  GUARD_END
}

// gemm_gptq(x, w_pre, scales, zeros, bias, perm, out)
PyObject* gemm_gptq(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(7);
  static Global fn("relax_b200.gemm_fp16_autogptq");
  const at::Tensor *x = as_tensor(a[0], "x"), *w = x ? as_tensor(a[1], "w_pre") : nullptr;
  Out out;
  if (!w || !out.take(a[6])) return nullptr;
  if (x->dim() < 1 || w->dim() < 2) return PyErr_SetString(PyExc_IndexError, "x needs one dimension, w_pre two"), nullptr;
  at::Tensor gathered;
  if (a[5] != Py_None) {
    if (!gather_into(*x, a[5], &gathered)) return nullptr;
    x = &gathered;
  }
  if (!out.given) out.t = empty_rows(*x, w->size(1));
  Frame f;
  if (!f.tensor(*x) || !f.tensor(*w) || !f.object(a[2]) || !f.object(a[3]) || !f.object(a[4]) || !f.tensor(out.t) ||
      !f.call(fn.get()))
    return nullptr;
  return out.give();
  GUARD_END
}

// moe_ft(x, w_pre, scales, indptr, zeros, out, first_expert)
PyObject* moe_ft(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(7);
  static Global fn("cutlass.moe_gemm");
  const at::Tensor *x = as_tensor(a[0], "x"), *w = as_tensor(a[1], "w_pre"), *s = as_tensor(a[2], "scales"),
                   *indptr = as_tensor(a[3], "indptr");
  int64_t first;
  Out out;
  if (!x || !w || !s || !indptr || !out.take(a[5]) || !as_int(a[6], &first)) return nullptr;
  if (x->dim() < 1 || w->dim() < 1 || s->dim() < 1 || indptr->dim() < 1)
    return PyErr_SetString(PyExc_IndexError, "x, w_pre, scales and indptr need a dimension"), nullptr;
  if (!out.given) out.t = empty_on({x->size(0), s->size(-1)}, c10::ScalarType::Half, *x);
  const int64_t local = w->size(0);
  at::Tensor view;
  if (first || local != indptr->size(0)) {
    view = indptr->slice(0, first, first + local);
    indptr = &view;
  }
  Frame f;
  if (!f.tensor(*x) || !f.tensor(*w) || !f.tensor(*s) || !f.object(a[4]) || !f.tensor(*indptr)) return nullptr;
  f.null();
  if (!f.tensor(out.t)) return nullptr;
  if (first) f.integer(1);
  if (!f.call(fn.get())) return nullptr;
  return out.give();
  GUARD_END
}

// moe_q4(x, w_pre, scales, indptr, zeros, group_size, zero_const, out)
PyObject* moe_q4(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(8);
  static Global fn("relax_b200.moe_gemm_q4f16");
  const at::Tensor *x = as_tensor(a[0], "x"), *w = as_tensor(a[1], "w_pre");
  int64_t group;
  double zero_const;
  Out out;
  if (!x || !w || !as_int(a[5], &group) || !as_real(a[6], &zero_const) || !out.take(a[7])) return nullptr;
  if (x->dim() < 1 || w->dim() < 2) return PyErr_SetString(PyExc_IndexError, "x needs one dimension, w_pre two"), nullptr;
  if (!out.given) out.t = empty_on({x->size(0), w->size(1)}, c10::ScalarType::Half, *x);
  Frame f;
  if (!f.tensor(*x) || !f.tensor(*w) || !f.object(a[2]) || !f.object(a[4]) || !f.object(a[3])) return nullptr;
  f.integer(group);
  f.real(zero_const);
  if (!f.tensor(out.t) || !f.call(fn.get())) return nullptr;
  return out.give();
  GUARD_END
}

// group_fp16(x, weight, indptr, workspace, out)
PyObject* group_fp16(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(5);
  static Global fn("cutlass.group_gemm_fp16_sm90");
  const at::Tensor *x = as_tensor(a[0], "x"), *w = as_tensor(a[1], "weight");
  Out out;
  if (!x || !w || !out.take(a[4])) return nullptr;
  if (x->dim() < 1 || w->dim() < 2) return PyErr_SetString(PyExc_IndexError, "x needs one dimension, weight two"), nullptr;
  if (!out.given) out.t = empty_on({x->size(0), w->size(1)}, c10::ScalarType::Half, *x);
  Frame f;
  if (!f.tensor(*x) || !f.tensor(*w) || !f.object(a[2]) || !f.object(a[3]) || !f.tensor(out.t) || !f.call(fn.get()))
    return nullptr;
  return out.give();
  GUARD_END
}

// ------------------------------------------------------------------ plain C entries (pointers, current stream)
void* current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// moe_route(logits, top_k, out | None, workspace | None)
PyObject* moe_route(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(4);
  const at::Tensor* given = as_tensor(a[0], "logits");
  int64_t top_k;
  if (!given || !as_int(a[1], &top_k)) return nullptr;
  if (given->dim() != 2) return PyErr_SetString(PyExc_ValueError, "logits must be [tokens, experts]"), nullptr;
  const int64_t t = given->size(0), e = given->size(1), r = t * top_k;
  at::Tensor o[4];
  if (a[2] == Py_None) {
    o[0] = empty_on({e}, c10::ScalarType::Long, *given);
    o[1] = empty_on({r}, c10::ScalarType::Int, *given);
    o[2] = empty_on({r}, c10::ScalarType::Float, *given);
    o[3] = empty_on({r}, c10::ScalarType::Int, *given);
  } else {
    PyObject* seq = PySequence_Fast(a[2], "out must be the four result tensors");
    if (!seq) return nullptr;
    bool fine = PySequence_Fast_GET_SIZE(seq) == 4;
    if (!fine) PyErr_SetString(PyExc_ValueError, "out must be the four result tensors");
    for (int i = 0; fine && i < 4; ++i) {
      const at::Tensor* p = as_tensor(PySequence_Fast_GET_ITEM(seq, i), "out");
      if (p) o[i] = *p;
      else fine = false;
    }
    Py_DECREF(seq);
    if (!fine) return nullptr;
  }
  const int64_t need = static_cast<int64_t>(lib.moe_route_workspace_bytes(t, top_k));
  at::Tensor ws;
  if (a[3] == Py_None) {
    ws = empty_on({need}, c10::ScalarType::Byte, *given);
  } else {
    const at::Tensor* p = as_tensor(a[3], "workspace");
    if (!p) return nullptr;
    ws = *p;
    if (ws.numel() < need) {
      PyErr_Format(PyExc_ValueError, "routing workspace holds %lld bytes, %lld needed", (long long)ws.numel(), (long long)need);
      return nullptr;
    }
  }
  at::Tensor logits = *given;
  if (logits.scalar_type() != c10::ScalarType::Float || !logits.is_contiguous())
    logits = logits.contiguous().to(c10::ScalarType::Float);
  if (lib.moe_route(logits.data_ptr(), t, e, top_k, o[0].data_ptr<int64_t>(), static_cast<int32_t*>(o[1].data_ptr()),
                    static_cast<float*>(o[2].data_ptr()), static_cast<int32_t*>(o[3].data_ptr()), ws.data_ptr(),
                    static_cast<size_t>(ws.numel()), current_stream()) != 0)
    return fail_library();
  PyObject* tup = PyTuple_New(4);
  for (int i = 0; tup && i < 4; ++i) PyTuple_SET_ITEM(tup, i, THPVariable_Wrap(o[i]));
  return tup;
  GUARD_END
}

// moe_gather(x, token_of_row, out | None)
PyObject* moe_gather(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(3);
  const at::Tensor *x = as_tensor(a[0], "x"), *tok = as_tensor(a[1], "token_of_row");
  Out out;
  if (!x || !tok || !out.take(a[2])) return nullptr;
  if (x->dim() < 2) return PyErr_SetString(PyExc_IndexError, "x must be [tokens, k]"), nullptr;
  if (!out.given) out.t = empty_on({tok->numel(), x->size(1)}, c10::ScalarType::Half, *x);
  const at::Tensor xc = x->contiguous();
  if (lib.moe_gather(xc.data_ptr(), static_cast<int32_t*>(tok->data_ptr()), out.t.data_ptr(), tok->numel(), x->size(1),
                     current_stream()) != 0)
    return fail_library();
  return out.give();
  GUARD_END
}

// moe_combine(y, row_of_flat, gate_of_row, top_k, out | None)
PyObject* moe_combine(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(5);
  const at::Tensor *y = as_tensor(a[0], "y"), *rof = as_tensor(a[1], "row_of_flat"), *gate = as_tensor(a[2], "gate_of_row");
  int64_t top_k;
  Out out;
  if (!y || !rof || !gate || !as_int(a[3], &top_k) || !out.take(a[4])) return nullptr;
  if (y->dim() < 2) return PyErr_SetString(PyExc_IndexError, "y must be [rows, n]"), nullptr;
  if (top_k == 0) return PyErr_SetString(PyExc_ZeroDivisionError, "top_k is zero"), nullptr;
  const int64_t tokens = rof->numel() / top_k;
  if (!out.given) out.t = empty_on({tokens, y->size(1)}, c10::ScalarType::Half, *y);
  const at::Tensor yc = y->contiguous();
  if (lib.moe_combine(yc.data_ptr(), static_cast<int32_t*>(rof->data_ptr()), static_cast<float*>(gate->data_ptr()),
                      out.t.data_ptr(), tokens, top_k, y->size(1), current_stream()) != 0)
    return fail_library();
  return out.give();
  GUARD_END
}

// encode_ft(y, weight_bits, group_size)
PyObject* encode_ft(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  GUARD_BEGIN
  NEED_ARGS(3);
  const at::Tensor* y = as_tensor(a[0], "y");
  int64_t bits, group;
  if (!y || !as_int(a[1], &bits) || !as_int(a[2], &group)) return nullptr;
  if (y->dim() != 2) return PyErr_SetString(PyExc_ValueError, "y must be [n, k]"), nullptr;
  const int64_t n = y->size(0), k = y->size(1);
  const bool per_row = group <= 0 || group >= k;
  at::Tensor packed = empty_on({k, bits == 4 ? n / 2 : n}, c10::ScalarType::Char, *y);
  at::Tensor scales = per_row ? empty_on({n}, c10::ScalarType::Half, *y) : empty_on({k / group, n}, c10::ScalarType::Half, *y);
  const at::Tensor yc = y->contiguous();
  if (lib.encode_ft(yc.data_ptr(), packed.data_ptr(), scales.data_ptr(), n, k, static_cast<int>(bits), group,
                    current_stream()) != 0)
    return fail_library();
  PyObject* tup = PyTuple_New(2);
  if (!tup) return nullptr;
  PyTuple_SET_ITEM(tup, 0, THPVariable_Wrap(std::move(packed)));
  PyTuple_SET_ITEM(tup, 1, THPVariable_Wrap(std::move(scales)));
  return tup;
  GUARD_END
}

// init(error_class, {symbol: address})
PyObject* init(PyObject*, PyObject* args) {
  PyObject *cls, *table;
  if (!PyArg_ParseTuple(args, "OO!", &cls, &PyDict_Type, &table)) return nullptr;
  Py_INCREF(cls);
  Py_XSETREF(error_class, cls);
#define TAKE(FIELD, SYMBOL)                                                             \
  {                                                                                     \
    PyObject* o = PyDict_GetItemString(table, SYMBOL);                                  \
    void* p = o ? PyLong_AsVoidPtr(o) : nullptr;                                        \
    if (!p) return PyErr_Format(PyExc_RuntimeError, "no address for %s", SYMBOL);       \
    lib.FIELD = reinterpret_cast<decltype(lib.FIELD)>(p);                               \
  }
  TAKE(last_error, "rb200_last_error")
  TAKE(set_stream, "rb200_set_stream")
  TAKE(func_call, "RB200FuncCall")
  TAKE(func_get_global, "RB200FuncGetGlobal")
  TAKE(encode_ft, "rb200_encode_ft")
  TAKE(moe_route, "rb200_moe_route")
  TAKE(moe_route_workspace_bytes, "rb200_moe_route_workspace_bytes")
  TAKE(moe_gather, "rb200_moe_gather")
  TAKE(moe_combine, "rb200_moe_combine")
#undef TAKE
  Py_RETURN_NONE;
}

#define FAST(NAME) {#NAME, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(NAME)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"init", init, METH_VARARGS, nullptr},
    FAST(call),      FAST(check),     FAST(call_like), FAST(gemm_ft),    FAST(gemm_q4),    FAST(gemm_gptq),   FAST(gather_columns),
    FAST(moe_ft),    FAST(moe_q4),    FAST(group_fp16), FAST(moe_route),  FAST(moe_gather),  FAST(moe_combine),
    FAST(encode_ft), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_host(void) {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "built_for", RB200_BUILT_FOR) != 0) Py_CLEAR(m);
  return m;
}
