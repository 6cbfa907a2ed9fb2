// The host side of the tensor-level wrappers (ops.py): allocates the outputs and the workspace of a call, passes their addresses
// to the C entry point and hands the tensors back, all in one native call.  From Python the same work (allocations, views,
// data pointers, a foreign call with up to twenty arguments) took 10 to 20 us per call beside 3 to 6 us for its launches, and a
// training step that is issued from Python makes 25 of them.  Checks of types and shapes stay in ops.py; the entry points are
// bound by address from the library that cabi.py has loaded, so this module links against torch only and needs no CUDA headers.
#include <Python.h>

#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/Tensor.h>
#include <ATen/ops/as_strided.h>
#include <ATen/ops/empty.h>
#include <c10/core/Stream.h>

#include <string.h>

#include "../../include/metis_nvfp4.h"

namespace {

// ---- entry points, by address -------------------------------------------------------------------------------

#define METIS_HOST_ENTRIES(X)                                                                                                  \
  X(metis_nvfp4_quantize) X(metis_nvfp4_quantize_workspace_bytes) X(metis_nvfp4_quantize_dual)                                  \
  X(metis_nvfp4_quantize_dual_workspace_bytes) X(metis_nvfp4_quantize_dual_finish) X(metis_rmsnorm_nvfp4_quantize)              \
  X(metis_col_mean) X(metis_col_mean_workspace_bytes) X(metis_nvfp4_gemv) X(metis_nvfp4_gemm) X(metis_nvfp4_gemm_scaled)       \
  X(metis_nvfp4_gemm_joined) X(metis_nvfp4_gemm_workspace_bytes) X(metis_lowrank_scale) X(metis_lowrank_factors)
struct Entries {
#define X(name) decltype(&::name) name = nullptr;
  METIS_HOST_ENTRIES(X)
#undef X
} lib;

// ---- arguments and results --------------------------------------------------------------------------------------

struct BadArguments {};

// While calls run that other threads need not wait for (as a foreign call from Python would have it).
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

struct Args {
  PyObject* const* v;
  Py_ssize_t n, at = 0;
  PyObject* next() {
    if (at >= n) {
      PyErr_SetString(PyExc_TypeError, "too few arguments");
      throw BadArguments();
    }
    return v[at++];
  }
  const at::Tensor& tensor() {
    PyObject* o = next();
    if (!THPVariable_Check(o)) {
      PyErr_Format(PyExc_TypeError, "argument %zd has to be a tensor", at - 1);
      throw BadArguments();
    }
    return THPVariable_Unpack(o);
  }
  at::Tensor optional() {
    if (at < n && v[at] == Py_None) { ++at; return at::Tensor(); }
    return tensor();
  }
  int64_t i64() {
    const long long x = PyLong_AsLongLong(next());
    if (x == -1 && PyErr_Occurred()) throw BadArguments();
    return x;
  }
  bool truth() {
    const int x = PyObject_IsTrue(next());
    if (x < 0) throw BadArguments();
    return x != 0;
  }
  uint64_t u64() {
    const unsigned long long x = PyLong_AsUnsignedLongLong(next());
    if (x == (unsigned long long)-1 && PyErr_Occurred()) throw BadArguments();
    return x;
  }
  double f64() {
    const double x = PyFloat_AsDouble(next());
    if (x == -1.0 && PyErr_Occurred()) throw BadArguments();
    return x;
  }
  void* address() { return reinterpret_cast<void*>(static_cast<uintptr_t>(u64())); }
};

template <typename T = void> T* ptr(const at::Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }

PyObject* result(int32_t rc, std::initializer_list<at::Tensor> tensors) {
  PyObject* out = PyTuple_New(1 + (Py_ssize_t)tensors.size());
  if (!out) return nullptr;
  PyTuple_SET_ITEM(out, 0, PyLong_FromLong(rc));
  Py_ssize_t i = 1;
  for (const at::Tensor& t : tensors) {
    PyObject* o = t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None);
    if (!o) { Py_DECREF(out); return nullptr; }
    PyTuple_SET_ITEM(out, i++, o);
  }
  return out;
}

#define METIS_HOST_BEGIN(args, nargs) HANDLE_TH_ERRORS try { Args a{args, nargs};
#define METIS_HOST_END } catch (const BadArguments&) { return nullptr; } END_HANDLE_TH_ERRORS

at::Tensor bytes_on(const at::Tensor& like, int64_t n) { return at::empty({n < 16 ? 16 : n}, at::TensorOptions().dtype(at::kByte).device(like.device())); }
at::Tensor floats_on(const at::Tensor& like, int64_t n) { return at::empty({n}, at::TensorOptions().dtype(at::kFloat).device(like.device())); }

// codes, scales and unit of one quantized [R, C] as views of a single allocation
struct Packed { at::Tensor codes, scales, unit; };
Packed packed(const at::Tensor& like, int64_t R, int64_t C, int64_t sf_bytes) {
  const int64_t half = C / 2, at_scales = (R * half + 255) & ~(int64_t)255, at_unit = (at_scales + sf_bytes + 255) & ~(int64_t)255;
  const at::Tensor buf = at::empty({at_unit + 16}, at::TensorOptions().dtype(at::kByte).device(like.device()));
  return {buf.as_strided({R, half}, {half, 1}), buf.as_strided({sf_bytes}, {1}, at_scales), buf.as_strided({4}, {1}, at_unit).view(at::kFloat)};
}

// ---- calls (positional arguments, in this order; each returns (status, tensors...)) ---------------------------

// x [rows, cols], dtype code, transposed, flags, seed, offset, sf_layout, bytes of the scales, extra workspace bytes, mean or None, stream
PyObject* quantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const at::Tensor& x = a.tensor();
  const int32_t dtype = (int32_t)a.i64();
  const bool transposed = a.truth();
  const uint32_t flags = (uint32_t)a.i64();
  const uint64_t seed = a.u64(), offset = a.u64();
  const int32_t layout = (int32_t)a.i64();
  const int64_t sf_bytes = a.i64(), extra = a.i64();
  const at::Tensor mean = a.optional();
  void* stream = a.address();
  const int64_t rows = x.size(0), cols = x.size(1), R = transposed ? cols : rows, C = transposed ? rows : cols;
  Packed q;
  int32_t rc;
  {
    NoGil free_;
    q = packed(x, R, C, sf_bytes);
    const at::Tensor ws = bytes_on(x, lib.metis_nvfp4_quantize_workspace_bytes(R, C) + extra);
    rc = lib.metis_nvfp4_quantize(x.data_ptr(), dtype, rows, cols, x.stride(0), ptr<float>(mean), flags, seed, offset, layout,
                                  ptr<uint8_t>(q.codes), ptr<uint8_t>(q.scales), ptr<float>(q.unit), ws.data_ptr(), ws.numel(), stream);
  }
  return result(rc, {q.codes, q.scales, q.unit});
  METIS_HOST_END
}

// x, dtype code, flags, seed, offset, sf_layout, bytes of the scales of Q and of Qt, mean or None, whether token sums, stream
// -> codes, scales, unit, codes_t, scales_t, unit_t, token sums or None, workspace
PyObject* quantize_dual(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const at::Tensor& x = a.tensor();
  const int32_t dtype = (int32_t)a.i64();
  const uint32_t flags = (uint32_t)a.i64();
  const uint64_t seed = a.u64(), offset = a.u64();
  const int32_t layout = (int32_t)a.i64();
  const int64_t sf_bytes = a.i64(), sf_bytes_t = a.i64();
  const at::Tensor mean = a.optional();
  const bool want_sums = a.truth();
  void* stream = a.address();
  const int64_t rows = x.size(0), cols = x.size(1);
  Packed q, qt;
  at::Tensor sums, ws;
  int32_t rc;
  {
    NoGil free_;
    q = packed(x, rows, cols, sf_bytes);
    qt = packed(x, cols, rows, sf_bytes_t);
    ws = bytes_on(x, lib.metis_nvfp4_quantize_dual_workspace_bytes(rows, cols));
    if (want_sums) sums = floats_on(x, cols);
    rc = lib.metis_nvfp4_quantize_dual(x.data_ptr(), dtype, rows, cols, x.stride(0), ptr<float>(mean), flags, seed, offset, layout,
                                       ptr<uint8_t>(q.codes), ptr<uint8_t>(q.scales), ptr<float>(q.unit), ptr<uint8_t>(qt.codes),
                                       ptr<uint8_t>(qt.scales), ptr<float>(qt.unit), ptr<float>(sums), ws.data_ptr(), ws.numel(), stream);
  }
  return result(rc, {q.codes, q.scales, q.unit, qt.codes, qt.scales, qt.unit, sums, ws});
  METIS_HOST_END
}

// rows, cols, which pass, sf_layout, scales, unit, codes_t, scales_t, unit_t, token sums or None, workspace, stream, then the
// stream as torch has it (id, device index, device type): every buffer is recorded as used there
PyObject* quantize_dual_finish(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const int64_t rows = a.i64(), cols = a.i64();
  const uint32_t which = (uint32_t)a.i64();
  const int32_t layout = (int32_t)a.i64();
  const at::Tensor &scales = a.tensor(), &unit = a.tensor(), &codes_t = a.tensor(), &scales_t = a.tensor(), &unit_t = a.tensor();
  const at::Tensor sums = a.optional();
  const at::Tensor& ws = a.tensor();
  void* stream = a.address();
  const int64_t id = a.i64(), index = a.i64(), type = a.i64();
  int32_t rc;
  {
    NoGil free_;
    rc = lib.metis_nvfp4_quantize_dual_finish(rows, cols, which, layout, ptr<uint8_t>(scales), ptr<float>(unit), ptr<uint8_t>(codes_t),
                                              ptr<uint8_t>(scales_t), ptr<float>(unit_t), ptr<float>(sums), ws.data_ptr(), ws.numel(), stream);
    if (rc == 0) {
      // one view of each allocation: Q's (scales), Qt's (codes_t), the workspace, the sums
      const c10::Stream st = c10::Stream::unpack3(id, (c10::DeviceIndex)index, (c10::DeviceType)type);
      scales.record_stream(st);
      codes_t.record_stream(st);
      ws.record_stream(st);
      if (sums.defined()) sums.record_stream(st);
    }
  }
  return result(rc, {});
  METIS_HOST_END
}

// x, dtype code, gamma, its dtype code, eps, sf_layout, bytes of the scales, extra workspace bytes, dtype code of the normalised tensor
// or -1, stream -> codes, scales, unit, normalised tensor or None
PyObject* rmsnorm_quantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const at::Tensor& x = a.tensor();
  const int32_t dtype = (int32_t)a.i64();
  const at::Tensor& gamma = a.tensor();
  const int32_t gamma_dtype = (int32_t)a.i64();
  const float eps = (float)a.f64();
  const int32_t layout = (int32_t)a.i64();
  const int64_t sf_bytes = a.i64(), extra = a.i64(), norm_dtype = a.i64();
  void* stream = a.address();
  const int64_t rows = x.size(0), cols = x.size(1);
  Packed q;
  at::Tensor norm;
  int32_t rc;
  {
    NoGil free_;
    q = packed(x, rows, cols, sf_bytes);
    if (norm_dtype >= 0)
      norm = at::empty({rows, cols}, at::TensorOptions().dtype(norm_dtype == METIS_DTYPE_BF16 ? at::kBFloat16 : at::kFloat).device(x.device()));
    const at::Tensor ws = bytes_on(x, lib.metis_nvfp4_quantize_workspace_bytes(rows, cols) + extra);
    rc = lib.metis_rmsnorm_nvfp4_quantize(x.data_ptr(), dtype, rows, cols, x.stride(0), gamma.data_ptr(), gamma_dtype, eps, layout,
                                          ptr<uint8_t>(q.codes), ptr<uint8_t>(q.scales), ptr<float>(q.unit), ptr(norm), ws.data_ptr(), ws.numel(), stream);
  }
  return result(rc, {q.codes, q.scales, q.unit, norm});
  METIS_HOST_END
}

// x, dtype code, stream -> mean
PyObject* col_mean(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const at::Tensor& x = a.tensor();
  const int32_t dtype = (int32_t)a.i64();
  void* stream = a.address();
  const int64_t rows = x.size(0), cols = x.size(1);
  at::Tensor mean;
  int32_t rc;
  {
    NoGil free_;
    mean = floats_on(x, cols);
    const at::Tensor ws = bytes_on(x, lib.metis_col_mean_workspace_bytes(rows, cols));
    rc = lib.metis_col_mean(x.data_ptr(), dtype, rows, cols, x.stride(0), ptr<float>(mean), ws.data_ptr(), ws.numel(), stream);
  }
  return result(rc, {mean});
  METIS_HOST_END
}

// codes, scales, unit, sf_layout, R, C, v or None, stream -> out
PyObject* gemv(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const at::Tensor &codes = a.tensor(), &scales = a.tensor(), &unit = a.tensor();
  const int32_t layout = (int32_t)a.i64();
  const int64_t R = a.i64(), C = a.i64();
  const at::Tensor v = a.optional();
  void* stream = a.address();
  at::Tensor out;
  int32_t rc;
  {
    NoGil free_;
    out = floats_on(codes, R);
    rc = lib.metis_nvfp4_gemv(ptr<uint8_t>(codes), ptr<uint8_t>(scales), ptr<float>(unit), layout, R, C, ptr<float>(v), ptr<float>(out), stream);
  }
  return result(rc, {out});
  METIS_HOST_END
}

// yv [M, r], s, its dtype code, unit_a, unit_b, stream -> out
PyObject* lowrank_scale(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const at::Tensor &yv = a.tensor(), &s = a.tensor();
  const int32_t s_dtype = (int32_t)a.i64();
  const at::Tensor &unit_a = a.tensor(), &unit_b = a.tensor();
  void* stream = a.address();
  const int64_t M = yv.size(0), r = yv.size(1);
  at::Tensor out;
  int32_t rc;
  {
    NoGil free_;
    out = at::empty({M, r}, yv.options());
    rc = lib.metis_lowrank_scale(yv.data_ptr(), M, r, yv.stride(0), s.data_ptr(), s_dtype, ptr<float>(unit_a), ptr<float>(unit_b), out.data_ptr(), stream);
  }
  return result(rc, {out});
  METIS_HOST_END
}

// yv [M, r] fp32, s, its dtype code, unit_a, unit_b, u [N, r] fp32, parts, stream -> t, u as bf16
PyObject* lowrank_factors(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const at::Tensor &yv = a.tensor(), &s = a.tensor();
  const int32_t s_dtype = (int32_t)a.i64();
  const at::Tensor &unit_a = a.tensor(), &unit_b = a.tensor(), &u = a.tensor();
  const int64_t parts = a.i64();
  void* stream = a.address();
  const int64_t M = yv.size(0), r = yv.size(1), N = u.size(0);
  at::Tensor t, u_out;
  int32_t rc;
  {
    NoGil free_;
    t = at::empty({M, parts * r}, yv.options().dtype(at::kBFloat16));
    u_out = at::empty({N, parts * r}, yv.options().dtype(at::kBFloat16));
    rc = lib.metis_lowrank_factors(ptr<float>(yv), M, r, yv.stride(0), s.data_ptr(), s_dtype, ptr<float>(unit_a), ptr<float>(unit_b), t.data_ptr(),
                                   ptr<float>(u), N, u.stride(0), u_out.data_ptr(), (int32_t)parts, stream);
  }
  return result(rc, {t, u_out});
  METIS_HOST_END
}

// M, N, K, alpha, codes, scales, unit of A, of B, T or None, U or None, cvec0, rvec0, cvec1, rvec1 (None where there is none), C or None,
// D or None, dtype code of D, debug bits, SM limit, status or None, rows_ready (address or 0), s or None, its dtype code, unit_a, unit_b,
// stream -> D, scaled copy or None, bytes of workspace the product was given (as a number behind the tensors)
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  metis_gemm_args g;
  memset(&g, 0, sizeof g);
  g.M = a.i64(); g.N = a.i64(); g.K = a.i64();
  g.alpha = (float)a.f64();
  const at::Tensor& codes_a = a.tensor();
  g.a_codes = ptr<uint8_t>(codes_a); g.a_scales = ptr<uint8_t>(a.tensor()); g.a_unit = ptr<float>(a.tensor());
  g.b_codes = ptr<uint8_t>(a.tensor()); g.b_scales = ptr<uint8_t>(a.tensor()); g.b_unit = ptr<float>(a.tensor());
  const at::Tensor t = a.optional(), u = a.optional();
  if (t.defined()) {
    g.rank = (int32_t)t.size(1);
    g.lr_t = ptr(t); g.ldt = t.stride(0);
    g.lr_u = ptr(u); g.ldu = u.stride(0);
  }
  g.cvec0 = ptr<float>(a.optional()); g.rvec0 = ptr<float>(a.optional());
  g.cvec1 = ptr<float>(a.optional()); g.rvec1 = ptr<float>(a.optional());
  const at::Tensor c = a.optional();
  if (c.defined()) { g.c = ptr(c); g.ldc = c.stride(0); }
  at::Tensor d = a.optional();
  g.d_dtype = (int32_t)a.i64();
  g.reserved = (int32_t)a.i64();
  g.sm_limit = (int32_t)a.i64();
  g.status = ptr<int32_t>(a.optional());
  void* rows_ready = a.address();
  const at::Tensor s = a.optional();
  const int32_t s_dtype = (int32_t)a.i64();
  const float *unit_a = ptr<float>(a.optional()), *unit_b = ptr<float>(a.optional());
  g.stream = a.address();
  at::Tensor scaled, ws;
  int64_t ws_bytes = 0;
  int32_t rc;
  {
    NoGil free_;
    if (!d.defined())
      d = at::empty({g.M, g.N}, at::TensorOptions().dtype(g.d_dtype == METIS_DTYPE_BF16 ? at::kBFloat16 : at::kFloat).device(codes_a.device()));
    g.d = d.data_ptr(); g.ldd = d.stride(0);
    if (g.M <= 128) ws_bytes = lib.metis_nvfp4_gemm_workspace_bytes(g.M, g.N, g.K);
    if (ws_bytes > 0) {                          // decode-sized product: scratch for its split-K partial sums
      ws = bytes_on(codes_a, ws_bytes);
      g.workspace = ws.data_ptr(); g.workspace_bytes = ws_bytes;
    }
    if (s.defined()) scaled = at::empty({g.M, g.N}, at::TensorOptions().dtype(at::kBFloat16).device(codes_a.device()));
    if (rows_ready)       rc = lib.metis_nvfp4_gemm_joined(&g, rows_ready, ptr(s), s_dtype, unit_a, unit_b, ptr(scaled));
    else if (s.defined()) rc = lib.metis_nvfp4_gemm_scaled(&g, ptr(s), s_dtype, unit_a, unit_b, ptr(scaled));
    else                  rc = lib.metis_nvfp4_gemm(&g);
  }
  PyObject* out = result(rc, {d, scaled, at::Tensor()});
  if (out) {
    PyObject* n = PyLong_FromLongLong(ws_bytes);
    PyObject* none = PyTuple_GET_ITEM(out, 3);
    PyTuple_SET_ITEM(out, 3, n);
    Py_DECREF(none);
  }
  return out;
  METIS_HOST_END
}

// name, address: binds an entry point; returns whether this module has a use for it
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  METIS_HOST_BEGIN(args, nargs)
  const char* name = PyUnicode_AsUTF8(a.next());
  if (!name) return nullptr;
  void* address = a.address();
#define X(entry) if (strcmp(name, #entry) == 0) { lib.entry = reinterpret_cast<decltype(lib.entry)>(address); Py_RETURN_TRUE; }
  METIS_HOST_ENTRIES(X)
#undef X
  Py_RETURN_FALSE;
  METIS_HOST_END
}

#define METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(quantize), METHOD(quantize_dual), METHOD(quantize_dual_finish), METHOD(rmsnorm_quantize), METHOD(col_mean),
                         METHOD(gemv), METHOD(lowrank_scale), METHOD(lowrank_factors), METHOD(gemm), METHOD(bind), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "metis_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_metis_host(void) { return PyModule_Create(&module); }
