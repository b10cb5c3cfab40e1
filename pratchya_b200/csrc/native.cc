// The host side of an op between Python and the C ABI of libpratchya_b200.so, as a CPython extension on torch's C++ API: output
// tensors are allocated, pointers taken and kernels launched in one call.  Through ctypes an op of one small kernel costs its
// caller 12 to 15 us, of which the launch is 2: every torch.empty from Python 2.5, the foreign call with its converted arguments 3
// to 4, shapes and data_ptr() the rest.  Here: 3 to 5.
//
// Two kinds of functions.  `pb_*` are the C entries as include/pratchya_b200.h declares them, a wrapper made from each declaration:
// a tensor stands for its data pointer, None for a null pointer, anything with a buffer (a ctypes structure) for its address; the
// trailing stream may be left out and is then the current one of the first tensor's device; a status other than PB_OK raises.  The
// others are whole ops of _qualia/_ops.py.  Those take only what needs no conversion and no refusal (plain contiguous CUDA
// tensors of the usual types, no dispatch mode watching) and return None for anything else, which the Python text then handles.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <initializer_list>
#include <numeric>
#include <optional>
#include <tuple>
#include <utility>

#include "pratchya_b200.h"

namespace {

PyObject* g_pb_error = nullptr;       // pratchya_b200._lib.PbError

// raises PbError(status, what the library says about it)
PyObject* raise_status(int status) {
  PyObject* exc = g_pb_error ? PyObject_CallFunction(g_pb_error, "is", status, pb_last_error()) : nullptr;
  if (exc) {
    PyErr_SetObject(g_pb_error, exc);
    Py_DECREF(exc);
  } else if (!PyErr_Occurred()) {
    PyErr_SetString(PyExc_RuntimeError, pb_last_error());
  }
  return nullptr;
}

template <typename F>
auto without_gil(F&& f) {
  struct Released {
    PyThreadState* state = PyEval_SaveThread();
    ~Released() { PyEval_RestoreThread(state); }
  } released;
  return f();
}

void* current_stream(c10::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

// ---- the C entries --------------------------------------------------------------------------------------------------
struct Taken {
  std::optional<c10::Device> device;
  Py_buffer buffers[4];
  int n_buffers = 0;
  ~Taken() { for (int i = 0; i < n_buffers; ++i) PyBuffer_Release(&buffers[i]); }
};

bool take(PyObject* o, Taken& t, void** out) {
  if (o == Py_None) { *out = nullptr; return true; }
  if (THPVariable_Check(o)) {
    const at::Tensor& x = THPVariable_Unpack(o);
    *out = x.data_ptr();
    if (!t.device && x.is_cuda()) t.device = x.device();
    return true;
  }
  if (PyLong_Check(o)) { *out = PyLong_AsVoidPtr(o); return !PyErr_Occurred(); }
  if (t.n_buffers == 4 || PyObject_GetBuffer(o, &t.buffers[t.n_buffers], PyBUF_SIMPLE) != 0) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "too many structure arguments");
    return false;
  }
  *out = t.buffers[t.n_buffers++].buf;
  return true;
}
template <typename T>
bool take_arg(PyObject* o, Taken& t, T* out) {
  if constexpr (std::is_pointer_v<T>) {
    void* p = nullptr;
    if (!take(o, t, &p)) return false;
    *out = static_cast<T>(p);
    return true;
  } else if constexpr (std::is_floating_point_v<T>) {
    const double v = PyFloat_AsDouble(o);
    *out = (T)v;
    return !(v == -1.0 && PyErr_Occurred());
  } else {
    const long long v = PyLong_AsLongLong(o);
    *out = (T)v;
    return !(v == -1 && PyErr_Occurred());
  }
}

template <auto Fn> struct Entry;
template <typename R, typename... A, R (*Fn)(A...)>
struct Entry<Fn> {
  static constexpr Py_ssize_t kArgs = sizeof...(A);
  static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    std::tuple<A...> v{};
    Taken t;
    PyObject* result = nullptr;
    if (fill(args, n, t, v, std::index_sequence_for<A...>{})) {
      c10::cuda::OptionalCUDAGuard guard;
      if (t.device) guard.set_device(*t.device);
      const R r = without_gil([&] { return std::apply(Fn, v); });
      if constexpr (std::is_same_v<R, int>) {
        if (r != PB_OK) raise_status(r);
        else { Py_INCREF(Py_None); result = Py_None; }
      } else {
        result = PyLong_FromSize_t(r);
      }
    }
    return result;
    END_HANDLE_TH_ERRORS
  }
  template <size_t... I>
  static bool fill(PyObject* const* args, Py_ssize_t n, Taken& t, std::tuple<A...>& v, std::index_sequence<I...>) {
    using Last = std::tuple_element_t<kArgs - 1, std::tuple<A...>>;
    const bool add_stream = n == kArgs - 1 && std::is_same_v<R, int> && std::is_same_v<Last, void*>;
    if (n != kArgs && !add_stream) {
      PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", kArgs, n);
      return false;
    }
    const bool ok = (((Py_ssize_t)I >= n || take_arg(args[I], t, &std::get<I>(v))) && ...);
    if (!ok || !add_stream) return ok;
    if (!t.device) { PyErr_SetString(PyExc_TypeError, "no CUDA tensor among the arguments"); return false; }
    if constexpr (std::is_same_v<Last, void*>) std::get<kArgs - 1>(v) = current_stream(*t.device);
    return true;
  }
};

// ---- whole ops --------------------------------------------------------------------------------------------------------
constexpr auto kE4M3 = at::kFloat8_e4m3fn;
constexpr auto kE5M2 = at::kFloat8_e5m2;
constexpr auto kE8M0 = at::kFloat8_e8m0fnu;

PyObject* none() { Py_INCREF(Py_None); return Py_None; }
PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* wrap(std::initializer_list<at::Tensor> ts) {
  PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
  Py_ssize_t i = 0;
  for (const at::Tensor& t : ts) PyTuple_SET_ITEM(r, i++, THPVariable_Wrap(t));
  return r;
}

// a tensor whose memory can be used as it is: contiguous, on a GPU, no wrapper or subclass, no lazy conjugate or negation
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.layout() != at::kStrided || !t.is_contiguous() || at::isTensorSubclassLike(t) || t.is_neg() || t.is_conj() || t._is_zerotensor()) return nullptr;
  return &t;
}
bool watched() { return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled(); }
bool fp8(const at::Tensor& t) { return t.scalar_type() == kE4M3 || t.scalar_type() == kE5M2; }
int format(const at::Tensor& t) { return t.scalar_type() == kE4M3 ? PB_E4M3 : PB_E5M2; }
bool dense(at::ScalarType t) { return t == at::kFloat || t == at::kBFloat16; }
int code(at::ScalarType t) { return t == at::kBFloat16 ? PB_BF16 : PB_F32; }
at::Tensor empty(at::IntArrayRef shape, at::ScalarType type, const at::Tensor& like) { return at::empty(shape, at::TensorOptions().device(like.device()).dtype(type)); }
at::Tensor scratch(size_t bytes, const at::Tensor& like) { return empty({(int64_t)bytes}, at::kByte, like); }

struct Grid {
  int64_t batch = 1, rows = 0, cols = 0, m = 0, k = 0;
  c10::SmallVector<int64_t, 8> sc8, sc32;
  // of [..., rows, cols] on (a, b); false: not divisible, empty or fewer than two dimensions
  bool of(at::IntArrayRef s, int64_t a, int64_t b) {
    if (s.size() < 2 || a <= 0 || b <= 0) return false;
    rows = s[s.size() - 2]; cols = s[s.size() - 1];
    if (rows <= 0 || cols <= 0 || rows % a || cols % b) return false;
    const int64_t nb = (rows * cols) / (a * b);
    k = std::gcd(std::max<int64_t>(1, a * b / 16), nb);
    m = nb / k;
    for (size_t i = 0; i + 2 < s.size(); ++i) { batch *= s[i]; sc8.push_back(s[i]); sc32.push_back(s[i]); }
    sc8.append({m, k}); sc32.append({m, 1, 1});
    return batch > 0;
  }
};

#define OP(name) PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t n)
#define NARGS(count)                                                                                        \
  if (n != (count)) return PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", (int)(count), n)
#define RUN(expr)                                                             \
  do {                                                                        \
    const int status_ = without_gil([&] { return (expr); });                  \
    if (status_ != PB_OK) return raise_status(status_);                       \
  } while (0)
// 0 for what is no integer: a block size or a count of 0 is left to the Python text
long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return 0; }
  return v;
}

// the same for what the C entries take as an int: beyond one it is left, too, not cut to its low bits
int small(PyObject* o) {
  const long long v = integer(o);
  return v == (int)v ? (int)v : 0;
}

// quantize(x, a, b, format) -> (q, sc8, sc32): quantize_impl
OP(quantize) {
  HANDLE_TH_ERRORS
  NARGS(4);
  const at::Tensor* x = plain(args[0]);
  const int a = small(args[1]), b = small(args[2]), fmt = small(args[3]);
  Grid g;
  if (!x || watched() || !dense(x->scalar_type()) || !g.of(x->sizes(), a, b)) return none();
  const c10::cuda::CUDAGuard guard(x->device());
  at::Tensor q = empty(x->sizes(), fmt == PB_E4M3 ? kE4M3 : kE5M2, *x), sc8 = empty(g.sc8, kE8M0, *x), sc32 = empty(g.sc32, at::kFloat, *x), ws;
  const size_t bytes = pb_quantize_workspace_size(g.batch, g.rows, g.cols, a, b);
  if (bytes) ws = scratch(bytes, *x);
  RUN(pb_quantize(x->data_ptr(), code(x->scalar_type()), g.batch, g.rows, g.cols, a, b, fmt, q.data_ptr(), (uint8_t*)sc8.data_ptr(), (float*)sc32.data_ptr(),
                  bytes ? ws.data_ptr() : nullptr, bytes, current_stream(x->device())));
  return wrap({q, sc8, sc32});
  END_HANDLE_TH_ERRORS
}

// quantize_transposed(x, b, format) -> (q, sc8, sc32): quantize_transposed_impl
OP(quantize_transposed) {
  HANDLE_TH_ERRORS
  NARGS(3);
  const at::Tensor* x = plain(args[0]);
  const int b = small(args[1]), fmt = small(args[2]);
  if (!x || watched() || !dense(x->scalar_type()) || x->dim() < 2) return none();
  c10::SmallVector<int64_t, 8> s(x->sizes().begin(), x->sizes().end());
  const int64_t rows = s[s.size() - 2], cols = s[s.size() - 1];
  s[s.size() - 2] = cols; s[s.size() - 1] = rows;
  Grid g;
  if (!g.of(s, 1, b)) return none();
  const c10::cuda::CUDAGuard guard(x->device());
  at::Tensor q = empty(s, fmt == PB_E4M3 ? kE4M3 : kE5M2, *x), sc8 = empty(g.sc8, kE8M0, *x), sc32 = empty(g.sc32, at::kFloat, *x), ws;
  const size_t bytes = pb_quantize_transposed_workspace_size(g.batch, rows, cols, b);
  if (bytes) ws = scratch(bytes, *x);
  RUN(pb_quantize_transposed(x->data_ptr(), code(x->scalar_type()), g.batch, rows, cols, b, fmt, q.data_ptr(), (uint8_t*)sc8.data_ptr(), (float*)sc32.data_ptr(),
                             bytes ? ws.data_ptr() : nullptr, bytes, current_stream(x->device())));
  return wrap({q, sc8, sc32});
  END_HANDLE_TH_ERRORS
}

// dequantize(q, sc8, sc32, dtype, a, b) -> out: dequantize_impl
OP(dequantize) {
  HANDLE_TH_ERRORS
  NARGS(6);
  const at::Tensor *q = plain(args[0]), *sc8 = plain(args[1]), *sc32 = plain(args[2]);
  const int a = small(args[4]), b = small(args[5]);
  if (!q || !sc8 || !sc32 || watched() || !THPDtype_Check(args[3]) || !fp8(*q) || sc8->dim() < 2) return none();
  const at::ScalarType type = reinterpret_cast<THPDtype*>(args[3])->scalar_type;
  Grid g;
  if (!dense(type) || !g.of(q->sizes(), a, b) || sc8->size(-2) != g.m || sc8->size(-1) != g.k) return none();
  const c10::cuda::CUDAGuard guard(q->device());
  at::Tensor out = empty(q->sizes(), type, *q);
  RUN(pb_dequantize(q->data_ptr(), format(*q), (const uint8_t*)sc8->data_ptr(), (const float*)sc32->data_ptr(), g.batch, g.rows, g.cols, a, b, code(type), out.data_ptr(),
                    current_stream(q->device())));
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// dequantize_bwd(sc8, sc32, g, a, b) -> cotangent: dequantize_impl_bwd
OP(dequantize_bwd) {
  HANDLE_TH_ERRORS
  NARGS(5);
  const at::Tensor *sc8 = plain(args[0]), *sc32 = plain(args[1]), *g_out = plain(args[2]);
  const int a = small(args[3]), b = small(args[4]);
  Grid g;
  if (!sc8 || !sc32 || !g_out || watched() || !dense(g_out->scalar_type()) || !g.of(g_out->sizes(), a, b)) return none();
  const c10::cuda::CUDAGuard guard(g_out->device());
  at::Tensor out = empty(g_out->sizes(), g_out->scalar_type(), *g_out);
  RUN(pb_dequantize_bwd(g_out->data_ptr(), code(g_out->scalar_type()), (const uint8_t*)sc8->data_ptr(), (const float*)sc32->data_ptr(), g.batch, g.rows, g.cols, a, b,
                        out.data_ptr(), current_stream(g_out->device())));
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// fake_quantize(x, a, b, dtype, format, scales) -> out, or (out, sc8, sc32) with scales: where one kernel or one call does it
OP(fake_quantize) {
  HANDLE_TH_ERRORS
  NARGS(6);
  const at::Tensor* x = plain(args[0]);
  const int a = small(args[1]), b = small(args[2]), fmt = small(args[4]);
  const bool scales = PyObject_IsTrue(args[5]) == 1;
  if (!x || watched() || !THPDtype_Check(args[3]) || x->scalar_type() != at::kFloat) return none();
  const at::ScalarType type = reinterpret_cast<THPDtype*>(args[3])->scalar_type;
  Grid g;
  if (!dense(type) || !g.of(x->sizes(), a, b)) return none();
  const c10::cuda::CUDAGuard guard(x->device());
  if (a == 1 && b == 128 && g.k == 8) {
    at::Tensor out = empty(x->sizes(), type, *x);
    if (!scales) {
      RUN(pb_fake_quantize(x->data_ptr(), PB_F32, g.batch, g.rows, g.cols, 1, 128, fmt, out.data_ptr(), code(type), current_stream(x->device())));
      return wrap(out);
    }
    at::Tensor sc8 = empty(g.sc8, kE8M0, *x), sc32 = empty(g.sc32, at::kFloat, *x);
    RUN(pb_fake_quantize_scales(x->data_ptr(), PB_F32, g.batch, g.rows, g.cols, 1, 128, fmt, out.data_ptr(), code(type), (uint8_t*)sc8.data_ptr(), (float*)sc32.data_ptr(),
                                current_stream(x->device())));
    return wrap({out, sc8, sc32});
  }
  if (scales || type != at::kFloat || fmt != PB_E4M3 || (reinterpret_cast<uintptr_t>(x->data_ptr()) & 15)) return none();
  const size_t bytes = pb_fake_quantize_blocks_workspace_size(g.batch, g.rows, g.cols, a, b);
  if (!bytes) return none();
  at::Tensor out = empty(x->sizes(), at::kFloat, *x), ws = scratch(bytes, *x);
  RUN(pb_fake_quantize_blocks((const float*)x->data_ptr(), g.batch, g.rows, g.cols, a, b, (float*)out.data_ptr(), ws.data_ptr(), bytes, current_stream(x->device())));
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// transpose_bytes(q) -> q^T
OP(transpose_bytes) {
  HANDLE_TH_ERRORS
  NARGS(1);
  const at::Tensor* q = plain(args[0]);
  if (!q || watched() || q->dim() != 2 || q->element_size() != 1 || q->numel() == 0) return none();
  const c10::cuda::CUDAGuard guard(q->device());
  at::Tensor out = empty({q->size(1), q->size(0)}, q->scalar_type(), *q);
  RUN(pb_transpose_bytes(q->data_ptr(), q->size(0), q->size(1), out.data_ptr(), current_stream(q->device())));
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// gemm(a_q, a_sc8, a_sc32, a_grid, b_q, b_sc8, b_sc32, b_grid, b_transposed, dtype) -> a [.., depth] times b [rows, depth], as _ops.gemm_tn;
// the grids are the block heights (blocks are 128 deep)
OP(gemm) {
  HANDLE_TH_ERRORS
  NARGS(10);
  const at::Tensor* t[6];
  for (int i = 0; i < 6; ++i)
    if (!(t[i] = plain(args[i < 3 ? i : i + 1]))) return none();
  const at::Tensor &aq = *t[0], &bq = *t[3];
  if (watched() || !THPDtype_Check(args[9]) || !fp8(aq) || !fp8(bq) || aq.dim() < 2 || bq.dim() != 2 || bq.size(1) != aq.size(-1) || aq.numel() == 0 || bq.numel() == 0) return none();
  const at::ScalarType type = reinterpret_cast<THPDtype*>(args[9])->scalar_type;
  if (!dense(type)) return none();
  const int64_t depth = aq.size(-1), rows = aq.numel() / depth, cols = bq.size(0);
  const pb_operand a{aq.data_ptr(), (const uint8_t*)t[1]->data_ptr(), (const float*)t[2]->data_ptr(), rows, depth, small(args[3]), 128, format(aq), 0};
  const pb_operand b{bq.data_ptr(), (const uint8_t*)t[4]->data_ptr(), (const float*)t[5]->data_ptr(), cols, depth, small(args[7]), 128, format(bq), small(args[8])};
  const c10::cuda::CUDAGuard guard(aq.device());
  c10::SmallVector<int64_t, 8> shape(aq.sizes().begin(), aq.sizes().end());
  shape.back() = cols;
  at::Tensor d = empty(shape, type, aq);
  const size_t bytes = pb_gemm_workspace_size(&a, &b);
  at::Tensor ws = scratch(bytes ? bytes : 1, aq);
  RUN(pb_gemm_tn(&a, &b, d.data_ptr(), code(type), cols, ws.data_ptr(), bytes, current_stream(aq.device())));
  return wrap(d);
  END_HANDLE_TH_ERRORS
}

// Whether `linear` takes an x (with x_q given, of its quantized rows) for a weight of [depth, cols] on (128, b)
bool linear_fits(PyObject* o, bool given, int64_t depth, int64_t cols, int b, bool fake, c10::Device device) {
  if (!THPVariable_CheckExact(o) || watched() || depth <= 0 || depth % 128 || (b != 128 && b != 1)) return false;
  const at::Tensor& x = THPVariable_Unpack(o);
  if (!dense(x.scalar_type()) || x.dim() < 2 || x.size(-1) != depth || x.numel() == 0) return false;
  const int64_t rows = x.numel() / depth;
  if ((rows * (depth / 128)) % 8 || (b == 128 ? cols % 128 : cols % 16)) return false;
  if (fake ? b != 128 || (rows * (cols / 128)) % 8 : x.scalar_type() != at::kFloat) return false;
  return given || (plain(o) && x.device() == device);
}
// linear_takes(x, x_q, weight, b, fake): the same before the weight is quantized and turned for the call
OP(linear_takes) {
  HANDLE_TH_ERRORS
  NARGS(5);
  if (!THPVariable_Check(args[2])) Py_RETURN_FALSE;
  const at::Tensor& w = THPVariable_Unpack(args[2]);
  if (!w.is_cuda() || w.dim() != 2) Py_RETURN_FALSE;
  return PyBool_FromLong(linear_fits(args[0], args[1] != Py_None, w.size(0), w.size(1), small(args[3]), PyObject_IsTrue(args[4]) == 1, w.device()));
  END_HANDLE_TH_ERRORS
}

// linear(x, x_q, x_sc8, x_sc32, w_sc8, w_sc32, w_t, b, fake) -> y: a Linear whose weight is on (128, b) and whose gradient nobody wants.  With
// x_q given x only lends its shape and type.  fake: the product is re-quantized on (1, b) and read back.
OP(linear) {
  HANDLE_TH_ERRORS
  NARGS(9);
  const bool given = args[1] != Py_None, fake = PyObject_IsTrue(args[8]) == 1;
  const at::Tensor *w8 = plain(args[4]), *w32 = plain(args[5]), *wt = plain(args[6]);
  const int b = small(args[7]);
  if (!w8 || !w32 || !wt || wt->dim() != 2 || !fp8(*wt) || !linear_fits(args[0], given, wt->size(1), wt->size(0), b, fake, wt->device())) return none();
  const at::Tensor& x = THPVariable_Unpack(args[0]);
  const int64_t depth = wt->size(1), cols = wt->size(0), rows = x.numel() / depth, blocks = rows * (depth / 128);
  at::Tensor q, s8, s32;
  const c10::cuda::CUDAGuard guard(wt->device());
  void* st = current_stream(wt->device());
  if (given) {
    const at::Tensor *gq = plain(args[1]), *g8 = plain(args[2]), *g32 = plain(args[3]);
    if (!gq || !g8 || !g32 || gq->dim() != 2 || gq->size(0) != rows || gq->size(1) != depth || !fp8(*gq)) return none();
    q = *gq; s8 = *g8; s32 = *g32;
  } else {
    q = empty({rows, depth}, kE4M3, x); s8 = empty({blocks / 8, 8}, kE8M0, x); s32 = empty({blocks / 8, 1, 1}, at::kFloat, x);
    at::Tensor ws;
    const size_t bytes = pb_quantize_workspace_size(1, rows, depth, 1, 128);
    if (bytes) ws = scratch(bytes, x);
    RUN(pb_quantize(x.data_ptr(), code(x.scalar_type()), 1, rows, depth, 1, 128, PB_E4M3, q.data_ptr(), (uint8_t*)s8.data_ptr(), (float*)s32.data_ptr(),
                    bytes ? ws.data_ptr() : nullptr, bytes, st));
  }
  const pb_operand oa{q.data_ptr(), (const uint8_t*)s8.data_ptr(), (const float*)s32.data_ptr(), rows, depth, 1, 128, format(q), 0};
  const pb_operand ob{wt->data_ptr(), (const uint8_t*)w8->data_ptr(), (const float*)w32->data_ptr(), cols, depth, b, 128, format(*wt), 1};
  c10::SmallVector<int64_t, 8> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = cols;
  at::Tensor d = empty(shape, at::kFloat, q);
  const size_t bytes = pb_gemm_workspace_size(&oa, &ob);
  at::Tensor ws = scratch(bytes ? bytes : 1, q);
  RUN(pb_gemm_tn(&oa, &ob, d.data_ptr(), PB_F32, cols, ws.data_ptr(), bytes, st));
  if (!fake) return wrap(d);
  at::Tensor out = empty(shape, x.scalar_type(), q);
  RUN(pb_fake_quantize(d.data_ptr(), PB_F32, 1, rows, cols, 1, 128, PB_E4M3, out.data_ptr(), code(x.scalar_type()), st));
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// ---- a Linear's training step: what _LinearFn's two passes call one by one, each in one call ----
struct Triple { at::Tensor q, s8, s32; };

int rows_form(const at::Tensor& x, int64_t rows, int64_t cols, int fmt, Triple* t, void* st) {       // on (1,128), whole groups of eight blocks
  const int64_t groups = rows * (cols / 128) / 8;
  *t = {empty({rows, cols}, fmt == PB_E4M3 ? kE4M3 : kE5M2, x), empty({groups, 8}, kE8M0, x), empty({groups, 1, 1}, at::kFloat, x)};
  at::Tensor ws;
  const size_t bytes = pb_quantize_workspace_size(1, rows, cols, 1, 128);
  if (bytes) ws = scratch(bytes, x);
  return without_gil([&] {
    return pb_quantize(x.data_ptr(), code(x.scalar_type()), 1, rows, cols, 1, 128, fmt, t->q.data_ptr(), (uint8_t*)t->s8.data_ptr(), (float*)t->s32.data_ptr(),
                       bytes ? ws.data_ptr() : nullptr, bytes, st);
  });
}
// x^T on (1,128): rows are a multiple of 1024
Triple tokens_form(const at::Tensor& x, int64_t rows, int64_t cols, int fmt) {
  const int64_t groups = rows * cols / 1024;
  return {empty({cols, rows}, fmt == PB_E4M3 ? kE4M3 : kE5M2, x), empty({groups, 8}, kE8M0, x), empty({groups, 1, 1}, at::kFloat, x)};
}
// both forms: quantize_dual_impl
int dual_form(const at::Tensor& x, int64_t rows, int64_t cols, int fmt, Triple* t, Triple* tt, void* st) {
  const size_t bytes = pb_quantize_transposed_workspace_size(1, rows, cols, 128);
  at::Tensor ws = scratch(bytes ? bytes : 1, x);
  if (x.scalar_type() == at::kBFloat16 && cols % 1024 == 0) {
    const int64_t groups = rows * cols / 1024;
    *t = {empty({rows, cols}, fmt == PB_E4M3 ? kE4M3 : kE5M2, x), empty({groups, 8}, kE8M0, x), empty({groups, 1, 1}, at::kFloat, x)};
    *tt = tokens_form(x, rows, cols, fmt);
    return without_gil([&] {
      return pb_quantize_dual(x.data_ptr(), PB_BF16, 1, rows, cols, fmt, t->q.data_ptr(), (uint8_t*)t->s8.data_ptr(), (float*)t->s32.data_ptr(), tt->q.data_ptr(),
                              (uint8_t*)tt->s8.data_ptr(), (float*)tt->s32.data_ptr(), ws.data_ptr(), bytes, st);
    });
  }
  if (int status = rows_form(x, rows, cols, fmt, t, st)) return status;
  *tt = tokens_form(x, rows, cols, fmt);
  return without_gil([&] {
    return pb_quantize_transposed(x.data_ptr(), code(x.scalar_type()), 1, rows, cols, 128, fmt, tt->q.data_ptr(), (uint8_t*)tt->s8.data_ptr(), (float*)tt->s32.data_ptr(),
                                  bytes ? ws.data_ptr() : nullptr, bytes, st);
  });
}
// d [rows of a, rows of b] f32, of operands whose blocks are 128 deep
int product(const Triple& a, const Triple& b, int b_height, int b_transposed, at::Tensor* d, void* st) {
  const int64_t depth = a.q.size(1), rows = a.q.size(0), cols = b.q.size(0);
  const pb_operand oa{a.q.data_ptr(), (const uint8_t*)a.s8.data_ptr(), (const float*)a.s32.data_ptr(), rows, depth, 1, 128, format(a.q), 0};
  const pb_operand ob{b.q.data_ptr(), (const uint8_t*)b.s8.data_ptr(), (const float*)b.s32.data_ptr(), cols, depth, b_height, 128, format(b.q), b_transposed};
  *d = empty({rows, cols}, at::kFloat, a.q);
  const size_t bytes = pb_gemm_workspace_size(&oa, &ob);
  at::Tensor ws = scratch(bytes ? bytes : 1, a.q);
  return without_gil([&] { return pb_gemm_tn(&oa, &ob, d->data_ptr(), PB_F32, cols, ws.data_ptr(), bytes, st); });
}
// _dense_dot; free: g's extent that is not summed over
int literal_dot(int tokens, const Triple& t, int a, int b, const at::Tensor& g, int64_t free, at::Tensor* out, void* st) {
  const int64_t rows = t.q.size(0), cols = t.q.size(1);
  const int type = code(g.scalar_type());
  *out = tokens ? empty({cols, free}, at::kFloat, g) : empty({free, rows}, at::kFloat, g);
  at::Tensor ws;
  size_t bytes = pb_dense_dot_workspace_best(tokens, rows, cols, a, b, free, type);
  try {
    if (bytes) ws = scratch(bytes, g);
  } catch (const c10::OutOfMemoryError&) {      // the form that takes less of it
    const size_t least = pb_dense_dot_workspace_size(tokens, rows, cols, a, b, free);
    if (least == bytes) throw;
    bytes = least;
    if (bytes) ws = scratch(bytes, g);
  }
  return without_gil([&] {
    return pb_dense_dot(tokens, (const uint8_t*)t.q.data_ptr(), (const uint8_t*)t.s8.data_ptr(), (const float*)t.s32.data_ptr(), rows, cols, a, b, g.data_ptr(), type, free,
                        (float*)out->data_ptr(), bytes ? ws.data_ptr() : nullptr, bytes, st);
  });
}

// linear_forward(x, w_sc8, w_sc32, w_t, b, fake, tokens) -> (y, x's triple[, the triple of x^T][, the scales of y]): _LinearFn.forward for a weight
// on (128, b).  tokens: the triple of x^T is wanted (rows a multiple of 1024).
OP(linear_forward) {
  HANDLE_TH_ERRORS
  NARGS(7);
  const bool fake = PyObject_IsTrue(args[5]) == 1, tokens = PyObject_IsTrue(args[6]) == 1;
  const at::Tensor *w8 = plain(args[1]), *w32 = plain(args[2]), *wt = plain(args[3]);
  const int b = small(args[4]);
  if (!w8 || !w32 || !wt || wt->dim() != 2 || !fp8(*wt) || !linear_fits(args[0], false, wt->size(1), wt->size(0), b, fake, wt->device())) return none();
  const at::Tensor& x = THPVariable_Unpack(args[0]);
  const int64_t depth = wt->size(1), cols = wt->size(0), rows = x.numel() / depth;
  if (tokens && rows % 1024) return none();
  const c10::cuda::CUDAGuard guard(wt->device());
  void* st = current_stream(wt->device());
  Triple q, t;
  int status = tokens ? dual_form(x, rows, depth, PB_E4M3, &q, &t, st) : rows_form(x, rows, depth, PB_E4M3, &q, st);
  if (status != PB_OK) return raise_status(status);
  at::Tensor d, s8, s32;
  if ((status = product(q, {*wt, *w8, *w32}, b, 1, &d, st)) != PB_OK) return raise_status(status);
  c10::SmallVector<int64_t, 8> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = cols;
  at::Tensor y;
  if (fake) {
    const int64_t groups = rows * (cols / 128) / 8;
    y = empty(shape, x.scalar_type(), x);
    s8 = empty({groups, 8}, kE8M0, x); s32 = empty({groups, 1, 1}, at::kFloat, x);
    RUN(pb_fake_quantize_scales(d.data_ptr(), PB_F32, 1, rows, cols, 1, 128, PB_E4M3, y.data_ptr(), code(x.scalar_type()), (uint8_t*)s8.data_ptr(), (float*)s32.data_ptr(), st));
  } else {
    y = d.view(shape);
  }
  if (tokens && fake) return wrap({y, q.q, q.s8, q.s32, t.q, t.s8, t.s32, s8, s32});
  if (tokens) return wrap({y, q.q, q.s8, q.s32, t.q, t.s8, t.s32});
  if (fake) return wrap({y, q.q, q.s8, q.s32, s8, s32});
  return wrap({y, q.q, q.s8, q.s32});
  END_HANDLE_TH_ERRORS
}

// linear_backward(g, x_q, x_sc8, x_sc32, w_q, w_sc8, w_sc32, t_q, t_sc8, t_sc32, y_sc8, y_sc32, b, format, x_dtype) -> (gx [rows, depth], gw):
// _LinearFn.backward for a weight on (128, b).  t: the triple of x^T, for products of fp8 gradients in `format`, or None: literal dots.  y: the
// scales of a fake-quantized output, or None.
OP(linear_backward) {
  HANDLE_TH_ERRORS
  NARGS(15);
  const at::Tensor* in[12];
  for (int i = 0; i < 12; ++i) {
    const bool may_miss = i >= 7;
    if (may_miss && args[i] == Py_None) { in[i] = nullptr; continue; }
    if (!(in[i] = plain(args[i]))) return none();
  }
  const bool tokens = in[7] && in[8] && in[9], fake = in[10] && in[11];
  const int b = small(args[12]), fmt = small(args[13]);
  const at::Tensor &xq = *in[1], &wq = *in[4];
  if (watched() || !THPDtype_Check(args[14]) || (b != 128 && b != 1) || (fake && b != 128) || (tokens && b != 128) || xq.dim() != 2 || wq.dim() != 2 || xq.scalar_type() != kE4M3 ||
      wq.scalar_type() != kE4M3 || xq.numel() == 0 || wq.numel() == 0 || !dense(in[0]->scalar_type()))
    return none();
  const at::ScalarType x_type = reinterpret_cast<THPDtype*>(args[14])->scalar_type;
  const int64_t rows = xq.size(0), depth = xq.size(1), cols = wq.size(1);
  if (!dense(x_type) || wq.size(0) != depth || depth % 128 || cols % (b == 128 ? 128 : 16) || (rows * (depth / 128)) % 8 || (fake && (rows * (cols / 128)) % 8) ||
      in[0]->dim() < 1 || in[0]->size(-1) != cols || in[0]->numel() != rows * cols || (tokens && (rows % 1024 || !fp8(*in[7]))) ||
      ((reinterpret_cast<uintptr_t>(in[0]->data_ptr()) | reinterpret_cast<uintptr_t>(xq.data_ptr()) | reinterpret_cast<uintptr_t>(wq.data_ptr())) & 15))
    return none();
  const size_t w_bytes = pb_fake_quantize_blocks_workspace_size(1, depth, cols, 128, b);
  if (!w_bytes) return none();
  const c10::cuda::CUDAGuard guard(xq.device());
  void* st = current_stream(xq.device());
  at::Tensor g = *in[0], gx, gw;
  int status = PB_OK;
  if (tokens) {
    Triple q, t;
    if (fake && g.scalar_type() == at::kFloat && cols % 1024 == 0) {
      const int64_t groups = rows * cols / 1024;
      q = {empty({rows, cols}, fmt == PB_E4M3 ? kE4M3 : kE5M2, g), empty({groups, 8}, kE8M0, g), empty({groups, 1, 1}, at::kFloat, g)};
      t = tokens_form(g, rows, cols, fmt);
      RUN(pb_dequantize_bwd_quantize_dual((const float*)g.data_ptr(), (const uint8_t*)in[10]->data_ptr(), (const float*)in[11]->data_ptr(), rows, cols, fmt, (uint8_t*)q.q.data_ptr(),
                                          (uint8_t*)q.s8.data_ptr(), (float*)q.s32.data_ptr(), (uint8_t*)t.q.data_ptr(), (uint8_t*)t.s8.data_ptr(), (float*)t.s32.data_ptr(), st));
    } else {
      if (fake) {
        at::Tensor scaled = empty(g.sizes(), g.scalar_type(), g);
        RUN(pb_dequantize_bwd(g.data_ptr(), code(g.scalar_type()), (const uint8_t*)in[10]->data_ptr(), (const float*)in[11]->data_ptr(), 1, rows, cols, 1, 128, scaled.data_ptr(), st));
        g = scaled;
      }
      if ((status = dual_form(g, rows, cols, fmt, &q, &t, st)) != PB_OK) return raise_status(status);
    }
    if ((status = product(q, {wq, *in[5], *in[6]}, 128, 0, &gx, st)) != PB_OK || (status = product({*in[7], *in[8], *in[9]}, t, 1, 0, &gw, st)) != PB_OK) return raise_status(status);
  } else {
    if (fake) {
      at::Tensor scaled = empty(g.sizes(), g.scalar_type(), g);
      RUN(pb_dequantize_bwd(g.data_ptr(), code(g.scalar_type()), (const uint8_t*)in[10]->data_ptr(), (const float*)in[11]->data_ptr(), 1, rows, cols, 1, 128, scaled.data_ptr(), st));
      g = scaled;
    }
    if ((status = literal_dot(0, {wq, *in[5], *in[6]}, 128, b, g, rows, &gx, st)) != PB_OK ||
        (status = literal_dot(1, {xq, *in[2], *in[3]}, 1, 128, g, cols, &gw, st)) != PB_OK)
      return raise_status(status);
  }
  at::Tensor dx = empty({rows, depth}, x_type, xq);
  RUN(pb_fake_quantize(gx.data_ptr(), PB_F32, 1, rows, depth, 1, 128, PB_E4M3, dx.data_ptr(), code(x_type), st));
  gx.reset();
  at::Tensor dw = empty({depth, cols}, at::kFloat, xq), ws = scratch(w_bytes, xq);
  RUN(pb_fake_quantize_blocks((const float*)gw.data_ptr(), 1, depth, cols, 128, b, (float*)dw.data_ptr(), ws.data_ptr(), w_bytes, st));
  return wrap({dx, dw});
  END_HANDLE_TH_ERRORS
}

// linear_step(x, rows, k, n, dtype, format, b operand, workspace, b prepared, relu2) -> (d, q, sc8, sc32): LinearStep.__call__
OP(linear_step) {
  HANDLE_TH_ERRORS
  NARGS(10);
  const at::Tensor *x = plain(args[0]), *ws = plain(args[7]);
  const int64_t rows = integer(args[1]), k = integer(args[2]), cols = integer(args[3]);
  const int fmt = small(args[5]);
  const bool ready = PyObject_IsTrue(args[8]) == 1, relu2 = PyObject_IsTrue(args[9]) == 1;
  if (!x || !ws || watched() || !THPDtype_Check(args[4]) || !dense(x->scalar_type()) || (relu2 && x->scalar_type() != at::kFloat) || x->dim() < 1 || x->numel() != rows * k ||
      x->size(-1) != k || x->numel() == 0 || x->device() != ws->device())
    return none();
  const at::ScalarType type = reinterpret_cast<THPDtype*>(args[4])->scalar_type;
  if (!dense(type)) return none();
  Taken taken;
  void* bp = nullptr;
  if (!take(args[6], taken, &bp)) return nullptr;
  const pb_operand b = *static_cast<const pb_operand*>(bp);
  const c10::cuda::CUDAGuard guard(x->device());
  const int64_t groups = rows * k / 1024;
  at::Tensor q = empty({rows, k}, fmt == PB_E4M3 ? kE4M3 : kE5M2, *x), sc8 = empty({groups, 8}, kE8M0, *x), sc32 = empty({groups, 1, 1}, at::kFloat, *x);
  at::Tensor d = empty({rows, cols}, type, *x);
  uint8_t* s8 = (uint8_t*)sc8.data_ptr();
  float* s32 = (float*)sc32.data_ptr();
  const size_t bytes = (size_t)ws->numel();
  void* st = current_stream(x->device());
  const pb_operand a{q.data_ptr(), s8, s32, rows, k, 1, 128, fmt, 0};
  RUN(relu2 ? pb_relu2_requantize(x->data_ptr(), rows, k, fmt, q.data_ptr(), s8, s32, &b, ws->data_ptr(), bytes, st)
            : pb_quantize_for_gemm(x->data_ptr(), code(x->scalar_type()), rows, k, fmt, q.data_ptr(), s8, s32, &b, ws->data_ptr(), bytes, st));
  RUN(pb_gemm_tn_ex(&a, &b, d.data_ptr(), code(type), cols, ws->data_ptr(), bytes, PB_GEMM_A_PREPARED | (ready ? PB_GEMM_B_PREPARED : 0), st));
  return wrap({d, q, sc8, sc32});
  END_HANDLE_TH_ERRORS
}

// dense_dot(tokens, q, sc8, sc32, a, b, g) -> out: _ops._dense_dot
OP(dense_dot) {
  HANDLE_TH_ERRORS
  NARGS(7);
  const at::Tensor *q = plain(args[1]), *sc8 = plain(args[2]), *sc32 = plain(args[3]), *g = plain(args[6]);
  const int tokens = small(args[0]), a = small(args[4]), b = small(args[5]);
  if (!q || !sc8 || !sc32 || !g || watched() || q->dim() != 2 || g->dim() != 2 || !dense(g->scalar_type()) || q->scalar_type() != kE4M3 ||
      g->size(tokens ? 0 : 1) != q->size(tokens ? 0 : 1))
    return none();
  const c10::cuda::CUDAGuard guard(g->device());
  at::Tensor out;
  if (const int status = literal_dot(tokens, {*q, *sc8, *sc32}, a, b, *g, g->size(tokens ? 1 : 0), &out, current_stream(g->device()))) return raise_status(status);
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// empty(shape, dtype, like) -> a tensor on the device of `like`; empties(like, count) -> a list of them, contiguous, of its shape and type
OP(empty_on) {
  HANDLE_TH_ERRORS
  NARGS(3);
  if (!PyTuple_Check(args[0]) || !THPDtype_Check(args[1]) || !THPVariable_Check(args[2])) return PyErr_Format(PyExc_TypeError, "empty(tuple, dtype, tensor)");
  c10::SmallVector<int64_t, 8> shape;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[0]); ++i) {
    shape.push_back(PyLong_AsLongLong(PyTuple_GET_ITEM(args[0], i)));
    if (PyErr_Occurred()) return nullptr;
  }
  return wrap(empty(shape, reinterpret_cast<THPDtype*>(args[1])->scalar_type, THPVariable_Unpack(args[2])));
  END_HANDLE_TH_ERRORS
}
OP(empties) {
  HANDLE_TH_ERRORS
  NARGS(2);
  if (!THPVariable_Check(args[0])) return PyErr_Format(PyExc_TypeError, "empties(tensor, count)");
  const at::Tensor& like = THPVariable_Unpack(args[0]);
  const long long count = PyLong_AsLongLong(args[1]);
  if (PyErr_Occurred()) return nullptr;
  PyObject* r = PyList_New(count);
  for (long long i = 0; r && i < count; ++i) {
    PyObject* t = THPVariable_Wrap(empty(like.sizes(), like.scalar_type(), like));
    if (!t) { Py_DECREF(r); return nullptr; }
    PyList_SET_ITEM(r, i, t);
  }
  return r;
  END_HANDLE_TH_ERRORS
}

PyObject* set_error(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  Py_XDECREF(g_pb_error);
  g_pb_error = cls;
  return none();
}

#define METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
#define ENTRY(name) METHOD(#name, &Entry<&name>::call)
PyMethodDef methods[] = {
    METHOD("quantize", quantize), METHOD("quantize_transposed", quantize_transposed), METHOD("dequantize", dequantize), METHOD("dequantize_bwd", dequantize_bwd),
    METHOD("fake_quantize", fake_quantize), METHOD("transpose_bytes", transpose_bytes), METHOD("gemm", gemm), METHOD("linear_step", linear_step), METHOD("linear", linear), METHOD("linear_takes", linear_takes),
    METHOD("linear_forward", linear_forward), METHOD("linear_backward", linear_backward),
    METHOD("dense_dot", dense_dot), METHOD("empty", empty_on), METHOD("empties", empties),
    ENTRY(pb_quantize_dual), ENTRY(pb_dequantize_bwd_quantize_dual), ENTRY(pb_relu2_requantize), ENTRY(pb_quantize_transposed_workspace_size),
    ENTRY(pb_wkv7_forward), ENTRY(pb_wkv7_backward), ENTRY(pb_wkv7_checkpoint_floats),
    ENTRY(pb_token_shift_lerp), ENTRY(pb_token_shift_lerp_bwd), ENTRY(pb_token_shift_lerp_bwd_workspace_size), ENTRY(pb_shift_lerp_quantize), ENTRY(pb_relu2_quantize_dual),
    ENTRY(pb_wkv_prepare), ENTRY(pb_wkv_prepare_bwd), ENTRY(pb_wkv_prepare_bwd_workspace_size),
    ENTRY(pb_rms_norm), ENTRY(pb_rms_norm_bwd), ENTRY(pb_rms_norm_bwd_workspace_size), ENTRY(pb_relu2), ENTRY(pb_relu2_bwd),
    ENTRY(pb_wkv_finish), ENTRY(pb_wkv_finish_workspace_size), ENTRY(pb_wkv_finish_bwd), ENTRY(pb_wkv_finish_bwd_workspace_size),
    ENTRY(pb_smoothed_xent), ENTRY(pb_smoothed_xent_bwd),
    {"set_error", set_error, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
