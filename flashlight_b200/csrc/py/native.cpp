// The host path of the Python mirror (extension.py, functions.py): argument checks, output and
// workspace allocation, descriptor set-up and the call into the C ABI, one native function per
// operator.  What bounds a small call is the host: an operator driven through ctypes took 10 to
// 20 us on the host for a 4 us kernel launch (stream lookup 3.3 us, an allocation 1.7 us each,
// descriptor and argument marshalling the rest), so that a 12-layer Transformer of one 128-token
// prompt ran at 25 us per kernel with the device idle two thirds of the time.  Here the same
// operator costs about 2 us over its launches (B200 box: that prompt 4.65 -> 1.88 ms, ResNet-50
// scoring 8 images 3.94 -> 1.94 ms).
//
// Plain CPython functions (METH_FASTCALL, no binding library between): tensors are unpacked in
// place, outputs come straight from torch's CUDA allocator on the current stream.  The Python
// modules keep the public signatures and their error texts; nothing here is computed by torch.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cuda_runtime.h>

#include <cstdint>
#include <initializer_list>

#include "flb200.h"

namespace {

using at::Tensor;
using at::ScalarType;

PyObject* g_check = nullptr;  // _lib.check: turns a status into the package's exceptions

struct PyRaised {};  // a Python exception is set

// ---------------------------------------------------------------- arguments
struct Args {
  PyObject* const* a;
  Py_ssize_t n;
  PyObject* at(Py_ssize_t i) const {
    if (i >= n) {
      PyErr_SetString(PyExc_TypeError, "too few arguments");
      throw PyRaised();
    }
    return a[i];
  }
  // null for None
  const Tensor* t(Py_ssize_t i) const {
    PyObject* o = at(i);
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) {
      PyErr_SetString(PyExc_TypeError, "expected a tensor or None");
      throw PyRaised();
    }
    return &THPVariable_Unpack(o);
  }
  const Tensor& tensor(Py_ssize_t i) const {
    const Tensor* v = t(i);
    if (!v) {
      PyErr_SetString(PyExc_TypeError, "expected a tensor");
      throw PyRaised();
    }
    return *v;
  }
  int64_t i(Py_ssize_t k) const {
    const int64_t v = PyLong_AsLongLong(at(k));
    if (v == -1 && PyErr_Occurred()) throw PyRaised();
    return v;
  }
  int n32(Py_ssize_t k) const { return (int)i(k); }
  double d(Py_ssize_t k) const {
    const double v = PyFloat_AsDouble(at(k));
    if (v == -1.0 && PyErr_Occurred()) throw PyRaised();
    return v;
  }
  bool b(Py_ssize_t k) const {
    const int v = PyObject_IsTrue(at(k));
    if (v < 0) throw PyRaised();
    return v != 0;
  }
};

[[noreturn]] void value_error(const char* text) {
  PyErr_SetString(PyExc_ValueError, text);
  throw PyRaised();
}

void check(int status) {
  if (status == FLB200_OK) return;
  PyObject* r = PyObject_CallFunction(g_check, "i", status);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "flb200 call failed");
  throw PyRaised();
}

// Other threads run while the library or the allocator does: a launch waits where the device's queue
// is full, an allocation may wait for the device.  The arguments are made before, with the lock held.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
template <class R, class... Params, class... A>
R unlocked(R (*f)(Params...), A... a) {
  const Unlocked u;
  return f(a...);
}

template <class F>
PyObject* guarded(F f) {
  HANDLE_TH_ERRORS
  try {
    return f();
  } catch (const PyRaised&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define NATIVE(name)                                                              \
  PyObject* name##_body(const Args& x);                                           \
  PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n) {                   \
    return guarded([&] { return name##_body(Args{a, n}); });                      \
  }                                                                               \
  PyObject* name##_body(const Args& x)

// ---------------------------------------------------------------- tensors
// Stored [N][H][W][C] with bytes that differ from the [N][C][H][W] order.
bool channels_last(const Tensor& t) {
  return t.dim() == 4 && !t.is_contiguous() && t.is_contiguous(at::MemoryFormat::ChannelsLast);
}
bool dense(const Tensor& t) { return t.is_contiguous() || channels_last(t); }
bool same_layout(const Tensor& a, const Tensor& b) {
  return a.sizes() == b.sizes() && channels_last(a) == channels_last(b);
}
int code_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case ScalarType::Float: return FLB200_F32;
    case ScalarType::Half: return FLB200_F16;
    case ScalarType::BFloat16: return FLB200_BF16;
    default:
      PyErr_Format(PyExc_ValueError, "dtype torch.%s is not supported by the B200 autograd extension",
                   torch::getTHPDtype(t.scalar_type())->name);
      throw PyRaised();
  }
}
ScalarType type_of(int code) {
  return code == FLB200_F32 ? ScalarType::Float
                            : (code == FLB200_F16 ? ScalarType::Half : ScalarType::BFloat16);
}

void* P(const Tensor* t) {
  if (!t) return nullptr;
  if (!t->is_cuda()) value_error("the B200 autograd extension needs device (CUDA) tensors");
  if (!dense(*t)) value_error("can't get device pointer of non-contiguous tensor");
  return t->data_ptr();
}
void* P(const Tensor& t) { return P(&t); }
float* Pf(const Tensor* t) { return static_cast<float*>(P(t)); }
bool aligned16(const Tensor* t) {
  return !t || (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15) == 0;
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

Tensor empty(at::IntArrayRef shape, ScalarType type, const Tensor& like, bool cl = false) {
  if (!like.is_cuda()) value_error("the B200 autograd extension needs device (CUDA) tensors");
  const Unlocked u;
  return at::detail::empty_cuda(shape, type, like.device(),
                                cl ? std::optional<at::MemoryFormat>(at::MemoryFormat::ChannelsLast)
                                   : std::nullopt);
}
Tensor empty_like(const Tensor& t) { return empty(t.sizes(), t.scalar_type(), t, channels_last(t)); }
Tensor floats(int64_t n, const Tensor& like) { return empty({n}, ScalarType::Float, like); }

// Scratch of a call: freed (stream-ordered, torch's caching allocator) when it goes out of scope.
struct Workspace {
  Tensor t;
  size_t bytes;
  Workspace(size_t n, const Tensor& like) : bytes(n) {
    if (n) t = empty({(int64_t)n}, ScalarType::Byte, like);
  }
  void* p() const { return bytes ? t.data_ptr() : nullptr; }
};

PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
PyObject* wrap(std::initializer_list<Tensor> ts) {
  PyObject* out = PyTuple_New((Py_ssize_t)ts.size());
  if (!out) throw PyRaised();
  Py_ssize_t k = 0;
  for (const Tensor& t : ts) PyTuple_SET_ITEM(out, k++, wrap(t));
  return out;
}

// ---------------------------------------------------------------- element-wise
enum { U_RELU, U_GELU, U_TANH };
enum { B_RELU, B_GELU, B_TANH, B_ADD };

NATIVE(unary) {  // (op, x)
  const Tensor& in = x.tensor(1);
  const int dt = code_of(in);
  Tensor out = empty_like(in);
  const int64_t n = in.numel();
  switch (x.n32(0)) {
    case U_RELU: check(unlocked(flb200_relu_forward, P(in), P(out), n, dt, stream())); break;
    case U_GELU: check(unlocked(flb200_gelu_forward, P(in), P(out), n, dt, stream())); break;
    default: check(unlocked(flb200_tanh_forward, P(in), P(out), n, dt, stream()));
  }
  return wrap(out);
}

NATIVE(binary) {  // (op, a, b, out or None)
  const Tensor &a = x.tensor(1), &b = x.tensor(2);
  if (!same_layout(a, b) || a.scalar_type() != b.scalar_type())
    value_error("operands must have the same shape, memory layout and dtype");
  const int dt = code_of(a);
  const Tensor* given = x.t(3);
  Tensor out = given ? *given : empty_like(a);
  const int64_t n = a.numel();
  switch (x.n32(0)) {
    case B_RELU: check(unlocked(flb200_relu_backward, P(a), P(b), P(out), n, dt, stream())); break;
    case B_GELU: check(unlocked(flb200_gelu_backward, P(a), P(b), P(out), n, dt, stream())); break;
    case B_TANH: check(unlocked(flb200_tanh_backward, P(a), P(b), P(out), n, dt, stream())); break;
    default: check(unlocked(flb200_add, P(a), P(b), P(out), n, dt, stream()));
  }
  return wrap(out);
}

// relu / relu(a + b) with the packed predicate (b: None for the plain relu)
NATIVE(relu_mask) {  // (a, b) -> (y, mask)
  const Tensor& a = x.tensor(0);
  const Tensor* b = x.t(1);
  if (b && !same_layout(a, *b)) value_error("operands must have the same shape and memory layout");
  const int dt = code_of(a);
  Tensor y = empty_like(a), mask = empty({(a.numel() + 7) / 8}, ScalarType::Byte, a);
  uint8_t* m = static_cast<uint8_t*>(mask.data_ptr());
  if (b)
    check(unlocked(flb200_add_relu_forward_mask, P(a), P(*b), P(y), m, a.numel(), dt, stream()));
  else
    check(unlocked(flb200_relu_forward_mask, P(a), P(y), m, a.numel(), dt, stream()));
  return wrap({y, mask});
}
NATIVE(relu_mask_backward) {  // (mask, ga, gb or None)
  const Tensor& ga = x.tensor(1);
  const Tensor* gb = x.t(2);
  if (gb && !same_layout(ga, *gb)) value_error("operands must have the same shape and memory layout");
  const int dt = code_of(ga);
  Tensor gx = empty_like(ga);
  const uint8_t* m = static_cast<const uint8_t*>(P(x.tensor(0)));
  if (gb)
    check(unlocked(flb200_relu_backward_mask_sum, m, P(ga), P(*gb), P(gx), ga.numel(), dt, stream()));
  else
    check(unlocked(flb200_relu_backward_mask, m, P(ga), P(gx), ga.numel(), dt, stream()));
  return wrap(gx);
}

NATIVE(dropout_apply) {  // (x, mask, scale)
  const Tensor &in = x.tensor(0), &mask = x.tensor(1);
  if (!same_layout(in, mask) || in.scalar_type() != mask.scalar_type())
    value_error("mask must match the tensor's shape, memory layout and dtype");
  Tensor out = empty_like(in);
  check(unlocked(flb200_dropout_apply, P(in), P(mask), P(out), (float)x.d(2), in.numel(), code_of(in), stream()));
  return wrap(out);
}

NATIVE(astype) {  // (x, dtype code)
  const Tensor& in = x.tensor(0);
  const int dst = x.n32(1);
  Tensor out = empty(in.sizes(), type_of(dst), in);
  check(unlocked(flb200_astype, P(in), code_of(in), P(out), dst, in.numel(), stream()));
  return wrap(out);
}

// x.reshape(shape).permute(perm) for a contiguous x; None where the 16-byte rules do not hold
NATIVE(reorder) {  // (x, shape tuple, perm tuple)
  const Tensor& in = x.tensor(0);
  PyObject *shape = x.at(1), *perm = x.at(2);
  if (!PyTuple_Check(shape) || !PyTuple_Check(perm) || PyTuple_GET_SIZE(shape) != PyTuple_GET_SIZE(perm)) {
    PyErr_SetString(PyExc_TypeError, "reorder: shape and perm are tuples of one length");
    throw PyRaised();
  }
  const int n = (int)PyTuple_GET_SIZE(shape);
  if (n < 2 || n > 5 || !in.is_contiguous()) Py_RETURN_NONE;
  int64_t ext[5], stride[5], out_shape[5], dims[4] = {1, 1, 1, 1}, st[4] = {0, 0, 0, 0};
  int p[5];
  for (int k = 0; k < n; ++k) {
    ext[k] = PyLong_AsLongLong(PyTuple_GET_ITEM(shape, k));
    p[k] = (int)PyLong_AsLong(PyTuple_GET_ITEM(perm, k));
    if (PyErr_Occurred()) throw PyRaised();
    if (p[k] < 0 || p[k] >= n) value_error("reorder: perm out of range");
  }
  if (p[n - 1] != n - 1) Py_RETURN_NONE;
  stride[n - 1] = 1;
  for (int k = n - 2; k >= 0; --k) stride[k] = stride[k + 1] * ext[k + 1];
  if (stride[0] * ext[0] != in.numel()) value_error("reorder: shape does not match the tensor");
  const int64_t es = (int64_t)in.element_size(), vec = 16 / es, inner = ext[n - 1];
  if (inner % vec || (reinterpret_cast<uintptr_t>(in.data_ptr()) & 15)) Py_RETURN_NONE;
  const int lead = 4 - (n - 1);
  for (int k = 0; k < n; ++k) {
    out_shape[k] = ext[p[k]];
    if (k < n - 1) {
      dims[lead + k] = ext[p[k]];
      st[lead + k] = stride[p[k]];
      if (stride[p[k]] % vec) Py_RETURN_NONE;
    }
  }
  Tensor out = empty(at::IntArrayRef(out_shape, n), in.scalar_type(), in);
  check(unlocked(flb200_reorder, P(in), P(out), dims, st, inner, code_of(in), stream()));
  return wrap(out);
}

NATIVE(bernoulli_mask) {  // (out, keep_prob, seed, offset)
  const Tensor& out = x.tensor(0);
  const uint64_t seed = PyLong_AsUnsignedLongLongMask(x.at(2));
  const uint64_t off = PyLong_AsUnsignedLongLongMask(x.at(3));
  if (PyErr_Occurred()) throw PyRaised();
  check(unlocked(flb200_bernoulli_mask, P(out), out.numel(), (float)x.d(1), seed, off, code_of(out), stream()));
  Py_RETURN_NONE;
}

NATIVE(channel_sum) {  // (x, outer, channels, inner)
  const Tensor& in = x.tensor(0);
  const int64_t o = x.i(1), c = x.i(2), n = x.i(3);
  if (in.numel() != o * c * n) value_error("channel_sum: geometry does not match the tensor");
  Tensor out = floats(c, in);
  Workspace ws(flb200_channel_sum_workspace_bytes(o, c, n), in);
  check(unlocked(flb200_channel_sum, P(in), Pf(&out), o, c, n, code_of(in), ws.p(), ws.bytes, stream()));
  return wrap(out);
}
NATIVE(channel_bias_add) {  // (x, bias, outer, channels, inner, out or None)
  const Tensor& in = x.tensor(0);
  const Tensor* given = x.t(5);
  Tensor out = given ? *given : empty_like(in);
  check(unlocked(flb200_channel_bias_add, P(in), Pf(x.t(1)), P(out), x.i(2), x.i(3), x.i(4), code_of(in), stream()));
  return wrap(out);
}

// ---------------------------------------------------------------- layernorm
NATIVE(layernorm) {  // (x contiguous, weight, bias, eps) -> (y, xhat, invstd)
  const Tensor& in = x.tensor(0);
  const int64_t feat = in.size(-1), rows = feat ? in.numel() / feat : 0;
  Tensor y = empty_like(in), xhat = empty_like(in), invstd = floats(rows, in);
  check(unlocked(flb200_layernorm_forward, P(in), Pf(x.t(1)), Pf(x.t(2)), P(y), P(xhat), nullptr, Pf(&invstd), rows,
                                 feat, x.d(3), code_of(in), stream()));
  return wrap({y, xhat, invstd});
}
NATIVE(layernorm_backward) {  // (grad_y contiguous, xhat, weight, invstd, need_x, need_params)
  const Tensor &gy = x.tensor(0), &xhat = x.tensor(1);
  const int64_t feat = xhat.size(-1), rows = feat ? xhat.numel() / feat : 0;
  Tensor gx, gw, gb;
  if (x.b(4)) gx = empty_like(xhat);
  if (x.b(5)) { gw = floats(feat, xhat); gb = floats(feat, xhat); }
  Workspace ws(flb200_layernorm_backward_workspace_bytes(rows, feat), xhat);
  check(unlocked(flb200_layernorm_backward, P(gy), P(xhat), Pf(x.t(2)), Pf(x.t(3)), gx.defined() ? P(gx) : nullptr,
                                  gw.defined() ? Pf(&gw) : nullptr, gb.defined() ? Pf(&gb) : nullptr, rows,
                                  feat, code_of(xhat), ws.p(), ws.bytes, stream()));
  return wrap({gx, gw, gb});
}

// ---------------------------------------------------------------- linear, matmul
struct LinearDims { int64_t O, I, cols; };
LinearDims linear_dims(const Tensor& weight, const Tensor& in) {
  LinearDims d;
  d.I = in.size(-1);
  d.cols = d.I ? in.numel() / d.I : 0;
  d.O = weight.size(1);
  if (weight.size(0) != d.I) {
    PyErr_Format(PyExc_ValueError, "linear: weight expects %lld input features, input has %lld",
                 (long long)weight.size(0), (long long)d.I);
    throw PyRaised();
  }
  return d;
}
Tensor rows_of(const Tensor& in, int64_t O) {
  auto s = in.sizes().vec();
  s.back() = O;
  return empty(s, in.scalar_type(), in);
}

NATIVE(linear) {  // (x, weight, bias or None, mode)
  const Tensor &in = x.tensor(0), &w = x.tensor(1);
  const LinearDims d = linear_dims(w, in);
  Tensor y = rows_of(in, d.O);
  Workspace ws(flb200_linear_workspace_bytes(d.O, d.I, d.cols, 0), in);
  check(unlocked(flb200_linear_forward, d.O, d.I, d.cols, P(w), P(in), P(x.t(2)), P(y), x.n32(3), ws.p(), ws.bytes,
                              stream()));
  return wrap(y);
}
NATIVE(linear_bias_act) {  // (x, weight, bias or None, gelu, mode) -> (y, pre) or None
  const Tensor &in = x.tensor(0), &w = x.tensor(1);
  const Tensor* bias = x.t(2);
  const bool gelu = x.b(3);
  const int mode = x.n32(4);
  const LinearDims d = linear_dims(w, in);
  if (d.O % 32 || !in.is_contiguous() || !w.is_contiguous() ||
      (in.scalar_type() == ScalarType::Float && mode == FLB200_MATH_STRICT_F32))
    Py_RETURN_NONE;
  Tensor y = rows_of(in, d.O), pre;
  if (gelu) pre = empty_like(y);
  flb200_matmul_desc m = {};  // the product that the call runs
  m.m = d.cols; m.n = d.O; m.k = d.I; m.batch = 1;
  m.a_row = d.I; m.a_col = 1; m.b_row = d.O; m.b_col = 1; m.c_row = d.O; m.c_col = 1;
  m.alpha = 1.f; m.dtype = code_of(in); m.math_mode = mode;
  Workspace ws(flb200_matmul_call_workspace_bytes(&m, P(in), P(w), P(y)), in);
  const int st = unlocked(
      flb200_linear_bias_act_forward, d.O, d.I, d.cols, P(w), P(in), Pf(bias), P(y), gelu ? P(pre) : nullptr,
      gelu ? FLB200_ACT_GELU : FLB200_ACT_NONE, code_of(in), mode, ws.p(), ws.bytes, stream());
  if (st == FLB200_UNSUPPORTED) Py_RETURN_NONE;
  check(st);
  return wrap({y, pre});
}
NATIVE(linear_backward) {  // (x, weight, grad_y, has_bias, need_x, need_w, mode) -> (gx, gw, gb)
  const Tensor &in = x.tensor(0), &w = x.tensor(1), &gy = x.tensor(2);
  const LinearDims d = linear_dims(w, in);
  const int mode = x.n32(6);
  Tensor gx, gw, gb;
  if (x.b(3)) {
    if (gy.numel() != d.cols * d.O) value_error("channel_sum: geometry does not match the tensor");
    gb = floats(d.O, gy);
    Workspace ws(flb200_channel_sum_workspace_bytes(d.cols, d.O, 1), in);
    check(unlocked(flb200_channel_sum, P(gy), Pf(&gb), d.cols, d.O, 1, code_of(gy), ws.p(), ws.bytes, stream()));
  }
  if (x.b(4)) {
    gx = empty_like(in);
    Workspace ws(flb200_linear_workspace_bytes(d.O, d.I, d.cols, 1), in);
    check(unlocked(flb200_linear_backward_input, d.O, d.I, d.cols, P(w), P(gy), P(gx), mode, ws.p(), ws.bytes,
                   stream()));
  }
  if (x.b(5)) {
    gw = empty_like(w);
    Workspace ws(flb200_linear_workspace_bytes(d.O, d.I, d.cols, 2), in);
    check(unlocked(flb200_linear_backward_weight, d.O, d.I, d.cols, P(gy), P(in), P(gw), mode, ws.p(), ws.bytes,
                   stream()));
  }
  return wrap({gx, gw, gb});
}
// (a, b, c or None, m, n, k, a_row, a_col, b_row, b_col, c_row, c_col, batch, a_batch, b_batch,
//  c_batch, alpha, beta, mode): c None = a new row-major result
NATIVE(matmul) {
  const Tensor &a = x.tensor(0), &b = x.tensor(1);
  const Tensor* given = x.t(2);
  const bool wide = x.b(19);  // an f32 result of 16-bit operands
  if (wide && given && given->scalar_type() != ScalarType::Float) value_error("matmul: a wide result is float32");
  flb200_matmul_desc d = {};
  d.m = x.i(3); d.n = x.i(4); d.k = x.i(5);
  d.a_row = x.i(6); d.a_col = x.i(7); d.b_row = x.i(8); d.b_col = x.i(9);
  d.batch = x.i(12);
  d.a_batch = x.i(13); d.b_batch = x.i(14);
  Tensor c;
  if (given) {
    c = *given;
    d.c_row = x.i(10); d.c_col = x.i(11); d.c_batch = x.i(15);
  } else {
    const ScalarType type = wide ? ScalarType::Float : a.scalar_type();
    if (d.batch > 1) c = empty({d.batch, d.m, d.n}, type, a);
    else c = empty({d.m, d.n}, type, a);
    d.c_row = d.n; d.c_col = 1; d.c_batch = d.m * d.n;
  }
  d.alpha = (float)x.d(16); d.beta = (float)x.d(17);
  d.dtype = code_of(a); d.math_mode = x.n32(18);
  Workspace ws(flb200_matmul_call_workspace_bytes(&d, P(a), P(b), P(c)), a);
  check(wide ? unlocked(flb200_matmul_wide, &d, P(a), P(b), Pf(&c), ws.p(), ws.bytes, stream())
             : unlocked(flb200_matmul, &d, P(a), P(b), P(c), ws.p(), ws.bytes, stream()));
  return wrap(c);
}

// ---------------------------------------------------------------- softmax and losses
void classes(const Tensor& t, int64_t* C, int64_t* X) {
  *C = t.size(-1);
  *X = *C ? t.numel() / *C : 0;
}
NATIVE(log_softmax) {  // (x)
  const Tensor& in = x.tensor(0);
  int64_t C, X;
  classes(in, &C, &X);
  Tensor y = empty_like(in);
  check(unlocked(flb200_log_softmax_forward, P(in), P(y), C, X, code_of(in), stream()));
  return wrap(y);
}
NATIVE(log_softmax_backward) {  // (y, grad_y)
  const Tensor& y = x.tensor(0);
  int64_t C, X;
  classes(y, &C, &X);
  Tensor gx = empty_like(y);
  check(unlocked(flb200_log_softmax_backward, P(y), P(x.tensor(1)), P(gx), C, X, code_of(y), stream()));
  return wrap(gx);
}
NATIVE(cce_forward) {  // (logp, targets int32, reduction, ignore_index) -> (loss, meta)
  const Tensor &logp = x.tensor(0), &tg = x.tensor(1);
  int64_t C, X;
  classes(logp, &C, &X);
  const int red = x.n32(2);
  Tensor loss = floats(red == FLB200_REDUCE_NONE ? X : 1, logp);
  Tensor meta = empty({2}, ScalarType::Int, logp);  // [count, bad-target flag]
  int32_t* m = static_cast<int32_t*>(meta.data_ptr());
  void* st = stream();
  if (unlocked(cudaMemsetAsync, m, 0, (size_t)8,
               static_cast<cudaStream_t>(st)) != cudaSuccess) check(FLB200_LAUNCH_FAILURE);
  Workspace ws(flb200_cce_workspace_bytes(X), logp);
  check(unlocked(flb200_cce_forward, P(logp), static_cast<const int32_t*>(P(tg)), Pf(&loss), m, m + 1, C, X, red,
                 x.n32(3),
                           code_of(logp), ws.p(), ws.bytes, st));
  return wrap({loss, meta});
}
// from the scores: (x, targets int32, reduction, ignore_index) -> (loss, meta, lse), or None where the
// library has no kernel for the rows
NATIVE(scores_cce_forward) {
  const Tensor &in = x.tensor(0), &tg = x.tensor(1);
  int64_t C, X;
  classes(in, &C, &X);
  if (C <= 1024 || C % 4 != 0 || X < 1 || X > 65535 || !in.is_contiguous() || !aligned16(&in)) Py_RETURN_NONE;
  const int red = x.n32(2);
  Tensor loss = floats(red == FLB200_REDUCE_NONE ? X : 1, in), lse = floats(X, in);
  Tensor meta = empty({2}, ScalarType::Int, in);  // [count, bad-target flag]
  int32_t* m = static_cast<int32_t*>(meta.data_ptr());
  void* st = stream();
  if (unlocked(cudaMemsetAsync, m, 0, (size_t)8, static_cast<cudaStream_t>(st)) != cudaSuccess)
    check(FLB200_LAUNCH_FAILURE);
  Workspace ws(flb200_cce_workspace_bytes(X), in);
  check(unlocked(flb200_scores_cce_forward, P(in), Pf(&lse), static_cast<const int32_t*>(P(tg)), Pf(&loss), m, m + 1,
                 C, X, red, x.n32(3), code_of(in), ws.p(), ws.bytes, st));
  return wrap({loss, meta, lse});
}
NATIVE(scores_cce_backward) {  // (x, lse, grad_loss, targets, meta, reduction, ignore_index)
  const Tensor &in = x.tensor(0), &tg = x.tensor(3), &meta = x.tensor(4);
  int64_t C, X;
  classes(in, &C, &X);
  Tensor gx = empty_like(in);
  check(unlocked(flb200_scores_cce_backward, P(in), Pf(x.t(1)), Pf(x.t(2)), static_cast<const int32_t*>(P(tg)),
                 static_cast<const int32_t*>(P(meta)), P(gx), C, X, x.n32(5), x.n32(6), code_of(in), stream()));
  return wrap(gx);
}
NATIVE(cce_backward) {  // (grad_loss, targets, meta, C, reduction, ignore_index, like)
  const Tensor &tg = x.tensor(1), &meta = x.tensor(2), &like = x.tensor(6);
  Tensor gx = empty_like(like);
  check(unlocked(flb200_cce_backward, Pf(x.t(0)), static_cast<const int32_t*>(P(tg)),
                            static_cast<const int32_t*>(P(meta)), P(gx), x.i(3), tg.numel(), x.n32(4), x.n32(5),
                            code_of(like), stream()));
  return wrap(gx);
}
NATIVE(log_softmax_cce_backward) {  // (y, grad_loss, targets, meta, reduction, ignore_index)
  const Tensor &y = x.tensor(0), &tg = x.tensor(2), &meta = x.tensor(3);
  int64_t C, X;
  classes(y, &C, &X);
  Tensor gx = empty_like(y);
  check(unlocked(flb200_log_softmax_cce_backward, P(y), Pf(x.t(1)), static_cast<const int32_t*>(P(tg)),
                                        static_cast<const int32_t*>(P(meta)), P(gx), C, X, x.n32(4), x.n32(5),
                                        code_of(y), stream()));
  return wrap(gx);
}
NATIVE(softmax) {  // (x, scale, causal_period, with_lse) -> y or (y, lse)
  const Tensor& in = x.tensor(0);
  int64_t C, X;
  classes(in, &C, &X);
  const float scale = (float)x.d(1);
  Tensor y = empty_like(in);
  if (!x.b(3)) {
    check(unlocked(flb200_softmax_forward, P(in), P(y), C, X, scale, x.i(2), code_of(in), stream()));
    return wrap(y);
  }
  Tensor lse = floats(X, in);
  check(unlocked(flb200_softmax_forward_lse, P(in), P(y), Pf(&lse), C, X, scale, x.i(2), code_of(in), stream()));
  return wrap({y, lse});
}
NATIVE(softmax_backward) {  // (y, grad_y, scale)
  const Tensor& y = x.tensor(0);
  int64_t C, X;
  classes(y, &C, &X);
  Tensor gx = empty_like(y);
  check(unlocked(flb200_softmax_backward, P(y), P(x.tensor(1)), P(gx), C, X, (float)x.d(2), code_of(y), stream()));
  return wrap(gx);
}
NATIVE(attention_backward) {  // (q, k, v, o, grad_o, lse, scale, causal) -> (dq, dk, dv)
  const Tensor& q = x.tensor(0);
  for (int i = 0; i < 5; ++i) {
    const Tensor& t = x.tensor(i);
    if (t.dim() != 3 || t.sizes() != q.sizes() || !t.is_contiguous() || t.scalar_type() != q.scalar_type())
      value_error("attention_backward: q, k, v, o and grad_o must be dense and alike");
  }
  const int64_t Z = q.size(0), T = q.size(1), hd = q.size(2);
  const Tensor all = empty({3, Z, T, hd}, q.scalar_type(), q);  // one after another (autograd.unbind)
  const Tensor dq = all.select(0, 0), dk = all.select(0, 1), dv = all.select(0, 2);
  Workspace ws(flb200_attention_backward_workspace_bytes(Z, T, hd), q);
  check(unlocked(flb200_attention_backward, P(q), P(x.t(1)), P(x.t(2)), P(x.t(3)), P(x.t(4)), Pf(x.t(5)), P(dq),
                 P(dk), P(dv),
                                  Z, T, hd, (float)x.d(6), x.b(7) ? 1 : 0, code_of(q), ws.p(), ws.bytes, stream()));
  return wrap({dq, dk, dv});
}

// (qkv [B * T, 3 * heads * hd] contiguous, B, T, heads, scale, causal) -> (out [B * T, heads * hd], lse), or
// None where the fused kernel is not built for it
NATIVE(attention_packed) {
  const Tensor& qkv = x.tensor(0);
  const int64_t B = x.i(1), T = x.i(2), h = x.i(3);
  if (qkv.dim() != 2 || !qkv.is_contiguous() || B < 1 || T < 1 || h < 1 || qkv.size(0) != B * T ||
      qkv.size(1) % (3 * h) != 0)
    value_error("attention_packed: qkv must be a dense (B * T, 3 * heads * head dim) tensor");
  const int64_t hd = qkv.size(1) / (3 * h);
  if (!flb200_attention_packed_supported(T, hd, code_of(qkv)) || (reinterpret_cast<uintptr_t>(P(qkv)) & 15))
    Py_RETURN_NONE;
  Tensor out = empty({B * T, h * hd}, qkv.scalar_type(), qkv), lse = floats(B * h * T, qkv);
  check(unlocked(flb200_attention_packed_forward, P(qkv), P(out), Pf(&lse), B, h, T, hd, (float)x.d(4), x.b(5) ? 1 : 0,
                                        code_of(qkv), stream()));
  return wrap({out, lse});
}
NATIVE(attention_packed_backward) {  // (qkv, out, grad_out contiguous, lse, B, T, heads, scale, causal)
  const Tensor &qkv = x.tensor(0), &out = x.tensor(1), &gy = x.tensor(2);
  const int64_t B = x.i(4), T = x.i(5), h = x.i(6), hd = out.size(1) / h;
  if (gy.sizes() != out.sizes() || !gy.is_contiguous() || gy.scalar_type() != qkv.scalar_type())
    value_error("attention_packed_backward: grad_out must be dense and like out");
  Tensor g = empty_like(qkv);
  Workspace ws(flb200_attention_backward_workspace_bytes(B * h, T, hd), qkv);
  check(unlocked(flb200_attention_packed_backward, P(qkv), P(out), P(gy), Pf(x.t(3)), P(g), B, h, T, hd, (float)x.d(7),
                                         x.b(8) ? 1 : 0, code_of(qkv), ws.p(), ws.bytes, stream()));
  return wrap(g);
}

// ---------------------------------------------------------------- embedding
int id_code(const Tensor& ids) {
  if (ids.scalar_type() == ScalarType::Long) return FLB200_IDS_I64;
  if (ids.scalar_type() == ScalarType::Int) return FLB200_IDS_I32;
  value_error("embedding: ids must be int32 or int64");
}
NATIVE(embedding) {  // (table, ids contiguous)
  const Tensor &table = x.tensor(0), &ids = x.tensor(1);
  const int code = id_code(ids);
  const int64_t vocab = table.size(0), dim = table.size(1), rows = ids.numel();
  Tensor out = empty({rows, dim}, table.scalar_type(), table);
  check(unlocked(flb200_embedding_forward, P(table), P(ids), code, P(out), rows, dim, vocab, code_of(table), stream()));
  return wrap(out);
}
NATIVE(embedding_backward) {  // (grad_out contiguous, ids contiguous, vocab)
  const Tensor &g = x.tensor(0), &ids = x.tensor(1);
  const int code = id_code(ids);
  const int64_t vocab = x.i(2), dim = g.size(-1);
  Tensor out = empty({vocab, dim}, ScalarType::Float, g);
  check(unlocked(flb200_embedding_backward, P(g), P(ids), code, Pf(&out), ids.numel(), dim, vocab, code_of(g),
                 stream()));
  return wrap(out);
}

// ---------------------------------------------------------------- images
// torch (.., N, C, H, W) with missing leading dims = 1
void shape4(const Tensor& t, int64_t* W, int64_t* H, int64_t* C, int64_t* N) {
  const int64_t n = t.dim();
  if (n > 4) value_error("expected at most 4 dimensions");
  *W = n > 0 ? t.size(n - 1) : 1;
  *H = n > 1 ? t.size(n - 2) : 1;
  *C = n > 2 ? t.size(n - 3) : 1;
  *N = n > 3 ? t.size(n - 4) : 1;
}
// args [at ..]: sx sy px py dx dy groups; y_cl: -1 = the layout of the input
flb200_conv2d_desc conv_desc(const Tensor& in, const Tensor& w, const Args& x, Py_ssize_t at, int y_cl, int mode) {
  const ScalarType ty = in.scalar_type();
  if ((ty != ScalarType::Float && ty != ScalarType::Half && ty != ScalarType::BFloat16) || w.scalar_type() != ty)
    value_error("conv2d: input and weights must share one of f32 / f16 / bf16");
  const bool x_cl = channels_last(in), out_cl = y_cl < 0 ? x_cl : y_cl != 0;
  if (x_cl && !out_cl) value_error("conv2d: a channels-last input gives a channels-last output");
  int64_t W, H, C, N, kW, kH, Cg, Cout;
  shape4(in, &W, &H, &C, &N);
  shape4(w, &kW, &kH, &Cg, &Cout);
  flb200_conv2d_desc d = {};
  d.groups = x.n32(at + 6);
  if (Cg * d.groups != C) {
    PyErr_Format(PyExc_ValueError, "conv2d: weight has %lld input channels per group x %d groups, input has %lld",
                 (long long)Cg, d.groups, (long long)C);
    throw PyRaised();
  }
  d.W = (int)W; d.H = (int)H; d.C = (int)C; d.N = (int)N;
  d.kW = (int)kW; d.kH = (int)kH; d.Cout = (int)Cout;
  d.sx = x.n32(at); d.sy = x.n32(at + 1); d.px = x.n32(at + 2); d.py = x.n32(at + 3);
  d.dx = x.n32(at + 4); d.dy = x.n32(at + 5);
  d.dtype = code_of(in);
  d.math_mode = mode;
  d.layout = x_cl ? FLB200_LAYOUT_NHWC : (out_cl ? FLB200_LAYOUT_NCHW_IN_NHWC_OUT : FLB200_LAYOUT_NCHW);
  return d;
}
flb200_conv2d_cache* cache_of(PyObject* o) {  // the address of a flb200_conv2d_cache, or None
  if (o == Py_None) return nullptr;
  void* p = PyLong_AsVoidPtr(o);
  if (!p && PyErr_Occurred()) throw PyRaised();
  return static_cast<flb200_conv2d_cache*>(p);
}

// (input, weights, sx sy px py dx dy groups, y_cl, mode) -> (bytes of the x copy, of the grad_y copy)
NATIVE(conv2d_cache_bytes) {
  const flb200_conv2d_desc d = conv_desc(x.tensor(0), x.tensor(1), x, 2, x.n32(9), x.n32(10));
  return Py_BuildValue("nn", (Py_ssize_t)flb200_conv2d_cache_bytes(&d, 0), (Py_ssize_t)flb200_conv2d_cache_bytes(&d, 1));
}
// (input, weights, bias or None, sx sy px py dx dy groups, y_cl, mode, cache, want_stats)
//   -> (y, statistics matrix or None, its groups)
NATIVE(conv2d) {
  const Tensor &in = x.tensor(0), &w = x.tensor(1);
  const Tensor* bias = x.t(2);
  const flb200_conv2d_desc d = conv_desc(in, w, x, 3, x.n32(10), x.n32(11));
  int32_t wo, ho;
  check(flb200_conv2d_output_dims(&d, &wo, &ho));
  if (bias && bias->numel() != d.Cout) value_error("conv2d: bias must have one element per output channel");
  Tensor out = empty({d.N, d.Cout, ho, wo}, in.scalar_type(), in, d.layout != FLB200_LAYOUT_NCHW), stats;
  Workspace ws(flb200_conv2d_workspace_bytes(&d, 0), in);
  flb200_conv2d_cache* cache = cache_of(x.at(12));
  int64_t groups = 0;
  size_t sbytes = 0;
  if (x.b(13)) {
    sbytes = flb200_conv2d_stats_bytes(&d, &groups);
    if (sbytes && !(aligned16(&in) && aligned16(&w) && aligned16(bias))) sbytes = 0;
  }
  if (sbytes) {
    stats = floats((int64_t)(sbytes / 4), in);
    check(unlocked(flb200_conv2d_forward_stats, &d, P(in), P(w), P(bias), P(out), Pf(&stats), sbytes, ws.p(),
                   ws.bytes, cache,
                                      stream()));
  } else {
    check(unlocked(flb200_conv2d_forward_cached, &d, P(in), P(w), P(bias), P(out), ws.p(), ws.bytes, cache, stream()));
  }
  PyObject* r = PyTuple_New(3);
  PyTuple_SET_ITEM(r, 0, wrap(out));
  PyTuple_SET_ITEM(r, 1, wrap(stats));
  PyTuple_SET_ITEM(r, 2, PyLong_FromLongLong(groups));
  return r;
}
// (grad_y, input, weight, sx sy px py dx dy groups, mode, cache, grad_x or None)
NATIVE(conv2d_backward_data) {
  const Tensor &gy = x.tensor(0), &in = x.tensor(1), &w = x.tensor(2);
  const flb200_conv2d_desc d = conv_desc(in, w, x, 3, channels_last(gy) || channels_last(in), x.n32(10));
  Tensor gx = empty_like(in);
  Workspace ws(flb200_conv2d_workspace_bytes(&d, 1), in);
  check(unlocked(flb200_conv2d_backward_data_cached, &d, P(gy), P(w), P(gx), ws.p(), ws.bytes, cache_of(x.at(11)),
                 stream()));
  return wrap(gx);
}
// (grad_y, input, weights, bias or None, sx sy px py dx dy groups, mode, cache) -> (grad_w, grad_b)
NATIVE(conv2d_backward_filter_bias) {
  const Tensor &gy = x.tensor(0), &in = x.tensor(1), &w = x.tensor(2);
  const Tensor* bias = x.t(3);
  const flb200_conv2d_desc d = conv_desc(in, w, x, 4, channels_last(gy) || channels_last(in), x.n32(11));
  Tensor gw = empty_like(w), gb;
  if (bias) gb = empty_like(*bias);
  Workspace ws(flb200_conv2d_workspace_bytes(&d, 2), in);
  check(unlocked(flb200_conv2d_backward_filter_bias_cached, &d, P(gy), P(in), P(gw), bias ? P(gb) : nullptr, ws.p(),
                 ws.bytes,
                                                  cache_of(x.at(12)), stream()));
  return wrap({gw, gb});
}

flb200_pool2d_desc pool_desc(const Tensor& in, const Args& x, Py_ssize_t at) {  // wx wy sx sy px py mode
  int64_t W, H, C, N;
  shape4(in, &W, &H, &C, &N);
  flb200_pool2d_desc d = {};
  d.W = (int)W; d.H = (int)H; d.C = (int)C; d.N = (int)N;
  d.wx = x.n32(at); d.wy = x.n32(at + 1); d.sx = x.n32(at + 2); d.sy = x.n32(at + 3);
  d.px = x.n32(at + 4); d.py = x.n32(at + 5); d.mode = x.n32(at + 6);
  d.dtype = code_of(in);
  d.layout = channels_last(in) ? FLB200_LAYOUT_NHWC : FLB200_LAYOUT_NCHW;
  return d;
}
NATIVE(pool2d) {  // (input, wx wy sx sy px py mode, want_argmax) -> (y, argmax or None)
  const Tensor& in = x.tensor(0);
  const flb200_pool2d_desc d = pool_desc(in, x, 1);
  int32_t wo, ho;
  check(flb200_pool2d_output_dims(&d, &wo, &ho));
  const bool cl = d.layout == FLB200_LAYOUT_NHWC;
  Tensor out = empty({d.N, d.C, ho, wo}, in.scalar_type(), in, cl), arg;
  if (x.b(8) && d.mode == FLB200_POOL_MAX) arg = empty({d.N, d.C, ho, wo}, ScalarType::Byte, in, cl);
  check(unlocked(flb200_pool2d_forward, &d, P(in), P(out),
                 arg.defined() ? static_cast<uint8_t*>(arg.data_ptr()) : nullptr,
                              stream()));
  return wrap({out, arg});
}
NATIVE(pool2d_backward) {  // (grad_y, input, argmax or None, wx wy sx sy px py mode)
  const Tensor &gy = x.tensor(0), &in = x.tensor(1);
  const flb200_pool2d_desc d = pool_desc(in, x, 3);
  Tensor gx = empty_like(in);
  check(unlocked(flb200_pool2d_backward, &d, P(gy), P(in), static_cast<const uint8_t*>(P(x.t(2))), P(gx), stream()));
  return wrap(gx);
}

// ---------------------------------------------------------------- batch-norm
flb200_batchnorm_desc bn_desc(const Tensor& in, PyObject* axes) {
  PyObject* seq = PySequence_Fast(axes, "batchnorm: axes must be a sequence");
  if (!seq) throw PyRaised();
  int32_t ax[8];
  const Py_ssize_t na = PySequence_Fast_GET_SIZE(seq);
  for (Py_ssize_t k = 0; k < na && k < 8; ++k) ax[k] = (int32_t)PyLong_AsLong(PySequence_Fast_GET_ITEM(seq, k));
  Py_DECREF(seq);
  if (PyErr_Occurred()) throw PyRaised();
  if (na > 8) value_error("batchnorm: too many axes");
  flb200_batchnorm_desc d = {};
  if (channels_last(in)) {
    // stored [N][H][W][C]: statistics per channel are column sums of a [pixels][C] matrix
    if (na != 1 || ax[0] != 2) value_error("batchnorm: a channels-last tensor is normalised over fl axis 2 only");
    d.outer = in.size(0) * in.size(2) * in.size(3);
    d.channels = in.size(1);
    d.inner = 1;
  } else {
    int64_t shape[16];
    const int nd = (int)in.dim();
    if (nd > 16) value_error("batchnorm: too many dimensions");
    for (int k = 0; k < nd; ++k) shape[k] = in.size(nd - 1 - k);
    check(flb200_batchnorm_geometry(shape, nd, ax, (int)na, &d));
  }
  d.dtype = code_of(in);
  return d;
}
void bn_params(const Args& x, Py_ssize_t at, int64_t channels) {  // weight bias running_mean running_var
  for (Py_ssize_t k = at; k < at + 4; ++k) {
    const Tensor* t = x.t(k);
    if (t && t->scalar_type() != ScalarType::Float)
      value_error("fl::batchnorm: non-input tensors must be of type f32");
  }
  if (x.t(at) && x.t(at)->numel() != channels) value_error("[BatchNorm] Invalid shape for weight.");
  if (x.t(at + 1) && x.t(at + 1)->numel() != channels) value_error("[BatchNorm] Invalid shape for bias.");
}
// (input, weight, bias, running_mean, running_var, axes, train, momentum, epsilon, relu, stats or None,
//  groups) -> (y, save_mean, save_invstd)
NATIVE(batchnorm) {
  const Tensor& in = x.tensor(0);
  const flb200_batchnorm_desc d = bn_desc(in, x.at(5));
  bn_params(x, 1, d.channels);
  const bool train = x.b(6), relu = x.b(9);
  const double mom = x.d(7), eps = x.d(8);
  const Tensor* stats = x.t(10);
  float *w = Pf(x.t(1)), *b = Pf(x.t(2)), *rm = Pf(x.t(3)), *rv = Pf(x.t(4));
  Tensor out = empty_like(in), sm, sv;
  if (train) { sm = floats(d.channels, in); sv = floats(d.channels, in); }
  float *pm = train ? Pf(&sm) : nullptr, *pv = train ? Pf(&sv) : nullptr;
  if (stats && train) {  // statistics from what the producing convolution took: no pass over x for them
    const int64_t groups = x.i(11);
    Workspace ws(flb200_batchnorm_from_stats_workspace_bytes(&d, groups), in);
    check(unlocked(flb200_batchnorm_forward_from_stats, &d, P(in), nullptr, relu ? 1 : 0, Pf(stats), groups, w, b,
                   rm, rv, pm, pv,
                                              mom, eps, P(out), nullptr, ws.p(), ws.bytes, stream()));
  } else {
    Workspace ws(flb200_batchnorm_workspace_bytes(&d), in);
    check(unlocked(
        relu ? flb200_batchnorm_relu_forward : flb200_batchnorm_forward, &d, P(in), w, b, rm, rv, pm, pv, train ? 1 : 0, mom, eps, P(out), ws.p(), ws.bytes, stream()));
  }
  return wrap({out, sm, sv});
}
NATIVE(batchnorm_add_relu_supported) {  // (input, addend, axes)
  const Tensor &in = x.tensor(0), &add = x.tensor(1);
  const flb200_batchnorm_desc d = bn_desc(in, x.at(2));
  const bool shape_ok = d.inner > 1 ? in.scalar_type() == ScalarType::Float
                                    : channels_last(in) && d.channels % 8 == 0;
  return PyBool_FromLong(shape_ok && same_layout(in, add) &&
                         add.scalar_type() == in.scalar_type() && dense(in) && aligned16(&in) && aligned16(&add));
}
// (input, addend, weight, bias, running_mean, running_var, axes, train, momentum, epsilon, stats or
//  None, groups) -> (y, mask, save_mean, save_invstd)
NATIVE(batchnorm_add_relu) {
  const Tensor &in = x.tensor(0), &add = x.tensor(1);
  const flb200_batchnorm_desc d = bn_desc(in, x.at(6));
  const bool train = x.b(7);
  const double mom = x.d(8), eps = x.d(9);
  const Tensor* stats = x.t(10);
  float *w = Pf(x.t(2)), *b = Pf(x.t(3)), *rm = Pf(x.t(4)), *rv = Pf(x.t(5));
  // elements per mask byte: 8 consecutive channels of a pixel for channels-last tensors
  const int64_t group = d.inner % 8 == 0 || d.inner == 1 ? 8 : (d.inner % 4 == 0 ? 4 : 1);
  Tensor out = empty_like(in), mask = empty({(in.numel() + group - 1) / group}, ScalarType::Byte, in), sm, sv;
  if (train) { sm = floats(d.channels, in); sv = floats(d.channels, in); }
  float *pm = train ? Pf(&sm) : nullptr, *pv = train ? Pf(&sv) : nullptr;
  uint8_t* m = static_cast<uint8_t*>(mask.data_ptr());
  if (stats && train) {
    const int64_t groups = x.i(11);
    Workspace ws(flb200_batchnorm_from_stats_workspace_bytes(&d, groups), in);
    check(unlocked(flb200_batchnorm_forward_from_stats, &d, P(in), P(add), 1, Pf(stats), groups, w, b, rm, rv, pm,
                   pv, mom, eps,
                                              P(out), m, ws.p(), ws.bytes, stream()));
  } else {
    Workspace ws(flb200_batchnorm_workspace_bytes(&d), in);
    check(unlocked(flb200_batchnorm_add_relu_forward, &d, P(in), P(add), w, b, rm, rv, pm, pv, train ? 1 : 0, mom,
                   eps, P(out), m,
                                            ws.p(), ws.bytes, stream()));
  }
  return wrap({out, mask, sm, sv});
}
// (grad_y, save_mean, save_invstd, input, weight, bias, axes, relu) -> (grad_x, grad_weight, grad_bias)
NATIVE(batchnorm_backward) {
  const Tensor &gy = x.tensor(0), &in = x.tensor(3);
  const flb200_batchnorm_desc d = bn_desc(in, x.at(6));
  float *sm = Pf(x.t(1)), *sv = Pf(x.t(2)), *w = Pf(x.t(4));
  Tensor gx = empty_like(in), gw = floats(d.channels, in), gb = floats(d.channels, in);
  Workspace ws(flb200_batchnorm_workspace_bytes(&d), in);
  if (x.b(7))
    check(unlocked(flb200_batchnorm_relu_backward, &d, P(gy), P(in), w, Pf(x.t(5)), sm, sv, P(gx), Pf(&gw), Pf(&gb),
                   ws.p(),
                                         ws.bytes, stream()));
  else
    check(unlocked(flb200_batchnorm_backward, &d, P(gy), P(in), w, sm, sv, P(gx), Pf(&gw), Pf(&gb), ws.p(), ws.bytes,
                   stream()));
  return wrap({gx, gw, gb});
}
// relu(batch-norm): (grad_a, grad_b or None, save_mean, save_invstd, input, weight, bias, axes, need_x)
//   -> (grad_x or None, grad_weight, grad_bias)
NATIVE(batchnorm_relu_backward_sum) {
  const Tensor &ga = x.tensor(0), &in = x.tensor(4);
  const Tensor* gb = x.t(1);
  const flb200_batchnorm_desc d = bn_desc(in, x.at(7));
  const bool need = x.b(8);
  Tensor gx, gs, gw = floats(d.channels, in), gb_out = floats(d.channels, in);
  if (need) gx = empty_like(in);
  if (need && gb) gs = empty_like(in);
  Workspace ws(flb200_batchnorm_workspace_bytes(&d), in);
  check(unlocked(flb200_batchnorm_relu_backward_sum, &d, P(ga), P(gb), P(in), Pf(x.t(5)), Pf(x.t(6)), Pf(x.t(2)),
                 Pf(x.t(3)), gs.defined() ? P(gs) : nullptr, gx.defined() ? P(gx) : nullptr, Pf(&gw), Pf(&gb_out),
                 ws.p(), ws.bytes, stream()));
  return wrap({gx, gw, gb_out});
}
// (mask, grad_a, grad_b or None, save_mean, save_invstd, input, weight, axes)
//   -> (grad_sum, grad_x, grad_weight, grad_bias)
NATIVE(batchnorm_add_relu_backward) {
  const Tensor& in = x.tensor(5);
  const flb200_batchnorm_desc d = bn_desc(in, x.at(7));
  Tensor gs = empty_like(in), gx = empty_like(in), gw = floats(d.channels, in), gb = floats(d.channels, in);
  Workspace ws(flb200_batchnorm_workspace_bytes(&d), in);
  check(unlocked(flb200_batchnorm_add_relu_backward, &d, static_cast<const uint8_t*>(P(x.t(0))), P(x.t(1)),
                 P(x.t(2)), P(in),
                                           Pf(x.t(6)), Pf(x.t(3)), Pf(x.t(4)), P(gs), P(gx), Pf(&gw), Pf(&gb), ws.p(),
                                           ws.bytes, stream()));
  return wrap({gs, gx, gw, gb});
}

NATIVE(set_check) {  // (callable)
  Py_XDECREF(g_check);
  g_check = x.at(0);
  Py_INCREF(g_check);
  Py_RETURN_NONE;
}

#define ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    ENTRY(set_check), ENTRY(unary), ENTRY(binary), ENTRY(relu_mask), ENTRY(relu_mask_backward),
    ENTRY(dropout_apply), ENTRY(astype), ENTRY(reorder), ENTRY(bernoulli_mask), ENTRY(channel_sum),
    ENTRY(channel_bias_add), ENTRY(layernorm), ENTRY(layernorm_backward), ENTRY(linear),
    ENTRY(linear_bias_act), ENTRY(linear_backward), ENTRY(matmul), ENTRY(log_softmax),
    ENTRY(log_softmax_backward), ENTRY(cce_forward), ENTRY(scores_cce_forward), ENTRY(scores_cce_backward), ENTRY(cce_backward),
    ENTRY(log_softmax_cce_backward), ENTRY(softmax), ENTRY(softmax_backward),
    ENTRY(attention_backward), ENTRY(attention_packed), ENTRY(attention_packed_backward),
    ENTRY(embedding), ENTRY(embedding_backward),
    ENTRY(conv2d_cache_bytes), ENTRY(conv2d), ENTRY(conv2d_backward_data),
    ENTRY(conv2d_backward_filter_bias), ENTRY(pool2d), ENTRY(pool2d_backward), ENTRY(batchnorm),
    ENTRY(batchnorm_add_relu_supported), ENTRY(batchnorm_add_relu), ENTRY(batchnorm_backward),
    ENTRY(batchnorm_add_relu_backward), ENTRY(batchnorm_relu_backward_sum), {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
