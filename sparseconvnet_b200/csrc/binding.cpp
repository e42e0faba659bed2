// The operator functions of SCN.py as native calls: argument checks, output sizing, the current stream and the C-ABI
// call in one step.  Through ctypes an operator costs 25 to 40 us of Python besides its launches (a U-Net forward 1.5
// of 4 ms); here it is 2 to 3 us.  Nothing else lives here: every function does what the function of the same name in
// SCN.py documents, with the same messages, and SCN.py keeps the forms it uses for profiling.
//
// Plain CPython calling convention (METH_FASTCALL), tensors through torch's own object layout.  The library itself has
// no torch types; this module is the only place where the two meet.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/scn_b200.h"

namespace {

struct Fail {};  // a Python exception is set

[[noreturn]] void fail(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  PyErr_FormatV(PyExc_RuntimeError, fmt, ap);
  va_end(ap);
  throw Fail{};
}

PyObject *g_check = nullptr;  // _lib.check: raises ScnError for a status
void check(int status) {
  if (status == SCN_OK) return;
  PyObject *r = PyObject_CallFunction(g_check, "i", status);
  if (r) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, "library call failed");
  }
  throw Fail{};
}

// A library call may launch dozens of kernels or wait for the GPU: other Python threads run meanwhile.
struct NoGil {
  PyThreadState *state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};
#define SCN_CALL(...)                    \
  do {                                   \
    int status_;                         \
    {                                    \
      const NoGil free_;                 \
      status_ = (__VA_ARGS__);           \
    }                                    \
    check(status_);                      \
  } while (0)

// ---- arguments ----------------------------------------------------------------------------------------------------
const at::Tensor &tensor(PyObject *o, const char *name) {
  if (!THPVariable_Check(o)) fail("%s must be a tensor", name);
  return THPVariable_Unpack(o);
}

const at::Tensor &features(PyObject *o, const char *name) {
  const at::Tensor &t = tensor(o, name);
  if (!t.is_cuda()) fail("%s must be a CUDA tensor: sparseconvnet_b200 has no CPU path", name);
  if (t.scalar_type() != at::kFloat) fail("%s must be float32", name);
  if (!t.is_contiguous()) fail("%s must be contiguous", name);
  return t;
}

// None or a 0-element tensor: absent
const float *optional(PyObject *o, const at::Tensor &like, const char *name) {
  if (o == Py_None) return nullptr;
  const at::Tensor &t0 = tensor(o, name);
  if (t0.numel() == 0) return nullptr;
  const at::Tensor &t = features(o, name);
  if (t.device() != like.device()) fail("%s is on another device than the features", name);
  return (const float *)t.data_ptr();
}

float *ptr(const at::Tensor &t) { return t.numel() ? (float *)t.data_ptr() : nullptr; }

// spatial size, filter size or stride: a CPU LongTensor, or any sequence of integers (copied to `own`)
struct Sizes {
  const int64_t *p = nullptr;
  int64_t own[16];
  int n = 0;
  explicit Sizes(PyObject *o) {
    if (THPVariable_Check(o)) {
      const at::Tensor &t = THPVariable_Unpack(o);
      if (t.scalar_type() == at::kLong && !t.is_cuda() && t.is_contiguous()) {
        p = (const int64_t *)t.data_ptr();
        n = (int)t.numel();
        return;
      }
    }
    PyObject *seq = PySequence_Fast(o, "a size must be a tensor or a sequence");
    if (!seq) throw Fail{};
    n = (int)std::min<Py_ssize_t>(PySequence_Fast_GET_SIZE(seq), 17);
    if (n > 16) {
      Py_DECREF(seq);
      fail("a size of more than 16 dimensions");
    }
    for (int i = 0; i < n; ++i) {
      PyObject *v = PyNumber_Long(PySequence_Fast_GET_ITEM(seq, i));
      own[i] = v ? PyLong_AsLongLong(v) : 0;
      Py_XDECREF(v);
    }
    Py_DECREF(seq);
    if (PyErr_Occurred()) throw Fail{};
    p = own;
  }
};

// The features' device made current for the call, and its current stream.
struct OnDevice {
  int previous = -1;
  void *stream;
  explicit OnDevice(const at::Tensor &f) {
    const int dev = f.get_device();
    const int current = c10::cuda::current_device();
    if (current != dev) {
      previous = current;
      c10::cuda::set_device((c10::DeviceIndex)dev);
    }
    stream = (void *)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  }
  ~OnDevice() {
    if (previous >= 0) c10::cuda::set_device((c10::DeviceIndex)previous);
  }
};

scn_metadata *md_of(PyObject *o) { return (scn_metadata *)PyLong_AsVoidPtr(o); }

int64_t n_active(scn_metadata *md, const Sizes &size) {
  int64_t n = 0;
  check(scn_md_n_active(md, size.p, &n));
  return n;
}

void same_rows(const at::Tensor &f, int64_t n) {
  if (f.size(0) != n)
    fail("features have %lld rows, metadata has %lld active sites", (long long)f.size(0), (long long)n);
}

struct Weight {
  const at::Tensor &w;
  int groups, cin, cout;
  Weight(PyObject *o, const at::Tensor &f) : w(features(o, "weight")) {
    if (w.dim() != 4) fail("weight must be [filter_volume, groups, nIn/groups, nOut/groups]");
    if (w.device() != f.device()) fail("weight and features are on different devices");
    groups = (int)w.size(1), cin = (int)w.size(2), cout = (int)w.size(3);
  }
};

// (scale, shift, leakiness) of a BatchNorm that rides in a convolution call, or None
struct Affine {
  const float *scale = nullptr, *shift = nullptr;
  double leak = 1.0;
  Affine(PyObject *o, const at::Tensor &f, int planes) {
    if (o == Py_None) return;
    if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 3) fail("a fused BatchNorm is a tuple (scale, shift, leakiness)");
    for (int i = 0; i < 2; ++i) {
      const at::Tensor &t = tensor(PyTuple_GET_ITEM(o, i), "scale / shift");
      if (!t.is_cuda() || t.scalar_type() != at::kFloat || t.numel() != planes || t.device() != f.device())
        fail("fused BatchNorm: scale / shift must be CUDA float32 [%d] on the features' device", planes);
      (i ? shift : scale) = (const float *)t.data_ptr();
    }
    leak = PyFloat_AsDouble(PyTuple_GET_ITEM(o, 2));
  }
};

// The multiply-add count of a convolution: a float, or (ticket, factor) while the rule totals are on their way.
PyObject *macs_result(scn_metadata *md, double macs) {
  if (macs >= 0) return PyFloat_FromDouble(macs);
  void *ticket = nullptr;
  check(scn_md_take_count_ticket(md, &ticket));
  if (!ticket) fail("count pending but no ticket");
  return Py_BuildValue("(Kd)", (unsigned long long)(uintptr_t)ticket, -macs);
}

struct Token {  // prepared weight images are kept under it while the call runs
  uint64_t t;
  explicit Token(PyObject *o) : t(PyLong_AsUnsignedLongLong(o)) {
    if (t) scn_set_weight_token(t);
  }
  ~Token() {
    if (t) scn_set_weight_token(0);
  }
};

// Rows in the tensor cores' split form that travel with a tensor from the convolution that makes them to the one that reads
// them: the input's (or None), and whether the result is wanted in that form too.
struct Split {
  at::Tensor made;
  bool want;
  Split(PyObject *in, PyObject *wanted) : want(PyObject_IsTrue(wanted) == 1) {
    in_ = in == Py_None ? nullptr : tensor(in, "split rows").data_ptr();
  }
  void begin(const at::Tensor &out, int precision) {
    if (!want && !in_) return;
    if (want) {
      const int64_t parts = precision == SCN_PRECISION_BF16 ? 1 : 2;
      made = at::empty({out.size(0), out.size(1) * 2 * parts}, out.options().dtype(at::kByte));
    }
    scn_set_split_rows(in_, want && made.numel() ? made.data_ptr() : nullptr);
    set_ = true;
  }
  // (output, count), or (output, count, split rows or None)
  PyObject *finish(PyObject *pair) {
    const bool written = set_ && scn_split_rows_written();
    set_ = false;
    if (!want || !pair || !PyTuple_Check(pair)) return pair;
    PyObject *three = PyTuple_New(3);
    for (int i = 0; i < 2; ++i) {
      PyObject *o = PyTuple_GET_ITEM(pair, i);
      Py_INCREF(o);
      PyTuple_SET_ITEM(three, i, o);
    }
    Py_DECREF(pair);
    if (!written) Py_INCREF(Py_None);
    PyTuple_SET_ITEM(three, 2, written ? THPVariable_Wrap(std::move(made)) : Py_None);
    return three;
  }
  ~Split() {
    if (set_) scn_split_rows_written();  // (an error on the way)
  }

 private:
  const void *in_ = nullptr;
  bool set_ = false;
};

void size_to(const at::Tensor &t, at::IntArrayRef shape) { const_cast<at::Tensor &>(t).resize_(shape); }

// The output of an operator: the caller's tensor, sized here, or (None) a new one that the call returns.
struct Output {
  at::Tensor t;
  const bool own;
  PyObject *given;
  Output(PyObject *o, const at::Tensor &like) : own(o == Py_None), given(o), like_(like) {}
  void size(at::IntArrayRef shape) {
    if (own) {
      t = at::empty(shape, like_.options());
    } else {
      t = tensor(given, "output_features");
      t.resize_(shape);
    }
  }
  float *ptr() { return t.numel() ? (float *)t.data_ptr() : nullptr; }
  PyObject *result() {
    if (!own) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(t));
  }
  PyObject *result(PyObject *value) {  // `value` alone, or (tensor, value)
    if (!own || !value) return value;
    PyObject *pair = PyTuple_New(2);
    PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(t)));
    PyTuple_SET_ITEM(pair, 1, value);
    return pair;
  }

 private:
  const at::Tensor &like_;
};

#define SCN_FN(name) PyObject *name(PyObject *, PyObject *const *a, Py_ssize_t n_args)
#define SCN_BEGIN(count)                                                                     \
  try {                                                                                      \
    if (n_args != (count)) fail("%s takes %d arguments, got %d", __func__, (count), (int)n_args);
#define SCN_END                                                                              \
  }                                                                                          \
  catch (const Fail &) {                                                                     \
    return nullptr;                                                                          \
  }                                                                                          \
  catch (const std::exception &e) {                                                          \
    PyErr_SetString(PyExc_RuntimeError, e.what());                                           \
    return nullptr;                                                                          \
  }

// ---- convolutions -------------------------------------------------------------------------------------------------
// Every forward call takes the output tensor it is to size and fill, or None: then it makes one and returns (output,
// count) instead of the count alone.
// (md, size, filter, features, out, weight, bias, epilogue, precision, token, prologue, split rows, want split rows)
SCN_FN(submanifold_convolution) {
  SCN_BEGIN(13)
  Split split(a[11], a[12]);
  scn_metadata *md = md_of(a[0]);
  const Sizes size(a[1]), filter(a[2]);
  const at::Tensor &f = features(a[3], "input_features");
  Output out(a[4], f);
  const Weight w(a[5], f);
  const int nin = w.groups * w.cin, nout = w.groups * w.cout;
  if (f.numel() && f.size(1) != nin) fail("features have %d planes, weight expects %d", (int)f.size(1), nin);
  const float *bias = optional(a[6], f, "bias");
  const Affine bn(a[7], f, nout), pre(a[10], f, nin);
  const int precision = (int)PyLong_AsLong(a[8]);
  const OnDevice on(f);
  const Token token(a[9]);
  const int64_t n = n_active(md, size);
  same_rows(f, n);
  out.size({n, nout});
  split.begin(out.t, precision);
  double macs = 0;
  if (pre.scale)
    SCN_CALL(scn_submanifold_convolution_joined_forward(md, size.p, filter.p, ptr(f), nin, nullptr, 0, out.ptr(), ptr(w.w), bias,
                                                        pre.scale, pre.shift, pre.leak, bn.scale, bn.shift, bn.leak, nout,
                                                        precision, on.stream, &macs));
  else if (bn.scale)
    SCN_CALL(scn_submanifold_convolution_bn_forward(md, size.p, filter.p, ptr(f), out.ptr(), ptr(w.w), bias, bn.scale,
                                                 bn.shift, bn.leak, nin, nout, w.groups, precision, on.stream, &macs));
  else
    SCN_CALL(scn_submanifold_convolution_forward(md, size.p, filter.p, ptr(f), out.ptr(), ptr(w.w), bias, nin, nout, w.groups,
                                              precision, on.stream, &macs));
  return split.finish(out.result(macs_result(md, macs)));
  SCN_END
}

// (md, size, filter, features_a, features_b, out, weight, bias, prologue, epilogue, precision, token, want split rows) -> None when the
// shapes are not ones the call takes
SCN_FN(submanifold_joined) {
  SCN_BEGIN(13)
  Split split(Py_None, a[12]);
  scn_metadata *md = md_of(a[0]);
  const Sizes size(a[1]), filter(a[2]);
  const at::Tensor &fa = features(a[3], "input_features"), &fb = features(a[4], "input_features");
  Output out(a[5], fa);
  const Weight w(a[6], fa);
  const int ca = (int)fa.size(1), cb = (int)fb.size(1);
  if (w.groups != 1 || fa.size(0) != fb.size(0) || ca % 8 || cb % 4 || fa.device() != fb.device() || w.cin != ca + cb)
    Py_RETURN_NONE;
  const float *bias = optional(a[7], fa, "bias");
  const Affine pre(a[8], fa, ca + cb), bn(a[9], fa, w.cout);
  const int precision = (int)PyLong_AsLong(a[10]);
  const OnDevice on(fa);
  const Token token(a[11]);
  const int64_t n = n_active(md, size);
  same_rows(fa, n);
  out.size({n, w.cout});
  split.begin(out.t, precision);
  double macs = 0;
  SCN_CALL(scn_submanifold_convolution_joined_forward(md, size.p, filter.p, ptr(fa), ca, ptr(fb), cb, out.ptr(), ptr(w.w), bias,
                                                   pre.scale, pre.shift, pre.leak, bn.scale, bn.shift, bn.leak, w.cout,
                                                   precision, on.stream, &macs));
  return split.finish(out.result(macs_result(md, macs)));
  SCN_END
}

// (md, in_size, out_size, filter, stride, features, out, weight, bias, epilogue, prologue, precision, token, split rows, want
// split rows)
SCN_FN(convolution) {
  SCN_BEGIN(15)
  Split split(a[13], a[14]);
  scn_metadata *md = md_of(a[0]);
  const Sizes in_size(a[1]), out_size(a[2]), filter(a[3]), stride(a[4]);
  const at::Tensor &f = features(a[5], "input_features");
  Output out(a[6], f);
  const Weight w(a[7], f);
  const int nin = w.groups * w.cin, nout = w.groups * w.cout;
  if (f.numel() && f.size(1) != nin) fail("features have %d planes, weight expects %d", (int)f.size(1), nin);
  const float *bias = optional(a[8], f, "bias");
  const Affine bn(a[9], f, nout), pre(a[10], f, nin);
  const int precision = (int)PyLong_AsLong(a[11]);
  const OnDevice on(f);
  const Token token(a[12]);
  same_rows(f, n_active(md, in_size));
  int64_t n_out = 0;
  SCN_CALL(scn_md_strided_rulebook(md, in_size.p, out_size.p, filter.p, stride.p, on.stream, &n_out, nullptr));
  out.size({n_out, nout});
  split.begin(out.t, precision);
  double macs = 0;
  if (pre.scale)
    SCN_CALL(scn_convolution_bn_bn_forward(md, in_size.p, out_size.p, filter.p, stride.p, ptr(f), out.ptr(), ptr(w.w), bias,
                                        pre.scale, pre.shift, pre.leak, bn.scale, bn.shift, bn.leak, nin, nout, w.groups,
                                        precision, on.stream, &macs));
  else if (bn.scale)
    SCN_CALL(scn_convolution_bn_forward(md, in_size.p, out_size.p, filter.p, stride.p, ptr(f), out.ptr(), ptr(w.w), bias,
                                     bn.scale, bn.shift, bn.leak, nin, nout, w.groups, precision, on.stream, &macs));
  else
    SCN_CALL(scn_convolution_forward(md, in_size.p, out_size.p, filter.p, stride.p, ptr(f), out.ptr(), ptr(w.w), bias, nin,
                                  nout, w.groups, precision, on.stream, &macs));
  return split.finish(out.result(macs_result(md, macs)));
  SCN_END
}

// (md, in_size, out_size, filter, stride, features, out, weight, bias, epilogue, precision, token, split rows, want split rows)
SCN_FN(deconvolution) {
  SCN_BEGIN(14)
  Split split(a[12], a[13]);
  scn_metadata *md = md_of(a[0]);
  const Sizes in_size(a[1]), out_size(a[2]), filter(a[3]), stride(a[4]);
  const at::Tensor &f = features(a[5], "input_features");
  Output out(a[6], f);
  const Weight w(a[7], f);
  const int nin = w.groups * w.cin, nout = w.groups * w.cout;
  if (f.numel() && f.size(1) != nin) fail("features have %d planes, weight expects %d", (int)f.size(1), nin);
  const float *bias = optional(a[8], f, "bias");
  const Affine bn(a[9], f, nout);
  const int precision = (int)PyLong_AsLong(a[10]);
  const OnDevice on(f);
  const Token token(a[11]);
  // same rulebook as the Convolution that made `in_size` out of `out_size`
  SCN_CALL(scn_md_strided_rulebook(md, out_size.p, in_size.p, filter.p, stride.p, on.stream, nullptr, nullptr));
  same_rows(f, n_active(md, in_size));
  out.size({n_active(md, out_size), nout});
  split.begin(out.t, precision);
  double macs = 0;
  if (bn.scale)
    SCN_CALL(scn_deconvolution_bn_forward(md, in_size.p, out_size.p, filter.p, stride.p, ptr(f), out.ptr(), ptr(w.w), bias,
                                       bn.scale, bn.shift, bn.leak, nin, nout, w.groups, precision, on.stream, &macs));
  else
    SCN_CALL(scn_deconvolution_forward(md, in_size.p, out_size.p, filter.p, stride.p, ptr(f), out.ptr(), ptr(w.w), bias, nin,
                                    nout, w.groups, precision, on.stream, &macs));
  return split.finish(out.result(macs_result(md, macs)));
  SCN_END
}

// (kind, md, in_size, out_size, filter, stride, features, d_features, d_out, weight, d_weight, d_bias); kind 0
// submanifold (out_size and stride None), 1 strided, 2 transposed
SCN_FN(convolution_backward) {
  SCN_BEGIN(12)
  const int kind = (int)PyLong_AsLong(a[0]);
  scn_metadata *md = md_of(a[1]);
  const Sizes in_size(a[2]), out_size(kind == 0 ? a[2] : a[3]), filter(a[4]), stride(kind == 0 ? a[4] : a[5]);
  const at::Tensor &f = features(a[6], "input_features"), &go = features(a[8], "d_output_features");
  const bool want_input = a[7] != Py_None;  // (the gradient of a network's input features is not wanted)
  float *df = nullptr;
  const Weight w(a[9], f);
  const int nin = w.groups * w.cin, nout = w.groups * w.cout;
  if (f.numel() && f.size(1) != nin) fail("features have %d planes, weight expects %d", (int)f.size(1), nin);
  const at::Tensor &dw = features(a[10], "d_weight");
  if (dw.sizes() != w.w.sizes()) fail("d_weight must have the shape of weight");
  float *db = a[11] == Py_None || tensor(a[11], "d_bias").numel() == 0 ? nullptr : ptr(features(a[11], "d_bias"));
  const OnDevice on(f);
  if (want_input) {
    const at::Tensor &t = tensor(a[7], "d_input_features");
    size_to(t, {f.size(0), nin});
    df = ptr(t);
  }
  if (kind == 0)
    SCN_CALL(scn_submanifold_convolution_backward(md, in_size.p, filter.p, ptr(f), df, ptr(go), ptr(w.w), ptr(dw), db, nin,
                                               nout, w.groups, on.stream));
  else
    SCN_CALL((kind == 1 ? scn_convolution_backward : scn_deconvolution_backward)(
        md, in_size.p, out_size.p, filter.p, stride.p, ptr(f), df, ptr(go), ptr(w.w), ptr(dw), db, nin, nout, w.groups,
        on.stream));
  Py_RETURN_NONE;
  SCN_END
}

// ---- BatchNorm ----------------------------------------------------------------------------------------------------
// (features, out, save_mean, save_invstd, running_mean, running_var, weight, bias, eps, momentum, train, leakiness)
SCN_FN(batchnorm_forward) {
  SCN_BEGIN(12)
  const at::Tensor &f = tensor(a[0], "input_features"), &out = tensor(a[1], "output_features");
  if (!f.is_cuda() || f.scalar_type() != at::kFloat || f.dim() != 2 || (f.numel() && f.stride(1) != 1))
    fail("input_features must be a CUDA float32 matrix with unit column stride");
  const int64_t n = f.size(0), c = f.size(1);
  const OnDevice on(f);
  size_to(out, {n, c});
  const at::Tensor &mean = tensor(a[2], "saveMean"), &invstd = tensor(a[3], "saveInvStd");
  size_to(mean, {c});
  size_to(invstd, {c});
  if (n == 0) Py_RETURN_NONE;
  float *running_mean = ptr(features(a[4], "runningMean")), *running_var = ptr(features(a[5], "runningVar"));
  const float *weight = optional(a[6], f, "weight"), *bias = optional(a[7], f, "bias");
  const double eps = PyFloat_AsDouble(a[8]), momentum = PyFloat_AsDouble(a[9]), leak = PyFloat_AsDouble(a[11]);
  const int train = PyObject_IsTrue(a[10]);
  if (PyErr_Occurred()) throw Fail{};
  SCN_CALL(scn_batchnorm_forward(ptr(f), ptr(out), n, (int)c, f.stride(0), out.stride(0), ptr(mean), ptr(invstd), running_mean,
                                 running_var, weight, bias, eps, momentum, train, leak, on.stream));
  Py_RETURN_NONE;
  SCN_END
}

// (features, d_features, out, d_out, save_mean, save_invstd, weight, d_weight, d_bias, leakiness)
SCN_FN(batchnorm_backward) {
  SCN_BEGIN(10)
  const at::Tensor &f = tensor(a[0], "input_features"), &df = tensor(a[1], "d_input_features");
  const at::Tensor &out = tensor(a[2], "output_features"), &go = tensor(a[3], "d_output_features");
  const int64_t n = f.size(0), c = f.size(1);
  const OnDevice on(f);
  size_to(df, {n, c});
  auto grad = [](PyObject *o) { return o == Py_None ? nullptr : ptr(tensor(o, "gradient")); };
  float *mean = ptr(tensor(a[4], "saveMean")), *invstd = ptr(tensor(a[5], "saveInvStd"));
  const float *weight = optional(a[6], f, "weight");
  float *dw = grad(a[7]), *db = grad(a[8]);
  const double leak = PyFloat_AsDouble(a[9]);
  if (PyErr_Occurred()) throw Fail{};
  SCN_CALL(scn_batchnorm_backward(ptr(f), ptr(df), ptr(out), ptr(go), n, (int)c, n ? f.stride(0) : c, n ? out.stride(0) : c,
                                  mean, invstd, weight, dw, db, leak, on.stream));
  Py_RETURN_NONE;
  SCN_END
}

// ---- pooling, SparseToDense ---------------------------------------------------------------------------------------
// (kind, md, in_size, out_size, pool, stride, features, out, drop); kind 0 max, 1 average, 2 unpooling
SCN_FN(pooling_forward) {
  SCN_BEGIN(9)
  const int kind = (int)PyLong_AsLong(a[0]), drop = (int)PyLong_AsLong(a[8]);
  scn_metadata *md = md_of(a[1]);
  const Sizes in_size(a[2]), out_size(a[3]), pool(a[4]), stride(a[5]);
  const at::Tensor &f = features(a[6], "input_features");
  Output out(a[7], f);
  const OnDevice on(f);
  int64_t n_out = 0;
  if (kind == 2)
    n_out = n_active(md, out_size);
  else
    SCN_CALL(scn_md_strided_rulebook(md, in_size.p, out_size.p, pool.p, stride.p, on.stream, &n_out, nullptr));
  out.size({n_out, f.size(1) - drop});
  SCN_CALL((kind == 0 ? scn_max_pooling_forward : kind == 1 ? scn_average_pooling_forward : scn_unpooling_forward)(
      md, in_size.p, out_size.p, pool.p, stride.p, ptr(f), out.ptr(), (int)f.size(1), drop, on.stream));
  return out.result();
  SCN_END
}

// (kind, md, in_size, out_size, pool, stride, features or None, d_features, out or None, d_out, planes, drop)
SCN_FN(pooling_backward) {
  SCN_BEGIN(12)
  const int kind = (int)PyLong_AsLong(a[0]), planes = (int)PyLong_AsLong(a[10]), drop = (int)PyLong_AsLong(a[11]);
  scn_metadata *md = md_of(a[1]);
  const Sizes in_size(a[2]), out_size(a[3]), pool(a[4]), stride(a[5]);
  const at::Tensor &df = tensor(a[7], "d_input_features"), &go = features(a[9], "d_output_features");
  const OnDevice on(go);
  if (a[6] != Py_None) size_to(df, {tensor(a[6], "input_features").size(0), planes});
  if (kind == 0) {
    const float *in = ptr(features(a[6], "input_features")), *out = ptr(features(a[8], "output_features"));
    SCN_CALL(scn_max_pooling_backward(md, in_size.p, out_size.p, pool.p, stride.p, in, ptr(df), out, ptr(go), planes, drop,
                                      on.stream));
  } else
    SCN_CALL((kind == 1 ? scn_average_pooling_backward : scn_unpooling_backward)(
        md, in_size.p, out_size.p, pool.p, stride.p, ptr(df), ptr(go), planes, drop, on.stream));
  Py_RETURN_NONE;
  SCN_END
}

// (md, size, features, out, planes)
SCN_FN(sparse_to_dense) {
  SCN_BEGIN(5)
  scn_metadata *md = md_of(a[0]);
  const Sizes size(a[1]);
  const at::Tensor &f = features(a[2], "input_features");
  Output out(a[3], f);
  const int planes = (int)PyLong_AsLong(a[4]);
  const OnDevice on(f);
  int64_t batch = 0;
  check(scn_md_batch_size(md, size.p, &batch));
  at::DimVector shape{batch, planes};
  for (int i = 0; i < size.n; ++i) shape.push_back(size.p[i]);
  out.size(shape);
  if (f.dim() != 2) {
    out.t.zero_();
    return out.result();
  }
  if (f.size(1) != planes) fail("features have %d planes, nPlanes is %d", (int)f.size(1), planes);
  SCN_CALL(scn_sparse_to_dense_forward(md, size.p, ptr(f), out.ptr(), planes, on.stream));
  return out.result();
  SCN_END
}

// ---- training: the same operators with their place in the autograd graph ----------------------------------------------
// One graph node per operator whose backward call runs on the engine's own threads without the interpreter.  (As a
// Python torch.autograd.Function an operator cost 15 us more in the forward pass and 20 in the backward pass: half a
// millisecond of a 2.3 ms training step of a small network.)  Gradients are defined once, as with the Python Functions.
namespace ag = torch::autograd;

struct Keep {  // a Python object that lives as long as the node
  PyObject *o;
  explicit Keep(PyObject *p) : o(p) { Py_INCREF(o); }
  Keep(const Keep &) = delete;
  ~Keep() {
    if (!Py_IsInitialized()) return;
    const PyGILState_STATE s = PyGILState_Ensure();
    Py_DECREF(o);
    PyGILState_Release(s);
  }
};

// check() for a thread that does not hold the interpreter lock
void check_free(int status) {
  if (status == SCN_OK) return;
  const PyGILState_STATE s = PyGILState_Ensure();
  python_error e;
  try {
    check(status);
  } catch (const Fail &) {
    e.persist();
  }
  PyGILState_Release(s);
  throw e;
}

std::vector<int64_t> list(const Sizes &s) { return std::vector<int64_t>(s.p, s.p + s.n); }

struct ConvolutionNode : ag::Node {
  ag::SavedVariable features_, weight_, bias_;
  int kind;
  scn_metadata *md;
  Keep keep;
  std::vector<int64_t> in_size, out_size, filter, stride;
  ConvolutionNode(int k, scn_metadata *m, PyObject *o) : kind(k), md(m), keep(o) {}
  std::string name() const override { return "SparseConvolutionBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    features_.reset_data();
    weight_.reset_data();
    bias_.reset_data();
  }
  ag::variable_list apply(ag::variable_list &&grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    ag::variable_list result(3);
    if (!grads[0].defined()) return result;
    const at::NoGradGuard no_grad;
    const at::Tensor f = features_.unpack(), w = weight_.unpack(), b = bias_.unpack(), go = grads[0].contiguous();
    TORCH_CHECK(go.is_cuda() && go.scalar_type() == at::kFloat, "the gradient must be CUDA float32");
    const OnDevice on(f);
    const int groups = (int)w.size(1), nin = groups * (int)w.size(2), nout = groups * (int)w.size(3);
    at::Tensor df, dw = at::empty_like(w), db;
    if (task_should_compute_output(0)) df = at::empty({f.size(0), nin}, go.options());
    if (b.defined() && b.numel()) db = at::empty_like(b);
    float *pf = df.defined() ? ptr(df) : nullptr, *pb = db.defined() ? ptr(db) : nullptr;
    if (kind == 0)
      check_free(scn_submanifold_convolution_backward(md, in_size.data(), filter.data(), ptr(f), pf, ptr(go), ptr(w), ptr(dw),
                                                      pb, nin, nout, groups, on.stream));
    else
      check_free((kind == 1 ? scn_convolution_backward : scn_deconvolution_backward)(
          md, in_size.data(), out_size.data(), filter.data(), stride.data(), ptr(f), pf, ptr(go), ptr(w), ptr(dw), pb, nin,
          nout, groups, on.stream));
    result[0] = df;
    if (task_should_compute_output(1)) result[1] = dw;
    if (db.defined() && task_should_compute_output(2)) result[2] = db;
    return result;
  }
};

struct BatchNormNode : ag::Node {
  ag::SavedVariable features_, out_, weight_;
  at::Tensor mean, invstd;
  double leak = 1;
  bool affine = false;
  std::string name() const override { return "SparseBatchNormBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    features_.reset_data();
    out_.reset_data();
    weight_.reset_data();
    mean.reset();
    invstd.reset();
  }
  ag::variable_list apply(ag::variable_list &&grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    ag::variable_list result(3);
    if (!grads[0].defined()) return result;
    const at::NoGradGuard no_grad;
    const at::Tensor f = features_.unpack(), out = out_.unpack(shared_from_this()), w = weight_.unpack();
    const at::Tensor go = grads[0].contiguous();
    TORCH_CHECK(go.is_cuda() && go.scalar_type() == at::kFloat, "the gradient must be CUDA float32");
    const OnDevice on(f);
    const int64_t n = f.size(0), c = f.size(1);
    at::Tensor df = at::empty({n, c}, go.options()), dw, db;
    if (affine) dw = at::empty_like(w), db = at::empty_like(w);
    check_free(scn_batchnorm_backward(ptr(f), ptr(df), ptr(out), ptr(go), n, (int)c, n ? f.stride(0) : c, n ? out.stride(0) : c,
                                      ptr(mean), ptr(invstd), affine ? ptr(w) : nullptr, affine ? ptr(dw) : nullptr,
                                      affine ? ptr(db) : nullptr, leak, on.stream));
    result[0] = df;
    if (affine && task_should_compute_output(1)) result[1] = dw;
    if (affine && task_should_compute_output(2)) result[2] = db;
    return result;
  }
};

struct PoolingNode : ag::Node {
  ag::SavedVariable features_, out_;
  int kind, drop;
  scn_metadata *md;
  Keep keep;
  std::vector<int64_t> in_size, out_size, pool, stride;
  PoolingNode(int k, int d, scn_metadata *m, PyObject *o) : kind(k), drop(d), md(m), keep(o) {}
  std::string name() const override { return "SparsePoolingBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    features_.reset_data();
    out_.reset_data();
  }
  ag::variable_list apply(ag::variable_list &&grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    ag::variable_list result(1);
    if (!grads[0].defined()) return result;
    const at::NoGradGuard no_grad;
    const at::Tensor f = features_.unpack(), out = out_.unpack(shared_from_this()), go = grads[0].contiguous();
    TORCH_CHECK(go.is_cuda() && go.scalar_type() == at::kFloat, "the gradient must be CUDA float32");
    const OnDevice on(f);
    at::Tensor df = at::empty_like(f);
    const int planes = (int)f.size(1);
    if (kind == 0)
      check_free(scn_max_pooling_backward(md, in_size.data(), out_size.data(), pool.data(), stride.data(), ptr(f), ptr(df),
                                          ptr(out), ptr(go), planes, drop, on.stream));
    else
      check_free((kind == 1 ? scn_average_pooling_backward : scn_unpooling_backward)(
          md, in_size.data(), out_size.data(), pool.data(), stride.data(), ptr(df), ptr(go), planes, drop, on.stream));
    result[0] = df;
    return result;
  }
};

bool has_tangent(const at::Tensor &t) { return t.defined() && t._fw_grad(0).defined(); }

// Forward-mode differentiation has no rule here, as a Python Function without jvp has none; a tangent must not get lost.
template <typename... T>
void no_tangents(const T &...t) {
  if ((has_tangent(t) || ...)) {
    PyErr_SetString(PyExc_NotImplementedError, "this operator has no forward-mode derivative");
    throw Fail{};
  }
}

at::Tensor contiguous_features(PyObject *o) {
  const at::Tensor &t = tensor(o, "input_features");
  if (!t.is_cuda()) fail("input_features must be a CUDA tensor: sparseconvnet_b200 has no CPU path");
  if (t.scalar_type() != at::kFloat) fail("input_features must be float32");
  return t.contiguous();
}

// (kind, metadata, md, in_size, out_size, filter, stride, features, weight, bias, precision) -> (output, count)
SCN_FN(convolution_train) {
  SCN_BEGIN(11)
  const int kind = (int)PyLong_AsLong(a[0]);
  scn_metadata *md = md_of(a[2]);
  const Sizes in_size(a[3]), out_size(kind == 0 ? a[3] : a[4]), filter(a[5]), stride(kind == 0 ? a[5] : a[6]);
  const at::Tensor &given = tensor(a[7], "input_features"), &bias_t = tensor(a[9], "bias");
  at::Tensor f, out;
  double macs = 0;
  const Weight w(a[8], given);
  no_tangents(given, w.w, bias_t);
  {
    const at::NoGradGuard no_grad;
    f = contiguous_features(a[7]);
    const int nin = w.groups * w.cin, nout = w.groups * w.cout;
    if (f.numel() && f.size(1) != nin) fail("features have %d planes, weight expects %d", (int)f.size(1), nin);
    const float *bias = optional(a[9], f, "bias");
    const int precision = (int)PyLong_AsLong(a[10]);
    const OnDevice on(f);
    int64_t n_out = 0;
    if (kind == 0) {
      n_out = n_active(md, in_size);
      same_rows(f, n_out);
    } else if (kind == 1) {
      same_rows(f, n_active(md, in_size));
      SCN_CALL(scn_md_strided_rulebook(md, in_size.p, out_size.p, filter.p, stride.p, on.stream, &n_out, nullptr));
    } else {
      SCN_CALL(scn_md_strided_rulebook(md, out_size.p, in_size.p, filter.p, stride.p, on.stream, nullptr, nullptr));
      same_rows(f, n_active(md, in_size));
      n_out = n_active(md, out_size);
    }
    out = at::empty({n_out, nout}, f.options());
    if (kind == 0)
      SCN_CALL(scn_submanifold_convolution_forward(md, in_size.p, filter.p, ptr(f), ptr(out), ptr(w.w), bias, nin, nout,
                                                   w.groups, precision, on.stream, &macs));
    else if (kind == 1)
      SCN_CALL(scn_convolution_forward(md, in_size.p, out_size.p, filter.p, stride.p, ptr(f), ptr(out), ptr(w.w), bias, nin,
                                       nout, w.groups, precision, on.stream, &macs));
    else
      SCN_CALL(scn_deconvolution_forward(md, in_size.p, out_size.p, filter.p, stride.p, ptr(f), ptr(out), ptr(w.w), bias, nin,
                                         nout, w.groups, precision, on.stream, &macs));
  }
  PyObject *count = macs_result(md, macs);
  if (ag::compute_requires_grad(given, w.w, bias_t)) {
    std::shared_ptr<ConvolutionNode> node(new ConvolutionNode(kind, md, a[1]), ag::deleteNode);
    node->set_next_edges(ag::collect_next_edges(given, w.w, bias_t));
    node->features_ = ag::SavedVariable(f, false);
    node->weight_ = ag::SavedVariable(w.w, false);
    node->bias_ = ag::SavedVariable(bias_t, false);
    node->in_size = list(in_size), node->out_size = list(out_size), node->filter = list(filter), node->stride = list(stride);
    ag::set_history(out, node);
  }
  PyObject *pair = PyTuple_New(2);
  PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(pair, 1, count);
  return pair;
  SCN_END
}

// (features, weight, bias, running_mean, running_var, eps, momentum, train, leakiness) -> output
SCN_FN(batchnorm_train) {
  SCN_BEGIN(9)
  const at::Tensor &given = tensor(a[0], "input_features"), &weight_t = tensor(a[1], "weight"), &bias_t = tensor(a[2], "bias");
  const double eps = PyFloat_AsDouble(a[5]), momentum = PyFloat_AsDouble(a[6]), leak = PyFloat_AsDouble(a[8]);
  const int train = PyObject_IsTrue(a[7]);
  if (PyErr_Occurred()) throw Fail{};
  no_tangents(given, weight_t, bias_t);
  at::Tensor f, out, mean, invstd;
  {
    const at::NoGradGuard no_grad;
    f = contiguous_features(a[0]);
    if (f.dim() != 2) fail("input_features must be a CUDA float32 matrix with unit column stride");
    const int64_t n = f.size(0), c = f.size(1);
    const OnDevice on(f);
    out = at::empty({n, c}, f.options());
    mean = at::empty({c}, f.options());
    invstd = at::empty({c}, f.options());
    float *running_mean = ptr(features(a[3], "runningMean")), *running_var = ptr(features(a[4], "runningVar"));
    const float *weight = optional(a[1], f, "weight"), *bias = optional(a[2], f, "bias");
    if (n)
      SCN_CALL(scn_batchnorm_forward(ptr(f), ptr(out), n, (int)c, f.stride(0), out.stride(0), ptr(mean), ptr(invstd),
                                     running_mean, running_var, weight, bias, eps, momentum, train, leak, on.stream));
  }
  if (ag::compute_requires_grad(given, weight_t, bias_t)) {
    std::shared_ptr<BatchNormNode> node(new BatchNormNode(), ag::deleteNode);
    node->set_next_edges(ag::collect_next_edges(given, weight_t, bias_t));
    node->features_ = ag::SavedVariable(f, false);
    node->weight_ = ag::SavedVariable(weight_t, false);
    node->mean = mean, node->invstd = invstd, node->leak = leak, node->affine = weight_t.numel() > 0;
    ag::set_history(out, node);
    node->out_ = ag::SavedVariable(out, true);
  }
  return THPVariable_Wrap(std::move(out));
  SCN_END
}

// rows @ weight (+ bias): the product on the library's kernel for narrow results, on torch's matrix product otherwise
bool rows_affine_takes(const at::Tensor &rows, int64_t nin, int64_t nout) {
  return nout <= 32 && nin % 4 == 0 && nin >= 4 && nin <= 256 && (uintptr_t)rows.data_ptr() % 16 == 0;
}

// Plain tensors that the node below is defined for; torch's own operators take everything else (subclasses, functional
// transforms, tracing, autocast, tangents, strided or misplaced operands and whatever torch has an error for).
// The weight gradient's kernel is ahead up to 16 k weights: with the whole pass on 100 k rows 64 -> 64 planes 177 us here,
// 291 on torch's products, 128 -> 128 438 and 516, 128 -> 256 924 and 699, 256 -> 512 3109 and 1804.
constexpr int64_t kMostAffineWeights = 16384;
bool rows_affine_native(PyObject *rows, PyObject *weight, PyObject *bias) {
  if (torch::jit::tracer::isTracing() || at::autocast::is_autocast_enabled(at::kCUDA)) return false;
  auto plain = [](PyObject *o) {
    if (!THPVariable_CheckTypeExact(Py_TYPE(o))) return false;
    const at::Tensor &t = THPVariable_Unpack(o);
    return t.is_cuda() && t.scalar_type() == at::kFloat && t.has_storage() && t.is_contiguous() && t.numel() > 0 && !has_tangent(t);
  };
  if (!plain(rows) || !plain(weight) || (bias != Py_None && !plain(bias))) return false;
  const at::Tensor &f = THPVariable_Unpack(rows), &w = THPVariable_Unpack(weight);
  if (f.dim() != 2 || w.dim() != 2 || f.size(1) != w.size(0) || f.device() != w.device() || w.numel() > kMostAffineWeights) return false;
  if (bias == Py_None) return true;
  const at::Tensor &b = THPVariable_Unpack(bias);
  return b.dim() == 1 && b.size(0) == w.size(1) && b.device() == f.device();
}

struct RowsAffineNode : ag::Node {
  ag::SavedVariable features_, weight_;
  bool with_bias = false;
  std::string name() const override { return "NetworkInNetworkBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    features_.reset_data();
    weight_.reset_data();
  }
  ag::variable_list apply(ag::variable_list &&grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    ag::variable_list result(3);
    if (!grads[0].defined()) return result;
    if (at::GradMode::is_enabled()) {  // the gradient is to be differentiated itself
      const at::Tensor f = features_.unpack(), w = weight_.unpack();
      if (task_should_compute_output(0)) result[0] = grads[0].mm(w.t());
      if (task_should_compute_output(1)) result[1] = f.t().mm(grads[0]);
      if (with_bias && task_should_compute_output(2)) result[2] = grads[0].sum(0);
      return result;
    }
    const at::Tensor f = features_.unpack(), w = weight_.unpack(), go = grads[0].contiguous();
    TORCH_CHECK(go.is_cuda() && go.scalar_type() == at::kFloat, "the gradient must be CUDA float32");
    const OnDevice on(f);
    const int64_t n = f.size(0), nin = w.size(0), nout = w.size(1);
    if (task_should_compute_output(0)) {
      if (rows_affine_takes(go, nout, nin)) {
        const at::Tensor wt = w.t().contiguous();
        result[0] = at::empty({n, nin}, go.options());
        check_free(scn_rows_affine_forward(ptr(go), ptr(result[0]), n, (int)nout, (int)nin, ptr(wt), nullptr, on.stream));
      } else {
        result[0] = at::mm(go, w.t());
      }
    }
    if (task_should_compute_output(1) || task_should_compute_output(2)) {
      at::Tensor dw = at::empty_like(w), db;
      if (with_bias) db = at::empty({nout}, go.options());
      check_free(scn_rows_affine_backward(ptr(f), ptr(go), n, (int)nin, (int)nout, ptr(dw), with_bias ? ptr(db) : nullptr,
                                          on.stream));
      result[1] = dw;
      result[2] = db;
    }
    return result;
  }
};

// (features, weight [nIn, nOut], bias or None) -> output, or None when the operands are not ones the call takes
SCN_FN(rows_affine_train) {
  SCN_BEGIN(3)
  if (!rows_affine_native(a[0], a[1], a[2])) Py_RETURN_NONE;
  const at::Tensor &f = THPVariable_Unpack(a[0]), &w = THPVariable_Unpack(a[1]);
  const at::Tensor bias = a[2] == Py_None ? at::Tensor() : THPVariable_Unpack(a[2]);
  at::Tensor out;
  {
    const at::NoGradGuard no_grad;
    const OnDevice on(f);
    const int64_t n = f.size(0), nin = w.size(0), nout = w.size(1);
    if (rows_affine_takes(f, nin, nout)) {
      out = at::empty({n, nout}, f.options());
      SCN_CALL(scn_rows_affine_forward(ptr(f), ptr(out), n, (int)nin, (int)nout, ptr(w), bias.defined() ? ptr(bias) : nullptr,
                                       on.stream));
    } else {
      out = bias.defined() ? at::addmm(bias, f, w) : at::mm(f, w);
    }
  }
  if (ag::compute_requires_grad(f, w, bias)) {
    std::shared_ptr<RowsAffineNode> node(new RowsAffineNode(), ag::deleteNode);
    node->set_next_edges(ag::collect_next_edges(f, w, bias));
    node->features_ = ag::SavedVariable(f, false);
    node->weight_ = ag::SavedVariable(w, false);
    node->with_bias = bias.defined();
    ag::set_history(out, node);
  }
  return THPVariable_Wrap(std::move(out));
  SCN_END
}

// (kind, metadata, md, in_size, out_size, pool, stride, features, drop) -> output
SCN_FN(pooling_train) {
  SCN_BEGIN(9)
  const int kind = (int)PyLong_AsLong(a[0]), drop = (int)PyLong_AsLong(a[8]);
  scn_metadata *md = md_of(a[2]);
  const Sizes in_size(a[3]), out_size(a[4]), pool(a[5]), stride(a[6]);
  const at::Tensor &given = tensor(a[7], "input_features");
  no_tangents(given);
  at::Tensor f, out;
  {
    const at::NoGradGuard no_grad;
    f = contiguous_features(a[7]);
    const OnDevice on(f);
    int64_t n_out = 0;
    if (kind == 2)
      n_out = n_active(md, out_size);
    else
      SCN_CALL(scn_md_strided_rulebook(md, in_size.p, out_size.p, pool.p, stride.p, on.stream, &n_out, nullptr));
    out = at::empty({n_out, f.size(1) - drop}, f.options());
    SCN_CALL((kind == 0 ? scn_max_pooling_forward : kind == 1 ? scn_average_pooling_forward : scn_unpooling_forward)(
        md, in_size.p, out_size.p, pool.p, stride.p, ptr(f), ptr(out), (int)f.size(1), drop, on.stream));
  }
  if (ag::compute_requires_grad(given)) {
    std::shared_ptr<PoolingNode> node(new PoolingNode(kind, drop, md, a[1]), ag::deleteNode);
    node->set_next_edges(ag::collect_next_edges(given));
    node->features_ = ag::SavedVariable(f, false);
    node->in_size = list(in_size), node->out_size = list(out_size), node->pool = list(pool), node->stride = list(stride);
    ag::set_history(out, node);
    node->out_ = ag::SavedVariable(out, true);
  }
  return THPVariable_Wrap(std::move(out));
  SCN_END
}

// (md, size, coords, features, batch_size, mode) -> output features: builds the site table of `coords`
// (CPU or CUDA LongTensor [n][d or d + 1]) and gathers the features of its sites
SCN_FN(input_layer) {
  SCN_BEGIN(6)
  scn_metadata *md = md_of(a[0]);
  const Sizes size(a[1]);
  const at::Tensor &f = features(a[3], "input_features");
  at::Tensor coords = tensor(a[2], "input_coords");
  if (coords.scalar_type() != at::kLong || coords.dim() != 2) fail("input_coords must be a 2-d LongTensor");
  if (coords.size(0) != f.size(0)) fail("input_coords and input_features disagree on the row count");
  const int64_t batch = PyLong_AsLongLong(a[4]);
  const int mode = (int)PyLong_AsLong(a[5]);
  if (PyErr_Occurred()) throw Fail{};
  const at::NoGradGuard no_grad;
  coords = coords.contiguous();
  if (coords.is_cuda() && coords.device() != f.device()) coords = coords.to(f.device());
  const OnDevice on(f);
  int64_t n_active = 0;
  SCN_CALL(scn_md_input_layer(md, size.p, coords.numel() ? (const int64_t *)coords.data_ptr() : nullptr, coords.is_cuda(),
                              coords.size(0), (int)coords.size(1), batch, mode, on.stream, &n_active));
  at::Tensor out = at::empty({n_active, f.size(1)}, f.options());
  SCN_CALL(scn_input_layer_forward(md, ptr(f), f.size(0), ptr(out), n_active, (int)f.size(1), on.stream));
  return THPVariable_Wrap(std::move(out));
  SCN_END
}

// (md, size, filter, stride, levels, features): the levels below `size` started on the side stream
SCN_FN(strided_chain_start) {
  SCN_BEGIN(6)
  scn_metadata *md = md_of(a[0]);
  const Sizes size(a[1]), filter(a[2]), stride(a[3]);
  const int levels = (int)PyLong_AsLong(a[4]);
  const OnDevice on(tensor(a[5], "features"));
  SCN_CALL(scn_md_strided_chain_start(md, size.p, filter.p, stride.p, levels, on.stream));
  Py_RETURN_NONE;
  SCN_END
}

// ---- small things the layers ask for on every call ----------------------------------------------------------------
// (md, size) -> active sites
SCN_FN(active_sites) {
  SCN_BEGIN(2)
  const Sizes size(a[1]);
  return PyLong_FromLongLong(n_active(md_of(a[0]), size));
  SCN_END
}

// filter and stride of as many dimensions as the size (the C entries read that many values)
void same_dimensions(const Sizes &size, const Sizes &filter, const Sizes &stride) {
  if (filter.n != size.n || stride.n != size.n)
    fail("spatial size, filter size and stride have %d, %d and %d dimensions", size.n, filter.n, stride.n);
}

// (size, filter, stride) -> LongTensor (size - filter) / stride + 1; None when the filter does not tile the size
SCN_FN(strided_size) {
  SCN_BEGIN(3)
  const Sizes size(a[0]), filter(a[1]), stride(a[2]);
  same_dimensions(size, filter, stride);
  for (int d = 0; d < size.n; ++d)
    if (stride.p[d] < 1) fail("stride %lld", (long long)stride.p[d]);  // (0 would end the process)
  at::Tensor out = at::empty({size.n}, at::kLong);
  int64_t *o = (int64_t *)out.data_ptr();
  for (int d = 0; d < size.n; ++d) {
    o[d] = (size.p[d] - filter.p[d]) / stride.p[d] + 1;
    if ((o[d] - 1) * stride.p[d] + filter.p[d] != size.p[d]) Py_RETURN_NONE;
  }
  return THPVariable_Wrap(std::move(out));
  SCN_END
}

// (size, filter, stride) -> LongTensor (size - 1) * stride + filter
SCN_FN(transposed_size) {
  SCN_BEGIN(3)
  const Sizes size(a[0]), filter(a[1]), stride(a[2]);
  same_dimensions(size, filter, stride);
  at::Tensor out = at::empty({size.n}, at::kLong);
  int64_t *o = (int64_t *)out.data_ptr();
  for (int d = 0; d < size.n; ++d) o[d] = (size.p[d] - 1) * stride.p[d] + filter.p[d];
  return THPVariable_Wrap(std::move(out));
  SCN_END
}

// (tensor or None, ...) -> bytes that change when one of them is written, replaced or moved
SCN_FN(versions) {
  try {
    std::string key;
    for (Py_ssize_t i = 0; i < n_args; ++i) {
      uint64_t v[2] = {0, 0};
      if (a[i] != Py_None) {
        const at::Tensor &t = tensor(a[i], "parameter");
        v[0] = (uint64_t)(uintptr_t)t.data_ptr();
        v[1] = (uint64_t)t._version();
      }
      key.append((const char *)v, sizeof(v));
    }
    return PyBytes_FromStringAndSize(key.data(), (Py_ssize_t)key.size());
  SCN_END
}

// (check function): how a failing status becomes an exception
SCN_FN(set_check) {
  SCN_BEGIN(1)
  Py_INCREF(a[0]);
  Py_XDECREF(g_check);
  g_check = a[0];
  Py_RETURN_NONE;
  SCN_END
}

#define SCN_METHOD(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    SCN_METHOD(submanifold_convolution), SCN_METHOD(submanifold_joined), SCN_METHOD(convolution), SCN_METHOD(deconvolution),
    SCN_METHOD(convolution_backward),    SCN_METHOD(batchnorm_forward),  SCN_METHOD(batchnorm_backward),
    SCN_METHOD(pooling_forward),         SCN_METHOD(pooling_backward),   SCN_METHOD(sparse_to_dense),
    SCN_METHOD(active_sites),            SCN_METHOD(strided_size),       SCN_METHOD(transposed_size),
    SCN_METHOD(convolution_train),       SCN_METHOD(batchnorm_train),    SCN_METHOD(pooling_train),
    SCN_METHOD(strided_chain_start),     SCN_METHOD(rows_affine_train),       SCN_METHOD(input_layer),             SCN_METHOD(versions),           SCN_METHOD(set_check),                    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding(void) { return PyModule_Create(&module); }
