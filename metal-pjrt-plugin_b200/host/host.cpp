// The Python front's per-call work in native code: tensor checks, the output's allocation and the C ABI's parameter
// structs.  The calls themselves are those of include/b200graft.h, reached through the addresses of the library that
// _lib.py has loaded; nothing is computed here.
//
// Why: a product of a few rows takes 3-8 us on the GPU, and filling the structs through ctypes took 12-17 us of host
// time per call (4096 x 6144 int4, one row: 16.8 us a call), so the host was the bound of every small call.
//
// Every function takes its arguments by position (the Python wrappers own names and defaults), releases the GIL around
// the library call as ctypes does, and reports a failing status through _lib.check, which raises B200Error.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "b200graft.h"

namespace {

struct Api {
  decltype(&b200_qmm_run) qmm_run;
  decltype(&b200_gemm) gemm;
  decltype(&b200_gemm_force_route) gemm_force_route;
  decltype(&b200_rownorm) rownorm;
  decltype(&b200_sample) sample;
  decltype(&b200_decoder_step) decoder_step;
} api;

PyObject* check_fn;             // _lib.check(status)
PyObject* default_context_fn;   // context.default_context(device) -> Context
constexpr int kDevices = 64;
b200_context* default_ctx[kDevices];

PyObject *s_q4, *s_q4h, *s_q, *s_s, *s_b, *s_handle, *s_value, *s_m, *s_n, *s_k, *s_a, *s_c, *s_batch_count, *s_alpha, *s_beta, *s_tensor,
    *s_ld, *s_batch_stride, *s_transpose, *s_act, *s_bias, *s_aux;

struct Raised {};   // a Python exception is set

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "expected a torch tensor, got %s", Py_TYPE(o)->tp_name);
    throw Raised();
  }
  return THPVariable_Unpack(o);
}
const at::Tensor* tensor_or_none(PyObject* o) { return o == Py_None ? nullptr : &tensor(o); }
void* data(const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }
int64_t as_int(PyObject* o) {
  const long long v = PyLong_Check(o) ? PyLong_AsLongLong(o) : [&] {
    PyObject* i = PyNumber_Index(o);
    if (i == nullptr) return -1ll;
    const long long r = PyLong_AsLongLong(i);
    Py_DECREF(i);
    return r;
  }();
  if (v == -1 && PyErr_Occurred()) throw Raised();
  return v;
}
double as_double(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Raised();
  return v;
}
bool as_bool(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw Raised();
  return v != 0;
}
// An owned reference to an attribute.
struct Attr {
  PyObject* o;
  Attr(PyObject* from, PyObject* name) : o(PyObject_GetAttr(from, name)) {
    if (o == nullptr) throw Raised();
  }
  ~Attr() { Py_DECREF(o); }
  Attr(const Attr&) = delete;
};

// A ctypes.c_void_p's (or int's) address; None is null.
void* address(PyObject* o) {
  if (o == Py_None) return nullptr;
  if (PyLong_Check(o)) return PyLong_AsVoidPtr(o);
  Attr v(o, s_value);
  return v.o == Py_None ? nullptr : PyLong_AsVoidPtr(v.o);
}
b200_context* context(PyObject* ctx, const at::Tensor& like) {
  if (ctx != Py_None) {
    Attr h(ctx, s_handle);
    return static_cast<b200_context*>(address(h.o));
  }
  const int dev = like.is_cuda() ? like.device().index() : 0;
  if (dev >= 0 && dev < kDevices && default_ctx[dev] != nullptr) return default_ctx[dev];
  PyObject* c = PyObject_CallFunction(default_context_fn, "i", dev);
  if (c == nullptr) throw Raised();
  b200_context* p = nullptr;
  try {
    Attr h(c, s_handle);
    p = static_cast<b200_context*>(address(h.o));
  } catch (const Raised&) {
    Py_DECREF(c);
    throw;
  }
  Py_DECREF(c);
  if (dev >= 0 && dev < kDevices) default_ctx[dev] = p;
  return p;
}
b200_stream stream_of(PyObject* stream) {
  if (stream != Py_None && as_bool(stream)) return static_cast<b200_stream>(address(stream));
  return reinterpret_cast<b200_stream>(c10::cuda::getCurrentCUDAStream().stream());
}
void check(b200_status s) {
  if (s == B200_OK) return;
  PyObject* r = PyObject_CallFunction(check_fn, "i", static_cast<int>(s));
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "b200: a call failed");
  throw Raised();
}
int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return B200_F32;
    case at::kHalf: return B200_F16;
    case at::kBFloat16: return B200_BF16;
    default: break;
  }
  PyErr_Format(PyExc_KeyError, "%s", c10::toString(t.scalar_type()));
  throw Raised();
}
at::Tensor empty(at::IntArrayRef size, at::ScalarType dtype, const at::Tensor& like) {
  return at::detail::empty_cuda(size, dtype, like.device(), std::nullopt);
}
PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
template <typename F>
void without_gil(F&& f) {
  b200_status s;
  Py_BEGIN_ALLOW_THREADS
  s = f();
  Py_END_ALLOW_THREADS
  check(s);
}
PyObject* item(PyObject* dict, PyObject* key) {
  PyObject* v = PyDict_GetItemWithError(dict, key);
  if (v == nullptr) {
    if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, key);
    throw Raised();
  }
  return v;
}

#define B200_TRY HANDLE_TH_ERRORS try {
#define B200_END                      \
  }                                   \
  catch (const Raised&) {             \
    return nullptr;                   \
  }                                   \
  END_HANDLE_TH_ERRORS
#define B200_ARGS(name, want)                                                           \
  if (n != (want)) {                                                                    \
    PyErr_Format(PyExc_TypeError, name " takes %d arguments, got %zd", want, n);        \
    return nullptr;                                                                     \
  }

// linear(x, w, residual, out_f32, rms_gain, eps, silu_mul, silu_pair, ctx, stream)
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  B200_ARGS("linear", 10)
  B200_TRY
  const at::Tensor& x = tensor(a[0]);
  b200_context* ctx = context(a[8], x);
  b200_qmm_params p = {};
  const at::Tensor *q, *s = nullptr, *b = nullptr;
  // the sizes below are read off the packed weights, so their rank is part of the format
  auto packed = [&](PyObject* o, int64_t dims) {
    const at::Tensor& t = tensor(o);
    if (t.dim() != dims) {
      PyErr_Format(PyExc_ValueError, "packed weights of this format have %lld dimensions, got %lld", static_cast<long long>(dims),
                   static_cast<long long>(t.dim()));
      throw Raised();
    }
    return &t;
  };
  if (PyDict_Check(a[1])) {
    PyObject* o;
    if ((o = PyDict_GetItemWithError(a[1], s_q4)) != nullptr) {
      q = packed(o, 2);
      p.bits = 4, p.group = 64, p.N = q->size(0), p.K = q->size(1) * 8;
    } else if ((o = PyDict_GetItemWithError(a[1], s_q4h)) != nullptr) {
      q = packed(o, 3);
      p.bits = 4, p.group = 64, p.nibble_order = 1, p.N = q->size(0), p.K = q->size(1) * 64;
    } else {
      q = packed(item(a[1], s_q), 2);
      p.bits = 8, p.N = q->size(0), p.K = q->size(1);
    }
    s = &tensor(item(a[1], s_s));
    if (p.bits == 4) {
      b = &tensor(item(a[1], s_b));
    } else {
      if (s->size(1) == 0) {
        PyErr_SetString(PyExc_ZeroDivisionError, "an int8 weight without scales");
        throw Raised();
      }
      p.group = static_cast<int32_t>(p.K / s->size(1));
    }
  } else {
    q = packed(a[1], 2);
    p.bits = 16, p.N = q->size(0), p.K = q->size(1);
  }
  const at::Tensor* residual = tensor_or_none(a[2]);
  const at::Tensor* gain = tensor_or_none(a[4]);
  const bool out_f32 = as_bool(a[3]), silu_mul = as_bool(a[6]), silu_pair = as_bool(a[7]);
  const int64_t width = silu_mul ? 2 * p.K : p.K, n_out = silu_pair ? p.N / 2 : p.N;
  if (x.numel() != 0 && (x.dim() == 0 || x.size(-1) != width)) {   // (the result has x's leading dimensions)
    PyErr_Format(PyExc_RuntimeError, "linear: the rows of x must have %lld elements", static_cast<long long>(width));
    throw Raised();
  }
  at::Tensor flat;
  const at::Tensor* x2 = &x;
  if (x.dim() != 2 || x.size(1) != width) flat = x.reshape({-1, width}), x2 = &flat;
  p.M = x2->size(0);
  at::Tensor out = empty({p.M, n_out}, out_f32 ? at::kFloat : at::kBFloat16, x);
  p.epilogue = silu_pair ? B200_QMM_OUT_SILU_PAIR
                         : (out_f32 ? B200_QMM_OUT_F32 : (residual != nullptr ? B200_QMM_ADD_RESIDUAL : B200_QMM_OUT_BF16));
  p.x = x2->data_ptr();
  p.q = q->data_ptr();
  p.scale = data(s);
  p.bias = data(b);
  p.residual = data(residual);
  p.out = out.data_ptr();
  p.ldx = p.M > 0 ? x2->stride(0) : 0;
  p.ldo = n_out;
  if (gain != nullptr) {
    p.prologue = B200_QMM_PRO_RMSNORM;
    p.eps = static_cast<float>(as_double(a[5]));
    p.prologue_gain = gain->data_ptr();
  } else if (silu_mul) {
    p.prologue = B200_QMM_PRO_SILU_MUL;
  }
  b200_stream st = stream_of(a[9]);
  without_gil([&] { return api.qmm_run(ctx, st, &p); });
  if (x.dim() == 2) return wrap(out);
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end() - 1);
  shape.push_back(n_out);
  return wrap(out.reshape(shape));
  B200_END
}

b200_operand operand(PyObject* o, const at::Tensor** t) {
  b200_operand r = {};
  Attr tn(o, s_tensor), ld(o, s_ld), bs(o, s_batch_stride), tr(o, s_transpose);
  *t = &tensor(tn.o);   // the operand keeps it alive
  r.ptr = (*t)->data_ptr();
  r.ld = as_int(ld.o);
  r.batch_stride = as_int(bs.o);
  r.dtype = dtype_code(**t);
  r.transpose = as_bool(tr.o);
  return r;
}
void run_gemm(b200_context* ctx, b200_stream st, const b200_gemm_params& p, const b200_epilogue& e, int route) {
  b200_status s;
  Py_BEGIN_ALLOW_THREADS
  api.gemm_force_route(ctx, route);
  s = api.gemm(ctx, st, &p, &e);
  api.gemm_force_route(ctx, 0);
  Py_END_ALLOW_THREADS
  check(s);
}

// run_steel_gemm(params, epilogue or None, ctx, stream, route)
PyObject* run_steel_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  B200_ARGS("run_steel_gemm", 5)
  B200_TRY
  b200_gemm_params p = {};
  b200_epilogue e = {};
  const at::Tensor *ta, *tb, *tc;
  {
    Attr m(a[0], s_m), nn(a[0], s_n), k(a[0], s_k), batch(a[0], s_batch_count), alpha(a[0], s_alpha), beta(a[0], s_beta);
    p.m = as_int(m.o), p.n = as_int(nn.o), p.k = as_int(k.o), p.batch = as_int(batch.o);
    p.alpha = as_double(alpha.o), p.beta = as_double(beta.o);
    Attr oa(a[0], s_a), ob(a[0], s_b), oc(a[0], s_c);
    p.a = operand(oa.o, &ta), p.b = operand(ob.o, &tb), p.c = operand(oc.o, &tc);
  }
  if (a[1] != Py_None) {
    Attr act(a[1], s_act), bias(a[1], s_bias), aux(a[1], s_aux);
    e.act = static_cast<int32_t>(as_int(act.o));
    e.bias = data(tensor_or_none(bias.o));
    e.aux = data(tensor_or_none(aux.o));
  }
  b200_context* ctx = context(a[2], *tc);
  run_gemm(ctx, stream_of(a[3]), p, e, static_cast<int>(as_int(a[4])));
  Py_RETURN_NONE;
  B200_END
}

// matmul(a, b, bias, act, out_dtype code or -1, transpose_b, ctx)
PyObject* matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  B200_ARGS("matmul", 7)
  B200_TRY
  const at::Tensor &A = tensor(a[0]), &B = tensor(a[1]);
  const at::Tensor* bias = tensor_or_none(a[2]);
  b200_context* ctx = context(a[6], A);
  const bool tb = as_bool(a[5]);
  if (A.dim() != 2) {
    PyErr_SetString(PyExc_ValueError, "matmul takes row-major 2-D tensors");
    throw Raised();
  }
  static const at::ScalarType types[3] = {at::kFloat, at::kHalf, at::kBFloat16};
  const int64_t code = as_int(a[4]);
  b200_gemm_params p = {};
  p.m = A.size(0), p.k = A.size(1), p.n = B.size(tb ? 0 : 1), p.batch = 1, p.alpha = 1.0;
  at::Tensor D = empty({p.m, p.n}, code >= 0 && code < 3 ? types[code] : A.scalar_type(), A);
  p.a = {A.data_ptr(), A.stride(0), 0, dtype_code(A), 0};
  p.b = {B.data_ptr(), B.stride(0), 0, dtype_code(B), tb};
  p.c = {D.data_ptr(), D.stride(0), 0, dtype_code(D), 0};
  b200_epilogue e = {static_cast<int32_t>(as_int(a[3])), data(bias), nullptr};
  run_gemm(ctx, stream_of(Py_None), p, e, 0);
  return wrap(D);
  B200_END
}

// rownorm(kind, x, gain, beta, eps, out, ctx, stream)
PyObject* rownorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  B200_ARGS("rownorm", 8)
  B200_TRY
  const at::Tensor& x = tensor(a[1]);
  b200_context* ctx = context(a[6], x);
  if (!x.is_contiguous()) {
    PyErr_SetString(PyExc_AssertionError, "rownorm takes a contiguous tensor");
    throw Raised();
  }
  const int64_t len = x.dim() > 0 ? x.size(-1) : 0, rows = len > 0 ? x.numel() / len : 0;
  const int dt = dtype_code(x);
  at::Tensor fresh;
  if (a[5] == Py_None) fresh = empty(x.sizes(), x.scalar_type(), x);
  void* y = a[5] == Py_None ? fresh.data_ptr() : tensor(a[5]).data_ptr();
  const void *gain = data(tensor_or_none(a[2])), *beta = data(tensor_or_none(a[3]));
  const double eps = as_double(a[4]);
  const int kind = static_cast<int>(as_int(a[0]));
  b200_stream st = stream_of(a[7]);
  without_gil([&] { return api.rownorm(ctx, st, kind, x.data_ptr(), gain, beta, y, rows, len, dt, eps); });
  if (a[5] == Py_None) return wrap(fresh);
  Py_INCREF(a[5]);
  return a[5];
  B200_END
}

// sample(logits, uniform, temperature, top_k, top_p, ctx, stream)
PyObject* sample(PyObject*, PyObject* const* a, Py_ssize_t n) {
  B200_ARGS("sample", 7)
  B200_TRY
  const at::Tensor& given = tensor(a[0]);
  b200_context* ctx = context(a[5], given);
  if (given.dim() != 2) {
    PyErr_SetString(PyExc_ValueError, "sample takes logits [batch, vocab]");
    throw Raised();
  }
  const at::Tensor logits = given.contiguous();
  const at::Tensor* uniform = tensor_or_none(a[1]);
  const int64_t B = logits.size(0), V = logits.size(1);
  at::Tensor out = empty({B}, at::kInt, logits);
  const float temperature = static_cast<float>(as_double(a[2])), top_p = static_cast<float>(as_double(a[4]));
  const int32_t top_k = static_cast<int32_t>(as_int(a[3]));
  b200_stream st = stream_of(a[6]);
  without_gil([&] {
    return api.sample(ctx, st, static_cast<const float*>(logits.data_ptr()), B, V, temperature, top_k, top_p,
                      static_cast<const float*>(data(uniform)), static_cast<int32_t*>(out.data_ptr()));
  });
  return wrap(out);
  B200_END
}

// decoder_step(decoder handle, tokens, pos, logits, stream)
PyObject* decoder_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  B200_ARGS("decoder_step", 5)
  B200_TRY
  b200_decoder* dec = static_cast<b200_decoder*>(address(a[0]));
  const at::Tensor &tokens = tensor(a[1]), &pos = tensor(a[2]), &logits = tensor(a[3]);
  const int batch = static_cast<int>(tokens.size(0));
  b200_stream st = stream_of(a[4]);
  without_gil([&] {
    return api.decoder_step(dec, st, static_cast<const int32_t*>(tokens.data_ptr()), static_cast<const int32_t*>(pos.data_ptr()),
                            static_cast<float*>(logits.data_ptr()), batch);
  });
  Py_RETURN_NONE;
  B200_END
}

// bind(addresses of the library's functions in Api's order, check, default_context)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  B200_ARGS("bind", 3)
  void** slot = reinterpret_cast<void**>(&api);
  if (!PyTuple_Check(a[0]) || PyTuple_GET_SIZE(a[0]) != static_cast<Py_ssize_t>(sizeof(Api) / sizeof(void*))) {
    PyErr_SetString(PyExc_TypeError, "bind: one address per function");
    return nullptr;
  }
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(a[0]); ++i) slot[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(a[0], i));
  if (PyErr_Occurred()) return nullptr;
  Py_INCREF(a[1]);
  Py_INCREF(a[2]);
  check_fn = a[1];
  default_context_fn = a[2];
  Py_RETURN_NONE;
}

// forget(context address): a context that is being closed is no longer anyone's default
PyObject* forget(PyObject*, PyObject* const* a, Py_ssize_t n) {
  B200_ARGS("forget", 1)
  const void* p = PyLong_AsVoidPtr(a[0]);
  for (b200_context*& c : default_ctx)
    if (c == p) c = nullptr;
  Py_RETURN_NONE;
}

#define B200_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {B200_METHOD(linear), B200_METHOD(run_steel_gemm), B200_METHOD(matmul), B200_METHOD(rownorm), B200_METHOD(sample),
                         B200_METHOD(decoder_step), B200_METHOD(bind), B200_METHOD(forget), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  struct {
    PyObject** to;
    const char* name;
  } names[] = {{&s_q4, "q4"}, {&s_q4h, "q4h"}, {&s_q, "q"}, {&s_s, "s"}, {&s_b, "b"}, {&s_handle, "handle"}, {&s_value, "value"},
               {&s_m, "m"}, {&s_n, "n"}, {&s_k, "k"}, {&s_a, "a"}, {&s_c, "c"}, {&s_batch_count, "batch_count"}, {&s_alpha, "alpha"},
               {&s_beta, "beta"}, {&s_tensor, "tensor"}, {&s_ld, "ld"}, {&s_batch_stride, "batch_stride"}, {&s_transpose, "transpose"},
               {&s_act, "act"}, {&s_bias, "bias"}, {&s_aux, "aux"}};
  for (auto& x : names)
    if ((*x.to = PyUnicode_InternFromString(x.name)) == nullptr) return nullptr;
  return PyModule_Create(&module);
}
