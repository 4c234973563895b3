// Native host path of the public calls: argument checks, output allocation and the C-ABI call of one op in one
// CPython extension function.
//
// What it is for: a decode step or a short prompt runs 2-10 us on the GPU, and the same checks written in Python with
// ctypes cost 20-25 us per call (a layer's token step of six calls: 135 us, all of it host time).  Each function here
// takes the arguments of one public op and handles the plain case -- CUDA tensors on the current device, storage types
// and layouts the kernels read as they are, no gradient wanted.  Anything else (casts, copies, wrong shapes, other
// devices) returns None, and the caller in Python goes the long way, which also raises the errors.  A negative DrStatus
// comes back as an int for the caller to raise.
//
// Functions are METH_FASTCALL on positional arguments: no keyword parsing, no per-argument type casters.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <exception>
#include <vector>

#include "deltarule_sm100.h"

namespace {

constexpr int kMaxDevices = 64;
constexpr int64_t kPackedScratch = (int64_t)1 << 30;   // varlen.PACKED_SCRATCH
int32_t* g_status[kMaxDevices] = {nullptr};   // device status words, registered by the Python side

struct Api {
  decltype(&dr_workspace_bytes) workspace_bytes;
  decltype(&dr_chunk_fwd) chunk_fwd;
  decltype(&dr_recurrent_fwd) recurrent_fwd;
  decltype(&dr_step) step;
  decltype(&dr_chunk_fwd_varlen) chunk_fwd_varlen;
  decltype(&dr_short_conv_silu) short_conv_silu;
  decltype(&dr_gate_activations) gate_activations;
  decltype(&dr_gated_rmsnorm) gated_rmsnorm;
  decltype(&dr_dplr_recurrent) dplr_recurrent;
  decltype(&dr_rwkv6_recurrent) rwkv6_recurrent;
  decltype(&dr_ssd_scan) ssd_scan;
  decltype(&dr_chunk_fwd_saving) chunk_fwd_saving;
  decltype(&dr_chunk_bwd_saved) chunk_bwd_saved;
} api;
bool g_open = false;

// Thrown (by value, never past a function below) when a call is not the plain case.
struct NotPlain {};
inline void need(bool ok) { if (!ok) throw NotPlain(); }

inline int dtype_code(const at::Tensor& t) {
  const auto s = t.scalar_type();
  if (s == at::kFloat) return DR_F32;
  if (s == at::kBFloat16) return DR_BF16;
  throw NotPlain();
}
inline at::ScalarType scalar_type(int code) { return code == DR_BF16 ? at::kBFloat16 : at::kFloat; }

// The arguments of one call.  Every tensor is a plain strided CUDA tensor of the current device.
struct Call {
  int dev = -1;
  bool grad = false;
  const at::Tensor* opt(PyObject* o) {
    if (o == Py_None) return nullptr;
    need(THPVariable_CheckExact(o));
    const at::Tensor& t = THPVariable_Unpack(o);
    need(t.is_cuda() && t.layout() == at::kStrided && !t.is_neg());
    if (dev < 0) {
      dev = t.device().index();
      need(dev < kMaxDevices && dev == c10::cuda::current_device() && g_status[dev]);
    } else {
      need(t.device().index() == dev);
    }
    grad |= t.requires_grad();
    return &t;
  }
  const at::Tensor& req(PyObject* o) {
    const at::Tensor* t = opt(o);
    need(t != nullptr);
    return *t;
  }
  void no_grad() const { need(!(grad && c10::GradMode::is_enabled())); }
  void* stream() const { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(); }
  int32_t* status() const { return g_status[dev]; }
  at::Tensor empty(at::IntArrayRef size, at::ScalarType st) const {
    return at::Tensor(at::detail::empty_cuda(size, st, c10::Device(c10::DeviceType::CUDA, (c10::DeviceIndex)dev), std::nullopt));
  }
  at::Tensor empty_strided(at::IntArrayRef size, at::IntArrayRef stride, at::ScalarType st) const {
    return at::Tensor(at::detail::empty_strided_cuda(
        size, stride, at::TensorOptions().dtype(st).device(c10::Device(c10::DeviceType::CUDA, (c10::DeviceIndex)dev))));
  }
};

inline const void* ptr(const at::Tensor* t) { return t ? t->const_data_ptr() : nullptr; }
inline const float* fptr(const at::Tensor* t) { return static_cast<const float*>(ptr(t)); }
inline const void* ptr(const at::Tensor& t) { return t.const_data_ptr(); }
inline float* fmut(const at::Tensor& t) { return static_cast<float*>(t.mutable_data_ptr()); }
inline bool is_shape(const at::Tensor& t, std::initializer_list<int64_t> s) {
  return t.sizes().equals(at::IntArrayRef(s.begin(), s.size()));
}
inline void need_f32(const at::Tensor* t) { if (t) need(t->scalar_type() == at::kFloat && t->is_contiguous()); }
inline long as_int(PyObject* o) { return PyLong_AsLong(o); }
inline double as_double(PyObject* o) { return PyFloat_AsDouble(o); }

// [B,H,T,...] given as a view of contiguous token-major storage [B,T,H,...]
bool is_bthd_view(const at::Tensor& t) {
  if (t.dim() < 3) return false;
  int64_t inner = 1;
  for (int64_t d = t.dim() - 1; d >= 3; --d) {
    if (t.size(d) != 1 && t.stride(d) != inner) return false;
    inner *= t.size(d);
  }
  const int64_t B = t.size(0), H = t.size(1), T = t.size(2);
  return (H == 1 || t.stride(1) == inner) && (T == 1 || t.stride(2) == inner * H) && (B == 1 || t.stride(0) == inner * H * T);
}

// Storage of the sequence tensors: all [B,H,T,..] contiguous, or all token-major views; anything else is not plain.
int common_layout(std::initializer_list<const at::Tensor*> ts) {
  bool contiguous = true, bthd = true;
  for (const at::Tensor* t : ts) {
    if (!t) continue;
    const bool c = t->is_contiguous();
    contiguous &= c;
    bthd &= !c && is_bthd_view(*t);
  }
  need(contiguous || bthd);
  return contiguous ? DR_LAYOUT_BHTD : DR_LAYOUT_BTHD;
}

at::Tensor sequence_out(const Call& c, int layout, int64_t B, int64_t H, int64_t T, int64_t D, at::ScalarType st) {
  if (layout == DR_LAYOUT_BHTD) return c.empty({B, H, T, D}, st);
  const std::array<int64_t, 4> size = {B, H, T, D}, stride = {T * H * D, D, H * D, 1};
  return c.empty_strided(size, stride, st);
}

PyObject* pair(const at::Tensor& a, PyObject* b_owned) {
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(a));
  PyTuple_SET_ITEM(r, 1, b_owned);
  return r;
}
PyObject* pair(const at::Tensor& a, const at::Tensor& b) { return pair(a, THPVariable_Wrap(b)); }

// q, k, v of one call: same storage type
int qkv_dtype(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
  const int dt = dtype_code(q);
  need(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type());
  return dt;
}

DrDesc make_desc(int variant, int layout, int64_t B, int64_t H, int64_t T, int64_t K, int64_t V, int64_t chunk, int qkv,
                 int g_dt, int out, bool l2norm, double scale, int path, int64_t Hq) {
  DrDesc d{};
  d.variant = variant; d.layout = layout;
  d.B = (int32_t)B; d.H = (int32_t)H; d.T = (int32_t)T; d.K = (int32_t)K; d.V = (int32_t)V; d.chunk = (int32_t)chunk;
  d.qkv_dtype = qkv; d.g_dtype = g_dt; d.out_dtype = out; d.use_qk_l2norm = l2norm; d.scale = (float)scale;
  d.path = path; d.qk_heads = (int32_t)Hq;
  return d;
}

// Runs `f` (which returns a new reference) and turns "not the plain case" into None, C++ errors into the Python exceptions that
// torch's own functions raise for them (an allocation that does not fit: torch.OutOfMemoryError, which callers catch).
template <class F>
PyObject* guarded(F f) {
  try {
    need(g_open);
    PyObject* r = f();
    return PyErr_Occurred() ? (Py_XDECREF(r), nullptr) : r;
  } catch (const NotPlain&) {
    if (PyErr_Occurred()) PyErr_Clear();   // an argument of another type: the Python path reports it
    Py_RETURN_NONE;
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

struct Unlocked {   // the launch may block on a full queue: other Python threads run meanwhile
  PyThreadState* s = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(s); }
};

// step(variant, q, k, v, g, beta, state, scale, l2norm, inplace) -> (o, state) | status | None
PyObject* py_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 10);
    Call c;
    const int variant = (int)as_int(a[0]);
    const at::Tensor &q = c.req(a[1]), &k = c.req(a[2]), &v = c.req(a[3]);
    const at::Tensor* g = c.opt(a[4]);
    const at::Tensor &beta = c.req(a[5]), &S = c.req(a[6]);
    const bool inplace = a[9] == Py_True;
    need(q.dim() == 3 && v.dim() == 3 && k.sizes().equals(q.sizes()) && v.size(0) == q.size(0));
    const int64_t B = q.size(0), Hq = q.size(1), K = q.size(2), H = v.size(1), V = v.size(2);
    need(Hq > 0 && H % Hq == 0 && is_shape(S, {B, H, K, V}) && is_shape(beta, {B, H}));
    const int dt = qkv_dtype(q, k, v);
    need(q.is_contiguous() && k.is_contiguous() && v.is_contiguous());
    need_f32(&beta);
    need_f32(&S);
    need((g != nullptr) == (variant != DR_DELTA));
    int g_dt = DR_F32;
    if (g) {
      need(g->is_contiguous() && (variant == DR_GATED ? is_shape(*g, {B, H}) : is_shape(*g, {B, H, K})));
      g_dt = dtype_code(*g);
    }
    const double scale = a[7] == Py_None ? 1.0 / std::sqrt((double)K) : as_double(a[7]);
    need(!PyErr_Occurred());
    const int out = variant == DR_KDA ? DR_F32 : dt;   // KDA answers in the state's type
    const at::Tensor o = c.empty({B, H, V}, scalar_type(out));
    const at::Tensor s_out = inplace ? S : c.empty({B, H, K, V}, at::kFloat);
    const DrDesc d = make_desc(variant, DR_LAYOUT_BHTD, B, H, 1, K, V, 0, dt, g_dt, out, a[8] == Py_True, scale, 0, Hq);
    void* stream = c.stream();
    int st;
    {
      Unlocked u;
      st = api.step(&d, ptr(q), ptr(k), ptr(v), ptr(g), fptr(&beta), fptr(&S), fmut(s_out), o.mutable_data_ptr(), c.status(), stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    if (inplace) { Py_INCREF(a[6]); return pair(o, a[6]); }
    return pair(o, s_out);
  });
}

// sequence(recurrent, variant, q, k, v, g, beta, h0, scale, chunk, l2norm, out_dtype, path) -> (o, hT) | status | None
PyObject* py_sequence(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 13);
    Call c;
    const bool recurrent = a[0] == Py_True;
    const int variant = (int)as_int(a[1]);
    const at::Tensor &q = c.req(a[2]), &k = c.req(a[3]), &v = c.req(a[4]);
    const at::Tensor* g = c.opt(a[5]);
    const at::Tensor& beta = c.req(a[6]);
    const at::Tensor* h0 = c.opt(a[7]);
    need(q.dim() == 4 && v.dim() == 4 && k.sizes().equals(q.sizes()));
    const int64_t B = q.size(0), Hq = q.size(1), T = q.size(2), K = q.size(3), H = v.size(1), V = v.size(3);
    need(v.size(0) == B && v.size(2) == T && Hq > 0 && H % Hq == 0 && is_shape(beta, {B, H, T}) && beta.scalar_type() == at::kFloat);
    const int dt = qkv_dtype(q, k, v);
    need((g != nullptr) == (variant != DR_DELTA));
    int g_dt = DR_F32;
    if (g) {
      need(variant == DR_GATED ? is_shape(*g, {B, H, T}) : is_shape(*g, {B, H, T, K}));
      g_dt = dtype_code(*g);
    }
    const int layout = common_layout({&q, &k, &v, g, &beta});
    need(layout == DR_LAYOUT_BHTD || (Hq > 1 && T > 1));
    if (h0) { need(is_shape(*h0, {B, H, K, V})); need_f32(h0); }
    const long out = as_int(a[11]), path = as_int(a[12]);
    need(out >= 0 && out <= DR_BF16 && path >= 0);
    const double scale = a[8] == Py_None ? 1.0 / std::sqrt((double)K) : as_double(a[8]);
    const DrDesc d = make_desc(variant, layout, B, H, T, K, V, as_int(a[9]), dt, g_dt, (int)out, a[10] == Py_True, scale, (int)path, Hq);
    need(!PyErr_Occurred());
    const at::Tensor o = sequence_out(c, layout, B, H, T, V, scalar_type((int)out));
    const at::Tensor hT = c.empty({B, H, K, V}, at::kFloat);
    void* stream = c.stream();
    int st;
    if (recurrent) {
      Unlocked u;
      st = api.recurrent_fwd(&d, ptr(q), ptr(k), ptr(v), ptr(g), fptr(&beta), fptr(h0), o.mutable_data_ptr(), fmut(hT), c.status(), stream);
    } else {
      const int64_t ws_bytes = api.workspace_bytes(&d, 2);
      if (ws_bytes < 0) return PyLong_FromLong((long)ws_bytes);
      at::Tensor ws;
      if (ws_bytes > 0) ws = c.empty({ws_bytes}, at::kByte);
      Unlocked u;
      st = api.chunk_fwd(&d, ptr(q), ptr(k), ptr(v), ptr(g), fptr(&beta), fptr(h0), o.mutable_data_ptr(), fmut(hT),
                         ws_bytes > 0 ? ws.mutable_data_ptr() : nullptr, (size_t)ws_bytes, c.status(), stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    return pair(o, hT);
  });
}

// What the two halves of a training step share: the inputs and their descriptor.
struct Training {
  Call c;
  const at::Tensor *q, *k, *v, *g, *beta;
  int64_t B, Hq, T, K, H, V;
  int dt, layout;
  DrDesc d;
  // a: variant, q, k, v, g, beta; out < 0: the inputs' storage type
  Training(PyObject* const* a, PyObject* scale_arg, PyObject* chunk, PyObject* l2norm, int out) {
    const int variant = (int)as_int(a[0]);
    q = &c.req(a[1]); k = &c.req(a[2]); v = &c.req(a[3]); g = c.opt(a[4]); beta = &c.req(a[5]);
    need(q->dim() == 4 && v->dim() == 4 && k->sizes().equals(q->sizes()));
    B = q->size(0); Hq = q->size(1); T = q->size(2); K = q->size(3); H = v->size(1); V = v->size(3);
    need(v->size(0) == B && v->size(2) == T && Hq > 0 && H % Hq == 0 && is_shape(*beta, {B, H, T}) && beta->scalar_type() == at::kFloat);
    dt = qkv_dtype(*q, *k, *v);
    need((g != nullptr) == (variant != DR_DELTA));
    int g_dt = DR_F32;
    if (g) {
      need(variant == DR_GATED ? is_shape(*g, {B, H, T}) : is_shape(*g, {B, H, T, K}));
      g_dt = dtype_code(*g);
    }
    layout = common_layout({q, k, v, g, beta});
    need(layout == DR_LAYOUT_BHTD || (Hq > 1 && T > 1));
    const double scale = scale_arg == Py_None ? 1.0 / std::sqrt((double)K) : as_double(scale_arg);
    d = make_desc(variant, layout, B, H, T, K, V, as_int(chunk), dt, g_dt, out < 0 ? dt : out, l2norm == Py_True, scale, 0, Hq);
    need(!PyErr_Occurred());
  }
  bool laid_out(const at::Tensor& t) const { return layout == DR_LAYOUT_BHTD ? t.is_contiguous() : is_bthd_view(t); }
  at::Tensor like(const at::Tensor& t, at::ScalarType st) const { return c.empty_strided(t.sizes(), t.strides(), st); }
};

// train_fwd(variant, q, k, v, g, beta, h0, scale, chunk, l2norm, out_dtype) -> (o, hT, workspace) | status | None
PyObject* py_train_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 11);
    const long out = as_int(a[10]);
    need(out >= 0 && out <= DR_BF16);
    Training t(a, a[7], a[8], a[9], (int)out);
    const at::Tensor* h0 = t.c.opt(a[6]);
    if (h0) { need(is_shape(*h0, {t.B, t.H, t.K, t.V})); need_f32(h0); }
    const int64_t ws_bytes = api.workspace_bytes(&t.d, 1);
    if (ws_bytes < 0) return PyLong_FromLong((long)ws_bytes);
    const at::Tensor ws = t.c.empty({ws_bytes}, at::kByte);
    const at::Tensor o = sequence_out(t.c, t.layout, t.B, t.H, t.T, t.V, scalar_type((int)out));
    const at::Tensor hT = t.c.empty({t.B, t.H, t.K, t.V}, at::kFloat);
    void* stream = t.c.stream();
    int st;
    {
      Unlocked u;
      st = api.chunk_fwd_saving(&t.d, ptr(*t.q), ptr(*t.k), ptr(*t.v), ptr(t.g), fptr(t.beta), fptr(h0), o.mutable_data_ptr(), fmut(hT),
                                ws.mutable_data_ptr(), (size_t)ws_bytes, t.c.status(), stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    PyObject* r = PyTuple_New(3);
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(o));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(hT));
    PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(ws));
    return r;
  });
}

// train_bwd(variant, q, k, v, g, beta, d_o, d_hT, scale, chunk, l2norm, workspace, want_dh0) -> (dq, dk, dv, dg, dbeta, dh0 | None) | status | None
PyObject* py_train_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 13);
    Training t(a, a[8], a[9], a[10], -1);
    const bool want_dh0 = a[12] == Py_True;
    const at::Tensor &given = t.c.req(a[6]), &ws = t.c.req(a[11]);
    const at::Tensor* d_hT = t.c.opt(a[7]);
    need(is_shape(given, {t.B, t.H, t.T, t.V}) && t.laid_out(given));
    if (d_hT) { need(is_shape(*d_hT, {t.B, t.H, t.K, t.V})); need_f32(d_hT); }
    const int64_t ws_bytes = api.workspace_bytes(&t.d, 1);
    if (ws_bytes < 0) return PyLong_FromLong((long)ws_bytes);
    need(ws.scalar_type() == at::kByte && ws.is_contiguous() && ws.numel() >= ws_bytes);
    const at::Tensor d_o = given.to(t.q->scalar_type());   // (keeps the layout; KDA's output is float32)
    const at::Tensor dq = t.like(*t.q, t.q->scalar_type()), dk = t.like(*t.k, t.q->scalar_type()), dv = t.like(*t.v, t.q->scalar_type());
    const at::Tensor dbeta = t.like(*t.beta, at::kFloat);
    at::Tensor dg, dh0;
    if (t.g) dg = t.like(*t.g, at::kFloat);
    if (want_dh0) dh0 = t.c.empty({t.B, t.H, t.K, t.V}, at::kFloat);
    void* stream = t.c.stream();
    int st;
    {
      Unlocked u;
      st = api.chunk_bwd_saved(&t.d, ptr(*t.q), ptr(*t.k), ptr(*t.v), ptr(t.g), fptr(t.beta), ptr(d_o), fptr(d_hT), dq.mutable_data_ptr(),
                               dk.mutable_data_ptr(), dv.mutable_data_ptr(), fmut(dbeta), t.g ? fmut(dg) : nullptr, want_dh0 ? fmut(dh0) : nullptr,
                               ws.mutable_data_ptr(), (size_t)ws.numel(), t.c.status(), stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    PyObject* r = PyTuple_New(6);
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(dq));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(dk));
    PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(dv));
    auto wrapped = [](bool there, const at::Tensor& x) -> PyObject* {
      if (there) return THPVariable_Wrap(x);
      Py_INCREF(Py_None);
      return Py_None;
    };
    PyTuple_SET_ITEM(r, 3, wrapped(t.g != nullptr, dg));
    PyTuple_SET_ITEM(r, 4, THPVariable_Wrap(dbeta));
    PyTuple_SET_ITEM(r, 5, wrapped(want_dh0, dh0));
    return r;
  });
}

// packed(variant, q, k, v, g, beta, cu (list of ints), h0, scale, chunk, l2norm, out_dtype) -> (o, hT) | status | None
PyObject* py_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 12);
    Call c;
    const int variant = (int)as_int(a[0]);
    const at::Tensor &q = c.req(a[1]), &k = c.req(a[2]), &v = c.req(a[3]);
    const at::Tensor* g = c.opt(a[4]);
    const at::Tensor& beta = c.req(a[5]);
    const at::Tensor* h0 = c.opt(a[7]);
    c.no_grad();   // with a gradient wanted the sequences go through the autograd ops
    need(q.dim() == 3 && v.dim() == 3 && k.sizes().equals(q.sizes()) && PyList_CheckExact(a[6]));
    const int64_t total = q.size(0), Hq = q.size(1), K = q.size(2), H = v.size(1), V = v.size(2);
    need(v.size(0) == total && Hq > 0 && H % Hq == 0 && is_shape(beta, {total, H}));
    const int dt = qkv_dtype(q, k, v);
    need(q.is_contiguous() && k.is_contiguous() && v.is_contiguous());
    need_f32(&beta);
    need((g != nullptr) == (variant != DR_DELTA));
    int g_dt = DR_F32;
    if (g) {
      need(g->is_contiguous() && (variant == DR_GATED ? is_shape(*g, {total, H}) : is_shape(*g, {total, H, K})));
      g_dt = dtype_code(*g);
    }
    const Py_ssize_t n_seqs = PyList_GET_SIZE(a[6]) - 1;
    need(n_seqs >= 1 && total < (int64_t)1 << 31);
    std::vector<int32_t> cu(n_seqs + 1);
    int64_t longest = 0;
    for (Py_ssize_t i = 0; i <= n_seqs; ++i) {
      PyObject* x = PyList_GET_ITEM(a[6], i);
      need(PyLong_CheckExact(x));
      const long y = PyLong_AsLong(x);
      need(y >= 0 && y <= total && (i == 0 ? y == 0 : y > cu[i - 1]));
      cu[i] = (int32_t)y;
      if (i) longest = std::max(longest, (int64_t)cu[i] - cu[i - 1]);
    }
    need(cu[n_seqs] == total);
    if (h0) { need(is_shape(*h0, {(int64_t)n_seqs, H, K, V})); need_f32(h0); }
    const long out = as_int(a[11]);
    need(out >= 0 && out <= DR_BF16);
    const double scale = a[8] == Py_None ? 1.0 / std::sqrt((double)K) : as_double(a[8]);
    const DrDesc d = make_desc(variant, DR_LAYOUT_BTHD, 1, H, longest, K, V, as_int(a[9]), dt, g_dt, (int)out, a[10] == Py_True, scale, 0, Hq);
    need(!PyErr_Occurred());
    // scratch for every sequence's chunks at once (one launch over all of them) up to kPackedScratch, past that in several launches;
    // the longest sequence's in any case
    DrDesc dw = d;
    dw.T = (int32_t)std::min<int64_t>(total + 64 * (int64_t)n_seqs, INT32_MAX);
    const int64_t all = api.workspace_bytes(&dw, 0);
    if (all < 0) return PyLong_FromLong((long)all);
    const int64_t ws_bytes = std::min(all, std::max(api.workspace_bytes(&d, 0), kPackedScratch));
    at::Tensor ws;
    if (ws_bytes > 0) ws = c.empty({ws_bytes}, at::kByte);
    const at::Tensor o = c.empty({total, H, V}, scalar_type((int)out));
    const at::Tensor hT = c.empty({(int64_t)n_seqs, H, K, V}, at::kFloat);
    void* stream = c.stream();
    int st;
    {
      Unlocked u;
      st = api.chunk_fwd_varlen(&d, ptr(q), ptr(k), ptr(v), ptr(g), fptr(&beta), cu.data(), (int32_t)n_seqs, fptr(h0), o.mutable_data_ptr(),
                                fmut(hT), ws_bytes > 0 ? ws.mutable_data_ptr() : nullptr, (size_t)ws_bytes, c.status(), stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    return pair(o, hT);
  });
}

// conv(x, weight, bias, cache, silu, cache_out) -> (y, new_cache) | status | None
PyObject* py_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 6);
    Call c;
    const at::Tensor &x = c.req(a[0]), &w = c.req(a[1]);
    const at::Tensor *bias = c.opt(a[2]), *cache = c.opt(a[3]), *cache_out = c.opt(a[5]);
    need(x.dim() == 3 && w.dim() == 2 && x.is_contiguous());
    const int dt = dtype_code(x);
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), W = w.size(0);
    need(W > 1 && w.size(1) == C);
    need_f32(&w);
    if (bias) { need(is_shape(*bias, {C})); need_f32(bias); }
    for (const at::Tensor* t : {cache, cache_out})
      if (t) need(is_shape(*t, {B, W - 1, C}) && t->scalar_type() == x.scalar_type() && t->is_contiguous());
    const at::Tensor y = c.empty({B, T, C}, x.scalar_type());
    const at::Tensor nc = cache_out ? *cache_out : c.empty({B, W - 1, C}, x.scalar_type());
    void* stream = c.stream();
    int st;
    {
      Unlocked u;
      st = api.short_conv_silu(ptr(x), fptr(&w), fptr(bias), ptr(cache), y.mutable_data_ptr(), nc.mutable_data_ptr(), (int)B, (int)T,
                               (int)C, (int)W, dt, a[4] == Py_True, stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    if (cache_out) { Py_INCREF(a[5]); return pair(y, a[5]); }
    return pair(y, nc);
  });
}

// gates(mode, a, b, A_log, bias, H, K, beta_scale, threshold) -> (g, beta | None) | status | None
PyObject* py_gates(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 9);
    Call c;
    const int mode = (int)as_int(a[0]);
    const at::Tensor& x = c.req(a[1]);
    const at::Tensor* b = c.opt(a[2]);
    const at::Tensor& A = c.req(a[3]);
    const at::Tensor* bias = c.opt(a[4]);
    const int64_t H = as_int(a[5]), K = as_int(a[6]);
    need(x.dim() == 3 && x.is_contiguous() && x.size(2) == H * K && is_shape(A, {H}));
    const int64_t B = x.size(0), T = x.size(1);
    need_f32(&A);
    if (bias) { need(bias->numel() == (mode == 0 ? H : H * K)); need_f32(bias); }
    if (b) need(b->is_contiguous() && is_shape(*b, {B, T, H}));
    const int adt = dtype_code(x), bdt = b ? dtype_code(*b) : DR_F32;
    const at::Tensor g = mode == 0 ? c.empty({B, T, H}, at::kFloat) : c.empty({B, T, H, K}, at::kFloat);
    at::Tensor beta;
    if (b) beta = c.empty({B, T, H}, at::kFloat);
    const double beta_scale = as_double(a[7]), threshold = as_double(a[8]);
    need(!PyErr_Occurred());
    void* stream = c.stream();
    int st;
    {
      Unlocked u;
      st = api.gate_activations(mode, ptr(x), ptr(b), fptr(&A), fptr(bias), fmut(g), b ? fmut(beta) : nullptr, (int)B, (int)T, (int)H,
                                (int)K, adt, bdt, (float)beta_scale, (float)threshold, stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    if (b) return pair(g, beta);
    Py_INCREF(Py_None);
    return pair(g, Py_None);
  });
}

// norm(o, weight, gate, eps, bthd, out_dtype (-1: o's)) -> y | status | None
PyObject* py_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 6);
    Call c;
    const at::Tensor &o = c.req(a[0]), &w = c.req(a[1]);
    const at::Tensor* gate = c.opt(a[2]);
    need(o.dim() == 4);
    bool bthd = a[4] == Py_True;
    const int64_t B = o.size(0), H = bthd ? o.size(2) : o.size(1), T = bthd ? o.size(1) : o.size(2), V = o.size(3);
    if (!o.is_contiguous()) {   // what the op returns for token-major inputs, taken as it is
      need(!bthd && is_bthd_view(o));
      bthd = true;
    }
    need(is_shape(w, {V}));
    need_f32(&w);
    if (gate) need(is_shape(*gate, {B, T, H, V}) && gate->is_contiguous());
    const int odt = dtype_code(o), gdt = gate ? dtype_code(*gate) : DR_F32;
    const long out_arg = as_int(a[5]);
    need(out_arg >= -1 && out_arg <= DR_BF16);
    const int ydt = out_arg < 0 ? odt : (int)out_arg;
    const double eps = as_double(a[3]);
    need(!PyErr_Occurred());
    const at::Tensor y = c.empty({B, T, H, V}, scalar_type(ydt));
    void* stream = c.stream();
    int st;
    {
      Unlocked u;
      st = api.gated_rmsnorm(ptr(o), ptr(gate), fptr(&w), y.mutable_data_ptr(), (int)B, (int)H, (int)T, (int)V,
                             bthd ? DR_LAYOUT_BTHD : DR_LAYOUT_BHTD, odt, gdt, ydt, (float)eps, stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    return THPVariable_Wrap(y);
  });
}

// scan(rule 0 RWKV-7 | 1 RWKV-6, q, k, v, a | u, b | None, gk | w, scale, h0) -> (o, hT) | status | None
PyObject* py_scan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 9);
    Call c;
    const bool dplr = as_int(a[0]) == 0;
    const at::Tensor &q = c.req(a[1]), &k = c.req(a[2]), &v = c.req(a[3]), &x = c.req(a[4]);
    const at::Tensor* b = c.opt(a[5]);
    const at::Tensor& w = c.req(a[6]);
    const at::Tensor* h0 = c.opt(a[8]);
    need(q.dim() == 4 && v.dim() == 4 && k.sizes().equals(q.sizes()) && w.sizes().equals(q.sizes()));
    const int64_t B = q.size(0), H = q.size(1), T = q.size(2), K = q.size(3), V = v.size(3);
    need(v.size(0) == B && v.size(1) == H && v.size(2) == T && T > 0);
    const int dt = qkv_dtype(q, k, v);
    need(w.scalar_type() == q.scalar_type());
    int layout;
    if (dplr) {
      need(b && x.sizes().equals(q.sizes()) && b->sizes().equals(q.sizes()) && x.scalar_type() == q.scalar_type() &&
           b->scalar_type() == q.scalar_type());
      layout = common_layout({&q, &k, &v, &x, b, &w});
    } else {
      need(!b && is_shape(x, {H, K}));
      need_f32(&x);
      layout = common_layout({&q, &k, &v, &w});
    }
    need(layout == DR_LAYOUT_BHTD || (H > 1 && T > 1));
    if (h0) { need(is_shape(*h0, {B, H, K, V})); need_f32(h0); }
    const double scale = as_double(a[7]);
    need(!PyErr_Occurred());
    const at::Tensor o = sequence_out(c, layout, B, H, T, V, q.scalar_type());
    const at::Tensor hT = c.empty({B, H, K, V}, at::kFloat);
    void* stream = c.stream();
    int st;
    {
      Unlocked u;
      st = dplr ? api.dplr_recurrent(ptr(q), ptr(k), ptr(v), ptr(x), ptr(b), ptr(w), fptr(h0), o.mutable_data_ptr(), fmut(hT), (int)B,
                                     (int)H, (int)T, (int)K, (int)V, (float)scale, dt, layout, c.status(), stream)
                : api.rwkv6_recurrent(ptr(q), ptr(k), ptr(v), ptr(w), fptr(&x), fptr(h0), o.mutable_data_ptr(), fmut(hT), (int)B, (int)H,
                                      (int)T, (int)K, (int)V, (float)scale, dt, layout, c.status(), stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    return pair(o, hT);
  });
}

// ssd(x, dt, A, B, C, D, n_groups, h0, dt_bias, lo, hi) -> (y, hT) | status | None
PyObject* py_ssd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n == 11);
    Call c;
    const at::Tensor &x = c.req(a[0]), &dt = c.req(a[1]), &A = c.req(a[2]), &Bm = c.req(a[3]), &Cm = c.req(a[4]), &D = c.req(a[5]);
    const int64_t G = as_int(a[6]);
    const at::Tensor *h0 = c.opt(a[7]), *bias = c.opt(a[8]);
    need(x.dim() == 4 && Bm.dim() == 4 && Cm.sizes().equals(Bm.sizes()));
    const int64_t Bt = x.size(0), T = x.size(1), H = x.size(2), P = x.size(3), N = Bm.size(3);
    need(T > 0 && Bm.size(0) == Bt && Bm.size(1) == T && Bm.size(2) == G && G > 0 && H % G == 0 && is_shape(dt, {Bt, T, H}));
    const int io = dtype_code(x);
    need(Bm.scalar_type() == x.scalar_type() && Cm.scalar_type() == x.scalar_type());
    need(x.is_contiguous() && Bm.is_contiguous() && Cm.is_contiguous());
    need_f32(&dt);
    for (const at::Tensor* t : {&A, &D, bias})
      if (t) { need(is_shape(*t, {H})); need_f32(t); }
    if (h0) { need(is_shape(*h0, {Bt, H, P, N})); need_f32(h0); }
    const double lo = as_double(a[9]), hi = as_double(a[10]);
    need(!PyErr_Occurred());
    const at::Tensor y = c.empty({Bt, T, H, P}, x.scalar_type());
    const at::Tensor hT = c.empty({Bt, H, P, N}, at::kFloat);
    void* stream = c.stream();
    int st;
    {
      Unlocked u;
      st = api.ssd_scan(ptr(x), ptr(dt), fptr(&A), ptr(Bm), ptr(Cm), fptr(&D), fptr(bias), fptr(h0), y.mutable_data_ptr(), fmut(hT), (int)Bt,
                        (int)T, (int)H, (int)P, (int)N, (int)G, (float)lo, (float)hi, io, c.status(), stream);
    }
    if (st < 0) return PyLong_FromLong(st);
    return pair(y, hT);
  });
}

// open(path of the kernel library)
PyObject* py_open(PyObject*, PyObject* arg) {
  const char* path = PyUnicode_AsUTF8(arg);
  if (!path) return nullptr;
  void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);   // the library ctypes has loaded already
  if (!h) { PyErr_SetString(PyExc_ImportError, dlerror()); return nullptr; }
#define DR_SYM(member, name)                                                                             \
  if (!(api.member = reinterpret_cast<decltype(api.member)>(dlsym(h, name)))) {                          \
    PyErr_SetString(PyExc_ImportError, "missing symbol " name);                                          \
    return nullptr;                                                                                      \
  }
  DR_SYM(workspace_bytes, "dr_workspace_bytes")
  DR_SYM(chunk_fwd, "dr_chunk_fwd")
  DR_SYM(recurrent_fwd, "dr_recurrent_fwd")
  DR_SYM(step, "dr_step")
  DR_SYM(chunk_fwd_varlen, "dr_chunk_fwd_varlen")
  DR_SYM(short_conv_silu, "dr_short_conv_silu")
  DR_SYM(gate_activations, "dr_gate_activations")
  DR_SYM(gated_rmsnorm, "dr_gated_rmsnorm")
  DR_SYM(dplr_recurrent, "dr_dplr_recurrent")
  DR_SYM(rwkv6_recurrent, "dr_rwkv6_recurrent")
  DR_SYM(ssd_scan, "dr_ssd_scan")
  DR_SYM(chunk_fwd_saving, "dr_chunk_fwd_saving")
  DR_SYM(chunk_bwd_saved, "dr_chunk_bwd_saved")
#undef DR_SYM
  g_open = true;
  Py_RETURN_NONE;
}

// set_status(device index, address of its status word)
PyObject* py_set_status(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) { PyErr_SetString(PyExc_TypeError, "set_status(index, address)"); return nullptr; }
  const long i = PyLong_AsLong(a[0]);
  const long long p = PyLong_AsLongLong(a[1]);
  if (PyErr_Occurred()) return nullptr;
  if (i >= 0 && i < kMaxDevices) g_status[i] = reinterpret_cast<int32_t*>(p);
  Py_RETURN_NONE;
}

#define DR_FN(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"open", py_open, METH_O, nullptr}, DR_FN(set_status), DR_FN(step), DR_FN(sequence), DR_FN(packed), DR_FN(conv), DR_FN(gates),
    DR_FN(norm), DR_FN(scan), DR_FN(ssd), DR_FN(train_fwd), DR_FN(train_bwd), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_calls(void) { return PyModule_Create(&module_def); }
