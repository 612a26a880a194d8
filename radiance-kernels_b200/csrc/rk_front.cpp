// Native front end of the Python package: what api.py's functions do between the caller's torch tensors and the C ABI
// (include/rk_mx_attn.h) -- checks of device, dtype and exact shape, allocation of outputs and workspace, the current
// stream, the call.  The small calls of this path are a few microseconds of GPU work, so this is what bounds them: the
// same steps written in Python over ctypes took 20 us per call (one decode step, three of them with the cache append,
// 38 us against 18 us of kernels); here a call costs 1-2 us plus its launches.
//
// CPython module with vectorcall functions over torch's C++ tensors.  Every function raises ValueError for a tensor the
// library must not be handed (past this point it is a raw pointer that TMA and bulk copies read with the sizes of the
// argument struct) and hands the library's own return code to the error function given by set_error.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstdio>
#include <initializer_list>

#include "../../include/rk_mx_attn.h"

namespace {

using at::Tensor;

struct PyFail {};                                      // a Python exception is set

PyObject* g_error = nullptr;                           // error(code, where): raises RkError

[[noreturn]] void fail(PyObject* type, const char* msg) {
  PyErr_SetString(type, msg);
  throw PyFail();
}
[[noreturn]] void value_error(const char* msg) { fail(PyExc_ValueError, msg); }

void check_code(int rc, const char* where) {
  if (rc == RK_OK) return;
  if (g_error) {
    PyObject* r = PyObject_CallFunction(g_error, "is", rc, where);
    Py_XDECREF(r);
  }
  if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s: code %d", where, rc);
  throw PyFail();
}

// ---- argument access -----------------------------------------------------------------------------------------
struct Args {
  PyObject* const* v;
  Py_ssize_t n;
  void expect(Py_ssize_t want) const {
    if (n != want) fail(PyExc_TypeError, "wrong number of arguments");
  }
  const Tensor* opt(Py_ssize_t i) const {              // None -> nullptr
    if (v[i] == Py_None) return nullptr;
    if (!THPVariable_Check(v[i])) fail(PyExc_TypeError, "expected a tensor");
    return &THPVariable_Unpack(v[i]);
  }
  const Tensor& tensor(Py_ssize_t i) const {
    const Tensor* t = opt(i);
    if (!t) fail(PyExc_TypeError, "expected a tensor, got None");
    return *t;
  }
  int64_t integer(Py_ssize_t i) const {
    const long long r = PyLong_AsLongLong(v[i]);
    if (r == -1 && PyErr_Occurred()) throw PyFail();
    return r;
  }
  int32_t i32(Py_ssize_t i) const {
    const int64_t r = integer(i);
    if (r < INT32_MIN || r > INT32_MAX) fail(PyExc_OverflowError, "integer argument out of the 32-bit range");
    return (int32_t)r;
  }
  float real(Py_ssize_t i) const {
    const double r = PyFloat_AsDouble(v[i]);
    if (r == -1.0 && PyErr_Occurred()) throw PyFail();
    return (float)r;
  }
  bool truth(Py_ssize_t i) const {
    const int r = PyObject_IsTrue(v[i]);
    if (r < 0) throw PyFail();
    return r != 0;
  }
};

using Dims = std::initializer_list<int64_t>;

void need_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t && (!t->is_cuda() || !t->is_contiguous())) value_error("expected contiguous CUDA tensors");
}

void expect(const Tensor* t, const char* name, at::ScalarType dtype, at::IntArrayRef shape) {
  if (!t) return;
  char msg[256];
  if (t->scalar_type() != dtype) {
    snprintf(msg, sizeof msg, "%s: expected dtype %s, got %s", name, c10::toString(dtype), c10::toString(t->scalar_type()));
    value_error(msg);
  }
  if (t->sizes() == shape) return;
  int n = snprintf(msg, sizeof msg, "%s: expected shape (", name);
  for (size_t i = 0; i < shape.size() && n < 200; ++i) n += snprintf(msg + n, sizeof msg - n, i ? ", %lld" : "%lld", (long long)shape[i]);
  snprintf(msg + n, sizeof msg - n, ")");
  value_error(msg);
}

// The shape of a tensor's leading axes followed by other ones, without an allocation for the usual ranks.
c10::SmallVector<int64_t, 6> shape_of(at::IntArrayRef lead, Dims tail) {
  c10::SmallVector<int64_t, 6> s(lead.begin(), lead.end());
  s.append(tail.begin(), tail.end());
  return s;
}
at::IntArrayRef lead_of(const Tensor& t, size_t drop) { return t.sizes().slice(0, t.dim() - drop); }

int64_t up(int64_t a, int64_t b) { return (a + b - 1) / b; }

// scale tensor of the [S][d] matrices of `lead` in a layout
c10::SmallVector<int64_t, 6> scale_shape(at::IntArrayRef lead, int64_t S, int64_t d, int layout) {
  if (layout == RK_SCALES_ROWMAJOR) return shape_of(lead, {S, d / 32});
  if (layout == RK_SCALES_GROUPMAJOR) return shape_of(lead, {d / 32, S});
  if (layout == RK_SCALES_SF_ATOMS) return shape_of(lead, {up(S, 128), up(d, 128), 512});
  value_error("scale layout must be SCALES_ROWMAJOR, SCALES_GROUPMAJOR or SCALES_SF_ATOMS");
}

Tensor empty_like_device(const Tensor& t, at::IntArrayRef shape, at::ScalarType dtype) {
  return Tensor(at::detail::empty_cuda(shape, dtype, t.device(), std::nullopt));
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

template <class T = uint8_t> T* ptr(const Tensor& t) { return static_cast<T*>(t.data_ptr()); }
template <class T = uint8_t> T* ptr(const Tensor* t) { return t ? static_cast<T*>(t->data_ptr()) : nullptr; }

PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* pair(Tensor a, Tensor b) {
  PyObject* x = wrap(std::move(a));
  PyObject* y = x ? wrap(std::move(b)) : nullptr;
  PyObject* r = y ? PyTuple_New(2) : nullptr;
  if (!r) { Py_XDECREF(x); Py_XDECREF(y); throw PyFail(); }
  PyTuple_SET_ITEM(r, 0, x);
  PyTuple_SET_ITEM(r, 1, y);
  return r;
}

// The library call without the interpreter lock: a launch can block while the stream's queue is full.  (f also asks the tensors
// for their pointers, which throws for those without storage: the lock is taken again on that way out, too.)
template <class F> int unlocked(F&& f) {
  struct Released {
    PyThreadState* state = PyEval_SaveThread();
    ~Released() { PyEval_RestoreThread(state); }
  } released;
  return f();
}

bool float_or_bf16(const Tensor& t) { return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16; }

// ---- quantizers ------------------------------------------------------------------------------------------------
PyObject* mx_quantize(const Args& a) {                 // x, fmt
  a.expect(2);
  const Tensor& x = a.tensor(0);
  const int fmt = a.i32(1);
  need_cuda({&x});
  if (!float_or_bf16(x) || x.dim() < 1) value_error("mx_quantize takes float32 or bfloat16");
  const int64_t cols = x.size(-1), rows = x.numel() / std::max<int64_t>(cols, 1);
  Tensor codes = empty_like_device(x, x.sizes(), at::kByte);
  Tensor scales = empty_like_device(x, shape_of(lead_of(x, 1), {cols / 32}), at::kByte);
  const bool bf16 = x.scalar_type() == at::kBFloat16;
  void* st = stream();
  check_code(unlocked([&] {
    return bf16 ? rk_mx_quantize_bf16(x.data_ptr(), rows, cols, fmt, ptr(codes), ptr(scales), st)
                : rk_mx_quantize(ptr<float>(x), rows, cols, fmt, ptr(codes), ptr(scales), st);
  }), "rk_mx_quantize");
  return pair(std::move(codes), std::move(scales));
}

PyObject* mx_quantize_ex(const Args& a) {              // x, fmt, scale_layout
  a.expect(3);
  const Tensor& x = a.tensor(0);
  const int fmt = a.i32(1), layout = a.i32(2);
  need_cuda({&x});
  if (!float_or_bf16(x) || x.dim() < 2) value_error("mx_quantize_ex takes float32 or bfloat16 [..., S, d]");
  const int64_t S = x.size(-2), d = x.size(-1), batch = x.numel() / std::max<int64_t>(S * d, 1);
  Tensor codes = empty_like_device(x, x.sizes(), at::kByte);
  Tensor scales = empty_like_device(x, scale_shape(lead_of(x, 2), S, d, layout), at::kByte);
  const bool bf16 = x.scalar_type() == at::kBFloat16;
  void* st = stream();
  check_code(unlocked([&] { return rk_mx_quantize_ex(x.data_ptr(), bf16, batch, S, d, fmt, ptr(codes), ptr(scales), layout, st); }),
             "rk_mx_quantize_ex");
  return pair(std::move(codes), std::move(scales));
}

PyObject* mx_quantize_keys(const Args& a) {            // x, fmt, scale_layout
  a.expect(3);
  const Tensor& x = a.tensor(0);
  const int fmt = a.i32(1), layout = a.i32(2);
  need_cuda({&x});
  if (x.scalar_type() != at::kFloat || x.dim() < 2) value_error("mx_quantize_keys takes float32 [..., rows, cols]");
  const int64_t rows = x.size(-2), cols = x.size(-1), batch = x.numel() / std::max<int64_t>(rows * cols, 1);
  Tensor codes = empty_like_device(x, x.sizes(), at::kByte);
  Tensor scales = empty_like_device(x, layout == RK_SCALES_ROWMAJOR ? shape_of(lead_of(x, 2), {up(rows, 32), cols})
                                                                     : scale_shape(lead_of(x, 2), rows, cols, RK_SCALES_SF_ATOMS), at::kByte);   // (no other: the library says so)
  void* st = stream();
  check_code(unlocked([&] { return rk_mx_quantize_keys_ex(ptr<float>(x), batch, rows, cols, fmt, ptr(codes), ptr(scales), layout, st); }),
             "rk_mx_quantize_keys");
  return pair(std::move(codes), std::move(scales));
}

PyObject* mx_rebase_v(const Args& a) {                 // codes, scales, fmt
  a.expect(3);
  const Tensor &codes = a.tensor(0), &scales = a.tensor(1);
  const int fmt = a.i32(2);
  need_cuda({&codes, &scales});
  if (codes.dim() < 2) value_error("mx_rebase_v takes codes [..., S, d]");
  const int64_t S = codes.size(-2), d = codes.size(-1), batch = codes.numel() / std::max<int64_t>(S * d, 1);
  if (scales.numel() < codes.numel() / 32) value_error("mx_rebase_v: fewer scales than blocks of codes");
  Tensor oc = empty_like_device(codes, codes.sizes(), codes.scalar_type());
  Tensor os = empty_like_device(codes, shape_of(lead_of(codes, 2), {up(S, 32), d}), at::kByte);
  void* st = stream();
  check_code(unlocked([&] { return rk_mx_rebase_v(ptr(codes), ptr(scales), batch, S, d, fmt, ptr(oc), ptr(os), st); }), "rk_mx_rebase_v");
  return pair(std::move(oc), std::move(os));
}

PyObject* rope_mx_quantize(const Args& a) {            // x, cos_half, sin_half, pos, pos0, fmt
  a.expect(6);
  const Tensor &x = a.tensor(0), &cos_half = a.tensor(1), &sin_half = a.tensor(2);
  const Tensor* pos = a.opt(3);
  const int pos0 = a.i32(4), fmt = a.i32(5);
  need_cuda({&x, &cos_half, &sin_half, pos});
  if (x.scalar_type() != at::kFloat || cos_half.scalar_type() != at::kFloat || sin_half.scalar_type() != at::kFloat)
    value_error("rope_mx_quantize takes float32");
  if (x.dim() < 2) value_error("rope_mx_quantize takes x [..., S, d]");
  const int64_t S = x.size(-2), d = x.size(-1), rows = x.numel() / std::max<int64_t>(d, 1);
  if (cos_half.dim() != 2 || cos_half.size(1) != d / 2 || sin_half.sizes() != cos_half.sizes())
    value_error("cos_half / sin_half must be [n_pos, d/2]");
  expect(pos, "pos", at::kInt, {rows});
  Tensor codes = empty_like_device(x, x.sizes(), at::kByte);
  Tensor scales = empty_like_device(x, shape_of(lead_of(x, 1), {d / 32}), at::kByte);
  void* st = stream();
  check_code(unlocked([&] {
    return rk_rope_mx_quantize(ptr<float>(x), rows, (int32_t)d, ptr<int32_t>(pos), (int32_t)S, pos0, ptr<float>(cos_half), ptr<float>(sin_half),
                               (int32_t)cos_half.size(0), fmt, ptr(codes), ptr(scales), st);
  }), "rk_rope_mx_quantize");
  return pair(std::move(codes), std::move(scales));
}

PyObject* rmsnorm_mx_quantize(const Args& a) {         // x, gamma, eps, fmt, unit_scale
  a.expect(5);
  const Tensor &x = a.tensor(0), &gamma = a.tensor(1);
  const float eps = a.real(2);
  const int fmt = a.i32(3);
  const bool unit = a.truth(4);
  need_cuda({&x, &gamma});
  if (!float_or_bf16(x) || x.dim() < 1 || gamma.scalar_type() != at::kFloat)
    value_error("rmsnorm_mx_quantize takes float32 or bfloat16 rows and a float32 gamma");
  const int64_t K = x.size(-1), rows = x.numel() / std::max<int64_t>(K, 1);
  expect(&gamma, "gamma", at::kFloat, {K});
  Tensor codes = empty_like_device(x, x.sizes(), at::kByte);
  Tensor scales = empty_like_device(x, shape_of(lead_of(x, 1), {K / 32}), at::kByte);
  const bool bf16 = x.scalar_type() == at::kBFloat16;
  void* st = stream();
  check_code(unlocked([&] {
    return rk_rmsnorm_mx_quantize(x.data_ptr(), bf16, rows, (int32_t)K, ptr<float>(gamma), eps, fmt, unit, ptr(codes), ptr(scales), st);
  }), "rk_rmsnorm_mx_quantize");
  return pair(std::move(codes), std::move(scales));
}

// ---- prefill ---------------------------------------------------------------------------------------------------
// The tensors of a prefill call against B / H / H_kv / S / d: exact dtypes and shapes.
void check_prefill(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& q_scale, const Tensor& k_scale, const Tensor& v_scale,
                   const Tensor* o, const Tensor* lse, int v_axis, int q_layout, int k_layout, int v_layout) {
  if (q.dim() != 4 || k.dim() != 4) value_error("q must be [B,H,S_q,d] and k/v [B,H_kv,S_kv,d]");
  const int64_t B = q.size(0), H = q.size(1), S_q = q.size(2), d = q.size(3), H_kv = k.size(1), S_kv = k.size(2);
  if (d % 32 != 0) value_error("d must be a multiple of 32");
  const int64_t kv_lead[2] = {B, H_kv}, q_lead[2] = {B, H};
  expect(&q, "q", at::kByte, {B, H, S_q, d});
  expect(&k, "k", at::kByte, {B, H_kv, S_kv, d});
  expect(&v, "v", at::kByte, {B, H_kv, S_kv, d});
  expect(&q_scale, "q_scale", at::kByte, scale_shape(q_lead, S_q, d, q_layout));
  expect(&k_scale, "k_scale", at::kByte, scale_shape(kv_lead, S_kv, d, k_layout));
  if (v_axis == RK_V_SCALES_ALONG_D) {
    if (v_layout != RK_SCALES_ROWMAJOR) value_error("V scales along d are row-major");
    expect(&v_scale, "v_scale", at::kByte, {B, H_kv, S_kv, d / 32});
  } else if (v_axis == RK_V_SCALES_ALONG_KEYS) {
    if (v_layout == RK_SCALES_ROWMAJOR) expect(&v_scale, "v_scale", at::kByte, {B, H_kv, up(S_kv, 32), d});
    else if (v_layout == RK_SCALES_SF_ATOMS) expect(&v_scale, "v_scale", at::kByte, scale_shape(kv_lead, S_kv, d, v_layout));
    else value_error("V scales along the keys are row-major or scale-factor atoms");
  } else {
    value_error("v_scale_axis must be V_SCALES_ALONG_KEYS or V_SCALES_ALONG_D");
  }
  expect(o, "out", at::kBFloat16, {B, H, S_q, d});
  expect(lse, "lse", at::kFloat, {B, H, S_q});
}

PyObject* check_prefill_tensors(const Args& a) {       // q, k, v, q_scale, k_scale, v_scale, o, lse, axis, three layouts
  a.expect(12);
  check_prefill(a.tensor(0), a.tensor(1), a.tensor(2), a.tensor(3), a.tensor(4), a.tensor(5), a.opt(6), a.opt(7), a.i32(8), a.i32(9),
                a.i32(10), a.i32(11));
  Py_RETURN_NONE;
}

// workspace (the caller's or one of this call, returned to the caching allocator when the call has been enqueued), launch
void launch_prefill(rk_prefill_args& p, const Tensor& q, const Tensor* workspace) {
  const size_t need = rk_attn_prefill_workspace_bytes(&p);
  Tensor own;
  if (!workspace) {
    own = empty_like_device(q, {(int64_t)std::max<size_t>(need, 1024)}, at::kByte);
    workspace = &own;
  } else if (workspace->scalar_type() != at::kByte) {
    value_error("workspace must be a uint8 tensor");
  }
  p.workspace = workspace->data_ptr();
  p.workspace_bytes = (size_t)workspace->numel();
  void* st = stream();
  check_code(unlocked([&] { return rk_attn_prefill(&p, st); }), "rk_attn_prefill");
}

// the options both prefill forms share, from argument i on: causal, softmax_scale, q_pos0, window, softcap, q_fmt, kv_fmt,
// q_scale_layout, k_scale_layout, v_scale_layout
void prefill_options(const Args& a, Py_ssize_t i, rk_prefill_args& p) {
  p.causal = a.truth(i);
  p.softmax_scale = a.real(i + 1);
  p.q_pos0 = a.i32(i + 2);
  p.window = a.i32(i + 3);
  p.softcap = a.real(i + 4);
  p.q_fmt = a.i32(i + 5);
  p.kv_fmt = a.i32(i + 6);
  p.q_scale_layout = a.i32(i + 7);
  p.k_scale_layout = a.i32(i + 8);
  p.v_scale_layout = a.i32(i + 9);
}

void prefill_pointers(rk_prefill_args& p, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& qs, const Tensor& ks,
                      const Tensor& vs, const Tensor& o, const Tensor* lse) {
  p.q = ptr(q); p.k = ptr(k); p.v = ptr(v);
  p.q_scale = ptr(qs); p.k_scale = ptr(ks); p.v_scale = ptr(vs);
  p.o = o.data_ptr(); p.lse = ptr<float>(lse);
}

PyObject* attn_prefill(const Args& a) {                // q, k, v, q_scale, k_scale, v_scale, out, lse, workspace, v_scale_axis, options
  a.expect(20);
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &qs = a.tensor(3), &ks = a.tensor(4), &vs = a.tensor(5);
  const Tensor *out = a.opt(6), *lse = a.opt(7), *ws = a.opt(8);
  rk_prefill_args p = {};
  p.v_scale_axis = a.i32(9);
  prefill_options(a, 10, p);
  need_cuda({&q, &k, &v, &qs, &ks, &vs, out, lse, ws});
  check_prefill(q, k, v, qs, ks, vs, out, lse, p.v_scale_axis, p.q_scale_layout, p.k_scale_layout, p.v_scale_layout);
  p.B = (int32_t)q.size(0); p.H = (int32_t)q.size(1); p.S_q = (int32_t)q.size(2); p.d = (int32_t)q.size(3);
  p.H_kv = (int32_t)k.size(1); p.S_kv = (int32_t)k.size(2);
  Tensor o = out ? *out : empty_like_device(q, q.sizes(), at::kBFloat16);
  prefill_pointers(p, q, k, v, qs, ks, vs, o, lse);
  launch_prefill(p, q, ws);
  return wrap(std::move(o));
}

PyObject* attn_prefill_packed(const Args& a) {         // q, k, vt, q_scale, k_scale, v_scale, out, lse, workspace, S_q, S_kv, d, options
  a.expect(22);
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &vt = a.tensor(2), &qs = a.tensor(3), &ks = a.tensor(4), &vs = a.tensor(5);
  const Tensor *out = a.opt(6), *lse = a.opt(7), *ws = a.opt(8);
  rk_prefill_args p = {};
  p.S_q = a.i32(9); p.S_kv = a.i32(10); p.d = a.i32(11);
  prefill_options(a, 12, p);
  p.v_scale_axis = RK_V_SCALES_ALONG_KEYS;
  p.q_packed = p.kv_packed = 1;
  need_cuda({&q, &k, &vt, &qs, &ks, &vs, out, lse, ws});
  if (q.dim() != 4 || k.dim() != 4 || vt.dim() != 4) value_error("q, k and vt are 4-d packed tensors");
  const int64_t B = q.size(0), H = q.size(1), H_kv = k.size(1), S_q = p.S_q, S_kv = p.S_kv, d = p.d;
  const int64_t q_lead[2] = {B, H}, kv_lead[2] = {B, H_kv};
  expect(&q, "q", at::kByte, {B, H, S_q, (int64_t)rk_mx_packed_rows_bytes(1, d, p.q_fmt)});
  expect(&k, "k", at::kByte, {B, H_kv, S_kv, (int64_t)rk_mx_packed_rows_bytes(1, d, p.kv_fmt)});
  expect(&vt, "vt", at::kByte, {B, H_kv, d, (int64_t)rk_mx_packed_vt_bytes(1, S_kv, 1, p.kv_fmt)});
  expect(&qs, "q_scale", at::kByte, scale_shape(q_lead, S_q, d, p.q_scale_layout));
  expect(&ks, "k_scale", at::kByte, scale_shape(kv_lead, S_kv, d, p.k_scale_layout));
  if (p.v_scale_layout == RK_SCALES_ROWMAJOR) expect(&vs, "v_scale", at::kByte, {B, H_kv, up(S_kv, 32), d});
  else if (p.v_scale_layout == RK_SCALES_SF_ATOMS) expect(&vs, "v_scale", at::kByte, scale_shape(kv_lead, S_kv, d, p.v_scale_layout));
  else value_error("V scales along the keys are row-major or scale-factor atoms");
  expect(out, "out", at::kBFloat16, {B, H, S_q, d});
  expect(lse, "lse", at::kFloat, {B, H, S_q});
  p.B = (int32_t)B; p.H = (int32_t)H; p.H_kv = (int32_t)H_kv;
  Tensor o = out ? *out : empty_like_device(q, {B, H, S_q, d}, at::kBFloat16);
  prefill_pointers(p, q, k, vt, qs, ks, vs, o, lse);
  launch_prefill(p, q, ws);
  return wrap(std::move(o));
}

// ---- KV cache and decode -----------------------------------------------------------------------------------------
PyObject* kv_cache_append(const Args& a) {             // k_new, v_new, pos, k_codes, k_scales, v_codes, v_scales, fmt
  a.expect(8);
  const Tensor &kn = a.tensor(0), &vn = a.tensor(1), &pos = a.tensor(2), &kc = a.tensor(3), &ks = a.tensor(4), &vc = a.tensor(5), &vs = a.tensor(6);
  const int fmt = a.i32(7);
  need_cuda({&kn, &vn, &pos, &kc, &ks, &vc, &vs});
  if (kn.scalar_type() != at::kFloat || vn.scalar_type() != at::kFloat || pos.scalar_type() != at::kInt)
    value_error("kv_cache_append takes float32 rows and int32 positions");
  if (kc.dim() != 4) value_error("k_codes must be [B,H_kv,L,d]");
  const int64_t B = kc.size(0), H_kv = kc.size(1), L = kc.size(2), d = kc.size(3);
  expect(&kn, "k_new", at::kFloat, {B, H_kv, d});
  expect(&vn, "v_new", at::kFloat, {B, H_kv, d});
  expect(&pos, "pos", at::kInt, {B});
  expect(&kc, "k_codes", at::kByte, {B, H_kv, L, d});
  expect(&vc, "v_codes", at::kByte, {B, H_kv, L, d});
  expect(&ks, "k_scales", at::kByte, {B, H_kv, L, d / 32});
  expect(&vs, "v_scales", at::kByte, {B, H_kv, L, d / 32});
  void* st = stream();
  check_code(unlocked([&] {
    return rk_kv_cache_append(ptr<float>(kn), ptr<float>(vn), (int32_t)B, (int32_t)H_kv, (int32_t)L, (int32_t)d, ptr<int32_t>(pos), fmt, ptr(kc),
                              ptr(ks), ptr(vc), ptr(vs), st);
  }), "rk_kv_cache_append");
  Py_RETURN_NONE;
}

void check_decode(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& ks, const Tensor& vs, const Tensor* kv_len,
                  const Tensor* out, const Tensor* lse) {
  if (q.dim() != 3 || k.dim() != 4) value_error("q must be [B,H,d] and k/v [B,H_kv,L,d]");
  const int64_t B = q.size(0), H = q.size(1), d = q.size(2), H_kv = k.size(1), L = k.size(2);
  expect(&k, "k", at::kByte, {B, H_kv, L, d});
  expect(&v, "v", at::kByte, {B, H_kv, L, d});
  expect(&ks, "k_scale", at::kByte, {B, H_kv, L, d / 32});
  expect(&vs, "v_scale", at::kByte, {B, H_kv, L, d / 32});
  expect(kv_len, "kv_len", at::kInt, {B});
  expect(out, "out", at::kBFloat16, {B, H, d});
  expect(lse, "lse", at::kFloat, {B, H});
}

PyObject* check_decode_tensors(const Args& a) {        // q, k, v, k_scale, v_scale, kv_len, out, lse
  a.expect(8);
  check_decode(a.tensor(0), a.tensor(1), a.tensor(2), a.tensor(3), a.tensor(4), a.opt(5), a.opt(6), a.opt(7));
  Py_RETURN_NONE;
}

PyObject* attn_decode(const Args& a) {                 // q, k, v, k_scale, v_scale, kv_len, out, lse, workspace, softmax_scale, kv_fmt, num_splits
  a.expect(12);
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &ks = a.tensor(3), &vs = a.tensor(4);
  const Tensor *kv_len = a.opt(5), *out = a.opt(6), *lse = a.opt(7), *ws = a.opt(8);
  rk_decode_args p = {};
  p.softmax_scale = a.real(9);
  p.kv_fmt = a.i32(10);
  p.num_splits = a.i32(11);
  need_cuda({&q, &k, &v, &ks, &vs, kv_len, out, lse, ws});
  if (q.scalar_type() != at::kBFloat16) value_error("decode query must be bfloat16");
  check_decode(q, k, v, ks, vs, kv_len, out, lse);
  p.B = (int32_t)q.size(0); p.H = (int32_t)q.size(1); p.d = (int32_t)q.size(2);
  p.H_kv = (int32_t)k.size(1); p.L = (int32_t)k.size(2);
  Tensor o = out ? *out : empty_like_device(q, q.sizes(), at::kBFloat16);
  p.q = q.data_ptr(); p.k = ptr(k); p.v = ptr(v); p.k_scale = ptr(ks); p.v_scale = ptr(vs);
  p.kv_len = ptr<int32_t>(kv_len); p.o = o.data_ptr(); p.lse = ptr<float>(lse);
  Tensor own;
  if (!ws) {
    own = empty_like_device(q, {(int64_t)std::max<size_t>(rk_attn_decode_workspace_bytes(&p), 16)}, at::kByte);
    ws = &own;
  }
  p.workspace = ws->data_ptr();
  p.workspace_bytes = (size_t)ws->numel();
  void* st = stream();
  check_code(unlocked([&] { return rk_attn_decode(&p, st); }), "rk_attn_decode");
  return wrap(std::move(o));
}

PyObject* set_error(const Args& a) {                   // error(code, where)
  a.expect(1);
  Py_INCREF(a.v[0]);
  Py_XSETREF(g_error, a.v[0]);
  Py_RETURN_NONE;
}

template <PyObject* (*F)(const Args&)>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  try {
    return F(Args{args, n});
  } catch (const PyFail&) {
    return nullptr;
  } catch (...) {                                      // a failed allocation and the like, as torch reports them
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

#define RK_FN(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {RK_FN(mx_quantize), RK_FN(mx_quantize_ex), RK_FN(mx_quantize_keys), RK_FN(mx_rebase_v), RK_FN(rope_mx_quantize),
                         RK_FN(rmsnorm_mx_quantize), RK_FN(attn_prefill), RK_FN(attn_prefill_packed), RK_FN(kv_cache_append), RK_FN(attn_decode),
                         RK_FN(check_prefill_tensors), RK_FN(check_decode_tensors), RK_FN(set_error), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_rk_front", "Native front end of the MX attention package.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__rk_front(void) { return PyModule_Create(&module); }
