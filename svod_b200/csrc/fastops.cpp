// The op layer's Python call path in compiled code: reads the operand tensors and the
// option objects of `svod_b200/ops.py`, fills the `svodb_*` structs of include/svodb.h and
// calls the library. Building those structs through ctypes took 15-30 us a call, more than
// most kernels of a small batch.
//
// Every function returns the result tensor(s), or None for anything out of the ordinary — an
// operand that is not a realized CUDA tensor, an option this file does not read, a call the
// library refuses. Nothing has been launched then: ops.py takes the same call through its
// general path, which converts or reports it.
//
// What torch throws underneath (an allocation that fails, a tensor without storage) comes back
// as the Python exception it is anywhere else, never through the interpreter's frames.
//
// The library's entry points come as addresses (`init`), so that SVODB_LIB_PATH keeps
// selecting the build that runs.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "svodb.h"

namespace {

decltype(&svodb_linear) p_linear = nullptr;
decltype(&svodb_attention) p_attention = nullptr;
decltype(&svodb_attention_packed) p_attention_packed = nullptr;
decltype(&svodb_layer_norm) p_layer_norm = nullptr;
decltype(&svodb_rms_norm) p_rms_norm = nullptr;
decltype(&svodb_add_layer_norm) p_add_layer_norm = nullptr;
decltype(&svodb_add_rms_norm) p_add_rms_norm = nullptr;

// Attribute names of the option dataclasses.
#define NAMES(X)                                                                                                      \
  X(bias) X(act) X(gated) X(residual) X(scale) X(rope) X(into) X(qkv) X(k_splits) X(w_static) X(cos) X(sin) X(heads)  \
  X(head_dim) X(kv_heads) X(q_norm) X(k_norm) X(eps) X(causal) X(keys) X(window) X(chunk) X(seg_start) X(splits)      \
  X(cache) X(want_lse) X(lens) X(mask) X(head_start) X(row_map) X(appended) X(app_lens)
#define DECL(n) PyObject* s_##n = nullptr;
NAMES(DECL)

// A borrowed-or-owned attribute, released at the end of the scope.
struct Ref {
  PyObject* o;
  explicit Ref(PyObject* p) : o(p) {}
  Ref(const Ref&) = delete;
  ~Ref() { Py_XDECREF(o); }
  bool none() const { return o == nullptr || o == Py_None; }
};
Ref attr(PyObject* o, PyObject* name) { return Ref(PyObject_GetAttr(o, name)); }

bool truth(PyObject* o) { return o != nullptr && PyObject_IsTrue(o) == 1; }

// The `svodb_tensor` of a CUDA tensor; false for anything else.
bool desc(PyObject* o, svodb_tensor& d) {
  if (o == nullptr || !THPVariable_Check(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.dim() > SVODB_MAX_RANK || t.layout() != at::kStrided) return false;
  switch (t.scalar_type()) {
    case at::kFloat: d.dtype = SVODB_F32; break;
    case at::kHalf: d.dtype = SVODB_F16; break;
    case at::kBFloat16: d.dtype = SVODB_BF16; break;
    case at::kInt: d.dtype = SVODB_I32; break;
    case at::kLong: d.dtype = SVODB_I64; break;
    case at::kByte: case at::kBool: d.dtype = SVODB_U8; break;
    default: return false;
  }
  d.data = t.data_ptr();
  d.rank = (int32_t)t.dim();
  for (int i = 0; i < d.rank; ++i) d.shape[i] = t.size(i), d.stride[i] = t.stride(i);
  return true;
}
void desc_of(const at::Tensor& t, svodb_tensor& d, int dtype) {
  d.data = t.data_ptr();
  d.dtype = dtype;
  d.rank = (int32_t)t.dim();
  for (int i = 0; i < d.rank; ++i) d.shape[i] = t.size(i), d.stride[i] = t.stride(i);
}

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }

// A library call with the interpreter let go, as ctypes does it: a launch waits while the
// device's queue is full, and other Python threads run on meanwhile.
template <typename F>
int unlocked(F&& call) {
  PyThreadState* state = PyEval_SaveThread();
  const int rc = call();
  PyEval_RestoreThread(state);
  return rc;
}

PyObject* none() {
  PyErr_Clear();
  Py_RETURN_NONE;
}

// linear(x, w, opts)
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || p_linear == nullptr) return none();
  svodb_tensor x{}, w{}, y{}, bias{}, res{}, cos{}, sin{}, qn{}, kn{};
  if (!desc(args[0], x) || !desc(args[1], w) || w.rank != 2 || x.rank < 1) return none();
  svodb_linear_opts o{};
  svodb_qkv_opts qo{};
  PyObject* opts = args[2];
  if (opts != Py_None) {
    Ref into = attr(opts, s_into), ks = attr(opts, s_k_splits);
    if (into.o == nullptr || !into.none() || ks.o == nullptr) return none();
    if (!ks.none() && PyLong_AsLong(ks.o) > 1) return none();
    Ref b = attr(opts, s_bias), r = attr(opts, s_residual), act = attr(opts, s_act), gated = attr(opts, s_gated);
    Ref scale = attr(opts, s_scale), rope = attr(opts, s_rope), qkv = attr(opts, s_qkv), st = attr(opts, s_w_static);
    if (!b.none()) {
      if (!desc(b.o, bias)) return none();
      o.bias = &bias;
    }
    if (!r.none()) {
      if (!desc(r.o, res)) return none();
      o.residual = &res;
    }
    o.act = (int32_t)PyLong_AsLong(act.o) | (truth(st.o) ? SVODB_LINEAR_W_STATIC : 0);
    o.gated = truth(gated.o);
    if (!scale.none()) o.has_scale = 1, o.scale = (float)PyFloat_AsDouble(scale.o);
    if (!rope.none()) {
      Ref c = attr(rope.o, s_cos), s = attr(rope.o, s_sin), h = attr(rope.o, s_heads), d = attr(rope.o, s_head_dim);
      if (!desc(c.o, cos) || !desc(s.o, sin) || h.o == nullptr || d.o == nullptr) return none();
      o.rope_cos = &cos, o.rope_sin = &sin;
      o.rope_heads = (int32_t)PyLong_AsLong(h.o), o.rope_head_dim = (int32_t)PyLong_AsLong(d.o);
    }
    if (!qkv.none()) {
      Ref h = attr(qkv.o, s_heads), hk = attr(qkv.o, s_kv_heads), d = attr(qkv.o, s_head_dim), e = attr(qkv.o, s_eps);
      Ref q = attr(qkv.o, s_q_norm), k = attr(qkv.o, s_k_norm), t = attr(qkv.o, s_rope);
      if (h.o == nullptr || hk.o == nullptr || d.o == nullptr || e.o == nullptr) return none();
      qo.heads = (int32_t)PyLong_AsLong(h.o), qo.kv_heads = (int32_t)PyLong_AsLong(hk.o);
      qo.head_dim = (int32_t)PyLong_AsLong(d.o), qo.eps = PyFloat_AsDouble(e.o);
      if (!q.none()) {
        if (!desc(q.o, qn)) return none();
        qo.q_norm = &qn;
      }
      if (!k.none()) {
        if (!desc(k.o, kn)) return none();
        qo.k_norm = &kn;
      }
      if (!t.none()) {
        if (!PyTuple_Check(t.o) || PyTuple_GET_SIZE(t.o) != 2) return none();
        if (!desc(PyTuple_GET_ITEM(t.o, 0), cos) || !desc(PyTuple_GET_ITEM(t.o, 1), sin)) return none();
        qo.rope_cos = &cos, qo.rope_sin = &sin;
      }
      o.qkv = &qo;
    }
    if (PyErr_Occurred()) return none();
  }
  const at::Tensor& xt = THPVariable_Unpack(args[0]);
  int64_t shape[SVODB_MAX_RANK];
  for (int i = 0; i < x.rank; ++i) shape[i] = x.shape[i];
  shape[x.rank - 1] = o.gated ? w.shape[0] / 2 : w.shape[0];
  at::Tensor out = at::empty(at::IntArrayRef(shape, x.rank), xt.options());
  desc_of(out, y, x.dtype);
  void* st = stream();
  if (unlocked([&] { return p_linear(&x, &w, &o, &y, st); }) != SVODB_OK) return none();
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// The options of an attention. `keep` holds the descriptors the struct points at.
struct AttnKeep {
  svodb_tensor lens{}, mask{}, seg{}, bias{}, row_map{}, app_k{}, app_v{}, app_lens{}, lse{};
};

bool contiguous(const svodb_tensor& t) {
  int64_t e = 1;
  for (int i = t.rank - 1; i >= 0; --i) {
    if (t.shape[i] != 1 && t.stride[i] != e) return false;
    e *= t.shape[i];
  }
  return true;
}
bool i32(PyObject* o, svodb_tensor& d) { return desc(o, d) && d.dtype == SVODB_I32 && contiguous(d); }

bool attn_opts(PyObject* opts, svodb_attn_opts& o, AttnKeep& k, bool& want_lse) {
  want_lse = false;
  if (opts == Py_None) return true;
  Ref splits = attr(opts, s_splits), chunk = attr(opts, s_chunk);
  if (splits.o == nullptr || !splits.none() || chunk.o == nullptr || !chunk.none()) return false;
  Ref causal = attr(opts, s_causal), keys = attr(opts, s_keys), window = attr(opts, s_window), seg = attr(opts, s_seg_start);
  Ref scale = attr(opts, s_scale), bias = attr(opts, s_bias), cache = attr(opts, s_cache), lse = attr(opts, s_want_lse);
  o.causal = truth(causal.o);
  want_lse = truth(lse.o);
  if (!keys.none()) {
    Ref lens = attr(keys.o, s_lens), mask = attr(keys.o, s_mask);
    if (!lens.none()) {
      if (!i32(lens.o, k.lens)) return false;
      o.key_lens = &k.lens;
    }
    if (!mask.none()) {
      if (!desc(mask.o, k.mask) || !contiguous(k.mask) || (k.mask.dtype != SVODB_U8 && k.mask.dtype != SVODB_I32)) return false;
      o.key_mask = &k.mask;
    }
  }
  if (!window.none()) {
    if (!PyTuple_Check(window.o) || PyTuple_GET_SIZE(window.o) != 2) return false;
    o.has_window = 1;
    o.window_left = PyLong_AsLongLong(PyTuple_GET_ITEM(window.o, 0));
    o.window_right = PyLong_AsLongLong(PyTuple_GET_ITEM(window.o, 1));
  }
  if (!seg.none()) {
    if (!i32(seg.o, k.seg)) return false;
    o.seg_start = &k.seg;
  }
  if (!scale.none()) o.has_scale = 1, o.scale = (float)PyFloat_AsDouble(scale.o);
  if (!bias.none()) {
    if (!desc(bias.o, k.bias) || !contiguous(k.bias)) return false;
    o.bias = &k.bias;
  }
  if (!cache.none()) {
    Ref hs = attr(cache.o, s_head_start), kv = attr(cache.o, s_kv_heads), rm = attr(cache.o, s_row_map);
    Ref app = attr(cache.o, s_appended), al = attr(cache.o, s_app_lens);
    if (hs.o == nullptr || kv.o == nullptr) return false;
    o.has_cache = 1;
    o.cache_head_start = (int32_t)PyLong_AsLong(hs.o), o.cache_kv_heads = (int32_t)PyLong_AsLong(kv.o);
    if (!rm.none()) {
      if (!i32(rm.o, k.row_map)) return false;
      o.cache_row_map = &k.row_map;
    }
    if (!app.none()) {
      if (!PyTuple_Check(app.o) || PyTuple_GET_SIZE(app.o) != 2) return false;
      if (!desc(PyTuple_GET_ITEM(app.o, 0), k.app_k) || !contiguous(k.app_k)) return false;
      if (!desc(PyTuple_GET_ITEM(app.o, 1), k.app_v) || !contiguous(k.app_v)) return false;
      o.cache_app_k = &k.app_k, o.cache_app_v = &k.app_v;
    }
    if (!al.none()) {
      if (!i32(al.o, k.app_lens)) return false;
      o.cache_app_lens = &k.app_lens;
    }
  }
  return !PyErr_Occurred();
}

at::Tensor lse_for(const at::Tensor& like, int64_t B, int64_t H, int64_t T, svodb_attn_opts& o, AttnKeep& k) {
  at::Tensor lse = at::empty({B, H, T}, like.options().dtype(at::kFloat));
  desc_of(lse, k.lse, SVODB_F32);
  o.lse = &k.lse;
  return lse;
}

PyObject* with_lse(at::Tensor&& out, at::Tensor&& lse, bool want) {
  PyObject* a = THPVariable_Wrap(std::move(out));
  if (!want || a == nullptr) return a;
  PyObject* b = THPVariable_Wrap(std::move(lse));
  PyObject* t = PyTuple_Pack(2, a, b);
  Py_DECREF(a);
  Py_XDECREF(b);
  return t;
}

// attention(q, k, v, opts)
PyObject* attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || p_attention == nullptr) return none();
  svodb_tensor q{}, k{}, v{}, y{};
  if (!desc(args[0], q) || !desc(args[1], k) || !desc(args[2], v) || q.rank != 4) return none();
  svodb_attn_opts o{};
  AttnKeep keep;
  bool want = false;
  if (!attn_opts(args[3], o, keep, want)) return none();
  const at::Tensor& qt = THPVariable_Unpack(args[0]);
  at::Tensor out = at::empty(qt.sizes(), qt.options()), lse;
  desc_of(out, y, q.dtype);
  if (want) lse = lse_for(qt, q.shape[0], q.shape[2], q.shape[1], o, keep);
  void* st = stream();
  if (unlocked([&] { return p_attention(&q, &k, &v, &o, &y, st); }) != SVODB_OK) return none();
  return with_lse(std::move(out), std::move(lse), want);
  END_HANDLE_TH_ERRORS
}

// attention_packed(qkv, heads, kv_heads, opts)
PyObject* attention_packed(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || p_attention_packed == nullptr) return none();
  svodb_tensor x{}, y{};
  if (!desc(args[0], x) || x.rank != 3) return none();
  const long heads = PyLong_AsLong(args[1]), kv = PyLong_AsLong(args[2]);
  if (PyErr_Occurred() || heads <= 0 || kv <= 0 || heads % kv != 0 || x.shape[2] % (heads + 2 * kv) != 0) return none();
  svodb_attn_opts o{};
  AttnKeep keep;
  bool want = false;
  if (!attn_opts(args[3], o, keep, want)) return none();
  const at::Tensor& xt = THPVariable_Unpack(args[0]);
  const int64_t d = x.shape[2] / (heads + 2 * kv);
  at::Tensor out = at::empty({x.shape[0], x.shape[1], heads, d}, xt.options()), lse;
  desc_of(out, y, x.dtype);
  if (want) lse = lse_for(xt, x.shape[0], heads, x.shape[1], o, keep);
  void* st = stream();
  if (unlocked([&] { return p_attention_packed(&x, (int32_t)heads, (int32_t)kv, &o, &y, st); }) != SVODB_OK)
    return none();
  return with_lse(std::move(out), std::move(lse), want);
  END_HANDLE_TH_ERRORS
}

// norm(x, residual | None, w, b | None, eps, layer): the norm, or (sum, norm) with a residual
PyObject* norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || p_layer_norm == nullptr) return none();
  svodb_tensor x{}, r{}, w{}, b{}, y{}, s{};
  if (!desc(args[0], x) || !desc(args[2], w)) return none();
  const bool res = args[1] != Py_None, bias = args[3] != Py_None;
  if ((res && !desc(args[1], r)) || (bias && !desc(args[3], b))) return none();
  const double eps = PyFloat_AsDouble(args[4]);
  if (PyErr_Occurred()) return none();
  const bool layer = truth(args[5]);
  const at::Tensor& xt = THPVariable_Unpack(args[0]);
  if (!xt.is_contiguous()) return none();
  at::Tensor out = at::empty(xt.sizes(), xt.options()), sum;
  desc_of(out, y, x.dtype);
  if (res) {
    sum = at::empty(xt.sizes(), xt.options());
    desc_of(sum, s, x.dtype);
  }
  const svodb_tensor* bp = bias ? &b : nullptr;
  void* st = stream();
  const int rc = unlocked([&] {
    if (layer) return res ? p_add_layer_norm(&x, &r, &w, bp, eps, &s, &y, st) : p_layer_norm(&x, &w, bp, eps, &y, st);
    return res ? p_add_rms_norm(&x, &r, &w, eps, &s, &y, st) : p_rms_norm(&x, &w, eps, &y, st);
  });
  if (rc != SVODB_OK) return none();
  if (!res) return THPVariable_Wrap(std::move(out));
  PyObject* a = THPVariable_Wrap(std::move(sum));
  PyObject* c = THPVariable_Wrap(std::move(out));
  PyObject* t = PyTuple_Pack(2, a, c);
  Py_XDECREF(a);
  Py_XDECREF(c);
  return t;
  END_HANDLE_TH_ERRORS
}

// init(address of svodb_linear, svodb_attention, svodb_attention_packed, svodb_layer_norm,
// svodb_rms_norm, svodb_add_layer_norm, svodb_add_rms_norm)
PyObject* init(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 7) {
    PyErr_SetString(PyExc_TypeError, "seven entry point addresses");
    return nullptr;
  }
  void* p[7];
  for (int i = 0; i < 7; ++i) p[i] = PyLong_AsVoidPtr(args[i]);
  if (PyErr_Occurred()) return nullptr;
  p_linear = (decltype(p_linear))p[0];
  p_attention = (decltype(p_attention))p[1];
  p_attention_packed = (decltype(p_attention_packed))p[2];
  p_layer_norm = (decltype(p_layer_norm))p[3];
  p_rms_norm = (decltype(p_rms_norm))p[4];
  p_add_layer_norm = (decltype(p_add_layer_norm))p[5];
  p_add_rms_norm = (decltype(p_add_rms_norm))p[6];
#define INTERN(n) s_##n = PyUnicode_InternFromString(#n);
  NAMES(INTERN)
  Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {FAST(init), FAST(linear), FAST(attention), FAST(attention_packed), FAST(norm), {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fastops", "compiled call path of svod_b200.ops", -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__fastops(void) {
  PyObject* m = PyModule_Create(&kModule);
  if (m != nullptr) PyModule_AddStringConstant(m, "torch", SVODB_TORCH);  // the torch it was built for
  return m;
}
