// hostops.cpp -- the operators of a decoded token as a CPython extension module (illatio_b200._hostops).
//
// A decode step is a few hundred launches of one to ten microseconds, so what the host spends on one decides the
// token: through ctypes an operator cost 9.4 us (3.2 of them torch.cuda.current_stream(), 0.8 the conversion of
// the arguments, the rest attribute look-ups and the launch itself at 2.4), here it costs 3 (a B200 box's Xeon,
// D.cmat_mul of 896 x 896).  They are cuda_dense.py's operators: they read its objects (CMat, QAct) and call the same C
// ABI.  What is rare or long -- prefill chunks, activations whose fp16 form is in use, errors -- goes to the Python
// functions registered with set_slow().
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/ExpandUtils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/illatio_b200.h"

namespace {

PyObject* g_slow = nullptr;   // name -> Python function
long long g_launches = 0;     // launches made from this module (counted under the GIL): what bench.py counts

// attribute names, interned once
#define NAMES(X) \
  X(type) X(rows) X(cols) X(qs) X(kind) X(xq) X(xs) X(xsum) X(_cf) X(w) X(act) X(y) X(n) X(bias) X(acc) X(x) X(f16_scale) X(d) X(eps) \
  X(h) X(wq) X(wk) X(wv) X(q) X(k) X(v) X(bq) X(bk) X(bv) X(g) X(u) X(fa) X(fb) X(emb) X(tokens) X(quant_q8) X(rmsnorm_q8) \
  X(cmat_mul) X(glu_mul) X(qkv_mul) X(error) X(vars) X(TC_MIN_TOKENS) X(dk_mv16) X(route) X(dk_shared) X(dk_ffn_tail) X(logits) X(nu) \
  X(mode) X(scale) X(sh_gate) X(sh_up) X(sh_down) X(norm) X(clamp) X(out) X(pool) X(norm2) X(sel) X(shared) X(moe) X(ff) X(gate_fmt) \
  X(down_fmt) X(gate_bytes) X(ptrs_all) X(slot_ptrs)
#define DECL(s) PyObject* S_##s;
NAMES(DECL)
#undef DECL

struct Failed {};  // a Python error is set
// What ends every operator: no C++ exception may reach the interpreter's C frames.  Tensors without storage (sparse, inside
// vmap) and a stream that cannot be had throw c10::Error, which becomes the exception that torch's Python functions raise.
#define CATCH_ERRORS                        \
  catch (const Failed&) { return nullptr; } \
  catch (const std::exception&) { torch::translate_exception_to_python(std::current_exception()); return nullptr; }

inline ill_stream cur_stream() { return (ill_stream)c10::cuda::getCurrentCUDAStream().stream(); }

inline bool capturing() {
  cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing((cudaStream_t)cur_stream(), &s) == cudaSuccess && s != cudaStreamCaptureStatusNone;
}

// the address of a tensor's data (None: 0)
inline ill_dptr ptr(PyObject* o) {
  if (o == Py_None) return 0;
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "expected a tensor or None, got %s", Py_TYPE(o)->tp_name);
    throw Failed();
  }
  return (ill_dptr)(uintptr_t)THPVariable_Unpack(o).data_ptr();
}
inline const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "expected a tensor, got %s", Py_TYPE(o)->tp_name);
    throw Failed();
  }
  return THPVariable_Unpack(o);
}

struct Ref {  // an owned reference
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) { if (!o) throw Failed(); }
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
};
inline long long as_int(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw Failed();
  return v;
}
inline double as_float(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Failed();
  return v;
}
inline int as_bool(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw Failed();
  return v;
}
inline long long attr_int(PyObject* o, PyObject* name) { Ref r(PyObject_GetAttr(o, name)); return as_int(r.p); }
inline ill_dptr attr_ptr(PyObject* o, PyObject* name) { Ref r(PyObject_GetAttr(o, name)); return ptr(r.p); }

// a CMat
struct Mat {
  int type, rows, cols;
  ill_dptr w;
  explicit Mat(PyObject* o)
      : type((int)attr_int(o, S_type)), rows((int)attr_int(o, S_rows)), cols((int)attr_int(o, S_cols)), w(attr_ptr(o, S_qs)) {}
};
// a QAct
struct Act {
  bool k;         // Q8_K super-blocks
  bool has_f16;   // its fp16 form is in use
  ill_dptr xq, xs, xsum;
  explicit Act(PyObject* o) : xq(attr_ptr(o, S_xq)), xs(attr_ptr(o, S_xs)), xsum(attr_ptr(o, S_xsum)) {
    Ref kind(PyObject_GetAttr(o, S_kind));
    k = !(PyUnicode_Check(kind.p) && PyUnicode_GetLength(kind.p) == 2);
    PyObject* cf = PyObject_GetAttr(o, S__cf);  // an object of the caller's own may lack it
    if (!cf) {
      if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw Failed();
      PyErr_Clear();
    }
    has_f16 = cf && cf != Py_None;
    Py_XDECREF(cf);
  }
};

PyObject* slow(PyObject* name) {
  PyObject* f = g_slow ? PyDict_GetItemWithError(g_slow, name) : nullptr;
  if (!f && !PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "illatio_b200._hostops: set_slow() has not been called");
  if (!f) throw Failed();
  return f;
}
[[noreturn]] void raise_status(const char* fn, int rc) {
  PyObject* r = PyObject_CallFunction(slow(S_error), "si", fn, rc);
  Py_XDECREF(r);
  if (r) PyErr_Format(PyExc_RuntimeError, "%s failed with status %d", fn, rc);
  throw Failed();
}
// FN(ARGS...) without the GIL, which the arguments were made under: a launch waits while its stream's queue is full, and
// other threads, and host functions queued before it, go on meanwhile.
template <class... P, class... A>
inline int launch(int (*fn)(P...), A... args) {
  PyThreadState* const ts = PyEval_SaveThread();
  const int rc = fn((P)args...);
  PyEval_RestoreThread(ts);
  return rc;
}
inline void check(const char* name, int rc) {
  if (rc) raise_status(name, rc);
  ++g_launches;
}
#define LAUNCH(FN, ...) check(#FN, launch(FN, __VA_ARGS__))

// positional and keyword arguments into OUT (absent: null); the first REQUIRED must be there
void parse(const char* fn, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames, PyObject* const* names, int n, int required,
           PyObject** out) {
  if (nargs > n) {
    PyErr_Format(PyExc_TypeError, "%s() takes at most %d arguments (%zd given)", fn, n, nargs);
    throw Failed();
  }
  for (int i = 0; i < n; ++i) out[i] = i < nargs ? args[i] : nullptr;
  const Py_ssize_t nk = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  for (Py_ssize_t j = 0; j < nk; ++j) {
    PyObject* key = PyTuple_GET_ITEM(kwnames, j);
    int at = -1;
    for (int i = 0; i < n && at < 0; ++i)
      if (key == names[i]) at = i;
    for (int i = 0; i < n && at < 0; ++i)  // a key that is not the interned string
      if (PyUnicode_Compare(key, names[i]) == 0) at = i;
    if (at < 0 || out[at]) {
      PyErr_Format(PyExc_TypeError, "%s(): %s argument '%U'", fn, at < 0 ? "unexpected" : "repeated", key);
      throw Failed();
    }
    out[at] = args[nargs + j];
  }
  for (int i = 0; i < required; ++i)
    if (!out[i]) {
      PyErr_Format(PyExc_TypeError, "%s(): missing argument '%U'", fn, names[i]);
      throw Failed();
    }
}
#define ARGS(FN, REQUIRED, ...)                                        \
  PyObject* const names_[] = {__VA_ARGS__};                            \
  constexpr int n_ = (int)(sizeof(names_) / sizeof(names_[0]));        \
  PyObject* a[n_];                                                     \
  parse(FN, args, nargs, kwnames, names_, n_, REQUIRED, a)
#define OPT_INT(o, dflt) ((o) ? as_int(o) : (dflt))
#define OPT_BOOL(o, dflt) ((o) ? as_bool(o) : (dflt))
#define OPT_PTR(o) ((o) ? ptr(o) : 0)

inline PyObject* ret(PyObject* o) { Py_INCREF(o); return o; }

// ---- the operators ------------------------------------------------------------------

PyObject* quant_q8(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("quant_q8", 2, S_x, S_act, S_f16_scale);
  const Act act(a[1]);
  if (act.has_f16) return PyObject_Vectorcall(slow(S_quant_q8), args, nargs, kwnames);
  const at::Tensor& x = tensor(a[0]);
  const ill_dptr xp = (ill_dptr)(uintptr_t)x.data_ptr();
  if (act.k) LAUNCH(ill_quant_q8_k, xp, act.xq, act.xs, act.xsum, x.numel() / 256, cur_stream());
  else LAUNCH(ill_quant_q8_0, xp, act.xq, act.xs, act.xsum, x.numel() / 32, OPT_BOOL(a[2], 1), cur_stream());
  return ret(a[1]);
} CATCH_ERRORS

PyObject* rmsnorm_q8(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("rmsnorm_q8", 5, S_x, S_w, S_act, S_d, S_eps, S_n, S_h, S_f16_scale);
  const Act act(a[2]);
  if (act.has_f16) return PyObject_Vectorcall(slow(S_rmsnorm_q8), args, nargs, kwnames);
  LAUNCH(ill_rmsnorm_q8, act.k ? 1 : 0, ptr(a[0]), ptr(a[1]), OPT_PTR(a[6]), act.xq, act.xs, act.xsum, (int)as_int(a[3]), (float)as_float(a[4]),
         OPT_INT(a[5], 1), OPT_BOOL(a[7], 1), cur_stream());
  return ret(a[2]);
} CATCH_ERRORS

// Y = W X for up to 16 tokens in one launch; false when the shape wants the tokens split (the Python form does that)
inline bool mul(const Mat& w, const Act& act, ill_dptr y, int n, ill_dptr bias, int acc) {
  const int rc = launch(ill_mv, w.type, w.w, w.rows, w.cols, act.xq, act.xs, act.k ? act.xsum : 0, y, bias, acc, n, cur_stream());
  if (rc == ILL_ERR_UNSUPPORTED && n > 1) return false;
  check("ill_mv", rc);
  return true;
}
// Whether N tokens are few; more are a chunk, and the Python form picks the kernel.  So it does from cuda_dense.TC_MIN_TOKENS on.
inline bool few(long long n) {
  if (n < 1 || n > 16) return false;
  PyObject* v = PyDict_GetItemWithError(slow(S_vars), S_TC_MIN_TOKENS);
  if (!v && PyErr_Occurred()) throw Failed();
  return !v || n < as_int(v);
}

PyObject* cmat_mul(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("cmat_mul", 3, S_w, S_act, S_y, S_n, S_bias, S_acc);
  const long long n = OPT_INT(a[3], 1);
  if (!few(n) || !mul(Mat(a[0]), Act(a[1]), ptr(a[2]), (int)n, OPT_PTR(a[4]), OPT_BOOL(a[5], 0)))
    return PyObject_Vectorcall(slow(S_cmat_mul), args, nargs, kwnames);
  return ret(a[2]);
} CATCH_ERRORS

void mul_any(PyObject* w, PyObject* act, PyObject* y, long long n, PyObject* bias) {
  if (few(n) && mul(Mat(w), Act(act), ptr(y), (int)n, bias ? ptr(bias) : 0, 0)) return;
  PyObject* nn = PyLong_FromLongLong(n);
  Ref hold(nn);
  PyObject* av[5] = {w, act, y, nn, bias ? bias : Py_None};
  Ref r(PyObject_Vectorcall(slow(S_cmat_mul), av, 5, nullptr));
}

// Up to three products of up to 16 tokens that share the activations, in one launch (C null: two); false where that is not to be had
inline bool mul_3(const Mat& a, const Mat& b, const Mat* c, const Act& x, ill_dptr ya, ill_dptr yb, ill_dptr yc, ill_dptr ba, ill_dptr bb,
                  ill_dptr bc, int n) {
  // (a Q8_0 matrix takes other activations than the K formats: not with them; a third of no rows, which ill_mv_3n would take for
  // none, is refused by the product of its own)
  if (c && c->rows < 1) return false;
  if ((a.type == 0) != (b.type == 0) || a.cols != b.cols || (c && ((c->type == 0) != (a.type == 0) || c->cols != a.cols))) return false;
  const int rc = launch(ill_mv_3n, a.type, b.type, c ? c->type : 0, a.w, b.w, c ? c->w : 0, a.rows, b.rows, c ? c->rows : 0, a.cols, x.xq, x.xs, x.k ? x.xsum : 0, ya, yb,
                        yc, ba, bb, bc, n, cur_stream());
  if (rc == ILL_ERR_UNSUPPORTED) return false;
  check("ill_mv_3n", rc);
  return true;
}

PyObject* qkv_mul(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("qkv_mul", 7, S_wq, S_wk, S_wv, S_act, S_q, S_k, S_v, S_bq, S_bk, S_bv, S_n);
  const long long n = OPT_INT(a[10], 1);
  if (n == 1) {
    const Mat q(a[0]), k(a[1]), v(a[2]);
    if (q.type == k.type) {
      const Act x(a[3]);
      const bool three = k.type == v.type;
      // Q4_K_M files keep V in Q6_K: V in a launch of its own.  In a stream that is being captured the Python form runs
      // it beside Q and K (a fork and a join cost a graph nothing: a 4B token 1.54 ms, 1.57 one after the other).  Launch
      // by launch, the fork's events and calls cost the host 21 us, and where the GPU is the bound all the same the overlap
      // gives nothing: a layer's products one after the other and with the fork take 26 and 45 us at a hidden size of
      // 1024, 41 and 47 at 2560, 58.4 and 58.5 at 4096, 81.6 and 82.3 at 5120, 137.2 and 137.4 at 8192.
      if (!three && capturing()) return PyObject_Vectorcall(slow(S_qkv_mul), args, nargs, kwnames);
      LAUNCH(ill_mv_3, q.type, q.w, k.w, three ? v.w : 0, q.rows, k.rows, three ? v.rows : 0, q.cols, x.xq, x.xs, x.k ? x.xsum : 0, ptr(a[4]),
             ptr(a[5]), three ? ptr(a[6]) : 0, OPT_PTR(a[7]), OPT_PTR(a[8]), three ? OPT_PTR(a[9]) : 0, cur_stream());
      if (!three) mul(v, x, ptr(a[6]), 1, OPT_PTR(a[9]), 0);
      Py_RETURN_NONE;
    }
  }
  if (n > 1 && !few(n)) return PyObject_Vectorcall(slow(S_qkv_mul), args, nargs, kwnames);  // a chunk
  int left = 0;
  if (n > 1) {
    const Mat q(a[0]), k(a[1]), v(a[2]);
    const Act x(a[3]);
    if (mul_3(q, k, &v, x, ptr(a[4]), ptr(a[5]), ptr(a[6]), OPT_PTR(a[7]), OPT_PTR(a[8]), OPT_PTR(a[9]), (int)n)) left = 3;
    else if (mul_3(q, k, nullptr, x, ptr(a[4]), ptr(a[5]), 0, OPT_PTR(a[7]), OPT_PTR(a[8]), 0, (int)n)) left = 2;
  }
  for (int i = left; i < 3; ++i) mul_any(a[i], a[3], a[4 + i], n, a[7 + i]);
  Py_RETURN_NONE;
} CATCH_ERRORS

PyObject* glu_mul(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("glu_mul", 4, S_g, S_u, S_act, S_fa, S_n, S_fb);
  const long long n = OPT_INT(a[4], 1);
  if (n == 1) {
    const Mat g(a[0]), u(a[1]);
    if (g.type == u.type) {
      const Act x(a[2]);
      LAUNCH(ill_mv_glu, g.type, g.w, u.w, g.rows, g.cols, x.xq, x.xs, x.k ? x.xsum : 0, ptr(a[3]), cur_stream());
      return ret(a[3]);
    }
  }
  if (n >= 1 && a[5] && a[5] != Py_None) {
    // the buffers may be longer than N tokens take (a serving loop's largest batch), but have to agree
    const at::Tensor &fa = tensor(a[3]), &fb = tensor(a[5]);
    const long long len = n * attr_int(a[0], S_rows);
    if (!at::is_expandable_to(fb.sizes(), fa.sizes()) || fa.numel() < len || fb.numel() < len) {
      PyErr_Format(PyExc_RuntimeError, "glu_mul(): FA of %lld values and FB of %lld do not agree, or hold fewer than N * ROWS = %lld",
                   (long long)fa.numel(), (long long)fb.numel(), len);
      throw Failed();
    }
    const Mat g(a[0]), u(a[1]);
    if (!(n > 1 && few(n) && g.rows == u.rows && g.type == u.type && mul_3(g, u, nullptr, Act(a[2]), ptr(a[3]), ptr(a[5]), 0, 0, 0, 0, (int)n))) {
      mul_any(a[0], a[2], a[3], n, nullptr);
      mul_any(a[1], a[2], a[5], n, nullptr);
    }
    const ill_dptr fp = ptr(a[3]);
    LAUNCH(ill_silu_mul, len, fp, ptr(a[5]), fp, cur_stream());
    return ret(a[3]);
  }
  return PyObject_Vectorcall(slow(S_glu_mul), args, nargs, kwnames);
} CATCH_ERRORS

PyObject* embed(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("embed", 3, S_emb, S_tokens, S_x);
  const Mat m(a[0]);
  const at::Tensor& t = tensor(a[1]);
  LAUNCH(ill_dequant_rows, m.type, m.w, m.cols, (ill_dptr)(uintptr_t)t.data_ptr(), 0, (int)t.numel(), ptr(a[2]), cur_stream());
  return ret(a[2]);
} CATCH_ERRORS

// ---- a token's mixture-of-experts layer (cuda_ds4f.py) --------------------------------------
// The Python forms' steps; what they do not take in one piece -- other types, shapes and layouts -- goes to those.

// device memory of a call's own: N bytes each, 256 apart, from one allocation on the current stream
struct Scratch {
  at::Tensor t;
  ill_dptr next;
  Scratch(const at::Tensor& like, long long bytes)
      : t(at::empty({bytes}, like.options().dtype(at::kByte).requires_grad(false))), next((ill_dptr)(uintptr_t)t.data_ptr()) {}
  ill_dptr take(long long bytes) {
    const ill_dptr p = next;
    next += (bytes + 255) / 256 * 256;
    return p;
  }
};
inline bool plain(const at::Tensor& t, at::ScalarType type) { return t.is_cuda() && t.scalar_type() == type && t.is_contiguous(); }

PyObject* dk_mv16(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("dk_mv16", 3, S_w, S_x, S_y, S_n);
  const at::Tensor& w = tensor(a[0]);
  const int type = w.scalar_type() == at::kFloat ? 0 : w.scalar_type() == at::kHalf ? 1 : w.scalar_type() == at::kBFloat16 ? 2 : -1;
  if (type < 0 || w.dim() != 2) return PyObject_Vectorcall(slow(S_dk_mv16), args, nargs, kwnames);
  LAUNCH(ill_mv_dense, type, ptr(a[0]), (int)w.size(0), (int)w.size(1), ptr(a[1]), ptr(a[2]), (int)OPT_INT(a[3], 1), w.size(0), cur_stream());
  return ret(a[2]);
} CATCH_ERRORS

PyObject* route(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("route", 2, S_logits, S_nu, S_mode, S_bias, S_scale);
  const at::Tensor& l = tensor(a[0]);
  const long long nu = as_int(a[1]);
  if (l.dim() != 2 || nu < 1) return PyObject_Vectorcall(slow(S_route), args, nargs, kwnames);
  at::Tensor sel = at::empty({l.size(0), nu}, l.options().dtype(at::kInt).requires_grad(false)),
             w = at::empty({l.size(0), nu}, l.options().dtype(at::kFloat).requires_grad(false));
  LAUNCH(ill_moe_route, (int)l.size(1), (int)nu, (int)OPT_INT(a[2], 2), (float)(a[4] ? as_float(a[4]) : 1.0), l.size(0), ptr(a[0]), OPT_PTR(a[3]),
         (ill_dptr)(uintptr_t)sel.data_ptr(), (ill_dptr)(uintptr_t)w.data_ptr(), cur_stream());
  Ref ps(THPVariable_Wrap(sel)), pw(THPVariable_Wrap(w));
  return PyTuple_Pack(2, ps.p, pw.p);
} CATCH_ERRORS

PyObject* dk_shared(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("dk_shared", 6, S_sh_gate, S_sh_up, S_sh_down, S_norm, S_clamp, S_out);
  const Mat g(a[0]), u(a[1]), d(a[2]);
  const at::Tensor& x = tensor(a[3]);
  if (g.type || u.type || d.type || u.rows != g.rows || u.cols != g.cols || d.cols != g.rows || x.numel() != g.cols || !plain(x, at::kFloat))
    return PyObject_Vectorcall(slow(S_dk_shared), args, nargs, kwnames);
  const long long c = g.cols, ff = g.rows;
  Scratch s(x, c + c / 8 + ff + ff / 8 + 12 * ff + 7 * 256);
  const ill_stream st = cur_stream();
  const ill_dptr xq = s.take(c), xs = s.take(c / 8), yg = s.take(4 * ff), yu = s.take(4 * ff), mid = s.take(4 * ff), mq = s.take(ff), ms = s.take(ff / 8);
  LAUNCH(ill_quant_q8_0, ptr(a[3]), xq, xs, 0, c / 32, 0, st);
  LAUNCH(ill_mv_3, 0, g.w, u.w, 0, g.rows, u.rows, 0, g.cols, xq, xs, 0, yg, yu, 0, 0, 0, 0, st);
  LAUNCH(ill_swiglu_w, ff, (int)ff, (float)as_float(a[4]), yg, yu, 0, mid, st);
  LAUNCH(ill_quant_q8_0, mid, mq, ms, 0, ff / 32, 0, st);
  LAUNCH(ill_mv, 0, d.w, d.rows, d.cols, mq, ms, 0, ptr(a[5]), 0, 0, 1, st);
  return ret(a[5]);
} CATCH_ERRORS

// Whether a pool's slot_ptrs() is ExpertPool's own, which reads its ptrs_all: not a subclass's, or an object's with a table elsewhere
inline bool own_slots(PyObject* pool) {
  Ref m(PyObject_GetAttr(pool, S_slot_ptrs));
  return PyMethod_Check(m.p) && PyMethod_GET_SELF(m.p) == pool && PyMethod_GET_FUNCTION(m.p) == slow(S_slot_ptrs);
}

PyObject* dk_ffn_tail(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) try {
  ARGS("dk_ffn_tail", 5, S_pool, S_norm2, S_sel, S_w, S_clamp, S_shared, S_moe);
  const at::Tensor &x = tensor(a[1]), &sel = tensor(a[2]);
  const long long d = attr_int(a[0], S_d), ff = attr_int(a[0], S_ff), k = sel.numel();
  if (!plain(x, at::kFloat) || !plain(sel, at::kInt) || x.numel() != d || d % 256 || ff % 256 || k < 1 || !own_slots(a[0]))
    return PyObject_Vectorcall(slow(S_dk_ffn_tail), args, nargs, kwnames);
  const Ref table(PyObject_GetAttr(a[0], S_ptrs_all));
  const at::Tensor& all = tensor(table.p);
  if (!plain(all, at::kLong) || all.dim() != 1 || all.device() != sel.device())
    return PyObject_Vectorcall(slow(S_dk_ffn_tail), args, nargs, kwnames);
  const long long gb = attr_int(a[0], S_gate_bytes), ne = all.numel();
  const ill_dptr ptrs = ptr(table.p), sp = ptr(a[2]);
  const ill_stream st = cur_stream();
  const auto f32 = x.options().requires_grad(false);
  Scratch s(x, d + d / 64 + d / 8 + k * (ff + ff / 64 + ff / 8) + 4 * k * d + 8 * 256);
  const ill_dptr xq = s.take(d), xs = s.take(d / 64), xsum = s.take(d / 8), mq = s.take(k * ff), ms = s.take(k * ff / 64),
                 msum = s.take(k * ff / 8), down = s.take(4 * k * d);
  at::Tensor mid = at::empty({k * ff}, f32);
  const ill_dptr mp = (ill_dptr)(uintptr_t)mid.data_ptr();
  LAUNCH(ill_quant_q8_k, ptr(a[1]), xq, xs, xsum, d / 256, st);
  LAUNCH(ill_moe_glu_sel, (int)attr_int(a[0], S_gate_fmt), (int)d, (int)ff, 0, gb, ptrs, (int)ne, sp, (int)k, xq, xs, xsum, 0, (float)as_float(a[4]),
         ptr(a[3]), mp, ff, st);
  // a slot's FF values are whole super-blocks: quantized apart (src/ds4f.lisp:1021-1022)
  LAUNCH(ill_quant_q8_k, mp, mq, ms, msum, k * ff / 256, st);
  LAUNCH(ill_moe_mv_sel, (int)attr_int(a[0], S_down_fmt), (int)ff, (int)d, 2 * gb, ptrs, (int)ne, sp, (int)k, mq, ms, msum, 1, down, d, st);
  Ref moe(a[6] && a[6] != Py_None ? ret(a[6]) : THPVariable_Wrap(at::empty({d}, f32)));
  LAUNCH(ill_moe_sum, (int)d, (int)k, 1, down, 0, OPT_PTR(a[5]), ptr(moe.p), st);
  Ref pm(THPVariable_Wrap(mid));
  return PyTuple_Pack(2, moe.p, pm.p);
} CATCH_ERRORS

PyObject* launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches); }

PyObject* set_slow(PyObject*, PyObject* d) {
  if (!PyDict_Check(d)) { PyErr_SetString(PyExc_TypeError, "set_slow() takes a dict"); return nullptr; }
  Py_INCREF(d);
  Py_XSETREF(g_slow, d);
  Py_RETURN_NONE;
}

#define FAST(name, text) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL | METH_KEYWORDS, text}
PyMethodDef methods[] = {
    FAST(quant_q8,
         "quant_q8(x, act, f16_scale=True)\n--\n\nX (float32, a whole number of blocks) quantized into ACT: the reference's quant_q8 launch\n"
         "(src/cuda-dense.lisp:366,417), in the kind ACT holds."),
    FAST(rmsnorm_q8,
         "rmsnorm_q8(x, w, act, d, eps, n=1, h=None, f16_scale=True)\n--\n\nRMSNORM-Q8 (src/cuda-dense.lisp:260-264): RMSNORM! of N rows of X\n"
         "(D wide) by W, quantized into ACT in the kind it holds; H, when given, also gets the floats."),
    FAST(cmat_mul,
         "cmat_mul(w, act, y, n=1, bias=None, acc=False)\n--\n\nCMAT-MUL (src/cuda-dense.lisp:220-248): Y = W X for N tokens (token t's X at\n"
         "t*cols, its Y at t*rows), or Y += it when ACC."),
    FAST(qkv_mul,
         "qkv_mul(wq, wk, wv, act, q, k, v, bq=None, bk=None, bv=None, n=1)\n--\n\nQKV-MUL (src/cuda-dense.lisp:309-324): for up to 16\n"
         "tokens one launch when the three formats agree (for several also when they are Q4_K and Q6_K), two when those of Q and\n"
         "K do; else three products."),
    FAST(glu_mul,
         "glu_mul(g, u, act, fa, n=1, fb=None)\n--\n\nGLU-MUL (src/cuda-dense.lisp:326-339): silu(G x) * (U x) into FA; FB, of\n"
         "FA's shape, is scratch for the products that one launch does not take."),
    FAST(embed,
         "embed(emb, tokens, x)\n--\n\nEMBED (src/cuda-dense.lisp:302-307): rows TOKENS (int32 on the device) of EMB as floats in X."),
    FAST(dk_mv16,
         "dk_mv16(w, x, y, n=1)\n--\n\nDK-MV16 (src/cuda-ds4f.lisp:767-771): Y = W X for an unquantized tensor W [rows, cols]\n"
         "(float32, float16 or bfloat16 on the device) and N tokens' float activations."),
    FAST(route,
         "route(logits, nu, mode=2, bias=None, scale=1.0)\n--\n\nD4-ROUTE / G53-ROUTE on the device for every row of LOGITS [n, ne]."),
    FAST(dk_shared,
         "dk_shared(sh_gate, sh_up, sh_down, norm, clamp, out)\n--\n\nThe shared expert as DK-FFN-HEAD runs it\n"
         "(src/cuda-ds4f.lisp:900-906): D4-SHARED! (src/ds4f.lisp:1039-1048)."),
    FAST(dk_ffn_tail,
         "dk_ffn_tail(pool, norm2, sel, w, clamp, shared=None, moe=None)\n--\n\nDK-FFN-TAIL (src/cuda-ds4f.lisp:908-956) for one token:\n"
         "the routed experts SEL (device int32 [k]) with weights W (device float [k]) on the FFN input NORM2, summed in SEL's order\n"
         "with the shared expert's output SHARED."),
    {"launches", launches, METH_NOARGS, "Launches made by this module since it was loaded."},
    {"set_slow", set_slow, METH_O, "Python functions for what this module leaves to Python: {name: function}."},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hostops", "Native host side of the decode operators.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__hostops(void) {
#define INTERN(s) if (!(S_##s = PyUnicode_InternFromString(#s))) return nullptr;
  NAMES(INTERN)
#undef INTERN
  return PyModule_Create(&module);
}
