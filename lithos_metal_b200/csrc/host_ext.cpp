// The native call path of the Python layer: tensors and knobs straight into the C ABI's argument structures.
//
// A call of a few rows lasts ~10 us on the GPU; filling a ctypes structure field by field, looking up streams and allocating the
// results from Python took ~25 us of host time around it, so the host was the bound of every small call. Each function here takes the
// ordinary case -- CUDA tensors of the right type, device and layout -- in one go and answers None for anything else; the Python
// function then does what it always did (conversions, copies, error messages). Measured on one FP32 row (top_k, top_p): see sampler.py.
//
// The ABI functions are called through addresses that the ctypes binding hands over (init), so that exactly one library is in use.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <mutex>
#include <tuple>

#include "../../include/lithos_b200.h"

namespace {

struct Abi {
  decltype(&lm_sample) sample = nullptr;
  decltype(&lm_argmax) argmax = nullptr;
  decltype(&lm_argmax_i64) argmax_i64 = nullptr;
  decltype(&lm_verify) verify = nullptr;
  decltype(&lm_draft_q) draft_q = nullptr;
  decltype(&lm_head) head = nullptr;
  decltype(&lm_workspace_bytes) workspace_bytes = nullptr;
  decltype(&lm_verify_workspace_bytes) verify_workspace_bytes = nullptr;
} abi;

PyObject *params_type = nullptr, *output_type = nullptr, *draft_type = nullptr, *check_fn = nullptr, *workspace_fn = nullptr;
// interned attribute names
PyObject *n_temperature, *n_top_k, *n_top_p, *n_min_p, *n_seed, *n_topp_in_topk, *n_rho, *n_pi, *n_draw, *n_exact_only, *n_grid_limit, *n_gumbel, *n_inverse_cdf;

struct Ref {                                                                // an owned reference
  PyObject* p;
  explicit Ref(PyObject* o = nullptr) : p(o) {}
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
  PyObject* release() { PyObject* o = p; p = nullptr; return o; }
};

inline PyObject* none() { Py_RETURN_NONE; }
inline const at::Tensor* as_tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }
inline int dtype_code(const at::Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? LM_DTYPE_BF16 : t.scalar_type() == at::kFloat ? LM_DTYPE_F32 : -1;
}
// [rows, vocab] on a CUDA device, a supported type, unit stride along the vocabulary
inline bool plain_rows(const at::Tensor& t) { return t.is_cuda() && t.dim() == 2 && dtype_code(t) >= 0 && t.stride(1) == 1; }
inline int64_t row_stride(const at::Tensor& t) { return t.size(0) > 1 ? t.stride(0) : std::max(t.stride(0), t.size(1)); }
inline bool plain_vector(const at::Tensor& t, at::ScalarType type, const at::Device& dev, int64_t n) {
  return t.scalar_type() == type && t.device() == dev && t.numel() == n && t.is_contiguous();
}
inline at::Tensor make(std::initializer_list<int64_t> sizes, at::ScalarType type, const at::Device& dev) {
  return at::detail::empty_cuda(at::IntArrayRef(sizes), type, dev, c10::nullopt);
}
inline void* ptr(const at::Tensor& t) { return const_cast<void*>(t.const_data_ptr()); }

// A knob: a number (scalar set) or a tensor of one value per row (*array set); false: not the ordinary case.
bool knob_f(PyObject* o, int64_t rows, const at::Device& dev, const float** array, float* scalar) {
  if (PyFloat_Check(o)) { *scalar = static_cast<float>(PyFloat_AS_DOUBLE(o)); return true; }
  if (PyLong_CheckExact(o)) { const double d = PyLong_AsDouble(o); if (d == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; } *scalar = static_cast<float>(d); return true; }
  const at::Tensor* t = as_tensor(o);
  if (!t || !plain_vector(*t, at::kFloat, dev, rows)) return false;
  *array = static_cast<const float*>(t->const_data_ptr());
  return true;
}
bool knob_i(PyObject* o, int64_t rows, const at::Device& dev, const int32_t** array, int32_t* scalar) {
  if (PyLong_CheckExact(o)) {
    int overflow = 0;
    const long v = PyLong_AsLongAndOverflow(o, &overflow);
    if (overflow || v < INT32_MIN || v > INT32_MAX) return false;
    *scalar = static_cast<int32_t>(v);
    return true;
  }
  const at::Tensor* t = as_tensor(o);
  if (!t || !plain_vector(*t, at::kInt, dev, rows)) return false;
  *array = static_cast<const int32_t*>(t->const_data_ptr());
  return true;
}
bool as_u64(PyObject* o, uint64_t* v) {                                     // an int, modulo 2^64
  if (!PyLong_Check(o)) return false;
  *v = PyLong_AsUnsignedLongLongMask(o);
  if (*v == static_cast<uint64_t>(-1) && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}

// The stream's scratch (one per device, kind and stream; made and owned by the Python layer, which keeps it for its own calls too).
// Remembered here with a reference of its own; asked for again when it is too small. A call is several launches that pass rows on in this
// scratch, and it runs without the GIL: two threads on one stream take turns.
struct Scratch { at::Tensor t; std::mutex turn; };
auto& scratches = *new std::map<std::tuple<int, int, void*>, Scratch>;     // (never destroyed: at exit the allocator may be gone before it)
struct Lease { at::Tensor t; std::mutex* turn = nullptr; };                  // (holds the buffer: another thread may replace it meanwhile)
bool scratch(const at::Device& dev, void* stream, int kind, size_t bytes, Lease* lease, void** p, size_t* n) {
  Scratch& s = scratches[std::make_tuple(static_cast<int>(dev.index()), kind, stream)];
  if (!s.t.defined() || static_cast<size_t>(s.t.numel()) < bytes) {
    Ref d(THPVariable_Wrap(at::detail::empty_cuda({0}, at::kByte, dev, c10::nullopt)));
    if (!d.p) return false;
    Ref device(PyObject_GetAttrString(d.p, "device"));
    if (!device.p) return false;
    Ref w(PyObject_CallFunction(workspace_fn, "Ons", device.p, static_cast<Py_ssize_t>(bytes), kind ? "verify" : "sample"));
    if (!w.p) return false;
    const at::Tensor* t = as_tensor(w.p);
    if (!t) { PyErr_SetString(PyExc_TypeError, "workspace"); return false; }
    s.t = *t;
  }
  lease->t = s.t; lease->turn = &s.turn;
  *p = ptr(s.t);
  *n = static_cast<size_t>(s.t.numel());
  return true;
}

// An ABI call, without the GIL as a ctypes call is: a launch can wait (a full launch queue, the first use of a kernel).
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};
template <class F>
int call(const at::Device& dev, std::mutex* turn, F f) {
  const NoGil released;                                                     // (taken back last, also when the guard throws)
  std::unique_lock<std::mutex> lock;
  if (turn) lock = std::unique_lock<std::mutex>(*turn);
  const c10::cuda::CUDAGuard guard(dev);
  return f();
}

PyObject* failed(int rc, const char* what) {                                // the Python layer's exception for an ABI error code
  Ref r(PyObject_CallFunction(check_fn, "is", rc, what));
  if (r.p) PyErr_SetString(PyExc_RuntimeError, what);
  return nullptr;
}

enum { kTau = 1, kStats = 2, kProbs = 4, kStatus = 8, kVmax = 16, kI64 = 32 };

// The outputs of a sampling call and the call itself; `a` holds everything else. Returns a SampleOutput, or the tokens alone (kI64).
PyObject* run_sample(lm_sample_args& a, const at::Tensor& x, PyObject* out, int want) {
  const at::Device dev = x.device();
  const int64_t rows = x.size(0), vocab = x.size(1);
  at::Tensor tokens, tau, stats, probs, status, vmax, mass;
  if (out == Py_None) tokens = make({rows}, (want & kI64) ? at::kLong : at::kInt, dev);
  else {
    const at::Tensor* t = as_tensor(out);
    if (!t || !plain_vector(*t, at::kInt, dev, rows)) return none();
    tokens = *t;
  }
  a.struct_size = sizeof(a);
  a.dtype = dtype_code(x);
  a.logits = ptr(x); a.rows = rows; a.vocab = vocab; a.row_stride = row_stride(x);
  a.out_tokens = static_cast<int32_t*>(ptr(tokens));
  if (want & kI64) a.flags |= LM_FLAG_TOKENS_I64;
  if (want & kTau) { tau = make({rows}, at::kFloat, dev); a.out_tau = static_cast<float*>(ptr(tau)); }
  if (want & kStats) { stats = make({rows, 2}, at::kFloat, dev); a.out_stats = static_cast<float*>(ptr(stats)); }
  if (want & kProbs) { probs = make({rows, vocab}, at::kFloat, dev); a.out_probs = static_cast<float*>(ptr(probs)); a.probs_stride = vocab; }
  if (want & kStatus) { status = make({rows}, at::kInt, dev); a.out_status = static_cast<uint32_t*>(ptr(status)); }
  if (want & kVmax) {
    vmax = make({rows}, at::kFloat, dev); a.out_vmax = static_cast<float*>(ptr(vmax));
    mass = make({rows}, at::kLong, dev); a.out_mass = static_cast<uint64_t*>(ptr(mass));
  }
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  a.stream = stream;
  Lease lease;
  if (!scratch(dev, stream, 0, abi.workspace_bytes(rows, vocab), &lease, &a.workspace, &a.workspace_bytes)) return nullptr;
  const int rc = call(dev, lease.turn, [&] { return abi.sample(&a); });
  if (rc != LM_OK) return failed(rc, "lm_sample");
  if (want & kI64) return THPVariable_Wrap(tokens);
  auto wrap = [](const at::Tensor& t) { if (t.defined()) return THPVariable_Wrap(t); Py_INCREF(Py_None); return Py_None; };
  Ref o0(out == Py_None ? THPVariable_Wrap(tokens) : (Py_INCREF(out), out)), o1(wrap(tau)), o2(wrap(stats)), o3(wrap(probs)), o4(wrap(status)), o5(wrap(vmax)), o6(wrap(mass));
  PyObject* args[7] = {o0.p, o1.p, o2.p, o3.p, o4.p, o5.p, o6.p};
  for (PyObject* o : args) if (!o) return nullptr;
  return PyObject_Vectorcall(output_type, args, 7, nullptr);
}

// sample(logits, params, history, uniforms, step, row_offset, want, out)
PyObject* py_sample(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8) { PyErr_SetString(PyExc_TypeError, "sample: 8 arguments"); return nullptr; }
  const at::Tensor* x = as_tensor(args[0]);
  PyObject* p = args[1];
  if (!x || !plain_rows(*x) || reinterpret_cast<PyObject*>(Py_TYPE(p)) != params_type) return none();
  const at::Device dev = x->device();
  const int64_t rows = x->size(0);
  lm_sample_args a{};
  Ref temperature(PyObject_GetAttr(p, n_temperature)), top_k(PyObject_GetAttr(p, n_top_k)), top_p(PyObject_GetAttr(p, n_top_p)), min_p(PyObject_GetAttr(p, n_min_p)),
      seed(PyObject_GetAttr(p, n_seed)), in_topk(PyObject_GetAttr(p, n_topp_in_topk)), rho(PyObject_GetAttr(p, n_rho)), pi(PyObject_GetAttr(p, n_pi)),
      draw(PyObject_GetAttr(p, n_draw)), exact(PyObject_GetAttr(p, n_exact_only)), limit(PyObject_GetAttr(p, n_grid_limit));
  if (!temperature.p || !top_k.p || !top_p.p || !min_p.p || !seed.p || !in_topk.p || !rho.p || !pi.p || !draw.p || !exact.p || !limit.p) { PyErr_Clear(); return none(); }
  if (!knob_f(temperature.p, rows, dev, &a.temperature, &a.temperature_s) || !knob_i(top_k.p, rows, dev, &a.top_k, &a.top_k_s) ||
      !knob_f(top_p.p, rows, dev, &a.top_p, &a.top_p_s) || !knob_f(min_p.p, rows, dev, &a.min_p, &a.min_p_s)) return none();
  if (!a.temperature && !(a.temperature_s >= 0.0f)) return none();
  bool inverse;
  if (draw.p == n_gumbel) inverse = false;
  else if (draw.p == n_inverse_cdf) inverse = true;
  else if (PyUnicode_Check(draw.p) && PyUnicode_CompareWithASCIIString(draw.p, "gumbel") == 0) inverse = false;
  else if (PyUnicode_Check(draw.p) && PyUnicode_CompareWithASCIIString(draw.p, "inverse_cdf") == 0) inverse = true;
  else return none();
  a.draw = inverse ? LM_DRAW_INVERSE_CDF : LM_DRAW_GUMBEL;
  if (!PyFloat_Check(rho.p) || !PyFloat_Check(pi.p) || !PyBool_Check(in_topk.p) || !PyBool_Check(exact.p) || !PyLong_Check(limit.p)) return none();
  a.repetition_penalty = static_cast<float>(PyFloat_AS_DOUBLE(rho.p)); a.presence_penalty = static_cast<float>(PyFloat_AS_DOUBLE(pi.p));
  if (!(PyFloat_AS_DOUBLE(rho.p) > 0.0)) return none();
  uint64_t grid = 0, step = 0, offset = 0;
  if (!as_u64(limit.p, &grid) || !as_u64(seed.p, &a.seed) || !as_u64(args[4], &step) || !as_u64(args[5], &offset)) return none();
  a.flags = (in_topk.p == Py_True ? LM_FLAG_TOPP_IN_TOPK : 0u) | (exact.p == Py_True ? LM_FLAG_EXACT_ONLY : 0u) | LM_FLAG_GRID_LIMIT(grid);
  a.step = static_cast<uint32_t>(step); a.row_offset = static_cast<int64_t>(offset);
  if (args[2] != Py_None) {
    const at::Tensor* h = as_tensor(args[2]);
    if (!h || h->dim() != 2 || h->size(0) != rows || h->device() != dev || h->scalar_type() != at::kInt || h->stride(1) != 1) return none();
    a.history = static_cast<const int32_t*>(h->const_data_ptr()); a.hist_len = h->size(1); a.hist_stride = row_stride(*h);
  }
  if (inverse && (a.temperature || a.temperature_s > 0.0f)) {
    const at::Tensor* u = as_tensor(args[3]);
    if (!u || !plain_vector(*u, at::kFloat, dev, rows)) return none();
    a.uniforms = static_cast<const float*>(u->const_data_ptr());
  }
  const long want = PyLong_AsLong(args[6]);
  return run_sample(a, *x, args[7], static_cast<int>(want));
  END_HANDLE_TH_ERRORS
}

// stochastic(logits, temperature, top_k, top_p, min_p, seed, topp_in_topk, step) -> int64 tokens
PyObject* py_stochastic(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8) { PyErr_SetString(PyExc_TypeError, "stochastic: 8 arguments"); return nullptr; }
  const at::Tensor* x = as_tensor(args[0]);
  if (!x || !plain_rows(*x)) return none();
  lm_sample_args a{};
  if (!PyFloat_Check(args[1]) || !PyFloat_Check(args[3]) || !PyFloat_Check(args[4]) || !PyBool_Check(args[6])) return none();
  a.temperature_s = static_cast<float>(PyFloat_AS_DOUBLE(args[1])); a.top_p_s = static_cast<float>(PyFloat_AS_DOUBLE(args[3])); a.min_p_s = static_cast<float>(PyFloat_AS_DOUBLE(args[4]));
  const int32_t* array = nullptr;
  uint64_t step = 0;
  if (!(a.temperature_s > 0.0f) || !PyLong_CheckExact(args[2]) || !knob_i(args[2], 0, x->device(), &array, &a.top_k_s) || !as_u64(args[5], &a.seed) || !as_u64(args[7], &step)) return none();
  a.step = static_cast<uint32_t>(step);
  a.flags = args[6] == Py_True ? LM_FLAG_TOPP_IN_TOPK : 0u;
  a.draw = LM_DRAW_GUMBEL; a.repetition_penalty = 1.0f;
  return run_sample(a, *x, Py_None, kI64);
  END_HANDLE_TH_ERRORS
}

// argmax(logits, out, i64): int32 tokens (or int64)
PyObject* py_argmax(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3) { PyErr_SetString(PyExc_TypeError, "argmax: 3 arguments"); return nullptr; }
  const at::Tensor* x = as_tensor(args[0]);
  if (!x || !plain_rows(*x)) return none();
  const bool i64 = args[2] == Py_True;
  const at::Device dev = x->device();
  const int64_t rows = x->size(0), vocab = x->size(1);
  at::Tensor tokens;
  if (args[1] == Py_None) tokens = make({rows}, i64 ? at::kLong : at::kInt, dev);
  else {
    const at::Tensor* t = as_tensor(args[1]);
    if (!t || i64 || !plain_vector(*t, at::kInt, dev, rows)) return none();
    tokens = *t;
  }
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int rc = call(dev, nullptr, [&] {
    return i64 ? abi.argmax_i64(ptr(*x), dtype_code(*x), rows, vocab, row_stride(*x), static_cast<int64_t*>(ptr(tokens)), stream)
               : abi.argmax(ptr(*x), dtype_code(*x), rows, vocab, row_stride(*x), static_cast<int32_t*>(ptr(tokens)), nullptr, 0, stream);
  });
  if (rc != LM_OK) return failed(rc, "lm_argmax");
  if (args[1] != Py_None) { Py_INCREF(args[1]); return args[1]; }
  return THPVariable_Wrap(tokens);
  END_HANDLE_TH_ERRORS
}

// draft_q(logits, temperature, seed, step, first_position, copy_logits) -> DraftQ
PyObject* py_draft_q(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6) { PyErr_SetString(PyExc_TypeError, "draft_q: 6 arguments"); return nullptr; }
  const at::Tensor* x = as_tensor(args[0]);
  if (!x || !plain_rows(*x) || x->size(0) < 1 || x->size(0) > LM_MAX_DRAFT + 1 || args[5] != Py_False) return none();
  const at::Device dev = x->device();
  const int64_t rows = x->size(0), vocab = x->size(1);
  lm_draft_q_args a{};
  uint64_t step = 0;
  const float* array = nullptr; const int32_t* iarray = nullptr;
  if (as_tensor(args[1]) || as_tensor(args[4]) || !knob_f(args[1], 0, dev, &array, &a.temperature) || !(a.temperature > 0.0f) || !as_u64(args[2], &a.seed) ||
      !as_u64(args[3], &step) || step > 0xFFFFFFFFull || !knob_i(args[4], 0, dev, &iarray, &a.first_position)) return none();
  a.struct_size = sizeof(a);
  a.dtype = dtype_code(*x); a.rows = static_cast<int32_t>(rows); a.logits = ptr(*x); a.vocab = vocab; a.row_stride = row_stride(*x); a.step = static_cast<uint32_t>(step);
  at::Tensor tokens = make({rows}, at::kInt, dev), lse = make({rows}, at::kFloat, dev), vmax = make({rows}, at::kFloat, dev), mass = make({rows}, at::kLong, dev),
             status = make({rows}, at::kInt, dev);
  a.out_tokens = static_cast<int32_t*>(ptr(tokens)); a.out_lse = static_cast<float*>(ptr(lse)); a.out_vmax = static_cast<float*>(ptr(vmax));
  a.out_mass = static_cast<uint64_t*>(ptr(mass)); a.out_status = static_cast<uint32_t*>(ptr(status));
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  a.stream = stream;
  Lease lease;
  if (!scratch(dev, stream, 1, abi.verify_workspace_bytes(static_cast<int32_t>(rows), vocab), &lease, &a.workspace, &a.workspace_bytes)) return nullptr;
  const int rc = call(dev, lease.turn, [&] { return abi.draft_q(&a); });
  if (rc != LM_OK) return failed(rc, "lm_draft_q");
  Ref fields(PyTuple_New(6));
  if (!fields.p) return nullptr;
  const at::Tensor* all[5] = {&tokens, &lse, &vmax, &mass, &status};
  for (int i = 0; i < 5; i++) { PyObject* o = THPVariable_Wrap(*all[i]); if (!o) return nullptr; PyTuple_SET_ITEM(fields.p, i, o); }
  Py_INCREF(Py_None);
  PyTuple_SET_ITEM(fields.p, 5, Py_None);
  Ref one(PyTuple_Pack(1, fields.p));                                       // tuple.__new__(DraftQ, fields): a NamedTuple without its Python constructor
  return one.p ? PyTuple_Type.tp_new(reinterpret_cast<PyTypeObject*>(draft_type), one.p, nullptr) : nullptr;
  END_HANDLE_TH_ERRORS
}

// verify(target, draft_ids, draft_probs, uniforms, u_resample, stochastic, temperature, tau, return_p_draft, draft_logits, draft_vmax, draft_mass,
//        seed, step, gumbel, out, target_vmax, target_mass) -> (accept, final, tokens[, p_draft])
PyObject* py_verify(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 18) { PyErr_SetString(PyExc_TypeError, "verify: 18 arguments"); return nullptr; }
  const at::Tensor *x = as_tensor(args[0]), *ids = as_tensor(args[1]);
  if (!x || !ids || !plain_rows(*x)) return none();
  const at::Device dev = x->device();
  const int64_t n = ids->numel(), vocab = x->size(1);
  if (x->size(0) != n + 1 || n < 1 || n > LM_MAX_DRAFT || !plain_vector(*ids, at::kInt, dev, n)) return none();
  lm_verify_args a{};
  const bool stochastic = args[5] == Py_True;
  a.struct_size = sizeof(a);
  a.mode = stochastic ? LM_VERIFY_STOCHASTIC : LM_VERIFY_GREEDY;
  a.dtype = dtype_code(*x); a.n_draft = static_cast<int32_t>(n);
  a.target_logits = ptr(*x); a.vocab = vocab; a.row_stride = row_stride(*x);
  a.draft_ids = static_cast<const int32_t*>(ids->const_data_ptr());
  uint64_t step = 0;
  if (!as_u64(args[12], &a.seed) || !as_u64(args[13], &step)) return none();
  a.step = static_cast<uint32_t>(step);
  a.residual_draw = args[14] == Py_True ? LM_RESIDUAL_GUMBEL : LM_RESIDUAL_INVERSE_CDF;
  // optional vectors on the device: true unless one is there that is not the ordinary case
  auto vec = [&](PyObject* o, at::ScalarType type, int64_t len, const void** p) {
    if (o == Py_None) return true;
    const at::Tensor* t = as_tensor(o);
    if (!t || !plain_vector(*t, type, dev, len)) return false;
    *p = t->const_data_ptr();
    return true;
  };
  const void *vmax = nullptr, *mass = nullptr, *ua = nullptr, *uf = nullptr, *tau = nullptr;
  if (!vec(args[16], at::kFloat, n + 1, &vmax) || !vec(args[17], at::kLong, n + 1, &mass)) return none();
  a.target_vmax = static_cast<const float*>(vmax);
  a.target_mass = vmax ? static_cast<const uint64_t*>(mass) : nullptr;
  const bool want_p = stochastic && args[8] == Py_True;
  if (stochastic) {
    const float* array = nullptr;
    if (as_tensor(args[6]) || !knob_f(args[6], 0, dev, &array, &a.temperature) || !(a.temperature > 0.0f)) return none();
    if (args[2] != Py_None) {
      const at::Tensor* q = as_tensor(args[2]);
      if (!q || !q->is_cuda() || q->device() != dev || q->dim() != 2 || q->size(0) != n || q->size(1) != vocab || q->scalar_type() != at::kFloat || q->stride(1) != 1) return none();
      a.draft_probs = static_cast<const float*>(q->const_data_ptr()); a.probs_stride = row_stride(*q);
    } else {
      const at::Tensor *q = as_tensor(args[9]), *qv = as_tensor(args[10]), *qm = as_tensor(args[11]);
      if (!q || !qv || !qm || q->device() != dev || q->dim() != 2 || q->size(0) != n || q->size(1) != vocab || q->scalar_type() != at::kBFloat16 || q->stride(1) != 1) return none();
      if (qv->device() != dev || qm->device() != dev || qv->scalar_type() != at::kFloat || qm->scalar_type() != at::kLong || !qv->is_contiguous() || !qm->is_contiguous() ||
          qv->dim() != 1 || qm->dim() != 1 || qv->numel() < n || qm->numel() < n) return none();
      a.draft_logits = q->const_data_ptr(); a.draft_logits_stride = row_stride(*q);
      a.draft_vmax = static_cast<const float*>(qv->const_data_ptr()); a.draft_mass = static_cast<const uint64_t*>(qm->const_data_ptr());
    }
    if (!vec(args[3], at::kFloat, n, &ua) || !vec(args[4], at::kFloat, 1, &uf) || !vec(args[7], at::kFloat, n + 1, &tau)) return none();
    a.u_accept = static_cast<const float*>(ua); a.u_final = static_cast<const float*>(uf); a.tau = static_cast<const float*>(tau);
  }
  at::Tensor out;
  if (args[15] == Py_None) out = make({n + 3}, at::kInt, dev);
  else {
    const at::Tensor* t = as_tensor(args[15]);
    if (!t || !plain_vector(*t, at::kInt, dev, n + 3)) return none();
    out = *t;
  }
  int32_t* o = static_cast<int32_t*>(ptr(out));
  a.out_accept = o; a.out_final = o + 1; a.out_tokens = o + 2;
  at::Tensor p_draft;
  if (want_p) { p_draft = make({n}, at::kFloat, dev); a.out_p_draft = static_cast<float*>(ptr(p_draft)); }
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  a.stream = stream;
  Lease lease;
  if (!scratch(dev, stream, 1, abi.verify_workspace_bytes(static_cast<int32_t>(n), vocab), &lease, &a.workspace, &a.workspace_bytes)) return nullptr;
  const int rc = call(dev, lease.turn, [&] { return abi.verify(&a); });
  if (rc != LM_OK) return failed(rc, "lm_verify");
  Ref res(PyTuple_New(want_p ? 4 : 3));
  if (!res.p) return nullptr;
  const int64_t at_[3] = {0, 1, 2}, len[3] = {1, 1, n + 1};
  for (int i = 0; i < 3; i++) { PyObject* t = THPVariable_Wrap(out.narrow(0, at_[i], len[i])); if (!t) return nullptr; PyTuple_SET_ITEM(res.p, i, t); }
  if (want_p) { PyObject* t = THPVariable_Wrap(p_draft); if (!t) return nullptr; PyTuple_SET_ITEM(res.p, 3, t); }
  return res.release();
  END_HANDLE_TH_ERRORS
}

// lm_head(hidden, weight, norm_weight, eps, one_plus, out) -> logits
PyObject* py_lm_head(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6) { PyErr_SetString(PyExc_TypeError, "lm_head: 6 arguments"); return nullptr; }
  const at::Tensor *x = as_tensor(args[0]), *w = as_tensor(args[1]), *g = args[2] == Py_None ? nullptr : as_tensor(args[2]);
  if (!x || !w || (args[2] != Py_None && !g)) return none();
  if (!x->is_cuda() || x->dim() != 2 || w->dim() != 2 || x->scalar_type() != at::kBFloat16 || w->scalar_type() != at::kBFloat16 || w->device() != x->device()) return none();
  const int64_t rows = x->size(0), H = x->size(1), V = w->size(0);
  if (rows > LM_HEAD_MAX_ROWS || w->size(1) != H || x->stride(1) != 1 || w->stride(1) != 1) return none();
  if (g && (g->dim() != 1 || !plain_vector(*g, at::kBFloat16, x->device(), H))) return none();
  if (!PyFloat_Check(args[3]) || !PyBool_Check(args[4])) return none();
  at::Tensor out;
  if (args[5] == Py_None) out = make({rows, V}, at::kBFloat16, x->device());
  else {
    const at::Tensor* t = as_tensor(args[5]);
    if (!t || t->dim() != 2 || t->size(0) != rows || t->size(1) != V || t->scalar_type() != at::kBFloat16 || t->stride(1) != 1 || t->device() != x->device()) return none();
    out = *t;
  }
  lm_head_args a{};
  a.struct_size = sizeof(a);
  a.rows = static_cast<int32_t>(rows); a.hidden = ptr(*x); a.hidden_stride = rows > 1 ? x->stride(0) : H;
  a.weight = ptr(*w); a.weight_stride = V > 1 ? w->stride(0) : H; a.hidden_dim = H; a.vocab = V;
  a.norm_weight = g ? ptr(*g) : nullptr;
  a.eps = static_cast<float>(PyFloat_AS_DOUBLE(args[3])); a.one_plus = args[4] == Py_True ? 1 : 0;
  a.logits = ptr(out); a.logits_stride = rows > 1 ? out.stride(0) : V;
  a.stream = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  const int rc = call(x->device(), nullptr, [&] { return abi.head(&a); });
  if (rc != LM_OK) return failed(rc, "lm_head");
  if (args[5] != Py_None) { Py_INCREF(args[5]); return args[5]; }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// init(addresses: dict of ABI function addresses, SamplingParams, SampleOutput, DraftQ, check, workspace)
PyObject* py_init(PyObject*, PyObject* args) {
  PyObject *addresses, *t0, *t1, *t2, *f0, *f1;
  if (!PyArg_ParseTuple(args, "O!OOOOO", &PyDict_Type, &addresses, &t0, &t1, &t2, &f0, &f1)) return nullptr;
  auto get = [&](const char* name) -> void* { PyObject* o = PyDict_GetItemString(addresses, name); return o ? PyLong_AsVoidPtr(o) : nullptr; };
  abi.sample = reinterpret_cast<decltype(abi.sample)>(get("lm_sample"));
  abi.argmax = reinterpret_cast<decltype(abi.argmax)>(get("lm_argmax"));
  abi.argmax_i64 = reinterpret_cast<decltype(abi.argmax_i64)>(get("lm_argmax_i64"));
  abi.verify = reinterpret_cast<decltype(abi.verify)>(get("lm_verify"));
  abi.draft_q = reinterpret_cast<decltype(abi.draft_q)>(get("lm_draft_q"));
  abi.head = reinterpret_cast<decltype(abi.head)>(get("lm_head"));
  abi.workspace_bytes = reinterpret_cast<decltype(abi.workspace_bytes)>(get("lm_workspace_bytes"));
  abi.verify_workspace_bytes = reinterpret_cast<decltype(abi.verify_workspace_bytes)>(get("lm_verify_workspace_bytes"));
  if (PyErr_Occurred()) return nullptr;
  if (!abi.sample || !abi.argmax || !abi.argmax_i64 || !abi.verify || !abi.draft_q || !abi.head || !abi.workspace_bytes || !abi.verify_workspace_bytes) {
    PyErr_SetString(PyExc_ValueError, "init: an address is missing");
    return nullptr;
  }
  for (PyObject* o : {t0, t1, t2, f0, f1}) Py_INCREF(o);
  params_type = t0; output_type = t1; draft_type = t2; check_fn = f0; workspace_fn = f1;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"init", py_init, METH_VARARGS, nullptr},
    {"sample", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_sample)), METH_FASTCALL, nullptr},
    {"stochastic", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_stochastic)), METH_FASTCALL, nullptr},
    {"argmax", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_argmax)), METH_FASTCALL, nullptr},
    {"draft_q", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_draft_q)), METH_FASTCALL, nullptr},
    {"verify", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_verify)), METH_FASTCALL, nullptr},
    {"lm_head", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_lm_head)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "lithos_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_lithos_host(void) {
  struct { PyObject** to; const char* name; } names[] = {{&n_temperature, "temperature"}, {&n_top_k, "top_k"}, {&n_top_p, "top_p"}, {&n_min_p, "min_p"}, {&n_seed, "seed"},
      {&n_topp_in_topk, "topp_in_topk"}, {&n_rho, "repetition_penalty"}, {&n_pi, "presence_penalty"}, {&n_draw, "draw"}, {&n_exact_only, "exact_only"},
      {&n_grid_limit, "grid_limit"}, {&n_gumbel, "gumbel"}, {&n_inverse_cdf, "inverse_cdf"}};
  for (auto& e : names) { *e.to = PyUnicode_InternFromString(e.name); if (!*e.to) return nullptr; }
  return PyModule_Create(&module);
}
