// The hot half of the Python binding: turns torch tensors into qb200_tensor descriptors, allocates the outputs and
// calls the C ABI, natively.
//
// What bounds a call is this code, not the kernel: the ctypes form of the same work (five descriptors filled field by
// field from Python, tensor attributes read one at a time) took 23.6 us for a 4096 -> 4096 linear whose kernel takes
// 4 us, and several hundred for the per-sequence cache lists of a decode tick.  The Python functions in __init__.py keep
// their names, defaults and docstrings and pass their arguments here by position; a status other than 0 raises
// qb200.Qb200Error.  The GIL is released around the library call, as ctypes does.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/qb200.h"

namespace {

PyObject* g_error_class = nullptr;   // qb200.Qb200Error, set once by the package

struct PyFail {};                    // a Python exception is already set

int q_dtype(at::ScalarType t) {
  switch (t) {
    case at::kBool: return QB200_BOOL;
    case at::kByte: return QB200_UINT8;
    case at::kUInt16: return QB200_UINT16;
    case at::kUInt32: return QB200_UINT32;
    case at::kChar: return QB200_INT8;
    case at::kShort: return QB200_INT16;
    case at::kInt: return QB200_INT32;
    case at::kLong: return QB200_INT64;
    case at::kHalf: return QB200_FLOAT16;
    case at::kFloat: return QB200_FLOAT32;
    case at::kDouble: return QB200_FLOAT64;
    case at::kBFloat16: return QB200_BFLOAT16;
    default: throw std::invalid_argument("qb200: a tensor of a dtype the library has no name for");
  }
}

// A descriptor and the tensor it describes.
struct T {
  qb200_tensor d;
  void fill(const at::Tensor& t, int dtype) {
    const auto sz = t.sizes();
    const auto st = t.strides();
    if (sz.size() > QB200_MAX_DIMS) throw std::invalid_argument("qb200: a tensor of more than 8 dimensions");
    d.data = t.numel() > 0 ? t.data_ptr() : nullptr;
    d.dtype = dtype;
    d.ndim = (int32_t)sz.size();
    for (size_t i = 0; i < sz.size(); ++i) { d.shape[i] = sz[i]; d.stride[i] = st[i]; }
  }
  void none() { d.data = nullptr; d.dtype = 0; d.ndim = 0; }
};

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) throw std::invalid_argument("qb200: a torch tensor was expected");
  return THPVariable_Unpack(o);
}
T plain(const at::Tensor& t) { T r; r.fill(t, q_dtype(t.scalar_type())); return r; }
T packed(const at::Tensor& t) { T r; r.fill(t, QB200_UINT32); return r; }   // uint32 payloads travel in int32 tensors
T plain(PyObject* o) {
  if (o == Py_None) { T r; r.none(); return r; }
  return plain(tensor(o));
}
T packed(PyObject* o) {
  if (o == Py_None) { T r; r.none(); return r; }
  return packed(tensor(o));
}

long as_long(PyObject* o) {
  const long v = PyLong_Check(o) ? PyLong_AsLong(o) : [&] {
    PyObject* i = PyNumber_Long(o);
    if (!i) return -1L;
    const long r = PyLong_AsLong(i);
    Py_DECREF(i);
    return r;
  }();
  if (v == -1 && PyErr_Occurred()) throw PyFail();
  return v;
}
double as_double(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyFail();
  return v;
}
bool as_bool(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyFail();
  return v != 0;
}
const char* as_str(PyObject* o) {
  const char* s = PyUnicode_AsUTF8(o);
  if (!s) throw PyFail();
  return s;
}
qb200_optional_int opt(PyObject* o) {
  if (o == Py_None) return {0, false};
  return {(int)as_long(o), true};
}
// Sizes of outputs follow Python's rules, as the callers see Python functions: whole numbers only, // rounds down, and a
// division by zero is an exception.  (The library checks bits and group size too, but after the output exists.)
int64_t as_index(PyObject* o) {
  const Py_ssize_t v = PyNumber_AsSsize_t(o, PyExc_OverflowError);
  if (v == -1 && PyErr_Occurred()) throw PyFail();
  return (int64_t)v;
}
int64_t floor_div(int64_t a, int64_t b) {
  if (b == 0) { PyErr_SetString(PyExc_ZeroDivisionError, "integer division or modulo by zero"); throw PyFail(); }
  const int64_t q = a / b;
  return a % b != 0 && (a < 0) != (b < 0) ? q - 1 : q;
}
int64_t bits_or_4(PyObject* o) { return o == Py_None ? 4 : as_index(o); }
int64_t gs_or_64(PyObject* o) { return o == Py_None ? 64 : as_index(o); }

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }

void check(int status) {
  if (status == 0) return;
  PyObject* e = g_error_class ? PyObject_CallFunction(g_error_class, "is", status, qb200_last_error()) : nullptr;
  if (e) {
    PyErr_SetObject(g_error_class, e);
    Py_DECREF(e);
  } else if (!PyErr_Occurred()) {
    PyErr_Format(PyExc_RuntimeError, "qb200 status %d: %s", status, qb200_last_error());
  }
  throw PyFail();
}
template <typename F>
void call(F&& f) {
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = f();
  Py_END_ALLOW_THREADS
  check(status);
}

at::Tensor empty(at::IntArrayRef shape, const at::Tensor& like) { return at::empty(shape, like.options().requires_grad(false)); }
at::Tensor empty(at::IntArrayRef shape, const at::Tensor& like, at::ScalarType dt) {
  return at::empty(shape, like.options().dtype(dt).requires_grad(false));
}
PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* ret(PyObject* o) { Py_INCREF(o); return o; }
using Shape = c10::SmallVector<int64_t, 8>;
Shape lead(const at::Tensor& t, int drop) { const auto s = t.sizes(); return Shape(s.begin(), s.end() - std::min<size_t>(drop, s.size())); }

// A list or tuple's items without a copy.
struct Seq {
  PyObject* o;
  explicit Seq(PyObject* s) : o(PySequence_Fast(s, "qb200: a list or tuple was expected")) { if (!o) throw PyFail(); }
  ~Seq() { Py_DECREF(o); }
  Seq(const Seq&) = delete;
  Py_ssize_t size() const { return PySequence_Fast_GET_SIZE(o); }
  PyObject* operator[](Py_ssize_t i) const {
    if (i >= size()) { PyErr_SetString(PyExc_IndexError, "qb200: the list is too short"); throw PyFail(); }
    return PySequence_Fast_GET_ITEM(o, i);
  }
  // one entry for each of n sequences or matrices (a shorter list fails where its missing entry is asked for)
  void at_most(Py_ssize_t n) const {
    if (size() > n) { PyErr_SetString(PyExc_IndexError, "qb200: the list is too long"); throw PyFail(); }
  }
};

// (codes, scales, biases) of every sequence as the ABI's three pointer lists.
struct Triples {
  std::vector<T> d;
  std::vector<qb200_tensor*> p[3];
  Triples(const Seq& list, Py_ssize_t n) {
    d.resize(3 * n);
    for (auto& v : p) v.resize(n);
    for (Py_ssize_t i = 0; i < n; ++i) {
      Seq t(list[i]);
      for (int j = 0; j < 3; ++j) {
        d[3 * i + j] = j == 0 ? packed(t[j]) : plain(t[j]);
        p[j][i] = &d[3 * i + j].d;
      }
    }
  }
  qb200_tensor* const* operator[](int j) { return p[j].data(); }
};

using Args = PyObject* const*;
// Turns what the body throws into a Python exception and checks the argument count.
template <int N, PyObject* (*F)(Args)>
PyObject* entry(PyObject*, Args a, Py_ssize_t n) {
  if (n != N) { PyErr_Format(PyExc_TypeError, "qb200._native: %d arguments expected, %zd given", N, n); return nullptr; }
  HANDLE_TH_ERRORS   // torch's own exceptions (out of memory, no device) become the classes Python code expects
  try {
    return F(a);
  } catch (const PyFail&) {
    return nullptr;
  } catch (const std::invalid_argument& e) {
    PyErr_SetString(PyExc_TypeError, e.what());
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// x, w, scales, biases, transpose, group_size, bits, mode, out
PyObject* quantized_matmul(Args a) {
  T x = plain(a[0]), w = packed(a[1]), s = plain(a[2]), b = plain(a[3]);
  const bool tr = as_bool(a[4]);
  const auto gs = opt(a[5]), nb = opt(a[6]);
  const char* mode = as_str(a[7]);
  at::Tensor made;
  if (a[8] == Py_None) {
    int64_t shp[QB200_MAX_DIMS];
    int32_t nd = 0;
    check(qb200_quantized_matmul_shape(&x.d, &w.d, &s.d, tr, gs, nb, shp, &nd));
    made = empty(at::IntArrayRef(shp, nd), tensor(a[0]));
  }
  T y = plain(made.defined() ? made : tensor(a[8]));
  void* st = stream();
  call([&] { return qb200_quantized_matmul(&y.d, &x.d, &w.d, &s.d, &b.d, tr, gs, nb, mode, st); });
  return made.defined() ? wrap(std::move(made)) : ret(a[8]);
}

// x, triples, outs, transpose, group_size, bits, mode
PyObject* quantized_matmul_batch(Args a) {
  T x = plain(a[0]);
  Seq tl(a[1]), ol(a[2]);
  const Py_ssize_t n = tl.size();
  ol.at_most(n);
  Triples w(tl, n);
  std::vector<T> y(n);
  std::vector<qb200_tensor*> yp(n);
  for (Py_ssize_t i = 0; i < n; ++i) { y[i] = plain(ol[i]); yp[i] = &y[i].d; }
  const bool tr = as_bool(a[3]);
  const auto gs = opt(a[4]), nb = opt(a[5]);
  const char* mode = as_str(a[6]);
  void* st = stream();
  call([&] { return qb200_quantized_matmul_batch(yp.data(), &x.d, w[0], w[1], w[2], (int)n, tr, gs, nb, mode, st); });
  return ret(a[2]);
}

at::Tensor gather_out(PyObject* out, const at::Tensor& x, const at::Tensor& w, PyObject* rhs) {
  if (out != Py_None) return tensor(out);
  const auto r = tensor(rhs).sizes();
  Shape s(r.begin(), r.end());
  s.push_back(x.size(-2));
  s.push_back(w.size(-2));
  return empty(s, x);
}

// x, w, scales, biases, lhs, rhs, transpose, group_size, bits, mode, sorted, out
PyObject* gather_qmm(Args a) {
  at::Tensor out = gather_out(a[11], tensor(a[0]), tensor(a[1]), a[5]);
  T y = plain(out), x = plain(a[0]), w = packed(a[1]), s = plain(a[2]), b = plain(a[3]), l = plain(a[4]), r = plain(a[5]);
  const bool tr = as_bool(a[6]), sorted = as_bool(a[10]);
  const auto gs = opt(a[7]), nb = opt(a[8]);
  const char* mode = as_str(a[9]);
  void* st = stream();
  call([&] { return qb200_gather_qmm(&y.d, &x.d, &w.d, &s.d, &b.d, &l.d, &r.d, tr, gs, nb, mode, sorted, st); });
  return a[11] == Py_None ? wrap(std::move(out)) : ret(a[11]);
}

// x, (w, scales, biases) gate, (w, scales, biases) up, lhs, rhs, group_size, bits, mode, sorted, out
PyObject* gather_qmm_swiglu(Args a) {
  at::Tensor out = gather_out(a[13], tensor(a[0]), tensor(a[1]), a[8]);
  T y = plain(out), x = plain(a[0]), g = packed(a[1]), gsc = plain(a[2]), gb = plain(a[3]), u = packed(a[4]), us = plain(a[5]), ub = plain(a[6]),
    l = plain(a[7]), r = plain(a[8]);
  const auto gs = opt(a[9]), nb = opt(a[10]);
  const char* mode = as_str(a[11]);
  const bool sorted = as_bool(a[12]);
  void* st = stream();
  call([&] { return qb200_gather_qmm_swiglu(&y.d, &x.d, &g.d, &gsc.d, &gb.d, &u.d, &us.d, &ub.d, &l.d, &r.d, gs, nb, mode, sorted, st); });
  return a[13] == Py_None ? wrap(std::move(out)) : ret(a[13]);
}

// act, w, scales, biases, inds, scores, group_size, bits, mode, out
PyObject* moe_down_reduce(Args a) {
  at::Tensor out;
  if (a[9] == Py_None) {
    Shape s = lead(tensor(a[5]), 1);
    s.push_back(tensor(a[1]).size(-2));
    out = empty(s, tensor(a[0]));
  } else {
    out = tensor(a[9]);
  }
  T y = plain(out), x = plain(a[0]), w = packed(a[1]), s = plain(a[2]), b = plain(a[3]), i = plain(a[4]), sc = plain(a[5]);
  const auto gs = opt(a[6]), nb = opt(a[7]);
  const char* mode = as_str(a[8]);
  void* st = stream();
  call([&] { return qb200_moe_down_reduce(&y.d, &x.d, &w.d, &s.d, &b.d, &i.d, &sc.d, gs, nb, mode, st); });
  return a[9] == Py_None ? wrap(std::move(out)) : ret(a[9]);
}

PyObject* pack(std::initializer_list<PyObject*> items) {   // takes the references
  PyObject* t = PyTuple_New((Py_ssize_t)items.size());
  Py_ssize_t i = 0;
  for (PyObject* o : items) PyTuple_SET_ITEM(t, i++, o);
  return t;
}

// logits, k
PyObject* moe_route(Args a) {
  const at::Tensor& l = tensor(a[0]);
  const int64_t k = as_index(a[1]);
  Shape s = lead(l, 1);
  s.push_back(k);
  at::Tensor inds = empty(s, l, at::kInt), scores = empty(s, l);
  T di = plain(inds), ds = plain(scores), dl = plain(l);
  void* st = stream();
  call([&] { return qb200_moe_route(&di.d, &ds.d, &dl.d, (int)k, st); });
  return pack({wrap(std::move(inds)), wrap(std::move(scores))});
}

// y, scores, inv_order, out
PyObject* moe_weighted_sum(Args a) {
  at::Tensor out;
  if (a[3] == Py_None) {
    Shape s = lead(tensor(a[1]), 1);
    s.push_back(tensor(a[0]).size(-1));
    out = empty(s, tensor(a[0]));
  } else {
    out = tensor(a[3]);
  }
  T r = plain(out), y = plain(a[0]), sc = plain(a[1]), inv = plain(a[2]);
  void* st = stream();
  call([&] { return qb200_moe_weighted_sum(&r.d, &y.d, &sc.d, &inv.d, st); });
  return a[3] == Py_None ? wrap(std::move(out)) : ret(a[3]);
}

// inds, num_experts, want_offsets
PyObject* moe_sort_by_expert(Args a) {
  const at::Tensor& in = tensor(a[0]);
  const long E = as_long(a[1]);
  const int64_t n = in.numel();
  at::Tensor o[5];
  for (int i = 0; i < 4; ++i) o[i] = empty({n}, in, at::kInt);
  const bool want = as_bool(a[2]);
  if (want) o[4] = empty({(int64_t)E + 1}, in, at::kInt);
  T d[5], di = plain(in);
  for (int i = 0; i < 4; ++i) d[i] = plain(o[i]);
  if (want) d[4] = plain(o[4]); else d[4].none();
  void* st = stream();
  call([&] { return qb200_moe_sort_by_expert(&d[0].d, &d[1].d, &d[2].d, &d[3].d, &d[4].d, &di.d, (int)E, st); });
  return pack({wrap(std::move(o[0])), wrap(std::move(o[1])), wrap(std::move(o[2])), wrap(std::move(o[3])),
               want ? wrap(std::move(o[4])) : ret(Py_None)});
}

// w, scales, biases, group_size, bits, mode, dtype, out
PyObject* dequantize(Args a) {
  const at::Tensor &w = tensor(a[0]), &s = tensor(a[1]);
  qb200_optional_dtype od = {0, false};
  at::ScalarType odt = s.scalar_type();
  if (a[6] != Py_None) {
    if (!THPDtype_Check(a[6])) throw std::invalid_argument("qb200: a torch dtype was expected");
    odt = reinterpret_cast<THPDtype*>(a[6])->scalar_type;
    od = {q_dtype(odt), true};
  }
  at::Tensor out;
  if (a[7] == Py_None) {
    Shape shp = lead(w, 1);
    shp.push_back(floor_div(w.size(-1) * 32, bits_or_4(a[4])));
    out = empty(shp, w, odt);
  } else {
    out = tensor(a[7]);
  }
  T y = plain(out), dw = packed(w), ds = plain(s), db = plain(a[2]), none;
  none.none();
  const auto gs = opt(a[3]), nb = opt(a[4]);
  const char* mode = as_str(a[5]);
  void* st = stream();
  call([&] { return qb200_dequantize(&y.d, &dw.d, &ds.d, &db.d, gs, nb, mode, &none.d, od, st); });
  return a[7] == Py_None ? wrap(std::move(out)) : ret(a[7]);
}

// w, group_size, bits, mode
PyObject* quantize(Args a) {
  const at::Tensor& w = tensor(a[0]);
  const int64_t gs = gs_or_64(a[1]), nb = bits_or_4(a[2]), D = w.size(-1);
  Shape sq = lead(w, 1), ss = sq;
  sq.push_back(floor_div(D * nb, 32));
  ss.push_back(floor_div(D, gs));
  at::Tensor q = empty(sq, w, at::kInt), s = empty(ss, w, at::kBFloat16), b = empty(ss, w, at::kBFloat16);
  T dq = packed(q), ds = plain(s), db = plain(b), dw = plain(w), none;
  none.none();
  const auto og = opt(a[1]), ob = opt(a[2]);
  const char* mode = as_str(a[3]);
  void* st = stream();
  call([&] { return qb200_quantize(&dq.d, &ds.d, &db.d, &dw.d, og, ob, mode, &none.d, st); });
  return pack({wrap(std::move(q)), wrap(std::move(s)), wrap(std::move(b))});
}

// cache_q, cache_scales, cache_biases, dense, offset, bits, group_size
PyObject* kv_append(Args a) {
  T q = packed(a[0]), s = plain(a[1]), b = plain(a[2]), d = plain(a[3]);
  const int64_t off = as_long(a[4]);
  const int nb = (int)as_long(a[5]), gs = (int)as_long(a[6]);
  void* st = stream();
  call([&] { return qb200_kv_append(&q.d, &s.d, &b.d, &d.d, off, nb, gs, st); });
  return ret(Py_None);
}

at::Tensor attn_out(PyObject* out, const at::Tensor& q, int64_t Tq, int64_t Dv) {
  if (out != Py_None) return tensor(out);
  return empty({q.size(0), q.size(1), Tq, Dv}, q);
}

// q, k_triple, v_triple, bits, group_size, scale, mask_mode, mask, kv_lens, workspace, out
PyObject* kv_decode_attention(Args a) {
  const at::Tensor& q = tensor(a[0]);
  Seq k(a[1]), v(a[2]);
  for (const Seq* s : {&k, &v})
    if (s->size() != 3) { PyErr_SetString(PyExc_ValueError, "qb200: (codes, scales, biases) were expected"); throw PyFail(); }
  const at::Tensor &kq = tensor(k[0]), &vq = tensor(v[0]);
  const int nb = (int)as_long(a[3]), gs = (int)as_long(a[4]);
  const float scale = (float)as_double(a[5]);
  const char* mm = as_str(a[6]);
  const int64_t B = q.size(0), Hq = q.size(1), Tq = q.size(2), Dv = floor_div(vq.size(3) * 32, as_index(a[3]));
  at::Tensor out = attn_out(a[10], q, Tq, Dv), ws;
  if (a[9] == Py_None) {
    const size_t need = qb200_kv_decode_attention_workspace_size(Tq > 1 ? Tq : B, Hq, kq.size(1), kq.size(2), Dv);
    ws = empty({(int64_t)(need > 16 ? need : 16)}, q, at::kByte);
  } else {
    ws = tensor(a[9]);
  }
  T y = plain(out), dq = plain(q), k0 = packed(kq), k1 = plain(k[1]), k2 = plain(k[2]), v0 = packed(vq), v1 = plain(v[1]), v2 = plain(v[2]),
    dm = plain(a[7]), dl = plain(a[8]);
  void* wp = ws.data_ptr();
  const size_t wn = (size_t)ws.numel();
  void* st = stream();
  call([&] {
    return qb200_kv_decode_attention(&y.d, &dq.d, &k0.d, &k1.d, &k2.d, &v0.d, &v1.d, &v2.d, nb, gs, scale, mm, &dm.d, &dl.d, wp, wn, st);
  });
  return a[10] == Py_None ? wrap(std::move(out)) : ret(a[10]);
}

// q, k_triple, v_triple, bits, group_size, scale, out, mask_mode, mask, kv_lens
PyObject* kv_decode_attention_noalloc(Args a) {
  Seq k(a[1]), v(a[2]);
  T y = plain(a[6]), dq = plain(a[0]), k0 = packed(k[0]), k1 = plain(k[1]), k2 = plain(k[2]), v0 = packed(v[0]), v1 = plain(v[1]), v2 = plain(v[2]),
    dm = plain(a[8]), dl = plain(a[9]);
  const int nb = (int)as_long(a[3]), gs = (int)as_long(a[4]);
  const float scale = (float)as_double(a[5]);
  const char* mm = as_str(a[7]);
  void* st = stream();
  call([&] {
    return qb200_kv_decode_attention_noalloc(&y.d, &dq.d, &k0.d, &k1.d, &k2.d, &v0.d, &v1.d, &v2.d, nb, gs, scale, mm, &dm.d, &dl.d, st);
  });
  return ret(a[6]);
}

// q, k_triples, v_triples, bits, group_size, scale, mask_mode, mask, kv_lens, workspace, out
PyObject* kv_decode_attention_ptrs(Args a) {
  const at::Tensor& q = tensor(a[0]);
  Seq kl(a[1]), vl(a[2]);
  const int nb = (int)as_long(a[3]), gs = (int)as_long(a[4]);
  const float scale = (float)as_double(a[5]);
  const char* mm = as_str(a[6]);
  const int64_t B = q.size(0), Hq = q.size(1);
  kl.at_most(B);
  vl.at_most(B);
  Seq k0(kl[0]), v0(vl[0]);
  const int64_t Hkv = tensor(k0[0]).size(1);
  const at::Tensor& vq = tensor(v0[0]);
  Triples k(kl, B), v(vl, B);
  int64_t tmax = 0;
  for (int64_t i = 0; i < B; ++i) {
    if (k[0][i]->ndim < 3) { PyErr_SetString(PyExc_IndexError, "qb200: a cache view of four dimensions was expected"); throw PyFail(); }
    tmax = std::max(tmax, k[0][i]->shape[2]);
  }
  const int64_t Dv = floor_div(vq.size(3) * 32, as_index(a[3]));
  at::Tensor out = attn_out(a[10], q, 1, Dv), ws;
  if (a[9] == Py_None) {
    const size_t need = qb200_kv_decode_attention_ptrs_workspace_size(B, Hq, Hkv, tmax, Dv);
    ws = empty({(int64_t)(need > 16 ? need : 16)}, q, at::kByte);
  } else {
    ws = tensor(a[9]);
  }
  T y = plain(out), dq = plain(q), dm = plain(a[7]), dl = plain(a[8]);
  void* wp = ws.data_ptr();
  const size_t wn = (size_t)ws.numel();
  void* st = stream();
  call([&] {
    return qb200_kv_decode_attention_ptrs(&y.d, &dq.d, k[0], k[1], k[2], v[0], v[1], v[2], (int)B, nb, gs, scale, mm, &dm.d, &dl.d, wp, wn, st);
  });
  return a[10] == Py_None ? wrap(std::move(out)) : ret(a[10]);
}

// a, b, weight, eps, sum_out, norm_out, want_norm
PyObject* add_rms_norm(Args a) {
  const at::Tensor& x = tensor(a[0]);
  const bool want = as_bool(a[6]);
  at::Tensor sum = a[4] == Py_None ? at::empty_like(x) : tensor(a[4]), norm;
  const bool make_norm = a[5] == Py_None && want;
  if (make_norm) norm = at::empty_like(x);
  T ds = plain(sum), dn, da = plain(x), db = plain(a[1]), dw;
  if (make_norm) dn = plain(norm); else dn = plain(a[5]);
  if (want) dw = plain(a[2]); else dw.none();
  const float eps = (float)as_double(a[3]);
  void* st = stream();
  call([&] { return qb200_add_rms_norm(&ds.d, &dn.d, &da.d, &db.d, &dw.d, eps, st); });
  return pack({a[4] == Py_None ? wrap(std::move(sum)) : ret(a[4]), make_norm ? wrap(std::move(norm)) : ret(a[5])});
}

// x, weight, eps, out
PyObject* rms_norm(Args a) {
  at::Tensor out = a[3] == Py_None ? at::empty_like(tensor(a[0])) : tensor(a[3]);
  T y = plain(out), x = plain(a[0]), w = plain(a[1]);
  const float eps = (float)as_double(a[2]);
  void* st = stream();
  call([&] { return qb200_rms_norm(&y.d, &x.d, &w.d, eps, st); });
  return a[3] == Py_None ? wrap(std::move(out)) : ret(a[3]);
}

// x, dims, base, scale, offsets, out
PyObject* rope(Args a) {
  at::Tensor out = a[5] == Py_None ? at::empty_like(tensor(a[0])) : tensor(a[5]);
  T y = plain(out), x = plain(a[0]), o = plain(a[4]), none;
  none.none();
  const int dims = (int)as_long(a[1]);
  const qb200_optional_float base = {(float)as_double(a[2]), true};
  const float scale = (float)as_double(a[3]);
  void* st = stream();
  call([&] { return qb200_rope(&y.d, &x.d, dims, false, base, scale, &o.d, &none.d, st); });
  return a[5] == Py_None ? wrap(std::move(out)) : ret(a[5]);
}

// x, seed, out
PyObject* turbo_rotate(Args a) {
  at::Tensor out = a[2] == Py_None ? at::empty_like(tensor(a[0])) : tensor(a[2]);
  T y = plain(out), x = plain(a[0]);
  const uint64_t seed = PyLong_AsUnsignedLongLongMask(a[1]);
  if (PyErr_Occurred()) throw PyFail();
  void* st = stream();
  call([&] { return qb200_turbo_rotate(&y.d, &x.d, seed, st); });
  return a[2] == Py_None ? wrap(std::move(out)) : ret(a[2]);
}

// gate, up, out
PyObject* swiglu(Args a) {
  at::Tensor out = a[2] == Py_None ? at::empty_like(tensor(a[0])) : tensor(a[2]);
  T y = plain(out), g = plain(a[0]), u = plain(a[1]);
  void* st = stream();
  call([&] { return qb200_swiglu(&y.d, &g.d, &u.d, st); });
  return a[2] == Py_None ? wrap(std::move(out)) : ret(a[2]);
}

// k_triples, v_triples, dense_k, dense_v, offsets, bits, group_size, rope_q, rope_dims, rope_base, rope_scale
PyObject* kv_append_seqs(Args a) {
  Seq kl(a[0]), vl(a[1]), ol(a[4]);
  const Py_ssize_t n = kl.size();
  vl.at_most(n);
  ol.at_most(n);
  Triples k(kl, n), v(vl, n);
  std::vector<int64_t> off((size_t)n);
  for (Py_ssize_t i = 0; i < n; ++i) off[i] = as_long(ol[i]);
  T dk = plain(a[2]), dv = plain(a[3]);
  const int nb = (int)as_long(a[5]), gs = (int)as_long(a[6]);
  if (a[7] != Py_None) {
    T q = plain(a[7]);
    const int dims = (int)as_long(a[8]);
    const float base = (float)as_double(a[9]), scale = (float)as_double(a[10]);
    void* st = stream();
    call([&] {
      return qb200_rope_kv_append_seqs(&q.d, dims, base, scale, k[0], k[1], k[2], v[0], v[1], v[2], &dk.d, &dv.d, off.data(), (int)n, nb, gs, st);
    });
  } else {
    void* st = stream();
    call([&] { return qb200_kv_append_seqs(k[0], k[1], k[2], v[0], v[1], v[2], &dk.d, &dv.d, off.data(), (int)n, nb, gs, st); });
  }
  return ret(Py_None);
}

PyObject* set_error_class(Args a) {
  Py_INCREF(a[0]);
  Py_XDECREF(g_error_class);
  g_error_class = a[0];
  return ret(Py_None);
}

#define QB_ENTRY(name, n) {#name, (PyCFunction)(void*)(&entry<n, name>), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    QB_ENTRY(quantized_matmul, 9), QB_ENTRY(quantized_matmul_batch, 7), QB_ENTRY(gather_qmm, 12), QB_ENTRY(gather_qmm_swiglu, 14),
    QB_ENTRY(moe_down_reduce, 10), QB_ENTRY(moe_route, 2), QB_ENTRY(moe_weighted_sum, 4), QB_ENTRY(moe_sort_by_expert, 3),
    QB_ENTRY(dequantize, 8), QB_ENTRY(quantize, 4), QB_ENTRY(kv_append, 7), QB_ENTRY(kv_decode_attention, 11),
    QB_ENTRY(kv_decode_attention_noalloc, 10), QB_ENTRY(kv_decode_attention_ptrs, 11), QB_ENTRY(add_rms_norm, 7), QB_ENTRY(rms_norm, 4),
    QB_ENTRY(rope, 6), QB_ENTRY(turbo_rotate, 3), QB_ENTRY(swiglu, 3), QB_ENTRY(kv_append_seqs, 11), QB_ENTRY(set_error_class, 1),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Native half of the qb200 Python binding", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
