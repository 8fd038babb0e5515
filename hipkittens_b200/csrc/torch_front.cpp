// The tensor front ends of hipkittens_b200 in native code: argument checks, output allocation and the C-ABI call for the
// entry points that a serving loop calls once per layer and token. In Python the checks of one call (about sixty
// attribute reads), the stream lookup and the ctypes conversions took 9 to 11 us; here they take under 2.
//
// Every function returns None when an argument is anything but a plain CUDA tensor that the call accepts as it is. The
// Python front end then runs its own checks, which raise what there is to raise (or accept, for instance, a tensor
// subclass); nothing is decided here that is not decided there. Otherwise: an int (an HK_E* code) when the
// library refused the call, else the outputs.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/hk_attn.h"

namespace {

using at::Tensor;

// A plain strided CUDA tensor, or null. The wrappers of torch.func's transforms are of the exact class too, but have no
// storage, and so no pointer to read.
const Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.has_storage() ? &t : nullptr;
}
bool is(const Tensor* t, at::ScalarType type, int64_t dim) { return t && t->scalar_type() == type && t->dim() == dim; }
bool dense(const Tensor* t, at::ScalarType type, int64_t dim) { return is(t, type, dim) && t->is_contiguous(); }
bool same_device(const Tensor& ref, std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->device() != ref.device()) return false;
  return true;
}
// An output: the caller's, or a new one. False: the Python front end is to look at it.
bool output(PyObject* o, const Tensor& ref, at::IntArrayRef shape, at::ScalarType type, Tensor& out) {
  if (o == Py_None) {
    out = at::empty(shape, ref.options().dtype(type).requires_grad(false));
    return out.has_storage();  // under a transform a new tensor is a wrapper as well
  }
  const Tensor* t = plain(o);
  if (!dense(t, type, int64_t(shape.size())) || t->sizes() != shape || t->device() != ref.device()) return false;
  out = *t;
  return true;
}
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
int i32(int64_t v) { return static_cast<int>(v); }
bool fits(std::initializer_list<int64_t> vs) {  // ctypes would refuse what an int does not hold
  for (int64_t v : vs)
    if (v > 0x7fffffffll) return false;
  return true;
}
bool number(PyObject* o, float& v) {
  if (o == Py_None) {
    v = 0.f;
    return true;
  }
  if (!PyFloat_CheckExact(o)) return false;
  v = static_cast<float>(PyFloat_AS_DOUBLE(o));
  return true;
}

// The device pointer of a tensor. data_ptr() can throw and must not race with a resize_ or set_ of another thread, so it
// is read while the interpreter lock is held.
template <typename T = void>
T* ptr(const Tensor& t) { return static_cast<T*>(t.data_ptr()); }

// The library call without the interpreter lock, as ctypes makes it. `call` must not throw: it holds pointers and numbers
// that were read before, and touches no tensor.
template <typename Call>
int unlocked(const Call& call) {
  int rc;
  Py_BEGIN_ALLOW_THREADS rc = call();
  Py_END_ALLOW_THREADS return rc;
}
PyObject* result(int rc, const Tensor& a, const Tensor& b) {
  if (rc != HK_OK) return PyLong_FromLong(rc);
  return Py_BuildValue("(NN)", THPVariable_Wrap(a), THPVariable_Wrap(b));
}

bool tma_strides(const Tensor& t, long long* st) {
  bool good = t.stride(3) == 1;
  for (int i = 0; i < 3; ++i) {
    st[i] = t.stride(i);
    good = good && st[i] > 0 && st[i] % 8 == 0;
  }
  return good;
}

// attn_fwd(q, k, v, causal, softmax_scale, out, lse, kv_lens)
PyObject* attn_fwd(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  float scale;
  if (n_args != 8 || !PyBool_Check(a[3]) || !number(a[4], scale)) Py_RETURN_NONE;
  const Tensor *q = plain(a[0]), *k = plain(a[1]), *v = plain(a[2]);
  for (const Tensor* t : {q, k, v})
    if (!is(t, at::kBFloat16, 4)) Py_RETURN_NONE;
  const int64_t b = q->size(0), n = q->size(1), h = q->size(2), d = q->size(3), nk = k->size(1), hkv = k->size(2);
  if (k->sizes() != v->sizes() || k->size(0) != b || k->size(3) != d || !same_device(*q, {k, v}) ||
      !fits({b, n, nk, h, hkv}))
    Py_RETURN_NONE;
  const bool strided = !(q->is_contiguous() && k->is_contiguous() && v->is_contiguous());
  long long qs[3], ks[3], vs[3];
  const bool q_ok = tma_strides(*q, qs), k_ok = tma_strides(*k, ks), v_ok = tma_strides(*v, vs);
  if (strided && !(q_ok && k_ok && v_ok)) Py_RETURN_NONE;
  const Tensor* lens = nullptr;
  if (a[7] != Py_None) {
    lens = plain(a[7]);
    if (!dense(lens, at::kInt, 1) || lens->size(0) != b || lens->device() != q->device()) Py_RETURN_NONE;
  }
  Tensor out, lse;
  if (!output(a[5], *q, q->sizes(), at::kBFloat16, out) || !output(a[6], *q, {b, h, 1, n}, at::kFloat, lse))
    Py_RETURN_NONE;
  void* st = stream_of(*q);
  const int causal = a[3] == Py_True, dev = q->device().index();
  const void *qp = ptr(*q), *kp = ptr(*k), *vp = ptr(*v);
  void* outp = ptr(out);
  float* lsep = ptr<float>(lse);
  const int32_t* lensp = lens ? ptr<int32_t>(*lens) : nullptr;
  const int rc = unlocked([&] {
    if (lens || nk != n || strided)
      return hk_attn_fwd_cross(qp, kp, vp, outp, lsep, i32(b), i32(n), i32(nk), i32(h), i32(hkv), i32(d), qs, ks, vs, lensp,
                               causal, scale, dev, st);
    return hk_attn_fwd(qp, kp, vp, outp, lsep, i32(b), i32(n), i32(h), i32(hkv), i32(d), causal, scale, dev, st);
  });
  return result(rc, out, lse);
  END_HANDLE_TH_ERRORS
}

// attn_bwd_strided(q, k, v, o, d_o, lse, dq, dk, dv, causal, softmax_scale, kv_lens): 0 when launched
PyObject* attn_bwd_strided(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  float scale;
  if (n_args != 12 || !PyBool_Check(a[9]) || !number(a[10], scale)) Py_RETURN_NONE;
  const Tensor *q = plain(a[0]), *k = plain(a[1]), *v = plain(a[2]), *o = plain(a[3]), *d_o = plain(a[4]),
               *lse = plain(a[5]), *dq = plain(a[6]), *dk = plain(a[7]), *dv = plain(a[8]);
  for (const Tensor* t : {q, k, v, dq, dk, dv})
    if (!is(t, at::kBFloat16, 4)) Py_RETURN_NONE;
  if (!dense(o, at::kBFloat16, 4) || !dense(d_o, at::kBFloat16, 4) || !dense(lse, at::kFloat, 4)) Py_RETURN_NONE;
  const int64_t b = q->size(0), n = q->size(1), h = q->size(2), d = q->size(3), nk = k->size(1), hkv = k->size(2);
  for (const Tensor* t : {o, d_o, dq})
    if (t->sizes() != q->sizes()) Py_RETURN_NONE;
  for (const Tensor* t : {v, dk, dv})
    if (t->sizes() != k->sizes()) Py_RETURN_NONE;
  if (k->size(0) != b || k->size(3) != d || lse->sizes() != at::IntArrayRef({b, h, 1, n}) ||
      !same_device(*q, {k, v, o, d_o, lse, dq, dk, dv}) || !fits({b, n, nk, h, hkv}))
    Py_RETURN_NONE;
  long long st[6][3];
  int i = 0;
  for (const Tensor* t : {q, k, v, dq, dk, dv})
    if (!tma_strides(*t, st[i++])) Py_RETURN_NONE;
  const Tensor* lens = nullptr;
  if (a[11] != Py_None) {
    lens = plain(a[11]);
    if (!dense(lens, at::kInt, 1) || lens->size(0) != b || lens->device() != q->device()) Py_RETURN_NONE;
  }
  const Tensor delta = at::empty({b, h, 1, n}, lse->options().requires_grad(false));
  if (!delta.has_storage()) Py_RETURN_NONE;
  void* stream = stream_of(*q);
  const int causal = a[9] == Py_True, dev = q->device().index();
  const void *qp = ptr(*q), *kp = ptr(*k), *vp = ptr(*v), *op = ptr(*o), *dop = ptr(*d_o);
  const float* lsep = ptr<float>(*lse);
  float* deltap = ptr<float>(delta);
  void *dqp = ptr(*dq), *dkp = ptr(*dk), *dvp = ptr(*dv);
  const int32_t* lensp = lens ? ptr<int32_t>(*lens) : nullptr;
  const int rc = unlocked([&] {
    return hk_attn_bwd_strided(qp, kp, vp, op, dop, lsep, deltap, dqp, dkp, dvp, i32(b), i32(n), i32(nk), i32(h),
                               i32(hkv), i32(d), st[0], st[1], st[2], st[3], st[4], st[5], lensp, causal, scale, dev,
                               stream);
  });
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

// rotary_bnhd(x, cos, sin, out, pos_offset)
PyObject* rotary_bnhd(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  if (n_args != 5 || !PyLong_CheckExact(a[4])) Py_RETURN_NONE;
  int overflow = 0;
  const long pos = PyLong_AsLongAndOverflow(a[4], &overflow);
  const Tensor *x = plain(a[0]), *cos = plain(a[1]), *sin = plain(a[2]);
  if (overflow || pos < 0 || !dense(x, at::kBFloat16, 4) || !dense(cos, at::kBFloat16, 2) ||
      !dense(sin, at::kBFloat16, 2))
    Py_RETURN_NONE;
  if (cos->sizes() != sin->sizes() || cos->size(0) < x->size(1) + pos || !same_device(*x, {cos, sin}) ||
      !fits({x->size(0), x->size(1), x->size(2), x->size(3), 2 * cos->size(1), pos}))
    Py_RETURN_NONE;
  Tensor out;
  if (!output(a[3], *x, x->sizes(), at::kBFloat16, out)) Py_RETURN_NONE;
  void* st = stream_of(*x);
  const int b = i32(x->size(0)), n = i32(x->size(1)), h = i32(x->size(2)), d = i32(x->size(3)), r = i32(2 * cos->size(1));
  const int dev = x->device().index();
  const void *xp = ptr(*x), *sinp = ptr(*sin), *cosp = ptr(*cos);
  void* outp = ptr(out);
  const int rc = unlocked([&] { return hk_rotary_bnhd(xp, outp, sinp, cosp, b, n, h, d, r, i32(pos), dev, st); });
  if (rc != HK_OK) return PyLong_FromLong(rc);
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// What the paged entries share: q [S,T,H,D], pools [P,page,H_KV,D], block_table [S,max_pages], lengths [S].
struct Paged {
  const Tensor *q, *kp, *vp, *table, *lens;
  int64_t s, t, h, d, pool, page, hkv, max_pages;
  void *q_ptr, *k_pages, *v_pages;
  const int32_t *table_ptr, *lens_ptr;
  int device;
  // What the library call needs of the tensors, read before the interpreter lock is given up.
  void read() {
    q_ptr = ptr(*q), k_pages = ptr(*kp), v_pages = ptr(*vp);
    table_ptr = ptr<int32_t>(*table), lens_ptr = ptr<int32_t>(*lens);
    device = q->device().index();
  }
  bool take(PyObject* const* a) {
    q = plain(a[0]), kp = plain(a[1]), vp = plain(a[2]), table = plain(a[3]), lens = plain(a[4]);
    if (!dense(q, at::kBFloat16, 4) || !dense(kp, at::kBFloat16, 4) || !dense(vp, at::kBFloat16, 4) ||
        !dense(table, at::kInt, 2) || !dense(lens, at::kInt, 1))
      return false;
    s = q->size(0), t = q->size(1), h = q->size(2), d = q->size(3);
    pool = kp->size(0), page = kp->size(1), hkv = kp->size(2), max_pages = table->size(1);
    return kp->size(3) == d && vp->sizes() == kp->sizes() && table->size(0) == s && lens->size(0) == s &&
           same_device(*q, {kp, vp, table, lens}) && fits({s, t, h, d, pool, page, hkv, max_pages});
  }
};

// paged_decode(q, k_pages, v_pages, block_table, ctx_lens, softmax_scale, out, lse, workspace)
PyObject* paged_decode(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  float scale;
  Paged p;
  if (n_args != 9 || !number(a[5], scale) || !p.take(a) || p.t != 1) Py_RETURN_NONE;
  const size_t need = hk_attn_paged_decode_workspace_bytes(i32(p.s), i32(p.h), i32(p.d), i32(p.max_pages), i32(p.page));
  Tensor out, lse, ws;
  if (need == 0 || !output(a[6], *p.q, p.q->sizes(), at::kBFloat16, out) ||
      !output(a[7], *p.q, {p.s, p.h, 1, 1}, at::kFloat, lse))
    Py_RETURN_NONE;
  if (a[8] == Py_None) {
    ws = at::empty({int64_t(need < 256 ? 256 : need)}, p.q->options().dtype(at::kByte).requires_grad(false));
    if (!ws.has_storage()) Py_RETURN_NONE;
  } else {
    const Tensor* t = plain(a[8]);
    if (!dense(t, at::kByte, 1) || t->device() != p.q->device()) Py_RETURN_NONE;
    ws = *t;
  }
  void* st = stream_of(*p.q);
  p.read();
  void *outp = ptr(out), *wsp = ptr(ws);
  float* lsep = ptr<float>(lse);
  const size_t ws_bytes = size_t(ws.numel());
  const int rc = unlocked([&] {
    return hk_attn_paged_decode(p.q_ptr, p.k_pages, p.v_pages, p.table_ptr, p.lens_ptr, outp, lsep, i32(p.s), i32(p.h),
                                i32(p.hkv), i32(p.d), i32(p.page), i32(p.max_pages), i32(p.pool), scale, wsp, ws_bytes,
                                p.device, st);
  });
  return result(rc, out, lse);
  END_HANDLE_TH_ERRORS
}

// attn_fwd_paged(q, k_pages, v_pages, block_table, ctx_lens, causal, softmax_scale, out, lse)
PyObject* attn_fwd_paged(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  float scale;
  Paged p;
  if (n_args != 9 || !PyBool_Check(a[5]) || !number(a[6], scale) || !p.take(a)) Py_RETURN_NONE;
  Tensor out, lse;
  if (!output(a[7], *p.q, p.q->sizes(), at::kBFloat16, out) ||
      !output(a[8], *p.q, {p.s, p.h, 1, p.t}, at::kFloat, lse))
    Py_RETURN_NONE;
  void* st = stream_of(*p.q);
  p.read();
  const int causal = a[5] == Py_True;
  void* outp = ptr(out);
  float* lsep = ptr<float>(lse);
  const int rc = unlocked([&] {
    return hk_attn_fwd_paged(p.q_ptr, p.k_pages, p.v_pages, p.table_ptr, p.lens_ptr, outp, lsep, i32(p.s), i32(p.t),
                             i32(p.h), i32(p.hkv), i32(p.d), i32(p.page), i32(p.max_pages), i32(p.pool), causal, scale,
                             p.device, st);
  });
  return result(rc, out, lse);
  END_HANDLE_TH_ERRORS
}

// paged_kv_append(k_new, v_new, k_pages, v_pages, block_table, start_pos[, cos, sin]): 0 when launched
PyObject* paged_kv_append(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  if (n_args != 6 && n_args != 8) Py_RETURN_NONE;
  const Tensor* v_new = plain(a[1]);
  PyObject* const shared[5] = {a[0], a[2], a[3], a[4], a[5]};
  Paged p;  // k_new in the place of q
  if (!p.take(shared) || !dense(v_new, at::kBFloat16, 4) || v_new->sizes() != p.q->sizes() || p.h != p.hkv ||
      v_new->device() != p.q->device())
    Py_RETURN_NONE;
  const Tensor *cos = nullptr, *sin = nullptr;
  if (n_args == 8) {
    cos = plain(a[6]), sin = plain(a[7]);
    if (!dense(cos, at::kBFloat16, 2) || !dense(sin, at::kBFloat16, 2) || cos->sizes() != sin->sizes() ||
        !same_device(*p.q, {cos, sin}) || !fits({cos->size(0), 2 * cos->size(1)}))
      Py_RETURN_NONE;
  }
  void* st = stream_of(*p.q);
  p.read();
  const void *vp = ptr(*v_new), *cosp = cos ? ptr(*cos) : nullptr, *sinp = cos ? ptr(*sin) : nullptr;
  const int rows = cos ? i32(cos->size(0)) : 0, rotary_dim = cos ? i32(2 * cos->size(1)) : 0;
  const int rc = unlocked([&] {
    if (n_args == 8)
      return hk_paged_kv_append_rotary(p.q_ptr, vp, p.k_pages, p.v_pages, p.table_ptr, p.lens_ptr, sinp, cosp, i32(p.s),
                                       i32(p.t), i32(p.h), i32(p.d), rotary_dim, rows, i32(p.page), i32(p.max_pages),
                                       i32(p.pool), p.device, st);
    return hk_paged_kv_append(p.q_ptr, vp, p.k_pages, p.v_pages, p.table_ptr, p.lens_ptr, i32(p.s), i32(p.t), i32(p.h),
                              i32(p.d), i32(p.page), i32(p.max_pages), i32(p.pool), p.device, st);
  });
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

#define HK_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {HK_METHOD(attn_fwd),       HK_METHOD(attn_bwd_strided), HK_METHOD(rotary_bnhd),
                         HK_METHOD(paged_decode),   HK_METHOD(attn_fwd_paged),   HK_METHOD(paged_kv_append),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_front", "Native tensor front ends of hipkittens_b200", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

// Looked for in the built file, before it is loaded, by whoever wants to know which torch it was compiled against.
extern "C" __attribute__((used, visibility("default"))) const char hk_torch_front_built_for[] =
    "built for torch " HK_TORCH_VERSION;

PyMODINIT_FUNC PyInit__torch_front(void) { return PyModule_Create(&module); }
