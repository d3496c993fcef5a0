// Host side of the operators that short passes are made of: tensor checks, output allocation and launch in one call.
//
// Why: a few-microsecond kernel was issued by 10 to 17 us of Python - attribute reads, ctypes conversions, `torch.empty` -
// around a launch that takes 3.5. Here the same work costs 1 to 2 us (norm 7.8 -> 4.0 us a call, few-rows GEMM 11.9 -> 5.5,
// attention half of a decoded block 34 -> 11.6, launches included). Every function returns None for anything but the
// plain case (dense bf16 CUDA tensors of the current device in the layouts the kernel takes); the Python front ends
// then go through their general path, which converts, falls back or raises. They also keep all rules about WHICH kernel runs:
// nothing in here chooses.
//
// The kernels are those of libb200llm.so, by the handle that the ctypes binding has already opened. The GIL is
// released around them, as ctypes does: a launch blocks while the device's queue is full.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <limits>
#include <optional>
#include <type_traits>

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
typedef const void* cptr;
typedef void* stream_t;

// The C entry points (csrc/*.cu) that are called from here.
struct Api {
  int (*rmsnorm_fwd)(cptr, cptr, void*, void*, int, int, float, stream_t);
  int (*rmsnorm_bwd)(cptr, cptr, cptr, cptr, cptr, void*, void*, void*, int, int, int, stream_t);
  int (*rmsnorm_bwd_partial_rows)(int);
  int (*embedding_fwd)(cptr, cptr, void*, int, int, int, int, stream_t);
  int (*gemm_skinny)(cptr, cptr, void*, cptr, int, int, int, int, int, int, int, int, int, float, stream_t);
  int (*gemm_bf16)(cptr, cptr, void*, cptr, int, int, int, int, int, int, int, int, int, int, float, int, int, int, stream_t);
  int (*gemm_bf16_2cta)(cptr, cptr, void*, cptr, int, int, int, int, int, int, int, int, int, int, float, stream_t);
  int (*gemm_bf16_2cta_split)(cptr, cptr, void*, cptr, int, int, int, int, int, int, int, int, int, int, float, void*, int,
                              stream_t);
  int (*gemm_bf16_2cta_rope)(cptr, cptr, void*, int, int, int, int, int, int, int, int, int, cptr, cptr, int, int, int, int,
                             stream_t);
  int (*gemm_bf16_2cta_swiglu)(cptr, cptr, void*, void*, int, int, int, int, int, int, int, int, stream_t);
  int (*flash_fwd_tc3)(cptr, cptr, cptr, void*, void*, cptr, const long long*, int, int, int, int, int, float, stream_t);
  int (*decode_attn_block)(cptr, cptr, cptr, cptr, void*, void*, void*, void*, void*, cptr, cptr, cptr, int, int, int, int,
                           int, int, int, int, int, float, stream_t);
  int (*mlp_few_rows)(cptr, cptr, cptr, cptr, void*, void*, int, int, int, int, int, stream_t);
};
Api api;

constexpr int MAX_DEVICES = 64;
std::atomic<bool> ready[MAX_DEVICES];          // the device's status block is registered with the library

// A tensor object of exactly torch.Tensor's type (subclasses take the general path); null otherwise.
const Tensor* plain(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

bool current_device(int* dev) {
  *dev = c10::cuda::current_device();
  return *dev >= 0 && *dev < MAX_DEVICES && ready[*dev].load(std::memory_order_relaxed);
}
bool on(const Tensor& t, int dev) { return t.is_cuda() && t.get_device() == dev && t.layout() == c10::kStrided; }
bool bf16_on(const Tensor& t, int dev) { return t.scalar_type() == at::kBFloat16 && on(t, dev); }
bool fits(int64_t v) { return v > 0 && v <= std::numeric_limits<int>::max(); }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
stream_t stream(int dev) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream(); }

// 2-D bf16 with rows that TMA and 16-byte loads can start on
bool tma_rows(const Tensor& t, int dev) {
  return bf16_on(t, dev) && t.dim() == 2 && t.stride(1) == 1 && t.stride(0) % 8 == 0 && aligned16(t.const_data_ptr()) &&
         fits(t.size(0)) && fits(t.size(1)) && fits(t.stride(0));
}
// An optional tensor argument: false when it is neither None nor a plain tensor.
bool optional(PyObject* o, const Tensor** t) {
  *t = o == Py_None ? nullptr : plain(o);
  return o == Py_None || *t != nullptr;
}
// [rows, cols] with unit column stride; *ld = its pitch
bool matrix(const Tensor& t, at::ScalarType dt, int dev, int64_t rows, int64_t cols, int* ld) {
  if (!on(t, dev) || t.scalar_type() != dt || t.dim() != 2 || t.size(0) != rows || t.size(1) != cols || t.stride(1) != 1)
    return false;
  const int64_t l = rows > 1 ? t.stride(0) : std::max(cols, t.stride(0));
  *ld = static_cast<int>(l);
  return fits(l);
}
Tensor empty(at::IntArrayRef size, const Tensor& like, at::ScalarType dt) { return at::empty(size, like.options().dtype(dt)); }
PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap2(const OptTensor& a, const OptTensor& b) {
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) return nullptr;
  for (int i = 0; i < 2; ++i) {
    const OptTensor& t = i == 0 ? a : b;
    PyObject* o = t ? wrap(*t) : Py_NewRef(Py_None);
    if (o == nullptr) {
      Py_DECREF(r);
      return nullptr;
    }
    PyTuple_SET_ITEM(r, i, o);
  }
  return r;
}
// After an error the general path makes the call again and raises. Of a call of several kernels the first ones may have
// been launched by then; made again they write the same: scratch, fresh outputs, the cache row of the new token. An output
// that is also the addend is written by the last kernel only.
template <class F>
bool launched(F call) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = call();
  Py_END_ALLOW_THREADS
  return rc == 0;
}
// Numbers of another type than int (or float) set an error, which CHECK_NUMBERS turns into the general path.
int as_int(PyObject* o) {
  if (PyLong_Check(o)) {
    const long v = PyLong_AsLong(o);
    if (v == static_cast<int>(v)) return static_cast<int>(v);
  }
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "int");
  return 0;
}
float as_float(PyObject* o) { return static_cast<float>(PyFloat_AsDouble(o)); }
bool as_bool(PyObject* o) { return PyObject_IsTrue(o) > 0; }

#define ARGS(count)                                                                        \
  HANDLE_TH_ERRORS                                                                         \
  if (n != (count)) {                                                                      \
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");                         \
    return nullptr;                                                                        \
  }                                                                                        \
  int dev;                                                                                 \
  if (!current_device(&dev)) Py_RETURN_NONE;
#define CHECK_NUMBERS     \
  if (PyErr_Occurred()) { \
    PyErr_Clear();        \
    Py_RETURN_NONE;       \
  }
#define END       \
  Py_RETURN_NONE; \
  END_HANDLE_TH_ERRORS

// rmsnorm_fwd(x, gamma, eps, keep_rstd) -> (y, rstd or None)
PyObject* rmsnorm_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(4)
  const Tensor *x = plain(a[0]), *g = plain(a[1]);
  const float eps = as_float(a[2]);
  const bool keep = as_bool(a[3]);
  CHECK_NUMBERS
  if (x && g && bf16_on(*x, dev) && bf16_on(*g, dev) && x->dim() >= 1 && x->is_contiguous() && g->is_contiguous()) {
    const int64_t H = x->size(-1), M = H > 0 ? x->numel() / H : 0;
    if (fits(H) && fits(M) && g->numel() == H) {
      Tensor y = empty(x->sizes(), *x, at::kBFloat16);
      OptTensor r;
      if (keep) r = empty({M}, *x, at::kFloat);
      if (launched([&] {
            return api.rmsnorm_fwd(x->const_data_ptr(), g->const_data_ptr(), y.mutable_data_ptr(),
                                   keep ? r->mutable_data_ptr() : nullptr, int(M), int(H), eps, stream(dev));
          }))
        return wrap2(y, r);
    }
  }
  END
}

// rmsnorm_bwd(dy, x, gamma, rstd, add or None) -> (dx, dgamma)
PyObject* rmsnorm_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(5)
  const Tensor *dy = plain(a[0]), *x = plain(a[1]), *g = plain(a[2]), *r = plain(a[3]), *add;
  if (dy && x && g && r && optional(a[4], &add) && bf16_on(*x, dev) && bf16_on(*dy, dev) && bf16_on(*g, dev) && on(*r, dev) &&
      r->scalar_type() == at::kFloat && x->dim() >= 1 && x->is_contiguous() && dy->is_contiguous() && g->is_contiguous() &&
      r->is_contiguous() && (!add || (bf16_on(*add, dev) && add->is_contiguous() && add->numel() == x->numel()))) {
    const int64_t H = x->size(-1), M = H > 0 ? x->numel() / H : 0;
    if (fits(H) && fits(M) && g->numel() == H && r->numel() == M && dy->numel() == x->numel()) {
      Tensor dx = empty(x->sizes(), *x, at::kBFloat16), dg = empty(g->sizes(), *x, at::kBFloat16);
      Tensor partial = empty({api.rmsnorm_bwd_partial_rows(int(M)), H}, *x, at::kFloat);
      if (launched([&] {
            return api.rmsnorm_bwd(dy->const_data_ptr(), x->const_data_ptr(), g->const_data_ptr(), r->const_data_ptr(),
                                   add ? add->const_data_ptr() : nullptr, dx.mutable_data_ptr(), dg.mutable_data_ptr(),
                                   partial.mutable_data_ptr(), int(M), int(H), 0, stream(dev));
          }))
        return wrap2(dx, dg);
    }
  }
  END
}

// embedding_fwd(W, idx, pad_id) -> out
PyObject* embedding_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(3)
  const Tensor *w = plain(a[0]), *idx = plain(a[1]);
  const int pad = as_int(a[2]);
  CHECK_NUMBERS
  if (w && idx && bf16_on(*w, dev) && w->dim() == 2 && w->is_contiguous() && on(*idx, dev) && idx->scalar_type() == at::kInt &&
      idx->is_contiguous() && fits(idx->numel()) && fits(w->size(0)) && fits(w->size(1))) {
    Tensor out = empty({idx->numel(), w->size(1)}, *w, at::kBFloat16);
    if (launched([&] {
          return api.embedding_fwd(w->const_data_ptr(), idx->const_data_ptr(), out.mutable_data_ptr(), int(idx->numel()),
                                   int(w->size(1)), pad, int(w->size(0)), stream(dev));
        }))
      return wrap(out);
  }
  END
}

enum Route { TILES = 0, SKINNY = 1, SMALL = 2 };

// gemm(a, b, trans_a, trans_b, out or None, add or None, fp32 output, alpha, whole-tiles and whole-K flags, route, K splits) -> out.
// Routes: CTA-pair tiles (splits > 1: over K), the few-rows kernel, single-CTA tiles.
PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(11)
  const Tensor *x = plain(a[0]), *w = plain(a[1]), *out, *add;
  const bool ta = as_bool(a[2]), tb = as_bool(a[3]), f32 = as_bool(a[6]);
  const float alpha = as_float(a[7]);
  const int whole = as_int(a[8]), route = as_int(a[9]), splits = as_int(a[10]);
  CHECK_NUMBERS
  if (!x || !w || !optional(a[4], &out) || !optional(a[5], &add) || !bf16_on(*x, dev) || !bf16_on(*w, dev) || x->dim() != 2 ||
      w->dim() != 2)
    Py_RETURN_NONE;
  int lda, ldb, ldd = 0, ldc = 0;
  for (const Tensor* t : {x, w})
    if (t->stride(1) != 1 || (t->size(0) > 1 && t->stride(0) < t->size(1)) || !aligned16(t->const_data_ptr()) ||
        !fits(t->size(0)) || !fits(t->size(1)))
      Py_RETURN_NONE;
  if (!matrix(*x, at::kBFloat16, dev, x->size(0), x->size(1), &lda) ||
      !matrix(*w, at::kBFloat16, dev, w->size(0), w->size(1), &ldb) || lda % 8 != 0 || ldb % 8 != 0)
    Py_RETURN_NONE;
  const int64_t M = x->size(ta ? 1 : 0), K = x->size(ta ? 0 : 1), N = w->size(tb ? 0 : 1);
  if (w->size(tb ? 1 : 0) != K || (route == SKINNY && ta)) Py_RETURN_NONE;
  const at::ScalarType dt = f32 ? at::kFloat : at::kBFloat16;
  if ((out && !matrix(*out, dt, dev, M, N, &ldd)) || (add && !matrix(*add, dt, dev, M, N, &ldc))) Py_RETURN_NONE;
  Tensor made;
  if (!out) {
    made = empty({M, N}, *x, dt);
    ldd = int(N);
  }
  const Tensor& d = out ? *out : made;
  void* dp = d.mutable_data_ptr();
  const void* cp = add ? add->const_data_ptr() : nullptr;
  const int flags = (f32 ? 1 : 0) | (add ? 2 : 0);
  const cptr xp = x->const_data_ptr(), wp = w->const_data_ptr();
  const int m = int(M), nn = int(N), k = int(K);
  const stream_t st = stream(dev);
  bool ok = false;
  if (route == SKINNY) {
    ok = launched([&] { return api.gemm_skinny(xp, wp, dp, cp, m, nn, k, lda, ldb, ldd, ldc, !tb, flags & 1, alpha, st); });
  } else if (route == SMALL) {
    ok = launched([&] {
      return api.gemm_bf16(xp, wp, dp, cp, m, nn, k, lda, ldb, ldd, ldc, ta, !tb, flags, alpha, 0, 0, 0, st);
    });
  } else {
    if (!aligned16(dp) || int64_t(ldd) * (f32 ? 4 : 2) % 16 != 0) Py_RETURN_NONE;
    if (splits > 1) {
      Tensor ws = empty({splits * ((M + 255) / 256 * 256) * ((N + 3) / 4 * 4)}, *x, at::kFloat);
      ok = launched([&] {
        return api.gemm_bf16_2cta_split(xp, wp, dp, cp, m, nn, k, lda, ldb, ldd, ldc, ta, !tb, flags, alpha,
                                        ws.mutable_data_ptr(), splits, st);
      });
    } else {
      ok = launched([&] {
        return api.gemm_bf16_2cta(xp, wp, dp, cp, m, nn, k, lda, ldb, ldd, ldc, ta, !tb, flags | whole, alpha, st);
      });
    }
  }
  if (ok) return out ? Py_NewRef(a[4]) : wrap(made);
  END
}

// tma_ok(tensor, ...) -> whether all are 2-D bf16 matrices of the current device with 16-byte aligned rows; None: not plain
PyObject* tma_ok(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int dev;
  if (!current_device(&dev)) Py_RETURN_NONE;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const Tensor* t = plain(a[i]);
    if (!t || !on(*t, dev)) Py_RETURN_NONE;
    if (t->scalar_type() != at::kBFloat16 || t->dim() != 2 || t->stride(1) != 1 || t->stride(0) % 8 != 0 ||
        !aligned16(t->const_data_ptr()))
      Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// gemm_rope(a, w, cos^T, sin^T, T, head_dim, rope_cols, flags) -> out
PyObject* gemm_rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(8)
  const Tensor *x = plain(a[0]), *w = plain(a[1]), *c = plain(a[2]), *s = plain(a[3]);
  const int T = as_int(a[4]), D = as_int(a[5]), cols = as_int(a[6]), flags = as_int(a[7]);
  CHECK_NUMBERS
  if (x && w && c && s && tma_rows(*x, dev) && tma_rows(*w, dev) && x->size(1) == w->size(0) && w->size(1) % 8 == 0 &&
      on(*c, dev) && on(*s, dev) && c->scalar_type() == at::kFloat && s->scalar_type() == at::kFloat && c->dim() == 2 &&
      c->is_contiguous() && s->is_contiguous() && s->sizes() == c->sizes() && c->size(0) == D / 2 && c->size(1) >= T &&
      fits(c->size(1))) {
    const int64_t M = x->size(0), N = w->size(1);
    Tensor out = empty({M, N}, *x, at::kBFloat16);
    if (launched([&] {
          return api.gemm_bf16_2cta_rope(x->const_data_ptr(), w->const_data_ptr(), out.mutable_data_ptr(), int(M), int(N),
                                         int(x->size(1)), int(x->stride(0)), int(w->stride(0)), int(N), 0, 1, flags,
                                         c->const_data_ptr(), s->const_data_ptr(), T, int(c->size(1)), cols, D, stream(dev));
        }))
      return wrap(out);
  }
  END
}

// gemm_swiglu(x, w_gate_val, keep_gv, flags) -> (gv or None, act)
PyObject* gemm_swiglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(4)
  const Tensor *x = plain(a[0]), *w = plain(a[1]);
  const bool keep = as_bool(a[2]);
  const int flags = as_int(a[3]);
  CHECK_NUMBERS
  if (x && w && tma_rows(*x, dev) && tma_rows(*w, dev) && x->size(1) == w->size(0) && w->size(1) % 16 == 0) {
    const int64_t M = x->size(0), I = w->size(1) / 2;
    Tensor act = empty({M, I}, *x, at::kBFloat16);
    OptTensor gv;
    if (keep) gv = empty({M, 2 * I}, *x, at::kBFloat16);
    if (launched([&] {
          return api.gemm_bf16_2cta_swiglu(x->const_data_ptr(), w->const_data_ptr(), keep ? gv->mutable_data_ptr() : nullptr,
                                           act.mutable_data_ptr(), int(M), int(I), int(x->size(1)), int(x->stride(0)),
                                           int(w->stride(0)), int(2 * I), int(I), flags, stream(dev));
        }))
      return wrap2(gv, act);
  }
  END
}

// flash_fwd(q, k, v, valid_len or None, scale) -> (o, lse); inputs already rotated, head_dim 64 or 128
PyObject* flash_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(5)
  const Tensor *q = plain(a[0]), *k = plain(a[1]), *v = plain(a[2]), *vl;
  const float scale = as_float(a[4]);
  CHECK_NUMBERS
  if (!q || !k || !v || !optional(a[3], &vl)) Py_RETURN_NONE;
  for (const Tensor* t : {q, k, v})
    if (!bf16_on(*t, dev) || t->dim() != 4 || t->stride(3) != 1) Py_RETURN_NONE;
  const int64_t B = q->size(0), T = q->size(1), QH = q->size(2), D = q->size(3), KVH = k->size(2);
  if (vl && (!on(*vl, dev) || vl->scalar_type() != at::kInt || !vl->is_contiguous() || vl->numel() != B)) Py_RETURN_NONE;
  if (k->sizes() != v->sizes() || k->size(0) != B || k->size(1) != T || k->size(3) != D || !fits(B) || !fits(T) ||
      !fits(QH) || !fits(KVH))
    Py_RETURN_NONE;
  Tensor o = empty({B, T, QH, D}, *q, at::kBFloat16), lse = empty({B, QH, T}, *q, at::kFloat);
  long long st[12];
  int i = 0;
  for (const Tensor* t : std::initializer_list<const Tensor*>{q, k, v, &o})
    for (int d = 0; d < 3; ++d) st[i++] = t->stride(d);
  if (launched([&] {
        return api.flash_fwd_tc3(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o.mutable_data_ptr(),
                                 lse.mutable_data_ptr(), vl ? vl->const_data_ptr() : nullptr, st, int(B), int(T), int(QH),
                                 int(KVH), int(D), scale, stream(dev));
      }))
    return wrap2(o, lse);
  END
}

// split_heads(kqv [B T, (KVH + QH + KVH) D], B, T, QH, KVH, D) -> (q, k, v) views [B, T, heads, D]
PyObject* split_heads(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(6)
  const Tensor* t = plain(a[0]);
  const int64_t B = as_int(a[1]), T = as_int(a[2]), QH = as_int(a[3]), KVH = as_int(a[4]), D = as_int(a[5]);
  CHECK_NUMBERS
  if (!t || !on(*t, dev) || t->dim() != 2 || B <= 0 || T <= 0 || t->size(0) != B * T || t->size(1) != (QH + 2 * KVH) * D)
    Py_RETURN_NONE;
  const int64_t s0 = t->stride(0), s1 = t->stride(1), off = t->storage_offset();
  auto view = [&](int64_t heads, int64_t first) {
    return at::as_strided(*t, {B, T, heads, D}, {T * s0, s0, D * s1, s1}, off + first * D * s1);
  };
  const Tensor q = view(QH, KVH), k = view(KVH, 0), v = view(KVH, KVH + QH);
  PyObject* r = PyTuple_New(3);
  if (r == nullptr) return nullptr;
  PyTuple_SET_ITEM(r, 0, wrap(q));
  PyTuple_SET_ITEM(r, 1, wrap(k));
  PyTuple_SET_ITEM(r, 2, wrap(v));
  return r;
  END_HANDLE_TH_ERRORS
}

// few rows: x in rows that start on 16 bytes, contiguous weights, a residual (or none) like the output
bool few_rows(const Tensor& x, const Tensor& w0, const Tensor& w1, const Tensor* res, int dev) {
  return tma_rows(x, dev) && tma_rows(w0, dev) && tma_rows(w1, dev) && w0.is_contiguous() && w1.is_contiguous() &&
         (!res || (bf16_on(*res, dev) && res->dim() == 2 && res->size(0) == x.size(0) && res->size(1) == w1.size(1) &&
                   res->stride(1) == 1 && fits(res->stride(0))));
}

// decode_attn_block(x, w_kqv, w_o, kcache, vcache, lens, pos, QH, KVH, cos, sin, scale, residual or None) -> out
PyObject* decode_attn_block(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(13)
  const Tensor *x = plain(a[0]), *w0 = plain(a[1]), *w1 = plain(a[2]), *kc = plain(a[3]), *vc = plain(a[4]),
               *lens = plain(a[5]), *c = plain(a[9]), *s = plain(a[10]), *res;
  const int64_t pos = as_int(a[6]);
  const int QH = as_int(a[7]), KVH = as_int(a[8]);
  const float scale = as_float(a[11]);
  CHECK_NUMBERS
  if (!x || !w0 || !w1 || !kc || !vc || !lens || !c || !s || !optional(a[12], &res) || !few_rows(*x, *w0, *w1, res, dev))
    Py_RETURN_NONE;
  if (!bf16_on(*kc, dev) || !bf16_on(*vc, dev) || kc->dim() != 4 || kc->sizes() != vc->sizes() || !kc->is_contiguous() ||
      !vc->is_contiguous() || !aligned16(kc->const_data_ptr()) || !aligned16(vc->const_data_ptr()) || !on(*lens, dev) ||
      lens->scalar_type() != at::kInt || !lens->is_contiguous())
    Py_RETURN_NONE;
  const int64_t B = x->size(0), H = x->size(1), Tmax = kc->size(2), D = kc->size(3), N = w0->size(1), HO = int64_t(QH) * D;
  if (QH <= 0 || KVH <= 0 || QH % KVH != 0 || (D != 32 && D != 64 && D != 128) || N != (QH + 2 * KVH) * D ||
      w0->size(0) != H || w1->size(0) != HO || w1->size(1) != H || kc->size(0) != B || kc->size(1) != KVH || pos < 0 ||
      pos >= Tmax || !fits(Tmax) || lens->numel() < B)
    Py_RETURN_NONE;
  for (const Tensor* t : {c, s})
    if (!on(*t, dev) || t->scalar_type() != at::kFloat || t->dim() != 2 || !t->is_contiguous() || t->size(0) <= pos ||
        t->size(1) != D / 2)
      Py_RETURN_NONE;
  Tensor scratch = empty({B, N + HO}, *x, at::kBFloat16), out = empty({B, H}, *x, at::kBFloat16);
  char* base = static_cast<char*>(scratch.mutable_data_ptr());
  if (launched([&] {
        return api.decode_attn_block(x->const_data_ptr(), w0->const_data_ptr(), w1->const_data_ptr(),
                                     res ? res->const_data_ptr() : nullptr, out.mutable_data_ptr(), base, base + 2 * B * N,
                                     kc->mutable_data_ptr(), vc->mutable_data_ptr(), lens->const_data_ptr(),
                                     c->const_data_ptr<float>() + pos * (D / 2), s->const_data_ptr<float>() + pos * (D / 2),
                                     int(B), int(H), QH, KVH, int(Tmax), int(D), int(x->stride(0)),
                                     res ? int(res->stride(0)) : 0, int(pos), scale, stream(dev));
      }))
    return wrap(out);
  END
}

// mlp_few_rows(x, w_gate_val, w_out, residual or None) -> out
PyObject* mlp_few_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(4)
  const Tensor *x = plain(a[0]), *w0 = plain(a[1]), *w1 = plain(a[2]), *res;
  if (!x || !w0 || !w1 || !optional(a[3], &res) || !few_rows(*x, *w0, *w1, res, dev)) Py_RETURN_NONE;
  const int64_t M = x->size(0), H = x->size(1), I = w1->size(0);
  if (w0->size(0) != H || w0->size(1) != 2 * I || w1->size(1) != H || I % 8 != 0) Py_RETURN_NONE;
  Tensor act = empty({M, I}, *x, at::kBFloat16), out = empty({M, H}, *x, at::kBFloat16);
  if (launched([&] {
        return api.mlp_few_rows(x->const_data_ptr(), w0->const_data_ptr(), w1->const_data_ptr(),
                                res ? res->const_data_ptr() : nullptr, out.mutable_data_ptr(), act.mutable_data_ptr(), int(M),
                                int(H), int(I), int(x->stride(0)), res ? int(res->stride(0)) : 0, stream(dev));
      }))
    return wrap(out);
  END
}

// memory_room(device index, bytes of the device) -> see ``native.memory_room``
PyObject* memory_room(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const auto dev = static_cast<c10::DeviceIndex>(n == 2 ? PyLong_AsLong(a[0]) : -1);
  const long long total = n == 2 ? PyLong_AsLongLong(a[1]) : 0;
  if (PyErr_Occurred()) return nullptr;
  const auto st = c10::cuda::CUDACachingAllocator::getDeviceStats(dev);
  const auto all = static_cast<size_t>(c10::CachingAllocator::StatType::AGGREGATE);
  const long long share = std::min(static_cast<long long>(c10::cuda::CUDACachingAllocator::getMemoryFraction(dev) * double(total)),
                                   total - total / 32);
  return Py_BuildValue("LL", std::max<long long>(share, st.reserved_bytes[all].current) - st.active_bytes[all].current,
                       static_cast<long long>(st.num_alloc_retries));
  END_HANDLE_TH_ERRORS
}

// bind(handle of libb200llm.so): looks the entry points up; raises when one is missing
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  void* lib = n == 1 ? PyLong_AsVoidPtr(a[0]) : nullptr;
  if (PyErr_Occurred()) return nullptr;
  auto get = [&](auto& f, const char* name) {
    f = reinterpret_cast<std::remove_reference_t<decltype(f)>>(dlsym(lib, name));
    TORCH_CHECK(f != nullptr, "native library without ", name);
  };
  get(api.rmsnorm_fwd, "b200_rmsnorm_fwd");
  get(api.rmsnorm_bwd, "b200_rmsnorm_bwd");
  get(api.rmsnorm_bwd_partial_rows, "b200_rmsnorm_bwd_partial_rows");
  get(api.embedding_fwd, "b200_embedding_fwd");
  get(api.gemm_skinny, "b200_gemm_skinny");
  get(api.gemm_bf16, "b200_gemm_bf16");
  get(api.gemm_bf16_2cta, "b200_gemm_bf16_2cta");
  get(api.gemm_bf16_2cta_split, "b200_gemm_bf16_2cta_split");
  get(api.gemm_bf16_2cta_rope, "b200_gemm_bf16_2cta_rope");
  get(api.gemm_bf16_2cta_swiglu, "b200_gemm_bf16_2cta_swiglu");
  get(api.flash_fwd_tc3, "b200_flash_fwd_tc3");
  get(api.decode_attn_block, "b200_decode_attn_block");
  get(api.mlp_few_rows, "b200_mlp_few_rows");
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// device_ready(index): tensors of this device may come here from now on
PyObject* device_ready(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const long i = n == 1 ? PyLong_AsLong(a[0]) : -1;
  if (PyErr_Occurred()) return nullptr;
  if (i >= 0 && i < MAX_DEVICES) ready[i] = true;
  Py_RETURN_NONE;
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(bind), METHOD(device_ready), METHOD(memory_room), METHOD(rmsnorm_fwd), METHOD(rmsnorm_bwd),
                         METHOD(embedding_fwd), METHOD(gemm), METHOD(tma_ok), METHOD(gemm_rope), METHOD(gemm_swiglu),
                         METHOD(flash_fwd), METHOD(split_heads), METHOD(decode_attn_block), METHOD(mlp_few_rows), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200host() { return PyModule_Create(&module); }
