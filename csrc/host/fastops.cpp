// The calls a training step makes hundreds of times, from Python to the kernel library without Python in between: check the
// tensors, allocate the result through torch's allocator, launch on the current stream.
//
// A step of a narrow model is some hundred launches of a few microseconds each, and the ctypes wrappers of
// zorse_b200/ops/sm100.py cost 7 to 16 us per call on the host (shapes, strides, data pointers, one torch.empty of 1.8 us
// per result, argument conversion), more than the GPU needs.  Here a call takes 3 to 5 us, most of it the launch itself.
//
// Every function returns None, having done nothing, for arguments it was not written for (other types, strides, devices or
// shapes; a device whose status word is not known yet): the caller then goes through the wrapper, which takes or refuses
// them as ever.  Nothing is kept between calls but the entry points and the addresses of the status words.  The GIL is
// released around the launches, which may wait for room in the stream's queue.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/SmallVector.h>

#include <cmath>
#include <cstdint>
#include <utility>

namespace {

using at::Tensor;

constexpr int GEMM_OUT_F32 = 1, GEMM_ACCUMULATE = 2, GEMM_LATE = 16;

// Entry points of the kernel library, in the order `init` gets them.
struct Entry {
  int (*gemm)(const void*, const void*, void*, int, int, int, int, int, int, int, int, const void*, const void*, int, int, int,
              int, int*, cudaStream_t);
  int (*gemm2)(const void*, const void*, void*, int, int, int, int, int, int, int, int, const void*, const void*, int, int, int,
               int*, cudaStream_t);
  int (*gemm2_split)(const void*, const void*, void*, int, int, int, int, int, int, int, int, const void*, const void*, int, int,
                     void*, long, int*, cudaStream_t);
  int (*gemm2_workspace)(int, int, int);
  int (*norm_fwd)(const void*, const void*, const void*, void*, float*, int, int, float, int, cudaStream_t);
  int (*norm_bwd2)(const void*, const void*, const void*, const float*, const void*, void*, float*, float*, void*, void*, int, int,
                   int, int, int, cudaStream_t);
  int (*norm_bwd2_rows)(int, int);
  int (*colsum)(const void*, int, int, int, float*, void*, int, int, cudaStream_t);
  int (*rope)(void*, const float*, int, int, int, int, int, int, cudaStream_t);
  int (*swiglu_fwd)(const void*, void*, long, int, cudaStream_t);
  int (*swiglu_bwd)(const void*, const void*, void*, long, int, cudaStream_t);
  int (*act_fwd)(const void*, void*, long, int, cudaStream_t);
  int (*act_bwd)(const void*, const void*, void*, long, int, cudaStream_t);
  int (*flash_fwd4)(const void*, void*, float*, int, int, int, int, int, int, int, float, int, int*, int, unsigned long long*, int,
                    cudaStream_t);
  int (*flash_bwd3)(const void*, const void*, const void*, const float*, void*, float*, int, int, int, int, int, int, int, float,
                    int*, int, unsigned long long*, int, cudaStream_t);
  int (*flash_stats_floats)(int, int, int);
  int (*gemm2_act_fwd)(const void*, const void*, const void*, void*, void*, int, int, int, int, int, int, int*, cudaStream_t);
  int (*gemm2_act_bwd)(const void*, const void*, const void*, void*, int, int, int, int, int, int, int*, cudaStream_t);
  int (*gemm2_rope_fwd)(const void*, const void*, const void*, const float*, void*, int, int, int, int, int, int, int, int, int*,
                        cudaStream_t);
  int (*column_sums)(const long*, int, int, cudaStream_t);
  const char* (*last_error)();
};
Entry lib;
bool ready = false;
PyObject* kernel_error = nullptr;
int* status_words[64] = {nullptr};
long long launches = 0;

constexpr auto BF16 = at::kBFloat16;
constexpr auto F32 = at::kFloat;

// The tensor behind a plain torch.Tensor (no subclass, which may mean something else by these operations), else nullptr.
const Tensor* tensor_of(PyObject* o) {
  return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr;
}
// ... or of None: `given` tells the two apart
bool optional_tensor(PyObject* o, const Tensor*& t) {
  t = nullptr;
  return o == Py_None || (t = tensor_of(o)) != nullptr;
}
bool strided(const Tensor* t, at::ScalarType type) {
  return t != nullptr && t->defined() && t->layout() == at::kStrided && t->is_cuda() && t->scalar_type() == type;
}
bool matrix(const Tensor* t, at::ScalarType type) {   // rows of any distance, each one contiguous
  return strided(t, type) && t->dim() == 2 && t->stride(1) == 1;
}
bool dense(const Tensor* t, at::ScalarType type) { return strided(t, type) && t->is_contiguous(); }
bool gradient(const Tensor* t) { return t != nullptr && (dense(t, F32) || dense(t, BF16)); }
bool on(const Tensor* t, const Tensor& like) { return t == nullptr || t->device() == like.device(); }
bool fits(int64_t v) { return v > 0 && v <= INT32_MAX; }

// The status word of the tensor's device if that is the current one (whose stream the launch goes to), else nullptr.
int* status_of(const Tensor& t) {
  const int d = t.get_device();
  return ready && d >= 0 && d < 64 && d == c10::cuda::current_device() ? status_words[d] : nullptr;
}
cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
Tensor empty(at::IntArrayRef sizes, const Tensor& like, at::ScalarType type) {
  return at::empty(sizes, like.options().dtype(type).requires_grad(false));
}
void* ptr(const Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }

// Runs `f` (the launches, 0 or an error code) without the GIL; counts `n` launches or raises KernelError.  An entry point
// answers 1, having done nothing, to what it was not written for: false without an error then where `declined` is given.
template <typename F>
bool launch(const char* what, int n, F&& f, bool* declined = nullptr) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  if (rc == 1 && declined != nullptr) {
    *declined = true;
    return false;
  }
  if (rc != 0) {   // (the error text is this thread's, and of an earlier error where this entry point set none)
    PyErr_Format(kernel_error, "%s: %s", what, rc == 1 ? "arguments it does not take" : lib.last_error());
    return false;
  }
  launches += n;
  return true;
}

bool int_arg(PyObject* o, int64_t& v) {
  v = PyLong_Check(o) ? PyLong_AsLongLong(o) : -1;
  if (PyErr_Occurred()) { PyErr_Clear(); return false; }
  return PyLong_Check(o);
}
bool truth(PyObject* o) { return PyObject_IsTrue(o) == 1; }

#define ZB_ARGS(n)                                                                          \
  if (nargs != n) {                                                                         \
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");                          \
    return nullptr;                                                                         \
  }

// Whether out[M, N] (+)= A B^T is a product for here.
bool product(const Tensor* a, const Tensor* b, const Tensor& out, bool a_mn, bool b_mn) {
  const int64_t M = out.size(0), N = out.size(1), K = a->size(a_mn ? 0 : 1);
  return a->size(a_mn ? 1 : 0) == M && b->size(b_mn ? 1 : 0) == N && b->size(b_mn ? 0 : 1) == K && fits(M) && fits(N) && fits(K) &&
         fits(a->stride(0)) && fits(b->stride(0)) && fits(out.stride(0));
}

// The workspace for a product whose last wave of tiles is to be cut along K; undefined where it is not.
Tensor split_workspace(int64_t M, int64_t N, int64_t K, const Tensor& like) {
  // (the same lines as in the wrapper: shorter reductions are never cut)
  const int bytes = M >= 256 && N >= 256 && K > 3000 ? lib.gemm2_workspace(int(M), int(N), int(K)) : 0;
  return bytes > 0 ? empty({bytes}, like, at::kByte) : Tensor();
}

// out[M, N] (+)= A B^T; `out` as the caller prepared it.  1: done, 0: not for here, -1: error set.
// more: flags, GEMM_LATE for one that starts under the kernel before it; workspace: what split_workspace gave, nullptr: gemm
// asks itself.
int gemm(const Tensor* a, const Tensor* b, const Tensor& out, bool a_mn, bool b_mn, const Tensor* bias, const Tensor* addend,
         bool accumulate, int* status, int more = 0, const Tensor* workspace = nullptr) {
  const int64_t M = out.size(0), N = out.size(1), K = a->size(a_mn ? 0 : 1);
  if (!product(a, b, out, a_mn, b_mn)) return 0;
  if (bias != nullptr && !(dense(bias, BF16) && bias->dim() == 1 && bias->size(0) == N)) return 0;
  if (addend != nullptr && !(matrix(addend, BF16) && addend->size(0) == M && addend->size(1) == N && fits(addend->stride(0))))
    return 0;
  const int flags = (out.scalar_type() == F32 ? GEMM_OUT_F32 : 0) | (accumulate ? GEMM_ACCUMULATE : 0) | more;
  const int lda = int(a->stride(0)), ldb = int(b->stride(0)), ldc = int(out.stride(0));
  const int ldx = addend == nullptr ? 0 : int(addend->stride(0));
  const void *pa = ptr(a), *pb = ptr(b), *pbias = ptr(bias), *px = ptr(addend);
  void* pc = out.data_ptr();
  const cudaStream_t s = stream();
  const int m = int(M), n = int(N), k = int(K);
  if (m < 256 || n < 256)
    return launch("gemm", 1, [&] {
      return lib.gemm(pa, pb, pc, m, n, k, lda, ldb, ldc, a_mn, b_mn, pbias, px, ldx, flags, 0, 0, status, s);
    }) ? 1 : -1;
  const Tensor ws = workspace != nullptr ? *workspace : split_workspace(m, n, k, *a);
  if (ws.defined()) {
    void* pw = ws.data_ptr();
    const long ws_bytes = ws.numel();
    return launch("gemm2_split", 1, [&] {
      return lib.gemm2_split(pa, pb, pc, m, n, k, lda, ldb, ldc, a_mn, b_mn, pbias, px, ldx, flags, pw, ws_bytes, status, s);
    }) ? 1 : -1;
  }
  return launch("gemm2", 1, [&] {
    return lib.gemm2(pa, pb, pc, m, n, k, lda, ldb, ldc, a_mn, b_mn, pbias, px, ldx, flags, 0, status, s);
  }) ? 1 : -1;
}

// Whether zb_column_sums takes this bf16 matrix.
bool summable(const Tensor& t) {
  return t.size(1) % 8 == 0 && t.stride(0) % 8 == 0 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}
bool later(PyObject* list, PyObject* entry) {   // (takes over `entry`)
  if (entry == nullptr) return false;
  const int rc = PyList_Append(list, entry);
  Py_DECREF(entry);
  return rc == 0;
}

PyObject* forward_like(PyObject* const* args, bool b_mn, PyObject* bias_o, PyObject* add_o) {
  const Tensor *x = tensor_of(args[0]), *w = tensor_of(args[1]), *bias, *add;
  if (!optional_tensor(bias_o, bias) || !optional_tensor(add_o, add) || !matrix(x, BF16) || !matrix(w, BF16)) Py_RETURN_NONE;
  if (!on(w, *x) || !on(bias, *x) || !on(add, *x)) Py_RETURN_NONE;
  int* status = status_of(*x);
  if (status == nullptr) Py_RETURN_NONE;
  if (x->size(1) != w->size(b_mn ? 0 : 1) || !fits(x->size(0)) || !fits(w->size(b_mn ? 1 : 0))) Py_RETURN_NONE;
  Tensor y = empty({x->size(0), w->size(b_mn ? 1 : 0)}, *x, BF16);
  const int done = gemm(x, w, y, false, b_mn, bias, add, false, status);
  if (done < 0) return nullptr;
  if (done == 0) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(y));
}

// linear_fwd(x, w, bias | None, addend | None) -> x w^T (+ bias) (+ addend)
PyObject* linear_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(4)
  return forward_like(args, false, args[2], args[3]);
  END_HANDLE_TH_ERRORS
}
// linear_dgrad(dy, w, addend | None) -> dy w (+ addend)
PyObject* linear_dgrad(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(3)
  return forward_like(args, true, Py_None, args[2]);
  END_HANDLE_TH_ERRORS
}
// linear_wgrad(dy, x, gw, gb | None, later | None): gw += dy^T x, gb += column sums of dy.  With a list `later` both are left
// to finish, (dy, x, gw, gb | None) appended.  True when done.
PyObject* linear_wgrad(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(5)
  const Tensor *dy = tensor_of(args[0]), *x = tensor_of(args[1]), *gw = tensor_of(args[2]), *gb;
  if (!optional_tensor(args[3], gb) || !matrix(dy, BF16) || !matrix(x, BF16)) Py_RETURN_NONE;
  if (!(matrix(gw, F32) || matrix(gw, BF16)) || !on(x, *dy) || !on(gw, *dy) || !on(gb, *dy)) Py_RETURN_NONE;
  if (gb != nullptr && !(gradient(gb) && gb->dim() == 1 && gb->size(0) == dy->size(1))) Py_RETURN_NONE;
  int* status = status_of(*dy);
  if (status == nullptr) Py_RETURN_NONE;
  if (PyList_Check(args[4]) && product(dy, x, *gw, true, true) && (gb == nullptr || summable(*dy)))
    return later(args[4], PyTuple_Pack(4, args[0], args[1], args[2], args[3])) ? Py_NewRef(Py_True) : nullptr;
  const int done = gemm(dy, x, *gw, true, true, nullptr, nullptr, true, status);
  if (done < 0) return nullptr;
  if (done == 0) Py_RETURN_NONE;
  if (gb != nullptr) {
    const int64_t T = dy->size(0), N = dy->size(1);
    const Tensor part = empty({T < 64 ? T : 64, N}, *dy, F32);
    const cudaStream_t s = stream();
    if (!launch("colsum", 1, [&] {
          return lib.colsum(dy->data_ptr(), int(T), int(N), int(dy->stride(0)), static_cast<float*>(part.data_ptr()),
                            gb->data_ptr(), gb->scalar_type() == F32, 1, s);
        }))
      return nullptr;
  }
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

constexpr int64_t ACT_SWIGLU = 3;   // the activation kinds of zb_gemm2_act_fwd: 0 - 2 as in act_fwd

// act_linear_fwd(x, w, bias | None, kind, keep) -> (act(x w^T + bias), pre-activations | None)
PyObject* act_linear_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(5)
  const Tensor *x = tensor_of(args[0]), *w = tensor_of(args[1]), *bias;
  int64_t kind;
  if (!optional_tensor(args[2], bias) || !matrix(x, BF16) || !matrix(w, BF16) || !int_arg(args[3], kind) || kind < 0 ||
      kind > ACT_SWIGLU || !on(w, *x) || !on(bias, *x))
    Py_RETURN_NONE;
  const int64_t M = x->size(0), K = x->size(1), W = w->size(0), N = kind == ACT_SWIGLU ? W / 2 : W;
  int* status = status_of(*x);
  if (status == nullptr || w->size(1) != K || !fits(M) || !fits(W) || !fits(K) || !fits(x->stride(0)) || !fits(w->stride(0)) ||
      (kind == ACT_SWIGLU && (bias != nullptr || W % 2)) || M < 256 || N < 256 || N % 8)
    Py_RETURN_NONE;
  if (bias != nullptr && !(dense(bias, BF16) && bias->dim() == 1 && bias->size(0) == W)) Py_RETURN_NONE;
  Tensor out = empty({M, N}, *x, BF16), pre;
  if (truth(args[4])) pre = empty({M, W}, *x, BF16);
  void* pp = pre.defined() ? pre.data_ptr() : nullptr;
  const cudaStream_t s = stream();
  bool declined = false;
  if (!launch("gemm2_act_fwd", 1, [&] {
        return lib.gemm2_act_fwd(ptr(x), ptr(w), ptr(bias), pp, out.data_ptr(), int(M), int(N), int(K), int(x->stride(0)),
                                 int(w->stride(0)), int(kind), status, s);
      }, &declined)) {
    if (declined) Py_RETURN_NONE;
    return nullptr;
  }
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(r, 1, pp != nullptr ? THPVariable_Wrap(std::move(pre)) : Py_NewRef(Py_None));
  return r;
  END_HANDLE_TH_ERRORS
}

// linear_rope_fwd(x, w, bias | None, cs, S, heads, d) -> x w^T + bias with its first `heads` heads rotated
PyObject* linear_rope_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(7)
  const Tensor *x = tensor_of(args[0]), *w = tensor_of(args[1]), *bias, *cs = tensor_of(args[3]);
  int64_t S, heads, d;
  if (!optional_tensor(args[2], bias) || !matrix(x, BF16) || !matrix(w, BF16) || !dense(cs, F32) || !int_arg(args[4], S) ||
      !int_arg(args[5], heads) || !int_arg(args[6], d) || !on(w, *x) || !on(bias, *x) || !on(cs, *x))
    Py_RETURN_NONE;
  const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
  int* status = status_of(*x);
  if (status == nullptr || w->size(1) != K || !fits(M) || !fits(N) || !fits(K) || !fits(x->stride(0)) || !fits(w->stride(0)) ||
      !fits(S) || M < 256 || N < 256 || (d != 64 && d != 128) || N % d || S <= 0 || heads <= 0 || heads > N / d ||
      cs->dim() != 2 || cs->size(0) < S || cs->size(1) != d || (reinterpret_cast<uintptr_t>(ptr(cs)) & 15))
    Py_RETURN_NONE;
  if (bias != nullptr && !(dense(bias, BF16) && bias->dim() == 1 && bias->size(0) == N)) Py_RETURN_NONE;
  Tensor out = empty({M, N}, *x, BF16);
  const cudaStream_t s = stream();
  bool declined = false;
  if (!launch("gemm2_rope_fwd", 1, [&] {
        return lib.gemm2_rope_fwd(ptr(x), ptr(w), ptr(bias), static_cast<const float*>(ptr(cs)), out.data_ptr(), int(M), int(N),
                                  int(K), int(x->stride(0)), int(w->stride(0)), int(S), int(heads), int(d), status, s);
      }, &declined)) {
    if (declined) Py_RETURN_NONE;
    return nullptr;
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// act_linear_dgrad(dy, w, pre, kind) -> (dy w) act'(pre)
PyObject* act_linear_dgrad(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(4)
  const Tensor *dy = tensor_of(args[0]), *w = tensor_of(args[1]), *pre = tensor_of(args[2]);
  int64_t kind;
  if (!matrix(dy, BF16) || !matrix(w, BF16) || !dense(pre, BF16) || pre->dim() != 2 || !int_arg(args[3], kind) || kind < 0 ||
      kind > ACT_SWIGLU || !on(w, *dy) || !on(pre, *dy))
    Py_RETURN_NONE;
  const int64_t M = dy->size(0), K = dy->size(1), N = w->size(1);
  int* status = status_of(*dy);
  if (status == nullptr || w->size(0) != K || pre->size(0) != M || pre->size(1) != (kind == ACT_SWIGLU ? 2 * N : N) || !fits(M) ||
      !fits(2 * N) || !fits(K) || !fits(dy->stride(0)) || !fits(w->stride(0)) || M < 256 || N < 256 || N % 8)
    Py_RETURN_NONE;
  Tensor dpre = empty(pre->sizes(), *dy, BF16);
  const cudaStream_t s = stream();
  bool declined = false;
  if (!launch("gemm2_act_bwd", 1, [&] {
        return lib.gemm2_act_bwd(ptr(dy), ptr(w), ptr(pre), dpre.data_ptr(), int(M), int(N), int(K), int(dy->stride(0)),
                                 int(w->stride(0)), int(kind), status, s);
      }, &declined)) {
    if (declined) Py_RETURN_NONE;
    return nullptr;
  }
  return THPVariable_Wrap(std::move(dpre));
  END_HANDLE_TH_ERRORS
}

// norm_fwd(x, w, b | None, eps, layernorm) -> (y, stats)
PyObject* norm_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(5)
  const Tensor *x = tensor_of(args[0]), *w = tensor_of(args[1]), *b;
  if (!optional_tensor(args[2], b) || !dense(x, BF16) || x->dim() != 2 || !dense(w, BF16) || !PyFloat_Check(args[3])) Py_RETURN_NONE;
  const int64_t T = x->size(0), H = x->size(1);
  if (!fits(T) || !fits(H) || w->numel() != H || !on(w, *x) || !on(b, *x)) Py_RETURN_NONE;
  if (b != nullptr && !(dense(b, BF16) && b->numel() == H)) Py_RETURN_NONE;
  if (status_of(*x) == nullptr) Py_RETURN_NONE;
  Tensor y = empty({T, H}, *x, BF16), stats = empty({T, 2}, *x, F32);
  const float eps = float(PyFloat_AS_DOUBLE(args[3]));
  const bool ln = truth(args[4]);
  const cudaStream_t s = stream();
  if (!launch("norm_fwd", 1, [&] {
        return lib.norm_fwd(ptr(x), ptr(w), ptr(b), y.data_ptr(), static_cast<float*>(stats.data_ptr()), int(T), int(H), eps, ln, s);
      }))
    return nullptr;
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(y)));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(stats)));
  return r;
  END_HANDLE_TH_ERRORS
}

// norm_bwd(dy, x, w, stats, dres | None, dw, db | None, layernorm, later | None) -> dx (+ dres); dw, db are added to, or,
// with a list `later`, left to finish as (partial sums, dw, db | None)
PyObject* norm_bwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(9)
  const Tensor *dy = tensor_of(args[0]), *x = tensor_of(args[1]), *w = tensor_of(args[2]), *stats = tensor_of(args[3]);
  const Tensor *dres, *dw = tensor_of(args[5]), *db;
  if (!optional_tensor(args[4], dres) || !optional_tensor(args[6], db) || !dense(dy, BF16) || !dense(x, BF16) ||
      x->dim() != 2 || !dense(w, BF16) || !dense(stats, F32) || !gradient(dw))
    Py_RETURN_NONE;
  const int64_t T = x->size(0), H = x->size(1);
  const bool ln = truth(args[7]);
  if (!fits(T) || !fits(H) || dy->sizes() != x->sizes() || w->numel() != H || stats->numel() != 2 * T || dw->numel() != H)
    Py_RETURN_NONE;
  if (dres != nullptr && !(dense(dres, BF16) && dres->sizes() == x->sizes())) Py_RETURN_NONE;
  if (db != nullptr && !(gradient(db) && db->numel() == H && db->scalar_type() == dw->scalar_type())) Py_RETURN_NONE;
  if (!on(dy, *x) || !on(w, *x) || !on(stats, *x) || !on(dres, *x) || !on(dw, *x) || !on(db, *x)) Py_RETURN_NONE;
  if (status_of(*x) == nullptr) Py_RETURN_NONE;
  const bool bias = ln && db != nullptr;
  const bool defer = PyList_Check(args[8]);
  const int64_t P = lib.norm_bwd2_rows(int(T), int(H));
  Tensor dx = empty({T, H}, *x, BF16);
  Tensor part = empty({bias ? 2 : 1, P, H}, *x, F32);
  float* part_dw = static_cast<float*>(part.data_ptr());
  float* part_db = bias ? part_dw + P * H : nullptr;
  const cudaStream_t s = stream();
  if (!launch("norm_bwd", 1, [&] {
        return lib.norm_bwd2(ptr(dy), ptr(x), ptr(w), static_cast<const float*>(ptr(stats)), ptr(dres), dx.data_ptr(), part_dw,
                             part_db, defer ? nullptr : ptr(dw), defer ? nullptr : ptr(db), int(T), int(H), ln,
                             dw->scalar_type() == F32, 1, s);
      }))
    return nullptr;
  if (defer) {
    PyObject* sums = THPVariable_Wrap(std::move(part));
    if (sums == nullptr) return nullptr;
    PyObject* entry = PyTuple_Pack(3, sums, args[5], bias ? args[6] : Py_None);
    Py_DECREF(sums);
    if (!later(args[8], entry)) return nullptr;
  }
  return THPVariable_Wrap(std::move(dx));
  END_HANDLE_TH_ERRORS
}

// finish(later): the products and column sums that linear_wgrad and norm_bwd have left in the list, which is emptied.
//
// No product reads what another one writes, so each but the first starts on the SMs that the one before it has done with,
// where one after the other every one ended with most of the GPU idle (a BERT block's four weight gradients are 54, 18, 72 and
// 72 tiles on 74 pairs), and the column sums take up SMs as the last product leaves them (such a list is 59 us, its products alone
// 47: the sources have left L2 by then).  All operands stay in the list until everything is
// launched, and the workspaces are taken ahead of the first launch (what the allocator hands out behind it may have been given
// back by another thread while kernels on this stream still use it): the rules of chain_late (ptx.cuh).
// Long products are cut along K as they are alone, for the same bits and the same accuracy: what a tensor core adds to an
// accumulator it truncates, so the error of an fp32 result grows with the tokens summed in one (9.1e-6 over 8192), and with
// whole products in the list weights of 512 columns, all of whose tiles are cut alone (512 x 512: 4.8e-7), lost up to a
// factor of 19.  But for the last, products with a side that is no multiple of 32, which no layer here has, stay whole: their
// results in a list have been held to the bits of whole tiles.
// A product whose gradient lies in memory that an earlier one of the list writes (two calls for one parameter) waits for it.
PyObject* finish(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(1)
  if (!PyList_Check(args[0]) || !ready) {
    PyErr_SetString(PyExc_TypeError, "finish takes the list that linear_wgrad and norm_bwd have filled");
    return nullptr;
  }
  auto refuse = [] {
    PyErr_SetString(PyExc_TypeError, "finish: an entry that linear_wgrad or norm_bwd did not make");
    return nullptr;
  };
  const Py_ssize_t entries = PyList_GET_SIZE(args[0]);
  Py_ssize_t last = -1, launched = 0;
  for (Py_ssize_t i = 0; i < entries; ++i) {
    PyObject* e = PyList_GET_ITEM(args[0], i);
    if (!PyTuple_Check(e) || (PyTuple_GET_SIZE(e) != 3 && PyTuple_GET_SIZE(e) != 4)) return refuse();
    if (PyTuple_GET_SIZE(e) == 4) last = i;
  }
  c10::SmallVector<Tensor, 8> workspaces;   // one per product, undefined for one that runs whole
  for (Py_ssize_t i = 0; i <= last; ++i) {
    PyObject* e = PyList_GET_ITEM(args[0], i);
    if (PyTuple_GET_SIZE(e) != 4) continue;
    const Tensor *dy = tensor_of(PyTuple_GET_ITEM(e, 0)), *gw = tensor_of(PyTuple_GET_ITEM(e, 2));
    if (dy == nullptr || gw == nullptr || dy->dim() != 2 || gw->dim() != 2 || !dy->is_cuda()) return refuse();
    const int64_t M = gw->size(0), N = gw->size(1);
    workspaces.push_back(i == last || (M % 32 == 0 && N % 32 == 0) ? split_workspace(M, N, dy->size(0), *dy) : Tensor());
  }
  constexpr int MAX = 8;   // sums per launch
  long desc[MAX][7];
  int n = 0;
  bool late = false;       // a product has been launched here: what the sums read was complete before it
  // Bytes that kernels launched here, or sums not launched yet, add to; `claim` answers whether none of them is in `out`,
  // which else has to wait: then all of them are done, and the record starts anew.
  c10::SmallVector<std::pair<uintptr_t, uintptr_t>, 16> written;
  auto claim = [&](const Tensor& out) {
    const uintptr_t lo = reinterpret_cast<uintptr_t>(out.data_ptr());
    const int64_t last = out.dim() == 2 ? (out.size(0) - 1) * out.stride(0) + out.size(1) : out.numel();
    const uintptr_t hi = lo + uintptr_t(last) * out.element_size();
    bool free = true;
    for (const auto& w : written) free = free && (hi <= w.first || w.second <= lo);
    if (!free) written.clear();
    written.emplace_back(lo, hi);
    return free;
  };
  const cudaStream_t s = stream();
  for (Py_ssize_t i = 0; i < entries; ++i) {
    PyObject* e = PyList_GET_ITEM(args[0], i);
    if (PyTuple_GET_SIZE(e) != 4) continue;
    const Tensor *dy = tensor_of(PyTuple_GET_ITEM(e, 0)), *x = tensor_of(PyTuple_GET_ITEM(e, 1)), *gw = tensor_of(PyTuple_GET_ITEM(e, 2));
    if (dy == nullptr || x == nullptr || gw == nullptr) return refuse();
    int* status = status_of(*dy);
    if (status == nullptr) return refuse();
    const bool free = claim(*gw);
    const int done = gemm(dy, x, *gw, true, true, nullptr, nullptr, true, status, launched == 0 || !free ? 0 : GEMM_LATE,
                          &workspaces[launched]);
    ++launched;
    if (done < 0) return nullptr;
    if (done == 0) return refuse();
    late = true;
  }
  auto run = [&] {
    const bool ok = n == 0 || launch("column_sums", 1, [&] { return lib.column_sums(desc[0], n, late, s); });
    n = 0;
    return ok;
  };
  auto add = [&](const Tensor& src, int64_t offset, int64_t rows, int64_t cols, int64_t ld, const Tensor& out) {
    if (n == MAX && !run()) return false;
    if (!claim(out)) {
      if (!run()) return false;
      late = false;
    }
    const bool f32 = src.scalar_type() == F32;
    const long d[7] = {reinterpret_cast<long>(src.data_ptr()) + long(offset * (f32 ? 4 : 2)), reinterpret_cast<long>(out.data_ptr()),
                       long(rows), long(cols), long(ld), f32, out.scalar_type() == F32};
    memcpy(desc[n++], d, sizeof(d));
    return true;
  };
  for (Py_ssize_t i = 0; i < entries; ++i) {
    PyObject* e = PyList_GET_ITEM(args[0], i);
    const Tensor* src = tensor_of(PyTuple_GET_ITEM(e, 0));
    if (src == nullptr) return refuse();
    if (PyTuple_GET_SIZE(e) == 4) {
      const Tensor* gb;
      if (!optional_tensor(PyTuple_GET_ITEM(e, 3), gb)) return refuse();
      if (gb != nullptr && !add(*src, 0, src->size(0), src->size(1), src->stride(0), *gb)) return nullptr;
    } else {
      const Tensor *out = tensor_of(PyTuple_GET_ITEM(e, 1)), *second;
      if (out == nullptr || !optional_tensor(PyTuple_GET_ITEM(e, 2), second) || src->dim() != 3) return refuse();
      const int64_t P = src->size(1), H = src->size(2);
      if (!add(*src, 0, P, H, H, *out) || (second != nullptr && !add(*src, P * H, P, H, H, *second))) return nullptr;
    }
  }
  if (!run()) return nullptr;
  if (PyList_SetSlice(args[0], 0, entries, nullptr) != 0) return nullptr;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// rope(buf, cs, S, nheads, d, backward): in place.  True when done.
PyObject* rope(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(6)
  const Tensor *buf = tensor_of(args[0]), *cs = tensor_of(args[1]);
  int64_t S, heads, d;
  if (!matrix(buf, BF16) || !dense(cs, F32) || !on(cs, *buf) || !int_arg(args[2], S) || !int_arg(args[3], heads) ||
      !int_arg(args[4], d) || !fits(S) || !fits(heads) || !fits(d) || !fits(buf->size(0)) || !fits(buf->stride(0)) ||
      heads * d > buf->size(1) || cs->dim() != 2 || cs->size(0) < S || cs->size(1) != d || status_of(*buf) == nullptr)
    Py_RETURN_NONE;
  const bool backward = truth(args[5]);
  const cudaStream_t s = stream();
  if (!launch("rope", 1, [&] {
        return lib.rope(ptr(buf), static_cast<const float*>(ptr(cs)), int(buf->size(0)), int(S), int(heads), int(d),
                        int(buf->stride(0)), backward, s);
      }))
    return nullptr;
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// swiglu_fwd(gu) -> silu(gate) * up
PyObject* swiglu_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(1)
  const Tensor* gu = tensor_of(args[0]);
  if (!dense(gu, BF16) || gu->dim() != 2 || gu->size(1) % 2 || !fits(gu->size(0)) || !fits(gu->size(1)) || status_of(*gu) == nullptr)
    Py_RETURN_NONE;
  const int64_t T = gu->size(0), F = gu->size(1) / 2;
  Tensor out = empty({T, F}, *gu, BF16);
  const cudaStream_t s = stream();
  if (!launch("swiglu_fwd", 1, [&] { return lib.swiglu_fwd(ptr(gu), out.data_ptr(), T, int(F), s); })) return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}
// swiglu_bwd(gu, dout) -> dgu
PyObject* swiglu_bwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(2)
  const Tensor *gu = tensor_of(args[0]), *dout = tensor_of(args[1]);
  if (!dense(gu, BF16) || gu->dim() != 2 || !dense(dout, BF16) || dout->dim() != 2 || !on(dout, *gu) ||
      dout->size(0) != gu->size(0) || 2 * dout->size(1) != gu->size(1) || !fits(gu->size(0)) || !fits(gu->size(1)) ||
      status_of(*gu) == nullptr)
    Py_RETURN_NONE;
  Tensor dgu = empty(gu->sizes(), *gu, BF16);
  const cudaStream_t s = stream();
  if (!launch("swiglu_bwd", 1, [&] {
        return lib.swiglu_bwd(ptr(gu), ptr(dout), dgu.data_ptr(), gu->size(0), int(dout->size(1)), s);
      }))
    return nullptr;
  return THPVariable_Wrap(std::move(dgu));
  END_HANDLE_TH_ERRORS
}
// act_fwd(x, kind) -> y
PyObject* act_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(2)
  const Tensor* x = tensor_of(args[0]);
  int64_t kind;
  if (!dense(x, BF16) || !int_arg(args[1], kind) || x->numel() == 0 || status_of(*x) == nullptr) Py_RETURN_NONE;
  Tensor y = empty(x->sizes(), *x, BF16);
  const cudaStream_t s = stream();
  if (!launch("act_fwd", 1, [&] { return lib.act_fwd(ptr(x), y.data_ptr(), x->numel(), int(kind), s); })) return nullptr;
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}
// act_bwd(x, dy, kind) -> dx
PyObject* act_bwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(3)
  const Tensor *x = tensor_of(args[0]), *dy = tensor_of(args[1]);
  int64_t kind;
  if (!dense(x, BF16) || !dense(dy, BF16) || !on(dy, *x) || dy->sizes() != x->sizes() || !int_arg(args[2], kind) ||
      x->numel() == 0 || status_of(*x) == nullptr)
    Py_RETURN_NONE;
  Tensor dx = empty(x->sizes(), *x, BF16);
  const cudaStream_t s = stream();
  if (!launch("act_bwd", 1, [&] { return lib.act_bwd(ptr(x), ptr(dy), dx.data_ptr(), x->numel(), int(kind), s); })) return nullptr;
  return THPVariable_Wrap(std::move(dx));
  END_HANDLE_TH_ERRORS
}

struct AttnArgs {
  int64_t B, S, Hq, Hkv, D, window;
  bool causal;
};
// B, S, Hq, Hkv, D, causal, window from args; the sizes of `qkv`
bool attn_args(PyObject* const* args, const Tensor* qkv, AttnArgs& a) {
  if (!int_arg(args[0], a.B) || !int_arg(args[1], a.S) || !int_arg(args[2], a.Hq) || !int_arg(args[3], a.Hkv) ||
      !int_arg(args[4], a.D) || !int_arg(args[6], a.window))
    return false;
  a.causal = truth(args[5]);
  if (!fits(a.B) || !fits(a.S) || !fits(a.Hq) || !fits(a.Hkv) || !fits(a.D) || a.window < 0) return false;
  if (a.window >= a.S) a.window = 0;   // every earlier key is visible
  return dense(qkv, BF16) && qkv->dim() == 2 && qkv->size(0) == a.B * a.S && qkv->size(1) == (a.Hq + 2 * a.Hkv) * a.D &&
         fits(qkv->size(0)) && fits(qkv->size(1)) && status_of(*qkv) != nullptr;
}

// attn_fwd(qkv, B, S, Hq, Hkv, D, causal, window, flags) -> (out, lse), the two-query-tile kernel
PyObject* attn_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(9)
  const Tensor* qkv = tensor_of(args[0]);
  AttnArgs a;
  int64_t flags;
  if (!attn_args(args + 1, qkv, a) || !int_arg(args[8], flags)) Py_RETURN_NONE;
  Tensor out = empty({a.B * a.S, a.Hq * a.D}, *qkv, BF16), lse = empty({a.B, a.Hq, a.S}, *qkv, F32);
  const float scale = float(1.0 / std::sqrt(double(a.D)));
  int* status = status_of(*qkv);
  const cudaStream_t s = stream();
  if (!launch("flash_fwd4", 1, [&] {
        return lib.flash_fwd4(ptr(qkv), out.data_ptr(), static_cast<float*>(lse.data_ptr()), int(a.B), int(a.S), int(a.Hq),
                              int(a.Hkv), int(a.D), a.causal, int(a.window), scale, int(a.Hq * a.D), status, int(flags), nullptr,
                              0, s);
      }))
    return nullptr;
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(lse)));
  return r;
  END_HANDLE_TH_ERRORS
}

// attn_bwd(do, qkv, o, lse, B, S, Hq, Hkv, D, causal, window) -> dqkv, the two-kernel form
PyObject* attn_bwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  ZB_ARGS(11)
  const Tensor *d_o = tensor_of(args[0]), *qkv = tensor_of(args[1]), *o = tensor_of(args[2]), *lse = tensor_of(args[3]);
  AttnArgs a;
  if (!attn_args(args + 4, qkv, a) || !dense(d_o, BF16) || !dense(o, BF16) || !dense(lse, F32) || !on(d_o, *qkv) ||
      !on(o, *qkv) || !on(lse, *qkv))
    Py_RETURN_NONE;
  if (d_o->numel() != a.B * a.S * a.Hq * a.D || o->numel() != d_o->numel() || lse->numel() != a.B * a.Hq * a.S) Py_RETURN_NONE;
  Tensor dqkv = empty(qkv->sizes(), *qkv, BF16);
  const Tensor stats = empty({lib.flash_stats_floats(int(a.B), int(a.S), int(a.Hq))}, *qkv, F32);
  const float scale = float(1.0 / std::sqrt(double(a.D)));
  int* status = status_of(*qkv);
  const cudaStream_t s = stream();
  if (!launch("flash_bwd3", 3, [&] {
        return lib.flash_bwd3(ptr(d_o), ptr(qkv), ptr(o), static_cast<const float*>(ptr(lse)), dqkv.data_ptr(),
                              static_cast<float*>(stats.data_ptr()), int(a.B), int(a.S), int(a.Hq), int(a.Hkv), int(a.D), a.causal,
                              int(a.window), scale, status, 3, nullptr, 0, s);
      }))
    return nullptr;
  return THPVariable_Wrap(std::move(dqkv));
  END_HANDLE_TH_ERRORS
}

// init(addresses of the entry points in Entry's order, KernelError)
PyObject* init(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  ZB_ARGS(2)
  constexpr Py_ssize_t N = sizeof(Entry) / sizeof(void*);
  if (!PyTuple_Check(args[0]) || PyTuple_GET_SIZE(args[0]) != N) {
    PyErr_Format(PyExc_ValueError, "init needs the addresses of %zd entry points", N);
    return nullptr;
  }
  void* table[N];
  for (Py_ssize_t i = 0; i < N; ++i) {
    table[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(args[0], i));
    if (PyErr_Occurred()) return nullptr;
  }
  static_assert(sizeof(table) == sizeof(lib), "one address per entry point");
  memcpy(&lib, table, sizeof(lib));
  Py_INCREF(args[1]);
  Py_XSETREF(kernel_error, args[1]);
  ready = true;
  Py_RETURN_NONE;
}
// set_status(device, address of its status word)
PyObject* set_status(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  ZB_ARGS(2)
  int64_t d;
  void* p = PyLong_AsVoidPtr(args[1]);
  if (PyErr_Occurred()) return nullptr;
  if (int_arg(args[0], d) && d >= 0 && d < 64) status_words[d] = static_cast<int*>(p);
  Py_RETURN_NONE;
}
PyObject* launch_count(PyObject*, PyObject* const*, Py_ssize_t) { return PyLong_FromLongLong(launches); }

#define ZB_FN(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ZB_FN(init), ZB_FN(set_status), ZB_FN(launch_count), ZB_FN(linear_fwd), ZB_FN(linear_dgrad),
                         ZB_FN(linear_wgrad), ZB_FN(act_linear_fwd), ZB_FN(act_linear_dgrad), ZB_FN(linear_rope_fwd),
                         ZB_FN(norm_fwd), ZB_FN(norm_bwd), ZB_FN(finish), ZB_FN(rope), ZB_FN(swiglu_fwd),
                         ZB_FN(swiglu_bwd), ZB_FN(act_fwd), ZB_FN(act_bwd), ZB_FN(attn_fwd), ZB_FN(attn_bwd),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "zorse_fastops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_zorse_fastops() { return PyModule_Create(&module); }
