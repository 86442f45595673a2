// Python side of the hot entry points: argument checks, tensor -> pointer, current stream and the C call in one
// native step.  A layer call through ctypes spent 12 - 20 us in the interpreter (one Python-level check per tensor,
// a stream object, twenty boxed arguments), several times the duration of the kernel on small layers; the same work
// here takes well under a microsecond.  The functions of the C ABI come in as addresses (bind), so this module is
// linked against nothing but Python and torch, and a library chosen at run time is honoured.
//
// Arguments mirror anode_b200/ops.py, which keeps the public signatures, defaults and error types.
// torch reports some conditions by C++ exceptions (no driver, a tensor without storage inside a function transform, a
// sparse one): every function turns them into Python errors (GUARDED), and nothing is asked of torch or CUDA once
// an argument was refused.
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

#include <stdint.h>

#include <exception>

// Exceptions become Python errors by torch's own translation, which runs only when there is one: HANDLE_TH_ERRORS around
// every call would set up a buffer for C++ warnings each time.
namespace {
PyObject *translated(std::exception_ptr e)
{
  HANDLE_TH_ERRORS
  std::rethrow_exception(e);
  END_HANDLE_TH_ERRORS
}
}  // namespace
#define GUARDED try {
#define END_GUARDED } catch (...) { return translated(std::current_exception()); }

namespace {

struct KernelConfig { uint32_t block_sz, max_block_ct; };

// addresses of the C ABI, in the order of kNames
enum { F_FWD, F_FWD_ACT, F_FWD_ADD, F_BWD, F_BWD_ACT, F_BWD_ADD, F_INFER, F_NORMALIZE, F_ADJOINT, F_COUNT };
const char *const kNames[F_COUNT] = {
    "anode_gpu_batch_norm_relu_fused_fwd_3d1_packed_f32", "anode_gpu_batch_norm_act_fused_fwd_3d1_packed_f32",
    "anode_gpu_batch_norm_add_act_fused_fwd_3d1_packed_f32", "anode_gpu_batch_norm_relu_fused_bwd_3d1_packed_f32",
    "anode_gpu_batch_norm_act_fused_bwd_3d1_packed_f32", "anode_gpu_batch_norm_add_act_fused_bwd_3d1_packed_f32",
    "anode_gpu_batch_norm_act_infer_3d1_packed_f32", "anode_gpu_batch_normalize_3d1_packed_f32",
    "anode_gpu_batch_normalize_adjoint_3d1_packed_f32"};
void *g_fn[F_COUNT] = {};

typedef const float *In;
typedef float *Out;
typedef int (*FwdFn)(uint32_t, uint32_t, uint32_t, float, float, int, In, In, In, Out, Out, Out, Out, Out, void *, size_t, const KernelConfig *, void *);
typedef int (*FwdActFn)(uint32_t, uint32_t, uint32_t, float, float, float, In, In, In, Out, Out, Out, Out, Out, void *, size_t, const KernelConfig *, void *);
typedef int (*FwdAddFn)(uint32_t, uint32_t, uint32_t, float, float, float, In, In, In, In, Out, Out, Out, Out, Out, void *, size_t, const KernelConfig *, void *);
typedef int (*BwdFn)(uint32_t, uint32_t, uint32_t, int, int, In, In, In, In, In, In, Out, Out, Out, void *, size_t, const KernelConfig *, void *);
typedef int (*BwdActFn)(uint32_t, uint32_t, uint32_t, float, int, In, In, In, In, In, In, Out, Out, Out, void *, size_t, const KernelConfig *, void *);
typedef int (*BwdAddFn)(uint32_t, uint32_t, uint32_t, float, int, In, In, In, In, In, In, In, Out, Out, Out, Out, void *, size_t, const KernelConfig *, void *);
typedef int (*InferFn)(uint32_t, uint32_t, uint32_t, float, In, In, In, In, In, Out, const KernelConfig *, void *);
typedef int (*NormalizeFn)(uint32_t, uint32_t, uint32_t, float, float, In, Out, Out, Out, Out, Out, const KernelConfig *, void *);
typedef int (*AdjointFn)(uint32_t, uint32_t, uint32_t, In, In, In, In, Out, Out, Out, const KernelConfig *, void *);

// The interpreter's lock is given back while this lives (exceptions included).
struct Unlocked {
  PyThreadState *state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// One call's arguments: the first failure sets the Python error and every later access does nothing.
struct Args {
  PyObject *const *v;
  bool ok = true;

  const at::Tensor *tensor(int i, bool null_ok)
  {
    if (!ok || (v[i] == Py_None && null_ok)) return nullptr;
    if (!THPVariable_Check(v[i])) {
      PyErr_SetString(PyExc_ValueError, "expected a contiguous float32 CUDA tensor");
      ok = false;
      return nullptr;
    }
    return &THPVariable_Unpack(v[i]);
  }
  // device pointer of a packed f32 array (the reference only implements packed arrays too, src/ops_gpu.rs:3777-3779)
  Out ptr(int i, bool null_ok = true)
  {
    const at::Tensor *t = tensor(i, null_ok);
    if (!t) return nullptr;
    if (!(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous())) {
      PyErr_SetString(PyExc_ValueError, "expected a contiguous float32 CUDA tensor");
      ok = false;
      return nullptr;
    }
    return static_cast<float *>(t->data_ptr());
  }
  float f(int i)
  {
    if (!ok) return 0.f;
    const double d = PyFloat_AsDouble(v[i]);
    if (d == -1.0 && PyErr_Occurred()) ok = false;
    return (float)d;
  }
  int truth(int i)
  {
    if (!ok) return 0;
    const int r = PyObject_IsTrue(v[i]);
    if (r < 0) ok = false;
    return r > 0;
  }
  size_t size(int i)
  {
    if (!ok) return 0;
    const size_t r = PyLong_AsSize_t(v[i]);
    if (r == (size_t)-1 && PyErr_Occurred()) ok = false;
    return r;
  }
  void *raw(int i)
  {
    const at::Tensor *t = tensor(i, true);
    return t ? t->data_ptr() : nullptr;
  }
  // a torch stream, or None for the current one
  void *stream(int i)
  {
    if (!ok) return nullptr;
    if (v[i] == Py_None) return c10::cuda::getCurrentCUDAStream().stream();
    PyObject *h = PyObject_GetAttrString(v[i], "cuda_stream");
    if (!h) { ok = false; return nullptr; }
    void *p = PyLong_AsVoidPtr(h);
    Py_DECREF(h);
    if (PyErr_Occurred()) ok = false;
    return p;
  }
  // [N, C, *spatial] -> (dim0, dim1, dim2) as the apply closures compute them (src/ops_gpu.rs:3764-3766, :4911-4913);
  // `axes` (None: not checked) must be the positions of the spatial dimensions (src/ops_gpu.rs:3736)
  void dims(int axes, int i, uint32_t d[3])
  {
    const at::Tensor *t = tensor(i, false);
    if (!t) return;
    const int64_t nd = t->dim();
    if (axes >= 0 && v[axes] != Py_None) {
      // any iterable whose items equal 0, 1, ...; the usual list of integers without making another one
      bool usual = PyList_CheckExact(v[axes]) && PyList_GET_SIZE(v[axes]) == (nd > 2 ? nd - 2 : 0);
      for (Py_ssize_t k = 0; usual && k + 2 < nd; ++k) {
        PyObject *e = PyList_GET_ITEM(v[axes], k);
        usual = PyLong_CheckExact(e) && PyLong_AsLong(e) == (long)k;
        if (PyErr_Occurred()) PyErr_Clear();      // (an integer beyond a long)
      }
      PyObject *got = usual ? nullptr : PySequence_List(v[axes]), *want = got ? PyList_New(0) : nullptr;
      int same = usual ? 2 : want ? 1 : -1;
      for (int64_t k = 0; same == 1 && k + 2 < nd; ++k) {
        PyObject *e = PyLong_FromLongLong(k);
        if (!e || PyList_Append(want, e)) same = -1;
        Py_XDECREF(e);
      }
      if (same == 1) same = PyObject_RichCompareBool(got, want, Py_EQ);
      if (same == 0) PyErr_Format(PyExc_ValueError, "axes must be %R for a %d-D batch array", want, (int)(nd - 2));
      Py_XDECREF(got); Py_XDECREF(want);
      if (same <= 0) { ok = false; return; }
    }
    if (nd < 2) { PyErr_SetString(PyExc_IndexError, "expected an array [N, C, *spatial]"); ok = false; return; }
    uint64_t d0 = 1;
    for (int64_t k = 2; k < nd; ++k) d0 *= (uint64_t)t->size(k);
    d[0] = (uint32_t)d0; d[1] = (uint32_t)t->size(1); d[2] = (uint32_t)t->size(0);
  }
};

bool want_args(Py_ssize_t n, Py_ssize_t want)
{
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
  return false;
}
bool bound(int which)
{
  if (g_fn[which]) return true;
  PyErr_SetString(PyExc_ImportError, "the CUDA library is not loaded");
  return false;
}
const KernelConfig kDefaultCfg = {1024, 148 * 32};     // ops.py's default launch hint (the kernels choose their own shapes)

// fwd(axes, epsilon, avg_rate, x, residual, y, mean, var, avg_mean, avg_var, gamma, beta, relu, neg_slope | None, ws, ws_bytes, stream)
PyObject *py_fwd(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 17)) return nullptr;
  Args a{v};
  uint32_t d[3] = {0, 0, 0};
  a.dims(0, 3, d);
  const float eps = a.f(1), rate = a.f(2);
  const bool add = v[4] != Py_None, act = add || v[13] != Py_None;
  const float slope = act ? a.f(13) : 0.f;      // (the residual epilogue always has one: None is refused)
  In x = a.ptr(3), res = a.ptr(4), gamma = a.ptr(10), beta = a.ptr(11);
  Out y = a.ptr(5), mean = a.ptr(6), var = a.ptr(7), rm = a.ptr(8), rv = a.ptr(9);
  const int relu = a.truth(12);
  void *ws = a.raw(14);
  const size_t bytes = a.size(15);
  void *s = a.stream(16);
  if (!a.ok) return nullptr;
  const int which = add ? F_FWD_ADD : act ? F_FWD_ACT : F_FWD;
  if (!bound(which)) return nullptr;
  int rc;
  {
    Unlocked unlocked;
    if (add) rc = ((FwdAddFn)g_fn[which])(d[0], d[1], d[2], eps, rate, slope, x, res, gamma, beta, y, mean, var, rm, rv, ws, bytes, &kDefaultCfg, s);
    else if (act) rc = ((FwdActFn)g_fn[which])(d[0], d[1], d[2], eps, rate, slope, x, gamma, beta, y, mean, var, rm, rv, ws, bytes, &kDefaultCfg, s);
    else rc = ((FwdFn)g_fn[which])(d[0], d[1], d[2], eps, rate, relu, x, gamma, beta, y, mean, var, rm, rv, ws, bytes, &kDefaultCfg, s);
  }
  return PyLong_FromLong(rc);
  END_GUARDED
}

// bwd(axes, dy, x, y | None, mean, var, dx, dresidual, gamma, beta, dgamma, dbeta, relu, neg_slope | None, accumulate, ws, ws_bytes, stream)
PyObject *py_bwd(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 18)) return nullptr;
  Args a{v};
  uint32_t d[3] = {0, 0, 0};
  a.dims(0, 2, d);
  const bool add = v[3] != Py_None, act = add || v[13] != Py_None;
  const float slope = act ? a.f(13) : 0.f;      // (the residual epilogue always has one: None is refused)
  In dy = a.ptr(1), x = a.ptr(2), y = a.ptr(3), mean = a.ptr(4), var = a.ptr(5), gamma = a.ptr(8), beta = a.ptr(9);
  Out dx = a.ptr(6), dres = a.ptr(7), dg = a.ptr(10), db = a.ptr(11);
  const int relu = a.truth(12), acc = a.truth(14);
  void *ws = a.raw(15);
  const size_t bytes = a.size(16);
  void *s = a.stream(17);
  if (!a.ok) return nullptr;
  const int which = add ? F_BWD_ADD : act ? F_BWD_ACT : F_BWD;
  if (!bound(which)) return nullptr;
  int rc;
  {
    Unlocked unlocked;
    if (add) rc = ((BwdAddFn)g_fn[which])(d[0], d[1], d[2], slope, acc, dy, x, y, mean, var, gamma, beta, dx, dres, dg, db, ws, bytes, &kDefaultCfg, s);
    else if (act) rc = ((BwdActFn)g_fn[which])(d[0], d[1], d[2], slope, acc, dy, x, mean, var, gamma, beta, dx, dg, db, ws, bytes, &kDefaultCfg, s);
    else rc = ((BwdFn)g_fn[which])(d[0], d[1], d[2], relu, acc, dy, x, mean, var, gamma, beta, dx, dg, db, ws, bytes, &kDefaultCfg, s);
  }
  return PyLong_FromLong(rc);
  END_GUARDED
}

// infer(axes, x, mean, var, y, gamma, beta, neg_slope, stream)
PyObject *py_infer(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 9)) return nullptr;
  Args a{v};
  uint32_t d[3] = {0, 0, 0};
  a.dims(0, 1, d);
  const float slope = a.f(7);
  In x = a.ptr(1), mean = a.ptr(2), var = a.ptr(3), gamma = a.ptr(5), beta = a.ptr(6);
  Out y = a.ptr(4);
  void *s = a.stream(8);
  if (!a.ok || !bound(F_INFER)) return nullptr;
  int rc;
  {
    Unlocked unlocked;
    rc = ((InferFn)g_fn[F_INFER])(d[0], d[1], d[2], slope, x, mean, var, gamma, beta, y, &kDefaultCfg, s);
  }
  return PyLong_FromLong(rc);
  END_GUARDED
}

// The outputs of the front end's composition are made here: three tensors through the interpreter took longer than the call.
at::Tensor like(const at::Tensor &x) { return at::empty_like(x); }
at::Tensor per_channel(const at::Tensor &x) { return at::empty({x.size(1)}, x.options()); }
Out data(const at::Tensor &t) { return static_cast<float *>(t.data_ptr()); }
// (status, a, b, c)
PyObject *answer(int rc, const at::Tensor &a, const at::Tensor &b, const at::Tensor &c)
{
  PyObject *t = PyTuple_New(4), *items[4] = {PyLong_FromLong(rc), THPVariable_Wrap(a), THPVariable_Wrap(b), THPVariable_Wrap(c)};
  bool ok = t != nullptr;
  for (int i = 0; i < 4; ++i) {
    ok = ok && items[i];
    if (t) PyTuple_SET_ITEM(t, i, items[i]); else Py_XDECREF(items[i]);
  }
  if (ok) return t;
  Py_XDECREF(t);
  return nullptr;
}

// normalize(axes, epsilon, avg_rate, x, avg_mean, avg_var, stream) -> status, y, mean, var
PyObject *py_normalize(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 7)) return nullptr;
  Args a{v};
  uint32_t d[3] = {0, 0, 0};
  a.dims(0, 3, d);
  const float eps = a.f(1), rate = a.f(2);
  In x = a.ptr(3, false);
  Out rm = a.ptr(4, false), rv = a.ptr(5, false);
  void *s = a.stream(6);
  if (!a.ok || !bound(F_NORMALIZE)) return nullptr;
  const at::Tensor &t = THPVariable_Unpack(v[3]);
  const at::Tensor mean = per_channel(t), var = per_channel(t), y = like(t);
  int rc;
  {
    Unlocked unlocked;
    rc = ((NormalizeFn)g_fn[F_NORMALIZE])(d[0], d[1], d[2], eps, rate, x, data(y), data(mean), data(var), rm, rv, &kDefaultCfg, s);
  }
  return answer(rc, y, mean, var);
  END_GUARDED
}

// adjoint(axes, dy, x, mean, var, stream) -> status, dx, dmean, dvar
PyObject *py_adjoint(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 6)) return nullptr;
  Args a{v};
  uint32_t d[3] = {0, 0, 0};
  a.dims(0, 2, d);
  In dy = a.ptr(1, false), x = a.ptr(2, false), mean = a.ptr(3, false), var = a.ptr(4, false);
  void *s = a.stream(5);
  if (!a.ok || !bound(F_ADJOINT)) return nullptr;
  const at::Tensor &t = THPVariable_Unpack(v[2]);
  const at::Tensor dvar = per_channel(t), dmean = per_channel(t), dx = like(t);
  int rc;
  {
    Unlocked unlocked;
    rc = ((AdjointFn)g_fn[F_ADJOINT])(d[0], d[1], d[2], dy, x, mean, var, data(dx), data(dmean), data(dvar), &kDefaultCfg, s);
  }
  return answer(rc, dx, dmean, dvar);
  END_GUARDED
}

// The tensors of one of the reference's own entry points: `lo` to `hi` of them, all required (these entry points have no
// status, and their kernels read and write what they are given).
struct Pointers {
  void *p[5] = {};
  Py_ssize_t k = 0;

  bool take(PyObject *tuple, Py_ssize_t lo, Py_ssize_t hi)
  {
    if (!PyTuple_Check(tuple)) { PyErr_SetString(PyExc_TypeError, "tensors: a tuple"); return false; }
    k = PyTuple_GET_SIZE(tuple);
    if (k < lo || k > hi) { PyErr_Format(PyExc_TypeError, "%zd to %zd tensors", lo, hi); return false; }
    PyObject *items[5];
    for (Py_ssize_t i = 0; i < k; ++i) items[i] = PyTuple_GET_ITEM(tuple, i);
    Args t{items};
    for (Py_ssize_t i = 0; i < k; ++i) {
      p[i] = t.ptr((int)i, false);
      if (t.ok && !p[i] && THPVariable_Unpack(items[i]).numel() != 0) {
        PyErr_SetString(PyExc_RuntimeError, "a tensor has no storage");
        t.ok = false;
      }
    }
    return t.ok;
  }
};
typedef void *P;
typedef const KernelConfig *K;

// The form of the C call is the function's, never read off the arguments' values.
// flat(address, tensors, stream): element count (of the first tensor) and 2 or 3 arrays
PyObject *py_flat(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 3)) return nullptr;
  void *fn = PyLong_AsVoidPtr(v[0]);
  if (PyErr_Occurred()) return nullptr;
  Args a{v};
  Pointers q;
  if (!q.take(v[1], 2, 3)) return nullptr;
  const uint32_t len = (uint32_t)THPVariable_Unpack(PyTuple_GET_ITEM(v[1], 0)).numel();
  void *s = a.stream(2);
  if (!a.ok) return nullptr;
  const KernelConfig *cfg = &kDefaultCfg;
  {
    Unlocked unlocked;
    if (q.k == 2) ((void (*)(uint32_t, P, P, K, P))fn)(len, q.p[0], q.p[1], cfg, s);
    else ((void (*)(uint32_t, P, P, P, K, P))fn)(len, q.p[0], q.p[1], q.p[2], cfg, s);
  }
  Py_RETURN_NONE;
  END_GUARDED
}

// packed(address, axes, like, tensors, stream): the dimensions of `like` and 2 to 5 arrays
PyObject *py_packed(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 5)) return nullptr;
  void *fn = PyLong_AsVoidPtr(v[0]);
  if (PyErr_Occurred()) return nullptr;
  Args a{v};
  uint32_t d[3] = {0, 0, 0};
  a.dims(1, 2, d);
  Pointers q;
  if (!a.ok || !q.take(v[3], 2, 5)) return nullptr;
  void *s = a.stream(4);
  if (!a.ok) return nullptr;
  const KernelConfig *cfg = &kDefaultCfg;
  {
    Unlocked unlocked;
    if (q.k == 2) ((void (*)(uint32_t, uint32_t, uint32_t, P, P, K, P))fn)(d[0], d[1], d[2], q.p[0], q.p[1], cfg, s);
    else if (q.k == 3) ((void (*)(uint32_t, uint32_t, uint32_t, P, P, P, K, P))fn)(d[0], d[1], d[2], q.p[0], q.p[1], q.p[2], cfg, s);
    else if (q.k == 4) ((void (*)(uint32_t, uint32_t, uint32_t, P, P, P, P, K, P))fn)(d[0], d[1], d[2], q.p[0], q.p[1], q.p[2], q.p[3], cfg, s);
    else ((void (*)(uint32_t, uint32_t, uint32_t, P, P, P, P, P, K, P))fn)(d[0], d[1], d[2], q.p[0], q.p[1], q.p[2], q.p[3], q.p[4], cfg, s);
  }
  Py_RETURN_NONE;
  END_GUARDED
}

// packed_eps(address, axes, like, tensors, epsilon, stream): the dimensions of `like`, epsilon and 3 arrays
PyObject *py_packed_eps(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 6)) return nullptr;
  void *fn = PyLong_AsVoidPtr(v[0]);
  if (PyErr_Occurred()) return nullptr;
  Args a{v};
  uint32_t d[3] = {0, 0, 0};
  a.dims(1, 2, d);
  const float eps = a.f(4);
  Pointers q;
  if (!a.ok || !q.take(v[3], 3, 3)) return nullptr;
  void *s = a.stream(5);
  if (!a.ok) return nullptr;
  {
    Unlocked unlocked;
    ((void (*)(uint32_t, uint32_t, uint32_t, float, P, P, P, K, P))fn)(d[0], d[1], d[2], eps, q.p[0], q.p[1], q.p[2], &kDefaultCfg, s);
  }
  Py_RETURN_NONE;
  END_GUARDED
}

// bind({name: address}): the C ABI's functions
PyObject *py_bind(PyObject *, PyObject *const *v, Py_ssize_t n)
{
  GUARDED
  if (!want_args(n, 1)) return nullptr;
  for (int i = 0; i < F_COUNT; ++i) {
    PyObject *e = PyDict_GetItemString(v[0], kNames[i]);
    if (!e) { PyErr_Format(PyExc_KeyError, "%s", kNames[i]); return nullptr; }
    g_fn[i] = PyLong_AsVoidPtr(e);
    if (PyErr_Occurred()) return nullptr;
  }
  Py_RETURN_NONE;
  END_GUARDED
}

PyMethodDef kMethods[] = {
    {"bind", (PyCFunction)(void *)py_bind, METH_FASTCALL, nullptr},
    {"fwd", (PyCFunction)(void *)py_fwd, METH_FASTCALL, nullptr},
    {"bwd", (PyCFunction)(void *)py_bwd, METH_FASTCALL, nullptr},
    {"infer", (PyCFunction)(void *)py_infer, METH_FASTCALL, nullptr},
    {"normalize", (PyCFunction)(void *)py_normalize, METH_FASTCALL, nullptr},
    {"adjoint", (PyCFunction)(void *)py_adjoint, METH_FASTCALL, nullptr},
    {"flat", (PyCFunction)(void *)py_flat, METH_FASTCALL, nullptr},
    {"packed", (PyCFunction)(void *)py_packed, METH_FASTCALL, nullptr},
    {"packed_eps", (PyCFunction)(void *)py_packed_eps, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Fast paths of anode_b200.ops into the C ABI.", -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__native(void)
{
  PyObject *m = PyModule_Create(&kModule);
  if (m && PyModule_AddStringConstant(m, "built_for", ANODE_BUILT_FOR) < 0) { Py_DECREF(m); return nullptr; }
  return m;
}
