// The GEMM and attention calls of kernels/__init__.py from Python in one native call each: operand checks, output and scratch
// allocation, launch.
//
// What it is for: a small call is shorter on the GPU than the interpreter needs to prepare it (328 x 1032 x 776: 7 us, and
// 12 us of Python and ctypes).  Each function takes the calls that need nothing but a launch and returns None for every
// other one: another type or device, tensor subclasses and tensors without storage (vmap, functionalisation), strides that
// need a copy, wrong shapes, the library baseline.  Those go on to the Python statements, which copy, refuse or explain.
// Host time per call, before / after: accumulating GEMM 10.3 / 3.4 us, attention forward 18.6 / 5.9, backward 38.7 / 12.6;
// the three GEMMs of a linear layer of 328 x 1032 x 776 36.4 / 23.6 us, attention of 2 x 459 tokens in both directions
// 62.2 / 34.2, which are their device times.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>
#include <cstdio>
#include <cstdlib>

#include "../native_calls.h"

namespace {

constexpr int MAX_DEVICES = 64;
int* g_status[MAX_DEVICES];        // status word of each device (owned by kernels/cuda.py)
PyObject* g_counter = nullptr;     // one-element list: kernels launched so far
PyObject* g_check = nullptr;       // callable(rc, what) that raises

bool baseline() {
  const char* e = std::getenv("KAREUS_B200_LIBRARY_BASELINE");
  return e && e[0] == '1' && e[1] == 0;
}

// A plain CUDA tensor of this type with storage of its own, on a device whose status word is known; null otherwise.
const at::Tensor* plain(PyObject* o, at::ScalarType type) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.scalar_type() != type || t.layout() != at::kStrided || !t.has_storage() ||
      t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::Functionalize})))
    return nullptr;
  const int dev = t.device().index();
  return dev >= 0 && dev < MAX_DEVICES && g_status[dev] ? &t : nullptr;
}

bool fits(int64_t v) { return v > 0 && v <= INT_MAX; }

// Rows that the kernels read where they lie: contiguous, 16-byte aligned, not overlapping.
bool rows_ok(const at::Tensor& t) {
  return t.dim() == 2 && t.stride(1) == 1 && t.stride(0) % 8 == 0 && t.stride(0) >= t.size(1) && t.stride(0) <= INT_MAX &&
         reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

// A view that the attention kernels read where it lies.
bool heads_ok(const at::Tensor& t) {
  if (t.stride(-1) != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) return false;
  for (int64_t i = 0; i + 1 < t.dim(); ++i)
    if (t.stride(i) % 8) return false;
  return true;
}

// Called with the GIL held; false with a Python error set.
bool finish(int rc, const char* what, long launches) {
  if (rc != 0) {
    PyObject* r = PyObject_CallFunction(g_check, "is", rc, what);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, what);
    return false;
  }
  const long n = PyLong_AsLong(PyList_GET_ITEM(g_counter, 0));
  return !PyErr_Occurred() && PyList_SetItem(g_counter, 0, PyLong_FromLong(n + launches)) == 0;
}

// The same with the shape in the error, as the Python statements have it.
bool finish_gemm(int rc, int64_t M, int64_t N, int64_t K, long launches) {
  char what[96] = "gemm";
  if (rc != 0)
    std::snprintf(what, sizeof(what), "gemm M=%lld N=%lld K=%lld", static_cast<long long>(M), static_cast<long long>(N),
                  static_cast<long long>(K));
  return finish(rc, what, launches);
}

template <typename F>
int without_gil(F f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  return rc;
}

// gemm(a, b, trans_a, trans_b, accumulate): bf16 output of its own, or accumulate += (fp32)
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5 || baseline()) Py_RETURN_NONE;
  const at::Tensor *a = plain(args[0], at::kBFloat16), *b = plain(args[1], at::kBFloat16);
  if (!a || !b || a->device() != b->device() || !rows_ok(*a) || !rows_ok(*b)) Py_RETURN_NONE;
  const int ta = PyObject_IsTrue(args[2]), tb = PyObject_IsTrue(args[3]);
  if (ta < 0 || tb < 0) return nullptr;
  const int64_t M = a->size(ta ? 1 : 0), K = a->size(ta ? 0 : 1), N = b->size(tb ? 0 : 1);
  if (K != b->size(tb ? 1 : 0) || !fits(M) || !fits(N) || !fits(K)) Py_RETURN_NONE;
  int* status = g_status[a->device().index()];
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const void *pa = a->data_ptr(), *pb = b->data_ptr();
  const int lda = static_cast<int>(a->stride(0)), ldb = static_cast<int>(b->stride(0));
  if (args[4] != Py_None) {
    const at::Tensor* c = plain(args[4], at::kFloat);
    if (!c || c->device() != a->device() || !c->is_contiguous() || c->dim() != 2 || c->size(0) != M || c->size(1) != N)
      Py_RETURN_NONE;
    // partial sums of a K split; nothing is split over fewer than 16 steps of 64
    const long n = K > 960 ? kb_gemm_accum_scratch_floats(M, N, K, 0) : 0;
    at::Tensor work;
    if (n) work = at::empty({n}, c->options().requires_grad(false));
    float* pw = n ? work.data_ptr<float>() : nullptr;
    float* pc = c->data_ptr<float>();
    const int rc = without_gil([&] {
      return kb_gemm_accum_bf16(pa, pb, pc, M, N, K, ta, lda, !tb, ldb, static_cast<int>(N), 0, pw, status, stream);
    });
    if (!finish_gemm(rc, M, N, K, n ? 2 : 1)) return nullptr;
    Py_INCREF(args[4]);
    return args[4];
  }
  at::Tensor out = at::empty({M, N}, a->options().requires_grad(false));
  void* pc = out.data_ptr();
  // partial sums of the last tiles' K parts, in rows that TMA can store; nothing is split over fewer than 16 steps of 64
  const long n = K >= 1024 && N % 8 == 0 ? kb_gemm_scratch_floats(M, N, K, !tb, 0) : 0;
  at::Tensor work;
  if (n) work = at::empty({n}, a->options().dtype(at::kFloat).requires_grad(false));
  float* pw = n ? work.data_ptr<float>() : nullptr;
  const int rc = without_gil([&] {
    return kb_gemm_work_bf16(pa, pb, pc, M, N, K, ta, lda, !tb, ldb, static_cast<int>(N), 0, pw, status, stream);
  });
  if (!finish_gemm(rc, M, N, K, n ? 2 : 1)) return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// Geometry of an attention call; `ok` is false for what the kernels do not take as it lies.
struct Heads {
  bool ok = false;
  const at::Tensor *q, *k, *v;
  int sq, skv, b, g, rep, q_offset, causal;
  long qs[4];
  double scale;
};

// args: q, k, v, scale, causal, q_offset
Heads heads(PyObject* const* args) {
  Heads h;
  h.q = plain(args[0], at::kBFloat16);
  h.k = plain(args[1], at::kBFloat16);
  h.v = plain(args[2], at::kBFloat16);
  if (!h.q || !h.k || !h.v || !PyFloat_Check(args[3]) || !PyBool_Check(args[4]) || !PyLong_Check(args[5])) return h;
  const at::Tensor &q = *h.q, &k = *h.k, &v = *h.v;
  if (q.device() != k.device() || q.device() != v.device() || k.dim() != 4 || k.sizes() != v.sizes() || k.size(3) != 128) return h;
  if (q.dim() == 5) {
    if (q.size(2) != k.size(2)) return h;
    h.rep = static_cast<int>(q.size(3));
    for (int i = 0; i < 4; ++i) h.qs[i] = q.stride(i);
  } else {
    if (q.dim() != 4 || k.size(2) == 0 || q.size(2) % k.size(2)) return h;
    h.rep = static_cast<int>(q.size(2) / k.size(2));
    h.qs[0] = q.stride(0);
    h.qs[1] = q.stride(1);
    h.qs[2] = q.stride(2) * h.rep;
    h.qs[3] = q.stride(2);
  }
  if (q.size(-1) != 128 || q.size(1) != k.size(1) || !heads_ok(q) || !heads_ok(k) || !heads_ok(v)) return h;
  if (q.numel() == 0 || k.numel() == 0 || !fits(q.size(0)) || !fits(k.size(0)) || !fits(k.size(1)) || !fits(q.numel() / 128)) return h;
  int overflow = 0;
  const long off = PyLong_AsLongAndOverflow(args[5], &overflow);
  if (overflow || off > INT_MAX || off < INT_MIN) return h;
  h.sq = static_cast<int>(q.size(0));
  h.skv = static_cast<int>(k.size(0));
  h.b = static_cast<int>(k.size(1));
  h.g = static_cast<int>(k.size(2));
  h.q_offset = static_cast<int>(off);
  h.causal = args[4] == Py_True;
  h.scale = PyFloat_AS_DOUBLE(args[3]);
  h.ok = true;
  return h;
}

// attention_fwd(q, k, v, scale, causal, q_offset) -> (out, lse)
PyObject* attention_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 6 || baseline()) Py_RETURN_NONE;
  const Heads h = heads(args);
  if (!h.ok) Py_RETURN_NONE;
  const at::Tensor &q = *h.q, &k = *h.k, &v = *h.v;
  const int64_t hq = static_cast<int64_t>(h.g) * h.rep;
  at::Tensor out = at::empty({h.sq, h.b, hq, 128}, q.options().requires_grad(false));
  at::Tensor lse = at::empty({h.b, hq, h.sq}, q.options().dtype(at::kFloat).requires_grad(false));
  int* status = g_status[q.device().index()];
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const void *pq = q.data_ptr(), *pk = k.data_ptr(), *pv = v.data_ptr();
  void* po = out.data_ptr();
  float* pl = lse.data_ptr<float>();
  const int rc = without_gil([&] {
    return kb_flash_attn_fwd(pq, h.qs[0], h.qs[1], h.qs[2], h.qs[3], pk, k.stride(0), k.stride(1), k.stride(2), pv, v.stride(0),
                             v.stride(1), v.stride(2), po, pl, h.sq, h.skv, h.b, h.g, h.rep, 128, static_cast<float>(h.scale),
                             h.causal, h.q_offset, status, stream);
  });
  if (!finish(rc, "flash_attn_fwd", 1)) return nullptr;
  PyObject* r = PyTuple_New(2);
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(lse)));
  return r;
  END_HANDLE_TH_ERRORS
}

// attention_bwd(q, k, v, scale, causal, q_offset, do, o, lse) -> (dq, dk, dv)
PyObject* attention_bwd(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 9 || baseline()) Py_RETURN_NONE;
  const Heads h = heads(args);
  const at::Tensor *dO = plain(args[6], at::kBFloat16), *o = plain(args[7], at::kBFloat16), *lse = plain(args[8], at::kFloat);
  if (!h.ok || !dO || !o || !lse) Py_RETURN_NONE;
  const at::Tensor &q = *h.q, &k = *h.k, &v = *h.v;
  for (const at::Tensor* t : {dO, o, lse})
    if (t->device() != q.device() || !t->is_contiguous()) Py_RETURN_NONE;
  if (o->numel() != q.numel() || dO->numel() != q.numel() || lse->numel() * 128 != q.numel()) Py_RETURN_NONE;
  const auto opts = q.options().requires_grad(false);
  at::Tensor dq = at::empty({h.sq, h.b, h.g, h.rep, 128}, opts), dk = at::empty(k.sizes(), opts), dv = at::empty(v.sizes(), opts);
  at::Tensor work = at::empty({kb_flash_attn_bwd_scratch_floats(h.sq, h.skv, h.b, h.g, h.rep, 128)}, opts.dtype(at::kFloat));
  int* status = g_status[q.device().index()];
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const void *pq = q.data_ptr(), *pk = k.data_ptr(), *pv = v.data_ptr(), *po = o->data_ptr(), *pdo = dO->data_ptr();
  const float* pl = lse->data_ptr<float>();
  void *pdq = dq.data_ptr(), *pdk = dk.data_ptr(), *pdv = dv.data_ptr();
  float* pw = work.data_ptr<float>();
  const int rc = without_gil([&] {
    return kb_flash_attn_bwd(pq, h.qs[0], h.qs[1], h.qs[2], h.qs[3], pk, k.stride(0), k.stride(1), k.stride(2), pv, v.stride(0),
                             v.stride(1), v.stride(2), po, pdo, pl, pdq, dq.stride(0), dq.stride(1), dq.stride(2), dq.stride(3),
                             pdk, dk.stride(0), dk.stride(1), dk.stride(2), pdv, dv.stride(0), dv.stride(1), dv.stride(2), pw,
                             h.sq, h.skv, h.b, h.g, h.rep, 128, static_cast<float>(h.scale), h.causal, h.q_offset, status,
                             stream);
  });
  if (!finish(rc, "flash_attn_bwd", 3)) return nullptr;
  PyObject* r = PyTuple_New(3);
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(q.dim() == 5 ? std::move(dq) : dq.view(q.sizes())));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(dk)));
  PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(std::move(dv)));
  return r;
  END_HANDLE_TH_ERRORS
}

// init(counter list, check callable); set_status(device index, address of the device's status word)
PyObject* init(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2 || !PyList_Check(args[0]) || PyList_GET_SIZE(args[0]) != 1 || !PyCallable_Check(args[1])) {
    PyErr_SetString(PyExc_TypeError, "init(counter, check)");
    return nullptr;
  }
  Py_INCREF(args[0]);
  Py_INCREF(args[1]);
  Py_XSETREF(g_counter, args[0]);
  Py_XSETREF(g_check, args[1]);
  Py_RETURN_NONE;
}

PyObject* set_status(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2) {
    PyErr_SetString(PyExc_TypeError, "set_status(device, address)");
    return nullptr;
  }
  const long dev = PyLong_AsLong(args[0]);
  void* p = PyLong_AsVoidPtr(args[1]);
  if (PyErr_Occurred()) return nullptr;
  if (dev < 0 || dev >= MAX_DEVICES || !g_counter) {
    PyErr_SetString(PyExc_ValueError, "set_status: bad device, or init() has not run");
    return nullptr;
  }
  g_status[dev] = static_cast<int*>(p);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gemm)), METH_FASTCALL, nullptr},
    {"attention_fwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(attention_fwd)), METH_FASTCALL, nullptr},
    {"attention_bwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(attention_bwd)), METH_FASTCALL, nullptr},
    {"init", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(init)), METH_FASTCALL, nullptr},
    {"set_status", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(set_status)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall() {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "torch_version", KB_TORCH_VERSION) != 0) Py_CLEAR(m);
  return m;
}
