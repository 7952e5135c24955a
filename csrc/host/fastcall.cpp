// CPython extension module `_fastcall`: the calls a training step or a codec user makes
// once per tensor or bucket, without ctypes.  A ctypes call with fifteen arguments costs
// about 5 us and filling a ctypes structure about 0.2 us per field, more than the
// kernels of a small tensor take; here a call costs well under a microsecond on top of
// the launch itself.  Only plain integers, floats and None cross the boundary (device
// addresses, sizes, stream handles), so the module needs no PyTorch headers.
//
// The C ABI of the CUDA library is reached through function pointers handed over by
// bind(), so whichever build of that library Python loaded is the one that runs.  The
// GIL is released around every call that may launch (a full launch queue blocks).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include <new>

#include "hipress/capi.h"
#include "hipress/common.h"

namespace {

using DenseEncode = int (*)(int, int, const void*, void*, const void*, void*, uint64_t, float, uint64_t, uint32_t,
                            uint32_t, uint32_t, uint64_t, int, void*);
using DenseDecode = int (*)(int, int, const void*, void*, uint64_t, float, float, int, int, void*);
using SparseEncode = int (*)(int, const void*, void*, void*, uint64_t, uint64_t, uint64_t, float, int, void*, void*,
                             uint64_t, int, void*);
using SparseDecode = int (*)(const void*, void*, uint64_t, uint64_t, float, int, void*);
using FusedDense = int (*)(int, int, int, const HpSeg*, int, const HpComm*, float, uint64_t, uint32_t, uint32_t, int,
                           void*);
using FusedSparse = int (*)(int, float, float, const HpSeg*, void* const*, int, const HpComm*, void*, int, void*);
using StreamOrder = int (*)(void*, void*, void*);

DenseEncode f_dense_encode;
DenseDecode f_dense_decode;
SparseEncode f_sparse_encode;
SparseDecode f_sparse_decode;
FusedDense f_fused_dense;
FusedSparse f_fused_sparse_ps, f_fused_sparse_ring;
StreamOrder f_stream_order;

struct Name {
  const char* name;
  void** slot;
};
const Name kNames[] = {
    {"hp_cuda_dense_encode", (void**)&f_dense_encode},
    {"hp_cuda_dense_decode", (void**)&f_dense_decode},
    {"hp_cuda_sparse_encode", (void**)&f_sparse_encode},
    {"hp_cuda_sparse_decode", (void**)&f_sparse_decode},
    {"hp_cuda_fused_dense", (void**)&f_fused_dense},
    {"hp_cuda_fused_sparse_ps", (void**)&f_fused_sparse_ps},
    {"hp_cuda_fused_sparse_ring", (void**)&f_fused_sparse_ring},
    {"hp_cuda_stream_order", (void**)&f_stream_order},
};

// ------------------------------------------------------------ argument readers
// Each leaves an exception set on a bad argument; callers check PyErr_Occurred() once,
// after all of them.
inline uint64_t as_u64(PyObject* o) { return PyLong_AsUnsignedLongLongMask(o); }
inline int as_int(PyObject* o) { return (int)PyLong_AsLong(o); }
inline float as_float(PyObject* o) { return (float)PyFloat_AsDouble(o); }
inline void* as_ptr(PyObject* o) { return o == Py_None ? nullptr : (void*)(uintptr_t)as_u64(o); }

bool arity(Py_ssize_t got, Py_ssize_t want, const char* what) {
  if (got == want) return true;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", what, want, got);
  return false;
}
bool bound(const void* f, const char* what) {
  if (f) return true;
  PyErr_Format(PyExc_RuntimeError, "%s: the CUDA library is not bound", what);
  return false;
}

// bind({symbol name: address})
PyObject* py_bind(PyObject*, PyObject* d) {
  if (!PyDict_Check(d)) {
    PyErr_SetString(PyExc_TypeError, "bind takes a dict");
    return nullptr;
  }
  for (const Name& n : kNames) {
    PyObject* v = PyDict_GetItemString(d, n.name);
    if (v) *n.slot = as_ptr(v);
  }
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// names bind() knows
PyObject* py_symbols(PyObject*, PyObject*) {
  PyObject* l = PyList_New(0);
  if (!l) return nullptr;
  for (const Name& n : kNames) {
    PyObject* s = PyUnicode_FromString(n.name);
    if (!s || PyList_Append(l, s) != 0) {
      Py_XDECREF(s);
      Py_DECREF(l);
      return nullptr;
    }
    Py_DECREF(s);
  }
  return l;
}

PyObject* py_dense_payload_bytes(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 3, "dense_payload_bytes")) return nullptr;
  const uint64_t b = hipress::dense_payload_bytes(as_int(a[0]), as_int(a[1]), as_u64(a[2]));
  return PyErr_Occurred() ? nullptr : PyLong_FromUnsignedLongLong(b);
}
PyObject* py_sparse_payload_bytes(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 1, "sparse_payload_bytes")) return nullptr;
  const uint64_t b = hipress::sparse_payload_bytes(as_u64(a[0]));
  return PyErr_Occurred() ? nullptr : PyLong_FromUnsignedLongLong(b);
}
PyObject* py_sparse_k(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 2, "sparse_k")) return nullptr;
  const uint64_t k = hipress::sparse_k(as_u64(a[0]), as_float(a[1]));
  return PyErr_Occurred() ? nullptr : PyLong_FromUnsignedLongLong(k);
}

#define LAUNCH(expr)                    \
  if (PyErr_Occurred()) return nullptr; \
  int rc;                               \
  Py_BEGIN_ALLOW_THREADS                \
  rc = (expr);                          \
  Py_END_ALLOW_THREADS                  \
  return PyLong_FromLong(rc)

PyObject* py_dense_encode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 15, "dense_encode") || !bound((void*)f_dense_encode, "dense_encode")) return nullptr;
  const int alg = as_int(a[0]), bits = as_int(a[1]), ctas = as_int(a[13]);
  void *g = as_ptr(a[2]), *r = as_ptr(a[3]), *in = as_ptr(a[4]), *out = as_ptr(a[5]), *st = as_ptr(a[14]);
  const uint64_t len = as_u64(a[6]), seed = as_u64(a[8]), off = as_u64(a[12]);
  const float tau = as_float(a[7]);
  const uint32_t step = (uint32_t)as_u64(a[9]), salt = (uint32_t)as_u64(a[10]), id = (uint32_t)as_u64(a[11]);
  LAUNCH(f_dense_encode(alg, bits, g, r, in, out, len, tau, seed, step, salt, id, off, ctas, st));
}
PyObject* py_dense_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 10, "dense_decode") || !bound((void*)f_dense_decode, "dense_decode")) return nullptr;
  const int alg = as_int(a[0]), bits = as_int(a[1]), acc = as_int(a[7]), ctas = as_int(a[8]);
  void *p = as_ptr(a[2]), *out = as_ptr(a[3]), *st = as_ptr(a[9]);
  const uint64_t len = as_u64(a[4]);
  const float tau = as_float(a[5]), scale = as_float(a[6]);
  LAUNCH(f_dense_decode(alg, bits, p, out, len, tau, scale, acc, ctas, st));
}
PyObject* py_sparse_encode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 14, "sparse_encode") || !bound((void*)f_sparse_encode, "sparse_encode")) return nullptr;
  const int alg = as_int(a[0]), update = as_int(a[8]), ctas = as_int(a[12]);
  void *g = as_ptr(a[1]), *acc = as_ptr(a[2]), *u = as_ptr(a[3]), *out = as_ptr(a[9]), *ws = as_ptr(a[10]),
       *st = as_ptr(a[13]);
  const uint64_t len = as_u64(a[4]), k = as_u64(a[5]), kmax = as_u64(a[6]), wsb = as_u64(a[11]);
  const float m = as_float(a[7]);
  LAUNCH(f_sparse_encode(alg, g, acc, u, len, k, kmax, m, update, out, ws, wsb, ctas, st));
}
PyObject* py_sparse_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 7, "sparse_decode") || !bound((void*)f_sparse_decode, "sparse_decode")) return nullptr;
  void *p = as_ptr(a[0]), *out = as_ptr(a[1]), *st = as_ptr(a[6]);
  const uint64_t len = as_u64(a[2]), kmax = as_u64(a[3]);
  const float scale = as_float(a[4]);
  const int acc = as_int(a[5]);
  LAUNCH(f_sparse_decode(p, out, len, kmax, scale, acc, st));
}

// stream_order(event, src, dst): what is launched on dst from here on runs behind what
// src holds now
PyObject* py_stream_order(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 3, "stream_order") || !bound((void*)f_stream_order, "stream_order")) return nullptr;
  void *ev = as_ptr(a[0]), *src = as_ptr(a[1]), *dst = as_ptr(a[2]);
  LAUNCH(f_stream_order(ev, src, dst));
}

// ---------------------------------------------------------------- bucket plans
// What stays the same between two launches of a fused bucket, laid out as the C ABI
// wants it; a launch only fills in the addresses.
struct Plan {
  int topo, alg, bits, ctas, nseg;
  float a, b;  // dense: tau; sparse: ratio, momentum
  uint64_t seed;
  void* ws;    // sparse scratch
  HpComm comm;
  uint64_t n[HP_MAX_SEGS];
};

const char* const kPlanName = "hipress.plan";

void plan_free(PyObject* cap) { delete static_cast<Plan*>(PyCapsule_GetPointer(cap, kPlanName)); }

// put(i, entry) for a sequence of n integers (or None); a None sequence puts None n times
template <typename F>
bool each(PyObject* seq, int n, const char* what, F put) {
  if (seq == Py_None) {
    for (int i = 0; i < n; ++i) put(i, Py_None);
    return true;
  }
  PyObject* fast = PySequence_Fast(seq, what);
  if (!fast) return false;
  if (PySequence_Fast_GET_SIZE(fast) != n) {
    PyErr_Format(PyExc_ValueError, "%s: %zd entries for %d", what, PySequence_Fast_GET_SIZE(fast), n);
    Py_DECREF(fast);
    return false;
  }
  PyObject** it = PySequence_Fast_ITEMS(fast);
  for (int i = 0; i < n; ++i) put(i, it[i]);
  Py_DECREF(fast);
  return PyErr_Occurred() == nullptr;
}

// plan(topo, alg, bits, ctas, a, b, seed, ws, sizes, nranks, rank, emulate, timeout_ns,
//      inbox_ptrs, flag_ptrs, status)
PyObject* py_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 16, "plan")) return nullptr;
  const Py_ssize_t nseg = PySequence_Size(a[8]);
  const int nranks = as_int(a[9]);
  if (PyErr_Occurred()) return nullptr;
  if (nseg < 1 || nseg > HP_MAX_SEGS || nranks < 1 || nranks > HP_MAX_RANKS) {
    PyErr_SetString(PyExc_ValueError, "plan: too many tensors or ranks");
    return nullptr;
  }
  Plan* p = new (std::nothrow) Plan();
  if (!p) return PyErr_NoMemory();
  p->topo = as_int(a[0]);
  p->alg = as_int(a[1]);
  p->bits = as_int(a[2]);
  p->ctas = as_int(a[3]);
  p->a = as_float(a[4]);
  p->b = as_float(a[5]);
  p->seed = as_u64(a[6]);
  p->ws = as_ptr(a[7]);
  p->nseg = (int)nseg;
  p->comm.nranks = nranks;
  p->comm.rank = as_int(a[10]);
  p->comm.emulate = as_int(a[11]);
  p->comm.timeout_ns = as_u64(a[12]);
  p->comm.status = as_ptr(a[15]);
  const bool ok =
      !PyErr_Occurred() && each(a[8], p->nseg, "sizes", [&](int i, PyObject* o) { p->n[i] = as_u64(o); }) &&
      each(a[13], nranks, "inbox addresses", [&](int i, PyObject* o) { p->comm.inbox[i] = as_ptr(o); }) &&
      each(a[14], nranks, "flag addresses", [&](int i, PyObject* o) { p->comm.flags[i] = as_ptr(o); });
  PyObject* cap = ok ? PyCapsule_New(p, kPlanName, plan_free) : nullptr;
  if (!cap) delete p;
  return cap;
}

// launch(plan, g, r, out, sr, ids or us, step, salt, epoch, trace, strides, stream)
// strides: None or (g, r, out, sr), the element strides between emulated ranks
PyObject* py_launch(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 12, "launch")) return nullptr;
  const Plan* p = static_cast<const Plan*>(PyCapsule_GetPointer(a[0], kPlanName));
  if (!p) return nullptr;
  const bool sparse = p->alg == hipress::kDgc || p->alg == hipress::kGradDrop;
  FusedSparse fs = p->topo == HP_TOPO_PS ? f_fused_sparse_ps : f_fused_sparse_ring;
  if (!bound(sparse ? (void*)fs : (void*)f_fused_dense, "launch")) return nullptr;
  const int m = p->nseg;
  HpSeg seg[HP_MAX_SEGS];   // of this call: several threads may launch one plan
  void* us[HP_MAX_SEGS];
  HpComm comm = p->comm;
  for (int i = 0; i < m; ++i) {
    seg[i].n = p->n[i];
    seg[i].id = (uint32_t)i;
    seg[i].pad = 0;
    us[i] = nullptr;
  }
  if (!each(a[1], m, "gradient addresses", [&](int i, PyObject* o) { seg[i].g = as_ptr(o); }) ||
      !each(a[2], m, "state addresses", [&](int i, PyObject* o) { seg[i].r = as_ptr(o); }) ||
      !each(a[3], m, "result addresses", [&](int i, PyObject* o) { seg[i].out = as_ptr(o); }) ||
      !each(a[4], m, "owner state addresses", [&](int i, PyObject* o) { seg[i].sr = as_ptr(o); }))
    return nullptr;
  if (!each(a[5], m, sparse ? "momentum addresses" : "tensor ids", [&](int i, PyObject* o) {
        if (sparse) us[i] = as_ptr(o);
        else if (o != Py_None) seg[i].id = (uint32_t)as_u64(o);
      }))
    return nullptr;
  const uint32_t step = (uint32_t)as_u64(a[6]), salt = (uint32_t)as_u64(a[7]);
  comm.epoch = (uint32_t)as_u64(a[8]);
  comm.trace = as_ptr(a[9]);
  int64_t st[4];
  if (!each(a[10], 4, "strides", [&](int i, PyObject* o) { st[i] = o == Py_None ? 0 : PyLong_AsLongLong(o); }))
    return nullptr;
  comm.emu_stride_g = st[0];
  comm.emu_stride_r = st[1];
  comm.emu_stride_out = st[2];
  comm.emu_stride_sr = st[3];
  void* stream = as_ptr(a[11]);
  void* const* pus = p->alg == hipress::kDgc ? us : nullptr;
  LAUNCH(sparse ? fs(p->alg, p->a, p->b, seg, pus, m, &comm, p->ws, p->ctas, stream)
                : f_fused_dense(p->topo, p->alg, p->bits, seg, m, &comm, p->a, p->seed, step, salt, p->ctas, stream));
}

#define FAST(name, fn, doc) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, doc}
PyMethodDef kMethods[] = {
    {"bind", py_bind, METH_O, "bind({symbol: address}): the CUDA library to call"},
    {"symbols", py_symbols, METH_NOARGS, "symbol names bind() takes"},
    FAST("dense_payload_bytes", py_dense_payload_bytes, "(alg, bits, n)"),
    FAST("sparse_payload_bytes", py_sparse_payload_bytes, "(kmax)"),
    FAST("sparse_k", py_sparse_k, "(n, ratio)"),
    FAST("dense_encode", py_dense_encode, "hp_cuda_dense_encode"),
    FAST("dense_decode", py_dense_decode, "hp_cuda_dense_decode"),
    FAST("sparse_encode", py_sparse_encode, "hp_cuda_sparse_encode"),
    FAST("sparse_decode", py_sparse_decode, "hp_cuda_sparse_decode"),
    FAST("stream_order", py_stream_order, "hp_cuda_stream_order"),
    FAST("plan", py_plan, "plan of a fused bucket"),
    FAST("launch", py_launch, "one fused launch of a plan"),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fastcall", "native calls without ctypes", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&kModule); }
