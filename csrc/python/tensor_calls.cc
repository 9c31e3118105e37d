// Python module `_uccl_tensor_calls`: the calls that a layer makes on every step, on torch tensors.
//
// A call through the pybind11 module spends more host time on looking at its tensors one Python attribute at a time and on
// converting ten arguments than on the launch.  Here the tensors are looked at natively.  Each function takes a call only
// if everything about it is ordinary -- plain dense CUDA tensors on the communicator's GPU, no Python-level override
// active, types and shapes as they have to be -- and returns whether it did; what it does not take, valid or not, is left
// untouched to the general path in the Python sources, which holds the checks, their order and their messages.  Errors of
// the library itself are raised as there.
//
// Kept apart from `_uccl_bindings`, which knows nothing of torch: without this module the general path serves all calls.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>

#include "uccl.h"

namespace {

PyObject* g_error = nullptr;       // UcclError of _uccl_bindings
PyObject* g_raw_stream = nullptr;  // torch._C._cuda_getCurrentRawStream
PyObject* g_device = nullptr;      // torch._C._cuda_getDevice

// The tensor behind `o`, or null if anything about it needs the general path.
const at::Tensor* dense(PyObject* o, int device) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined()) return nullptr;
  using K = c10::DispatchKey;
  const c10::DispatchKeySet keys = t.key_set();
  constexpr c10::DispatchKeySet special({K::Python, K::PythonTLSSnapshot, K::Functionalize, K::FuncTorchBatched, K::FuncTorchGradWrapper,
                                         K::Batched, K::Conjugate, K::Negative, K::ZeroTensor});
  if (!keys.has(K::CUDA) || keys.has_any(special) || !t.has_storage()) return nullptr;
  return t.get_device() == device ? &t : nullptr;
}
const at::Tensor* flat(PyObject* o, int device) {
  const at::Tensor* t = dense(o, device);
  return t && t->is_contiguous() ? t : nullptr;
}
const at::Tensor* flat(PyObject* o, int device, at::ScalarType type) {
  const at::Tensor* t = flat(o, device);
  return t && t->scalar_type() == type ? t : nullptr;
}
bool reducible(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16 || t == at::kFloat; }
bool dataType(at::ScalarType t, ucclDataType_t* d) {
  switch (t) {
    case at::kHalf: *d = ucclFloat16; return true;
    case at::kBFloat16: *d = ucclBfloat16; return true;
    case at::kFloat: *d = ucclFloat32; return true;
    case at::kFloat8_e4m3fn: *d = ucclFloat8e4m3; return true;
    case at::kByte: *d = ucclUint8; return true;
    default: return false;
  }
}

bool overridden() { return at::impl::torch_function_mode_enabled(); }

// The raw handle of the stream that is current on a device.  False: a Python error is set.
bool streamOf(int device, void** stream) {
  PyObject* d = PyLong_FromLong(device);
  PyObject* s = d ? PyObject_CallOneArg(g_raw_stream, d) : nullptr;
  Py_XDECREF(d);
  if (!s) return false;
  *stream = PyLong_AsVoidPtr(s);
  Py_DECREF(s);
  return !PyErr_Occurred();
}
bool handle(PyObject* o, void** p) {
  if (!PyLong_CheckExact(o)) return false;
  *p = PyLong_AsVoidPtr(o);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return *p != nullptr;
}
bool whole(PyObject* o, long lo, long hi, long* v) {
  if (!PyLong_CheckExact(o)) return false;
  *v = PyLong_AsLong(o);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return *v >= lo && *v <= hi;
}
// an index of a GPU; -1 (the CPU backend) and anything else are not for here
bool gpu(PyObject* o, int* device) {
  long v;
  if (!whole(o, 0, 1023, &v)) return false;
  *device = static_cast<int>(v);
  return true;
}
bool number(PyObject* o, float* v) {
  if (!PyFloat_CheckExact(o)) return false;
  *v = static_cast<float>(PyFloat_AS_DOUBLE(o));
  return true;
}

PyObject* finish(ucclResult_t r, const char* what, ucclComm_t comm) {
  if (r == ucclSuccess) Py_RETURN_TRUE;
  std::string msg = std::string(what) + ": " + ucclGetErrorString(r);
  if (comm) {
    const char* last = ucclGetLastError(comm);
    if (last && *last) msg += std::string(" (") + last + ")";
  }
  PyErr_SetString(g_error, msg.c_str());
  return nullptr;
}

// gemm(a, b, out, swiglu)
PyObject* gemm(PyObject* const* v, Py_ssize_t n) {
  if (n != 4 || overridden() || (v[3] != Py_True && v[3] != Py_False)) Py_RETURN_FALSE;
  if (!THPVariable_CheckExact(v[0]) || !THPVariable_Unpack(v[0]).is_cuda()) Py_RETURN_FALSE;
  const int device = static_cast<int>(THPVariable_Unpack(v[0]).get_device());
  const at::Tensor *a = dense(v[0], device), *b = dense(v[1], device), *c = dense(v[2], device);
  if (!a || !b || !c || a->dim() != 2 || b->dim() != 2 || c->dim() != 2) Py_RETURN_FALSE;
  if (a->scalar_type() != at::kBFloat16 || b->scalar_type() != at::kBFloat16 || c->scalar_type() != at::kBFloat16) Py_RETURN_FALSE;
  const bool swiglu = v[3] == Py_True;
  const int64_t M = a->size(0), K = a->size(1), N = b->size(0), most = INT32_MAX;
  const int64_t lda = a->stride(0), ldb = b->stride(0), ldc = c->stride(0);
  if (b->size(1) != K || a->stride(1) != 1 || b->stride(1) != 1 || c->stride(1) != 1) Py_RETURN_FALSE;
  if (c->size(0) != M || c->size(1) != (swiglu ? N / 2 : N)) Py_RETURN_FALSE;
  if (M > most || N > most || K > most || lda > most || ldb > most || ldc > most) Py_RETURN_FALSE;
  PyObject* cur = PyObject_CallNoArgs(g_device);
  if (!cur) return nullptr;
  const long current = PyLong_AsLong(cur);
  Py_DECREF(cur);
  if (current != device) Py_RETURN_FALSE;
  void* stream;
  if (!streamOf(device, &stream)) return nullptr;
  return finish(ucclGemmBf16(a->data_ptr(), b->data_ptr(), c->data_ptr(), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K),
                             static_cast<int>(lda), static_cast<int>(ldb), static_cast<int>(ldc), swiglu ? 1 : 0, stream),
                "ucclGemmBf16", nullptr);
}

// norm(comm, device, x, residual, gamma, eps, out, residual_out)
PyObject* norm(PyObject* const* v, Py_ssize_t n) {
  void *comm, *stream;
  int device;
  float eps;
  if (n != 8 || overridden() || !handle(v[0], &comm) || !gpu(v[1], &device) || !number(v[5], &eps)) Py_RETURN_FALSE;
  const at::Tensor *x = flat(v[2], device, at::kBFloat16), *res = flat(v[3], device, at::kBFloat16), *gamma = flat(v[4], device, at::kBFloat16),
                   *out = flat(v[6], device, at::kBFloat16), *resOut = flat(v[7], device, at::kBFloat16);
  if (!x || !res || !gamma || !out || !resOut || x->dim() != 2 || x->size(0) > INT32_MAX || x->size(1) > INT32_MAX) Py_RETURN_FALSE;
  void *px = x->data_ptr(), *pr = res->data_ptr(), *pg = gamma->data_ptr(), *po = out->data_ptr(), *pro = resOut->data_ptr();
  const int tokens = static_cast<int>(x->size(0)), hidden = static_cast<int>(x->size(1));
  if (!streamOf(device, &stream)) return nullptr;
  ucclResult_t r;
  Py_BEGIN_ALLOW_THREADS
  r = ucclAllReduceResidualRMSNorm(px, pr, pg, po, pro, tokens, hidden, eps, static_cast<ucclComm_t>(comm), stream);
  Py_END_ALLOW_THREADS
  return finish(r, "ucclAllReduceResidualRMSNorm", static_cast<ucclComm_t>(comm));
}

// reduce_scatter / allgather(comm, device, world_size, send, recv)
PyObject* exchange(PyObject* const* v, Py_ssize_t n, bool gather) {
  void *comm, *stream;
  int device;
  long world;
  if (n != 5 || overridden() || !handle(v[0], &comm) || !gpu(v[1], &device) || !whole(v[2], 1, 1 << 20, &world)) Py_RETURN_FALSE;
  const at::Tensor *send = flat(v[3], device), *recv = flat(v[4], device);
  ucclDataType_t type;
  if (!send || !recv || !dataType(send->scalar_type(), &type) || recv->scalar_type() != send->scalar_type()) Py_RETURN_FALSE;
  if (!gather && !reducible(send->scalar_type())) Py_RETURN_FALSE;
  const at::Tensor *part = gather ? send : recv, *all = gather ? recv : send;
  if (all->numel() != part->numel() * world) Py_RETURN_FALSE;
  const size_t count = static_cast<size_t>(part->numel());
  void *ps = send->data_ptr(), *pr = recv->data_ptr();
  if (!streamOf(device, &stream)) return nullptr;
  ucclResult_t r;
  Py_BEGIN_ALLOW_THREADS
  if (gather) r = ucclAllGather(ps, pr, count, type, static_cast<ucclComm_t>(comm), stream);
  else r = ucclReduceScatter(ps, pr, count, type, ucclSum, static_cast<ucclComm_t>(comm), stream);
  Py_END_ALLOW_THREADS
  return finish(r, gather ? "ucclAllGather" : "ucclReduceScatter", static_cast<ucclComm_t>(comm));
}
PyObject* reduceScatter(PyObject* const* v, Py_ssize_t n) { return exchange(v, n, false); }
PyObject* allGather(PyObject* const* v, Py_ssize_t n) { return exchange(v, n, true); }

// reduce_scatter_cast / allreduce_cast(comm, device, world_size, send, out, factor, scales); scales None: not fp8
PyObject* cast(PyObject* const* v, Py_ssize_t n, bool all) {
  void *comm, *stream;
  int device;
  long world;
  float factor;
  if (n != 7 || overridden() || !handle(v[0], &comm) || !gpu(v[1], &device) || !whole(v[2], 1, 1 << 20, &world) || !number(v[5], &factor)) Py_RETURN_FALSE;
  const at::Tensor *send = flat(v[3], device), *out = flat(v[4], device);
  ucclDataType_t in, to;
  if (!send || !out || !reducible(send->scalar_type()) || !dataType(send->scalar_type(), &in) || !dataType(out->scalar_type(), &to)) Py_RETURN_FALSE;
  if (to == ucclUint8 || send->numel() != out->numel() * (all ? 1 : world)) Py_RETURN_FALSE;
  float* scales = nullptr;
  if (to == ucclFloat8e4m3) {
    const at::Tensor* s = flat(v[6], device, at::kFloat);
    if (!s || s->numel() * 128 != out->numel() || (all ? out->numel() / world : out->numel()) % 128) Py_RETURN_FALSE;
    scales = static_cast<float*>(s->data_ptr());
  } else if (v[6] != Py_None) {
    Py_RETURN_FALSE;
  }
  const size_t count = static_cast<size_t>(out->numel());
  void *ps = send->data_ptr(), *po = out->data_ptr();
  if (!streamOf(device, &stream)) return nullptr;
  ucclResult_t r;
  Py_BEGIN_ALLOW_THREADS
  if (all) r = ucclAllReduceEx(ps, po, count, in, to, factor, scales, static_cast<ucclComm_t>(comm), stream);
  else r = ucclReduceScatterEx(ps, po, count, in, to, factor, scales, static_cast<ucclComm_t>(comm), stream);
  Py_END_ALLOW_THREADS
  return finish(r, all ? "ucclAllReduceEx" : "ucclReduceScatterEx", static_cast<ucclComm_t>(comm));
}
PyObject* reduceScatterCast(PyObject* const* v, Py_ssize_t n) { return cast(v, n, false); }
PyObject* allReduceCast(PyObject* const* v, Py_ssize_t n) { return cast(v, n, true); }

// moe_dispatch(ctx, device, hidden, topk, x, topk_idx)
PyObject* moeDispatch(PyObject* const* v, Py_ssize_t n) {
  void *ctx, *stream;
  int device;
  long hidden, topk;
  if (n != 6 || overridden() || !handle(v[0], &ctx) || !gpu(v[1], &device) || !whole(v[2], 1, INT32_MAX, &hidden) || !whole(v[3], 1, INT32_MAX, &topk))
    Py_RETURN_FALSE;
  const at::Tensor *x = flat(v[4], device, at::kBFloat16), *idx = flat(v[5], device, at::kInt);
  if (!x || !idx || x->dim() != 2 || idx->dim() != 2 || x->size(1) != hidden || x->size(0) > INT32_MAX) Py_RETURN_FALSE;
  if (idx->size(0) != x->size(0) || idx->size(1) != topk) Py_RETURN_FALSE;
  const int tokens = static_cast<int>(x->size(0));
  void *px = x->data_ptr(), *pi = idx->data_ptr();
  if (!streamOf(device, &stream)) return nullptr;
  ucclResult_t r;
  Py_BEGIN_ALLOW_THREADS
  r = ucclMoeDispatch(static_cast<ucclMoeContext_t>(ctx), px, static_cast<const int32_t*>(pi), tokens, stream);
  Py_END_ALLOW_THREADS
  return finish(r, "ucclMoeDispatch", nullptr);
}

// moe_combine(ctx, device, tokens, hidden, topk, topk_weight, out)
PyObject* moeCombine(PyObject* const* v, Py_ssize_t n) {
  void *ctx, *stream;
  int device;
  long tokens, hidden, topk;
  if (n != 7 || overridden() || !handle(v[0], &ctx) || !gpu(v[1], &device)) Py_RETURN_FALSE;
  if (!whole(v[2], 0, INT32_MAX, &tokens) || !whole(v[3], 1, INT32_MAX, &hidden) || !whole(v[4], 1, INT32_MAX, &topk)) Py_RETURN_FALSE;
  const at::Tensor *w = flat(v[5], device, at::kFloat), *out = flat(v[6], device, at::kBFloat16);
  if (!w || !out || w->dim() != 2 || w->size(0) != tokens || w->size(1) != topk) Py_RETURN_FALSE;
  if (out->dim() != 2 || out->size(0) != tokens || out->size(1) != hidden) Py_RETURN_FALSE;
  void *pw = w->data_ptr(), *po = out->data_ptr();
  if (!streamOf(device, &stream)) return nullptr;
  ucclResult_t r;
  Py_BEGIN_ALLOW_THREADS
  r = ucclMoeCombine(static_cast<ucclMoeContext_t>(ctx), static_cast<const float*>(pw), static_cast<int>(tokens), po, stream);
  Py_END_ALLOW_THREADS
  return finish(r, "ucclMoeCombine", nullptr);
}

// No C++ exception leaves into Python: what a tensor answers with one (a storage without data) is for the general path.
template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyObject* entry(PyObject*, PyObject* const* v, Py_ssize_t n) {
  try {
    return F(v, n);
  } catch (...) {
    Py_RETURN_FALSE;
  }
}

template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyMethodDef method(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<F>)), METH_FASTCALL, nullptr};
}
PyMethodDef methods[] = {method<gemm>("gemm"), method<norm>("norm"), method<reduceScatter>("reduce_scatter"), method<allGather>("allgather"),
                         method<reduceScatterCast>("reduce_scatter_cast"), method<allReduceCast>("allreduce_cast"),
                         method<moeDispatch>("moe_dispatch"), method<moeCombine>("moe_combine"), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_uccl_tensor_calls", "Per-step calls on torch tensors", -1, methods, nullptr, nullptr, nullptr, nullptr};

// The layout of a tensor is compiled in.  A torch that was exchanged after the build may have another one and all the symbols.
bool builtForThisTorch() {
  PyObject* v = PyImport_ImportModule("torch.version");
  PyObject* number = v ? PyObject_GetAttrString(v, "__version__") : nullptr;
  PyObject* git = number ? PyObject_GetAttrString(v, "git_version") : nullptr;
  PyObject* here = git ? PyUnicode_FromFormat("%S_%S", number, git) : nullptr;
  const bool same = here && PyUnicode_CompareWithASCIIString(here, UCCL_TORCH_VERSION) == 0;
  if (here && !same) PyErr_Format(PyExc_ImportError, "built for torch %s, this is %U", UCCL_TORCH_VERSION, here);
  Py_XDECREF(here);
  Py_XDECREF(git);
  Py_XDECREF(number);
  Py_XDECREF(v);
  return same;
}

}  // namespace

PyMODINIT_FUNC PyInit__uccl_tensor_calls() {
  if (!builtForThisTorch()) return nullptr;
  PyObject* bindings = PyImport_ImportModule("unified_ccl_b200._uccl_bindings");
  PyObject* torch = bindings ? PyImport_ImportModule("torch._C") : nullptr;
  if (torch) {
    g_error = PyObject_GetAttrString(bindings, "UcclError");
    g_raw_stream = g_error ? PyObject_GetAttrString(torch, "_cuda_getCurrentRawStream") : nullptr;
    g_device = g_raw_stream ? PyObject_GetAttrString(torch, "_cuda_getDevice") : nullptr;
  }
  Py_XDECREF(bindings);
  Py_XDECREF(torch);
  if (!g_device) {
    PyErr_SetString(PyExc_ImportError, "needs a torch with CUDA");
    return nullptr;
  }
  return PyModule_Create(&module);
}
