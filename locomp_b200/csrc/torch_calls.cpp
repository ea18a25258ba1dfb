// The host path of the operators for torch CUDA tensors, in native code: one Python call checks the
// operands, makes the output, finds the stream and its workspace and calls the C ABI
// (include/locomp_b200.h).  A small kernel of this library runs 2-4 us; the same steps written in
// Python (operand objects, attribute reads, a size query, a device context, ctypes conversions) took
// 20 us per call, so a decode loop that is not captured in a graph was bound by them.
//
// Every function returns NotImplemented for whatever is not the ordinary case (NumPy arrays,
// DeviceTensor, foreign objects, non-contiguous or CPU tensors, wrong types or sizes): the caller then
// takes the general path in Python, which handles it or raises the error that names what is wrong.
// The GIL is released around the C ABI call only (a full launch queue makes it wait).  The scratch of a stream
// is locked from its lookup until the call has returned: threads that share a stream (each thread's current stream
// is the default one unless it changed it) would otherwise mix the launches of calls that use the same scratch, or
// replace it under a call that has not launched yet.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>

#include <map>
#include <mutex>
#include <utility>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/locomp_b200.h"

namespace {

// The C ABI, looked up in the library that the Python side loaded.
struct Api {
  decltype(&lcq_matmul_int4) matmul[2];
  decltype(&lcq_dequant_int4) dequant[2];
  decltype(&lcq_quantize_int4) quantize[2];
  decltype(&lcq_rms_norm) rms_norm;
  decltype(&lcq_residual_rms_norm) residual_rms_norm;
  decltype(&lcq_silu_mul) silu_mul;
  decltype(&lcq_add_inplace) add_inplace;
  decltype(&lcq_embed_lookup) embed_lookup;
  decltype(&lcq_argmax) argmax;
  decltype(&lcq_matmul_workspace_bytes) workspace_bytes;
} api;
PyObject* raise_status = nullptr;      // callable(status): raises the exception of a negative status
PyObject* make_workspace = nullptr;    // callable(nbytes, device, stream): allocates (or grows) and reports it through set_workspace

// The scratch of a (device, stream).  The lock is taken without the GIL (and may be held while the GIL is taken, never
// the other way round), the table is touched with the GIL only.  Recursive: the allocation below it may run
// other Python code of the same thread.
struct Scratch {
  std::recursive_mutex lock;
  PyObject* tensor = nullptr;          // owns the memory
  void* ptr = nullptr;
  size_t bytes = 0;
};
std::map<std::pair<int, uintptr_t>, Scratch> scratches;
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  void end() { if (state) PyEval_RestoreThread(state); state = nullptr; }
  void again() { state = PyEval_SaveThread(); }
  ~NoGil() { end(); }
};

constexpr int NOT_FLOAT = -1;
int float_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return LCQ_F32;
    case at::kHalf: return LCQ_F16;
    case at::kBFloat16: return LCQ_BF16;
    default: return NOT_FLOAT;
  }
}
at::ScalarType float_type(int code) { return code == LCQ_F32 ? at::kFloat : code == LCQ_F16 ? at::kHalf : at::kBFloat16; }

// A contiguous CUDA tensor, or nullptr.
const at::Tensor* cuda_tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() ? &t : nullptr;
}
bool as_int(PyObject* o, long long& v) {
  if (!PyLong_Check(o)) return false;
  int overflow = 0;
  v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}
PyObject* not_implemented() { Py_RETURN_NOTIMPLEMENTED; }
PyObject* fail(int status) {
  PyObject* r = PyObject_CallFunction(raise_status, "i", status);
  if (r) {      // the callable raises; this is reached only if it does not
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, "locomp_b200: a call failed without a message");
  }
  return nullptr;
}
PyObject* finish(int status, at::Tensor&& out) { return status < 0 ? fail(status) : THPVariable_Wrap(std::move(out)); }
PyObject* finish(int status, PyObject* given) {
  if (status < 0) return fail(status);
  Py_INCREF(given);
  return given;
}
template <typename F>
int unlocked(const F& call) {
  NoGil released;
  return call();
}
void* current_stream(int device) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream(); }
at::Tensor empty(at::IntArrayRef shape, at::ScalarType type, const at::Tensor& like) {
  return at::detail::empty_cuda(shape, type, like.device(), c10::nullopt);
}

// matmul(x, w, scales, group_size, bits, out | None, workspace | None)
PyObject* matmul(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 7) return not_implemented();
  const at::Tensor *x = cuda_tensor(args[0]), *w = cuda_tensor(args[1]), *s = cuda_tensor(args[2]);
  long long group, bits;
  if (!x || !w || !s || !as_int(args[3], group) || !as_int(args[4], bits) || (bits != 4 && bits != 8)) return not_implemented();
  const int xk = float_code(x->scalar_type()), sk = float_code(s->scalar_type());
  if (xk == NOT_FLOAT || sk == NOT_FLOAT || w->scalar_type() != (bits == 4 ? at::kByte : at::kChar)) return not_implemented();
  const bool row = x->dim() == 1;
  if ((!row && x->dim() != 2) || w->dim() != 2 || w->device() != x->device() || s->device() != x->device()) return not_implemented();
  const int64_t M = row ? 1 : x->size(0), K = x->size(-1), N = w->size(0);
  constexpr int64_t most = 2000000000;
  if (w->size(1) * (bits == 4 ? 2 : 1) != K || group <= 0 || group > most || K % group != 0 || s->numel() != N * (K / group) ||
      M > most || N > most || K > most)
    return not_implemented();
  at::Tensor made;
  const at::Tensor* out = &made;
  int ok = xk;
  const c10::cuda::OptionalCUDAGuard guard(x->device());
  if (args[5] == Py_None) {
    made = row ? empty({N}, x->scalar_type(), *x) : empty({M, N}, x->scalar_type(), *x);
  } else {
    out = cuda_tensor(args[5]);
    if (!out || out->device() != x->device() || out->numel() != M * N || (ok = float_code(out->scalar_type())) == NOT_FLOAT)
      return not_implemented();
  }
  const int dev = x->device().index();
  void* stream = current_stream(dev);
  const void *xp = x->data_ptr(), *wp = w->data_ptr(), *sp = s->data_ptr();
  void* op = out->data_ptr();
  const auto call = [&](void* ws, size_t ws_bytes) {       // without the GIL
    return api.matmul[bits == 8](xp, wp, sp, op, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), static_cast<int>(group),
                                 xk, sk, ok, LCQ_ALGO_AUTO, ws, ws_bytes, stream);
  };
  int rc = LCQ_ERR_WORKSPACE;
  if (args[6] != Py_None) {
    const at::Tensor* ws = cuda_tensor(args[6]);
    if (!ws || ws->device() != x->device()) return not_implemented();
    void* ws_ptr = ws->data_ptr();
    const size_t ws_bytes = ws->nbytes();
    rc = unlocked([&] { return call(ws_ptr, ws_bytes); });
    if (rc == LCQ_ERR_WORKSPACE) return not_implemented();
  } else if (bits == 8 || xk == LCQ_F32 || sk != LCQ_F16) {
    rc = unlocked([&] { return call(nullptr, 0); });         // no kernel of these types has scratch
  }
  if (args[6] == Py_None && rc == LCQ_ERR_WORKSPACE) {
    Scratch& scratch = scratches[{dev, reinterpret_cast<uintptr_t>(stream)}];
    NoGil released;
    const std::lock_guard<std::recursive_mutex> held(scratch.lock);
    // The call itself says whether the scratch this stream has is enough: no size query on the ordinary path.
    rc = call(scratch.ptr, scratch.bytes);
    if (rc == LCQ_ERR_WORKSPACE) {
      released.end();
      const size_t need = api.workspace_bytes(static_cast<int>(bits), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K),
                                              static_cast<int>(group), xk, sk, ok, LCQ_ALGO_AUTO);
      PyObject* r = PyObject_CallFunction(make_workspace, "niK", static_cast<Py_ssize_t>(need), dev,
                                          static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)));
      if (!r) return nullptr;
      Py_DECREF(r);
      released.again();
      rc = call(scratch.ptr, scratch.bytes);
    }
  }
  return args[5] == Py_None ? finish(rc, std::move(made)) : finish(rc, args[5]);
}

// dequantize(w, scales, N, K, group_size, bits, out dtype code)
PyObject* dequantize(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 7) return not_implemented();
  const at::Tensor *w = cuda_tensor(args[0]), *s = cuda_tensor(args[1]);
  long long N, K, group, bits, ok;
  if (!w || !s || !as_int(args[2], N) || !as_int(args[3], K) || !as_int(args[4], group) || !as_int(args[5], bits) || !as_int(args[6], ok))
    return not_implemented();
  const int sk = float_code(s->scalar_type());
  if ((bits != 4 && bits != 8) || w->scalar_type() != (bits == 4 ? at::kByte : at::kChar) || sk == NOT_FLOAT || s->device() != w->device())
    return not_implemented();
  if (N < 0 || K <= 0 || group <= 0 || group > 2000000000 || K % group != 0 || (bits == 4 && K % 2 != 0) ||
      w->numel() != N * (bits == 4 ? K / 2 : K) || s->numel() != N * (K / group))
    return not_implemented();
  const c10::cuda::OptionalCUDAGuard guard(w->device());
  at::Tensor out = empty({N, K}, float_type(static_cast<int>(ok)), *w);
  void* stream = current_stream(w->device().index());
  const int rc = unlocked([&] {
    return api.dequant[bits == 8](w->data_ptr(), s->data_ptr(), out.data_ptr(), N, K, static_cast<int>(group), sk, static_cast<int>(ok), stream);
  });
  return finish(rc, std::move(out));
}

// quantize(weights, group_size, bits, style) -> (packed, scales)
PyObject* quantize(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 4) return not_implemented();
  const at::Tensor* w = cuda_tensor(args[0]);
  long long group, bits, style;
  if (!w || !as_int(args[1], group) || !as_int(args[2], bits) || !as_int(args[3], style) || w->dim() != 2) return not_implemented();
  const int wk = float_code(w->scalar_type());
  const int64_t N = w->size(0), K = w->size(1);
  if (wk == NOT_FLOAT || (bits != 4 && bits != 8) || group <= 0 || group > 2000000000 || K <= 0 || K % group != 0 || (bits == 4 && group % 2 != 0))
    return not_implemented();
  const c10::cuda::OptionalCUDAGuard guard(w->device());
  at::Tensor q = bits == 4 ? empty({N, K / 2}, at::kByte, *w) : empty({N, K}, at::kChar, *w);
  at::Tensor s = empty({N, K / group}, at::kFloat, *w);
  void* stream = current_stream(w->device().index());
  const int rc = unlocked([&] {
    return api.quantize[bits == 8](w->data_ptr(), q.data_ptr(), s.data_ptr(), N, K, static_cast<int>(group), wk, static_cast<int>(style), stream);
  });
  if (rc < 0) return fail(rc);
  PyObject* pair = PyTuple_New(2);
  if (!pair) return nullptr;
  PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(q)));
  PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::move(s)));
  return pair;
}

// Operands that must share type and device; the type's code, or NOT_FLOAT.
int shared_code(const at::Tensor& a, const at::Tensor& b) {
  return a.scalar_type() == b.scalar_type() && a.device() == b.device() ? float_code(a.scalar_type()) : NOT_FLOAT;
}
// The result tensor of an operator whose result is shaped like `like`: `given`, or a new one in `made`.
const at::Tensor* result(PyObject* given, const at::Tensor& like, at::Tensor& made) {
  if (given == Py_None) {
    made = empty(like.sizes(), like.scalar_type(), like);
    return &made;
  }
  const at::Tensor* out = cuda_tensor(given);
  return out && out->numel() == like.numel() && shared_code(*out, like) != NOT_FLOAT ? out : nullptr;
}

// rms_norm(x, weight, eps, out | None)
PyObject* rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 4) return not_implemented();
  const at::Tensor *x = cuda_tensor(args[0]), *w = cuda_tensor(args[1]);
  if (!x || !w || !PyFloat_Check(args[2]) || x->dim() < 1 || x->numel() == 0) return not_implemented();
  const int code = shared_code(*x, *w);
  const int64_t n = x->size(-1);
  if (code == NOT_FLOAT || w->numel() != n || n > 2000000000) return not_implemented();
  const c10::cuda::OptionalCUDAGuard guard(x->device());
  at::Tensor made;
  const at::Tensor* out = result(args[3], *x, made);
  if (!out) return not_implemented();
  void* stream = current_stream(x->device().index());
  const float eps = static_cast<float>(PyFloat_AS_DOUBLE(args[2]));
  const int rc = unlocked([&] {
    return api.rms_norm(x->data_ptr(), w->data_ptr(), out->data_ptr(), x->numel() / n, static_cast<int>(n), eps, code, stream);
  });
  return args[3] == Py_None ? finish(rc, std::move(made)) : finish(rc, args[3]);
}

// residual_rms_norm(hidden, delta, weight, eps, out | None)
PyObject* residual_rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 5) return not_implemented();
  const at::Tensor *h = cuda_tensor(args[0]), *d = cuda_tensor(args[1]), *w = cuda_tensor(args[2]);
  if (!h || !d || !w || !PyFloat_Check(args[3]) || h->dim() < 1 || h->numel() == 0) return not_implemented();
  const int code = shared_code(*h, *d);
  const int64_t n = h->size(-1);
  if (code == NOT_FLOAT || shared_code(*h, *w) == NOT_FLOAT || d->numel() != h->numel() || w->numel() != n || n > 2000000000)
    return not_implemented();
  const c10::cuda::OptionalCUDAGuard guard(h->device());
  at::Tensor made;
  const at::Tensor* out = result(args[4], *h, made);
  if (!out) return not_implemented();
  void* stream = current_stream(h->device().index());
  const float eps = static_cast<float>(PyFloat_AS_DOUBLE(args[3]));
  const int rc = unlocked([&] {
    return api.residual_rms_norm(h->data_ptr(), d->data_ptr(), w->data_ptr(), out->data_ptr(), h->numel() / n, static_cast<int>(n), eps, code, stream);
  });
  return args[4] == Py_None ? finish(rc, std::move(made)) : finish(rc, args[4]);
}

// silu_mul(gate, up, out | None)
PyObject* silu_mul(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 3) return not_implemented();
  const at::Tensor *g = cuda_tensor(args[0]), *u = cuda_tensor(args[1]);
  if (!g || !u || g->numel() != u->numel()) return not_implemented();
  const int code = shared_code(*g, *u);
  if (code == NOT_FLOAT) return not_implemented();
  const c10::cuda::OptionalCUDAGuard guard(g->device());
  at::Tensor made;
  const at::Tensor* out = result(args[2], *g, made);
  if (!out) return not_implemented();
  void* stream = current_stream(g->device().index());
  const int rc = unlocked([&] { return api.silu_mul(g->data_ptr(), u->data_ptr(), out->data_ptr(), g->numel(), code, stream); });
  return args[2] == Py_None ? finish(rc, std::move(made)) : finish(rc, args[2]);
}

// add_inplace(a, b)
PyObject* add_inplace(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 2) return not_implemented();
  const at::Tensor *a = cuda_tensor(args[0]), *b = cuda_tensor(args[1]);
  if (!a || !b || a->numel() != b->numel()) return not_implemented();
  const int code = shared_code(*a, *b);
  if (code == NOT_FLOAT) return not_implemented();
  const c10::cuda::OptionalCUDAGuard guard(a->device());
  void* stream = current_stream(a->device().index());
  return finish(unlocked([&] { return api.add_inplace(a->data_ptr(), b->data_ptr(), a->numel(), code, stream); }), args[0]);
}

// embed_lookup(token_ids, table, out, seq_len, dim)
PyObject* embed_lookup(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 5) return not_implemented();
  const at::Tensor *ids = cuda_tensor(args[0]), *table = cuda_tensor(args[1]), *out = cuda_tensor(args[2]);
  long long tokens, dim;
  if (!ids || !table || !out || !as_int(args[3], tokens) || !as_int(args[4], dim)) return not_implemented();
  const int code = shared_code(*table, *out);
  if (code == NOT_FLOAT || ids->scalar_type() != at::kInt || ids->device() != table->device() || tokens < 0 || dim <= 0 || dim > 2000000000 ||
      ids->numel() < tokens || table->numel() % dim != 0 || table->numel() / dim > 2000000000 || out->numel() / dim < tokens)
    return not_implemented();
  const c10::cuda::OptionalCUDAGuard guard(table->device());
  void* stream = current_stream(table->device().index());
  const int rc = unlocked([&] {
    return api.embed_lookup(ids->data_ptr(), table->data_ptr(), out->data_ptr(), tokens, static_cast<int>(table->numel() / dim),
                            static_cast<int>(dim), code, stream);
  });
  return finish(rc, Py_None);
}

// argmax(x, out | None)
PyObject* argmax(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 2) return not_implemented();
  const at::Tensor* x = cuda_tensor(args[0]);
  if (!x || x->dim() < 1 || x->numel() == 0) return not_implemented();
  const int code = float_code(x->scalar_type());
  const int64_t n = x->size(-1), rows = x->numel() / n;
  if (code == NOT_FLOAT || n > 2000000000) return not_implemented();
  const c10::cuda::OptionalCUDAGuard guard(x->device());
  at::Tensor made;
  const at::Tensor* out = &made;
  if (args[1] == Py_None) {
    made = empty(x->sizes().slice(0, x->dim() - 1), at::kInt, *x);
  } else {
    out = cuda_tensor(args[1]);
    if (!out || out->scalar_type() != at::kInt || out->numel() != rows || out->device() != x->device()) return not_implemented();
  }
  void* stream = current_stream(x->device().index());
  const int rc = unlocked([&] { return api.argmax(x->data_ptr(), out->data_ptr(), rows, static_cast<int>(n), code, stream); });
  return args[1] == Py_None ? finish(rc, std::move(made)) : finish(rc, args[1]);
}

bool stream_key(PyObject* const* args, std::pair<int, uintptr_t>& key) {      // (device, stream)
  const long dev = PyLong_AsLong(args[0]);
  const unsigned long long stream = PyErr_Occurred() ? 0 : PyLong_AsUnsignedLongLong(args[1]);
  key = {static_cast<int>(dev), static_cast<uintptr_t>(stream)};
  return !PyErr_Occurred();
}
// set_workspace(device, stream, tensor): the scratch that calls on this stream use from now on; its lock is held
PyObject* set_workspace(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  std::pair<int, uintptr_t> key;
  if (n_args != 3 || !THPVariable_Check(args[2])) return PyErr_Format(PyExc_TypeError, "set_workspace(device, stream, tensor)");
  if (!stream_key(args, key)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(args[2]);
  Scratch& scratch = scratches[key];
  scratch.ptr = t.data_ptr();
  scratch.bytes = t.nbytes();
  PyObject* old = scratch.tensor;
  Py_INCREF(args[2]);
  scratch.tensor = args[2];
  Py_XDECREF(old);
  Py_RETURN_NONE;
}
// lock_workspace(device, stream), unlock_workspace(device, stream): for the general path
PyObject* lock_workspace(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  std::pair<int, uintptr_t> key;
  if (n_args != 2) return PyErr_Format(PyExc_TypeError, "lock_workspace(device, stream)");
  if (!stream_key(args, key)) return nullptr;
  Scratch& scratch = scratches[key];
  unlocked([&] { scratch.lock.lock(); return 0; });
  Py_RETURN_NONE;
}
PyObject* unlock_workspace(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  std::pair<int, uintptr_t> key;
  if (n_args != 2) return PyErr_Format(PyExc_TypeError, "unlock_workspace(device, stream)");
  if (!stream_key(args, key)) return nullptr;
  scratches[key].lock.unlock();
  Py_RETURN_NONE;
}

// bind(path of the library, raise_status, make_workspace)
PyObject* bind(PyObject*, PyObject* args) {
  const char* path;
  PyObject *raise_fn, *workspace_fn;
  if (!PyArg_ParseTuple(args, "sOO", &path, &raise_fn, &workspace_fn)) return nullptr;
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!lib) return PyErr_Format(PyExc_ImportError, "%s: %s", path, dlerror());
  bool all = true;
  const auto find = [&](auto& slot, const char* name) {
    void* p = dlsym(lib, name);
    slot = reinterpret_cast<std::remove_reference_t<decltype(slot)>>(p);
    all = all && p;
  };
  find(api.matmul[0], "lcq_matmul_int4");
  find(api.matmul[1], "lcq_matmul_int8");
  find(api.dequant[0], "lcq_dequant_int4");
  find(api.dequant[1], "lcq_dequant_int8");
  find(api.quantize[0], "lcq_quantize_int4");
  find(api.quantize[1], "lcq_quantize_int8");
  find(api.rms_norm, "lcq_rms_norm");
  find(api.residual_rms_norm, "lcq_residual_rms_norm");
  find(api.silu_mul, "lcq_silu_mul");
  find(api.add_inplace, "lcq_add_inplace");
  find(api.embed_lookup, "lcq_embed_lookup");
  find(api.argmax, "lcq_argmax");
  find(api.workspace_bytes, "lcq_matmul_workspace_bytes");
  if (!all) return PyErr_Format(PyExc_ImportError, "%s lacks an entry point", path);
  Py_INCREF(raise_fn);
  Py_INCREF(workspace_fn);
  raise_status = raise_fn;
  make_workspace = workspace_fn;
  Py_RETURN_NONE;
}

// The base class of QuantLinear: the call itself in native code, so that it enters no Python frame.  The layer's weights
// are ordinary attributes of the instance (it is copied, pickled and changed as any Python object) and are owned here
// for the duration of the call: another thread may rebind them while the GIL is released.  What is not `linear(x)`
// or `linear(x, out)` goes to the method _general of the subclass.
PyObject* general_name = nullptr;
PyObject* operand_names[4];            // w, scales, group_size, bits

struct Owned {
  PyObject* p = nullptr;
  ~Owned() { Py_XDECREF(p); }
};

PyObject* linear_call(PyObject* self, PyObject* args, PyObject* kwargs) {
  const Py_ssize_t n = PyTuple_GET_SIZE(args);
  if (raise_status && (kwargs == nullptr || PyDict_GET_SIZE(kwargs) == 0) && (n == 1 || n == 2)) {
    Owned of_layer[4];
    bool all = true;
    for (int i = 0; i < 4 && all; ++i) all = (of_layer[i].p = PyObject_GetAttr(self, operand_names[i])) != nullptr;
    if (all) {
      PyObject* const a[7] = {PyTuple_GET_ITEM(args, 0), of_layer[0].p, of_layer[1].p, of_layer[2].p, of_layer[3].p,
                              n == 2 ? PyTuple_GET_ITEM(args, 1) : Py_None, Py_None};
      PyObject* r;
      {
        HANDLE_TH_ERRORS
        r = matmul(nullptr, a, 7);
        END_HANDLE_TH_ERRORS
      }
      if (r != Py_NotImplemented) return r;
      Py_DECREF(r);
    } else {
      PyErr_Clear();                   // (_general raises it)
    }
  }
  PyObject* method = PyObject_GetAttr(self, general_name);
  if (!method) return nullptr;
  PyObject* r = PyObject_Call(method, args, kwargs);
  Py_DECREF(method);
  return r;
}
PyType_Slot linear_slots[] = {{Py_tp_call, reinterpret_cast<void*>(linear_call)}, {0, nullptr}};
PyType_Spec linear_spec = {"locomp_b200._torch_calls.LinearBase", 0, 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE, linear_slots};

// A C++ exception (out of memory, a CUDA error seen by torch) becomes the Python exception torch gives it.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, args, n);
  END_HANDLE_TH_ERRORS
}
#define LCQ_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    LCQ_METHOD(matmul), LCQ_METHOD(dequantize), LCQ_METHOD(quantize), LCQ_METHOD(rms_norm), LCQ_METHOD(residual_rms_norm),
    LCQ_METHOD(silu_mul), LCQ_METHOD(add_inplace), LCQ_METHOD(embed_lookup), LCQ_METHOD(argmax), LCQ_METHOD(set_workspace),
    LCQ_METHOD(lock_workspace), LCQ_METHOD(unlock_workspace),
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_calls(void) {
  general_name = PyUnicode_InternFromString("_general");
  const char* const names[4] = {"w", "scales", "group_size", "bits"};
  bool all = general_name != nullptr;
  for (int i = 0; i < 4; ++i) all = (operand_names[i] = PyUnicode_InternFromString(names[i])) != nullptr && all;
  PyObject* m = PyModule_Create(&module);
  PyObject* type = PyType_FromSpec(&linear_spec);      // a heap type without fields of its own, like a class of Python
  if (!all || !m || !type || PyModule_AddObject(m, "LinearBase", type) < 0) return nullptr;
  return m;
}
