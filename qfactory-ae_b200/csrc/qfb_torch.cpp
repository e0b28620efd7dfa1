// CPython module `_qfb_torch`: the per-call host work of the layers and of the decoder's element-wise neighbours
// between a Python call and the C ABI (include/qfactory_b200.h).
//
// What bounds it: a call on a small layer occupies the GPU for 4-5 us, while argument checks, torch.empty,
// the stream look-up and a ctypes call written in Python take 11 us, so a loop over small layers waits for the
// host.  Here the same steps are C++ on the tensors themselves.
//
// Every entry serves the plain case (dense fp16 CUDA tensors on the current device, contiguous) and returns
// NotImplemented for anything else; the Python code that called it then takes its general path, which also raises
// the errors.  A status other than QFB_OK comes back as an int.  What torch throws (no memory for an output, a tensor
// without storage) becomes the Python exception torch's own bindings raise: no C++ exception reaches the interpreter's
// frames.  The C ABI is reached through function addresses that the binding passes in, so this module does not link
// the library.
#include <Python.h>
#include <structmember.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/PyInterpreter.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/object_ptr.h>

#include "../../include/qfactory_b200.h"

namespace {

typedef int (*linear_fn)(const qfb_layer*, const void*, int, void*, void*, size_t, unsigned, void*);
typedef int (*rmsnorm_fn)(const void*, const void*, void*, int, int, float, void*);
typedef int (*add_rmsnorm_fn)(void*, const void*, const void*, void*, int, int, float, void*);
typedef int (*silu_mul_fn)(const void*, void*, int, int, void*);
typedef int (*attention_rope_fn)(const void*, const void*, const void*, const void*, void*, void*, void*, int, int, int, int,
                                 int, void*);

struct Abi {
  linear_fn linear, linear_silu_mul;
  rmsnorm_fn rmsnorm;
  add_rmsnorm_fn add_rmsnorm;
  silu_mul_fn silu_mul;
  attention_rope_fn attention_rope;
} abi = {};

// what a native call of one layer needs; `hold` keeps the packed tensors and the workspace alive (a new workspace comes
// with a new tuple)
struct LayerCall {
  PyObject_HEAD
  qfb_layer desc;
  void* ws;
  unsigned long long ws_bytes;
  unsigned flags;
  int silu_rows;      // most rows the fused silu(gate) * up form serves in one launch
  int device;
  PyObject* hold;
};

inline PyObject* general() { Py_RETURN_NOTIMPLEMENTED; }

// the GIL given up for the time of a launch, and taken back on any way out
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// the plain tensor behind `o`, or null where a subclass or another object needs the general path
inline const at::Tensor* plain(PyObject* o) {
  return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr;
}
inline bool dense_half(const at::Tensor& t, int device) {
  return t.is_cuda() && t.scalar_type() == at::kHalf && t.get_device() == device && t.is_contiguous();
}
// Something looks at torch's operations (a tracer, functorch, a dispatch or function mode): the Python path, whose
// operations it sees.  A default device is a function mode too, but concerns only factory calls that name no device.
PyObject* device_context_type = nullptr;
inline bool observed() {
  if (torch::jit::tracer::isTracing()) return true;
  const c10::DispatchKeySet included = c10::impl::tls_local_dispatch_key_set().included_;
  if (!(included - c10::default_included_set).empty()) return true;
  for (int64_t i = at::impl::PythonTorchFunctionTLS::stack_len() - 1; i >= 0; --i) {
    PyObject* mode = at::impl::PythonTorchFunctionTLS::get_stack_at(i)->ptr(getPyInterpreter());
    if (reinterpret_cast<PyObject*>(Py_TYPE(mode)) != device_context_type) return true;
  }
  return false;
}
// launches go to the current device: the plain case is the one where it is the tensors' own
inline bool ordinary(int device) { return c10::cuda::current_device() == device && !observed(); }
inline void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

inline at::Tensor empty_half(c10::IntArrayRef sizes, int device) {
  return at::Tensor(at::detail::empty_cuda(sizes, at::kHalf, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), std::nullopt));
}

// One linear: x [..., width] -> y [..., n].  `fused` = x is [gate | up] and the layer's input is silu(gate) * up.
PyObject* run_linear(LayerCall* L, PyObject* xo, PyObject* outo, bool fused) {
  const at::Tensor* x = plain(xo);
  if (!x || !dense_half(*x, L->device) || !ordinary(L->device)) return general();
  const int64_t width = (int64_t)L->desc.k * (fused ? 2 : 1), n = L->desc.n;
  const auto sizes = x->sizes();
  if (sizes.empty() || sizes.back() != width) return general();
  const int64_t rows = x->numel() / width;
  if (rows > INT32_MAX || (fused && (rows < 1 || rows > L->silu_rows))) return general();
  at::Tensor y;
  if (outo && outo != Py_None) {
    const at::Tensor* o = plain(outo);
    if (!o || !dense_half(*o, L->device) || o->numel() != rows * n || sizes.size() != 2) return general();
    if (fused && (o->dim() != 2 || o->size(1) != n)) return general();  // (comes back in the shape of the rows)
    y = *o;
  } else if (sizes.size() == 2) {
    const int64_t shape[2] = {rows, n};
    y = empty_half(shape, L->device);
  } else {
    c10::SmallVector<int64_t, 6> shape(sizes.begin(), sizes.end());
    shape.back() = n;
    y = empty_half(shape, L->device);
  }
  const void* xp = x->data_ptr();
  void *yp = y.mutable_data_ptr(), *st = stream_of(L->device);
  const linear_fn fn = fused ? abi.linear_silu_mul : abi.linear;
  // (read, and held, while no other thread can change them)
  void* const ws = L->ws;
  const size_t ws_bytes = (size_t)L->ws_bytes;
  const unsigned flags = L->flags;
  const THPObjectPtr hold(Py_XNewRef(L->hold));
  int status;
  {
    WithoutGil released;  // a launch waits where the stream's queue is full
    status = fn(&L->desc, xp, (int)rows, yp, ws, ws_bytes, flags, st);
  }
  if (outo && outo != Py_None && status == 0) {
    Py_INCREF(outo);
    return outo;
  }
  return status == 0 ? THPVariable_Wrap(std::move(y)) : PyLong_FromLong(status);
}

int layer_init(PyObject* self, PyObject* args, PyObject*) {
  LayerCall* L = reinterpret_cast<LayerCall*>(self);
  unsigned long long w, s, z, ws, ws_bytes;
  int n, k, bits, group, layout, device, silu_rows;
  unsigned flags;
  PyObject* hold;
  if (!PyArg_ParseTuple(args, "KKKiiiiiKKIiiO", &w, &s, &z, &n, &k, &bits, &group, &layout, &ws, &ws_bytes, &flags, &silu_rows,
                        &device, &hold))
    return -1;
  L->desc = qfb_layer{reinterpret_cast<const void*>(w), reinterpret_cast<const void*>(s), reinterpret_cast<const void*>(z), n, k,
                      bits, group, layout};
  L->ws = reinterpret_cast<void*>(ws);
  L->ws_bytes = ws_bytes;
  L->flags = flags;
  L->silu_rows = silu_rows;
  L->device = device;
  Py_INCREF(hold);
  Py_XSETREF(L->hold, hold);
  return 0;
}
void layer_dealloc(PyObject* self) {
  Py_XDECREF(reinterpret_cast<LayerCall*>(self)->hold);
  Py_TYPE(self)->tp_free(self);
}

PyObject* layer_forward(PyObject* self, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  if (na < 1 || na > 2) return general();
  return run_linear(reinterpret_cast<LayerCall*>(self), a[0], na > 1 ? a[1] : nullptr, false);
  END_HANDLE_TH_ERRORS
}
PyObject* layer_forward_silu_mul(PyObject* self, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  if (na < 1 || na > 2) return general();
  return run_linear(reinterpret_cast<LayerCall*>(self), a[0], na > 1 ? a[1] : nullptr, true);
  END_HANDLE_TH_ERRORS
}

PyMethodDef layer_methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(layer_forward), METH_FASTCALL, "y = x @ dequant(W)^T"},
    {"forward_silu_mul", reinterpret_cast<PyCFunction>(layer_forward_silu_mul), METH_FASTCALL, "y = (silu(gate) * up) @ dequant(W)^T"},
    {nullptr, nullptr, 0, nullptr}};
PyMemberDef layer_members[] = {{"flags", T_UINT, offsetof(LayerCall, flags), 0, "QFB_FLAG_* of every call"},
                               {"ws_ptr", T_ULONGLONG, offsetof(LayerCall, ws), 0, "workspace address"},
                               {"hold", T_OBJECT, offsetof(LayerCall, hold), 0, "what the pointers point into: (w, s, z, workspace)"},
                               {"ws_bytes", T_ULONGLONG, offsetof(LayerCall, ws_bytes), 0, "workspace size"},
                               {nullptr, 0, 0, 0, nullptr}};
PyTypeObject LayerType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- `layer(x)` without torch.nn.Module.__call__ -------------------------------------------------------------
// nn.Module's call walks several Python frames to find that a layer has no hooks (1-2 us).  This function is the
// layers' `__call__`: where the call that a layer inherits, its `_call_impl` and its `forward` are the ones they were
// when the classes were made, and neither the module nor torch as a whole has a hook or a compiled call, it runs the
// layer; anything else goes to the inherited call as it is at that moment, so that a replaced nn.Module.__call__ (as
// torch.fx's tracer does) or `forward` is seen.
PyObject *layer_call_method = nullptr;   // this function, as it stands in the classes
PyObject *served = nullptr;              // ((class, its forward, its _call_impl), ...)
PyObject *plain_call = nullptr;          // nn.Module's own __call__
PyObject *global_hooks = nullptr, *hook_keys = nullptr;
PyObject *key_native = nullptr, *key_forward = nullptr, *key_call = nullptr, *key_call_impl = nullptr;

inline bool empty_container(PyObject* o) {
  return o == nullptr || o == Py_None || (PyDict_Check(o) && PyDict_Size(o) == 0);
}

// the `__call__` behind this module's own in the order of the type's bases (borrowed)
PyObject* inherited_call(PyTypeObject* type) {
  bool own = false;
  PyObject* mro = type->tp_mro;
  for (Py_ssize_t i = 0; mro && i < PyTuple_GET_SIZE(mro); ++i) {
    PyObject* dict = reinterpret_cast<PyTypeObject*>(PyTuple_GET_ITEM(mro, i))->tp_dict;
    PyObject* call = dict ? PyDict_GetItem(dict, key_call) : nullptr;
    if (own && call && call != layer_call_method) return call;
    own = own || call == layer_call_method;
  }
  return nullptr;
}

// the call object of a layer that nobody has hooked, wrapped or replaced a part of; null otherwise
THPObjectPtr unhooked(PyObject* self, PyObject* inherited) {
  if (inherited != plain_call) return THPObjectPtr();
  bool ok = false;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(served) && !ok; ++i) {
    PyObject* entry = PyTuple_GET_ITEM(served, i);
    ok = reinterpret_cast<PyObject*>(Py_TYPE(self)) == PyTuple_GET_ITEM(entry, 0) &&
         _PyType_Lookup(Py_TYPE(self), key_forward) == PyTuple_GET_ITEM(entry, 1) &&
         _PyType_Lookup(Py_TYPE(self), key_call_impl) == PyTuple_GET_ITEM(entry, 2);
  }
  for (Py_ssize_t i = 0; ok && i < PyTuple_GET_SIZE(global_hooks); ++i) ok = empty_container(PyTuple_GET_ITEM(global_hooks, i));
  if (!ok) return THPObjectPtr();
  PyObject** dictp = _PyObject_GetDictPtr(self);
  THPObjectPtr dict(dictp && *dictp ? Py_NewRef(*dictp) : PyObject_GenericGetDict(self, nullptr));
  if (!dict) {
    PyErr_Clear();
    return THPObjectPtr();
  }
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(hook_keys); ++i)
    if (!empty_container(PyDict_GetItem(dict.get(), PyTuple_GET_ITEM(hook_keys, i)))) return THPObjectPtr();
  PyObject* native = PyDict_GetItem(dict.get(), key_native);
  return native && Py_TYPE(native) == &LayerType ? THPObjectPtr(Py_NewRef(native)) : THPObjectPtr();
}

PyObject* call_layer(PyObject*, PyObject* const* a, Py_ssize_t na, PyObject* kwnames) {
  HANDLE_TH_ERRORS
  if (!served || na < 1) {
    PyErr_SetString(PyExc_RuntimeError, "_qfb_torch: no layer, or bind has not been called");
    return nullptr;
  }
  PyObject *self = a[0], *inherited = inherited_call(Py_TYPE(self));
  if (!inherited) {
    PyErr_Format(PyExc_TypeError, "'%.200s' object is not a layer", Py_TYPE(self)->tp_name);
    return nullptr;
  }
  // layer(x), layer(x, out) or layer(x, out=...)
  const Py_ssize_t nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  if ((na == 2 && nkw == 0) || (na == 3 && nkw == 0) ||
      (na == 2 && nkw == 1 && PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, 0), "out") == 0)) {
    THPObjectPtr native = unhooked(self, inherited);
    if (native) {
      PyObject* y = run_linear(reinterpret_cast<LayerCall*>(native.get()), a[1], na + nkw > 2 ? a[2] : nullptr, false);
      if (!y || THPVariable_Check(y)) return y;
      Py_DECREF(y);  // NotImplemented or a status: the Python path repeats the call and raises what is wrong
    }
  }
  THPObjectPtr call(Py_NewRef(inherited));
  if (PyType_HasFeature(Py_TYPE(call.get()), Py_TPFLAGS_METHOD_DESCRIPTOR))
    return PyObject_Vectorcall(call.get(), a, (size_t)na, kwnames);
  const descrgetfunc get = Py_TYPE(call.get())->tp_descr_get;
  THPObjectPtr bound(get ? get(call.get(), self, reinterpret_cast<PyObject*>(Py_TYPE(self))) : Py_NewRef(call.get()));
  return bound ? PyObject_Vectorcall(bound.get(), a + 1, (size_t)(na - 1), kwnames) : nullptr;
  END_HANDLE_TH_ERRORS
}

// ---- element-wise neighbours ---------------------------------------------------------------------------------
inline bool out_tensor(PyObject* o, c10::IntArrayRef sizes, int device, at::Tensor* y) {
  if (!o || o == Py_None) {
    *y = empty_half(sizes, device);
    return true;
  }
  const at::Tensor* t = plain(o);
  if (!t || !dense_half(*t, device) || t->numel() != c10::multiply_integers(sizes)) return false;
  *y = *t;
  return true;
}
inline PyObject* give(int st, PyObject* o, at::Tensor& y) {
  if (st != 0) return PyLong_FromLong(st);
  if (o && o != Py_None) {
    Py_INCREF(o);
    return o;
  }
  return THPVariable_Wrap(std::move(y));
}

// `ro`: the residual, or null for the norm alone
PyObject* run_rmsnorm(PyObject* xo, PyObject* ro, PyObject* wo, PyObject* epso, PyObject* outo) {
  const at::Tensor *x = plain(xo), *w = plain(wo);
  const bool add = ro != nullptr;
  const at::Tensor* r = add ? plain(ro) : nullptr;
  if (!x || !w || (add && !r) || !x->is_cuda() || x->dim() < 1) return general();
  const int dev = x->get_device();
  if (!dense_half(*x, dev) || w->scalar_type() != at::kHalf || !w->is_cuda() || !ordinary(dev)) return general();
  if (add && (!dense_half(*r, dev) || r->sizes() != x->sizes())) return general();
  if (!PyFloat_Check(epso) && !PyLong_Check(epso)) return general();  // (what is no number is for ctypes to refuse)
  const double eps = PyFloat_AsDouble(epso);
  if (eps == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return general();
  }
  const int64_t d = x->sizes().back(), rows = d ? x->numel() / d : 0;
  at::Tensor y;
  if (rows > INT32_MAX || d > INT32_MAX || !out_tensor(outo, x->sizes(), dev, &y)) return general();
  void *xp = x->data_ptr(), *yp = y.mutable_data_ptr(), *st = stream_of(dev);
  const void *wp = w->data_ptr(), *rp = add ? r->data_ptr() : nullptr;
  int status;
  {
    WithoutGil released;
    status = add ? abi.add_rmsnorm(xp, rp, wp, yp, (int)rows, (int)d, (float)eps, st)
                 : abi.rmsnorm(xp, wp, yp, (int)rows, (int)d, (float)eps, st);
  }
  return give(status, outo, y);
}

// rmsnorm(x, weight, eps, out | None)
PyObject* py_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  return na == 4 ? run_rmsnorm(a[0], nullptr, a[1], a[2], a[3]) : general();
  END_HANDLE_TH_ERRORS
}

// add_rmsnorm(x, residual, weight, eps, out | None)
PyObject* py_add_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  return na == 5 ? run_rmsnorm(a[0], a[1], a[2], a[3], a[4]) : general();
  END_HANDLE_TH_ERRORS
}

// silu_mul(gate_up, out | None)
PyObject* py_silu_mul(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  if (na != 2) return general();
  const at::Tensor* x = plain(a[0]);
  if (!x || !x->is_cuda() || x->dim() < 1) return general();
  const int dev = x->get_device();
  const int64_t half = x->sizes().back() / 2;
  if (!dense_half(*x, dev) || !ordinary(dev) || half < 1) return general();
  const int64_t rows = x->numel() / (2 * half);
  c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
  shape.back() = half;
  at::Tensor y;
  if (rows > INT32_MAX || half > INT32_MAX || !out_tensor(a[1], shape, dev, &y)) return general();
  const void* xp = x->data_ptr();
  void *yp = y.mutable_data_ptr(), *st = stream_of(dev);
  int status;
  {
    WithoutGil released;
    status = abi.silu_mul(xp, yp, (int)rows, (int)half, st);
  }
  return give(status, a[1], y);
  END_HANDLE_TH_ERRORS
}

// decode_attention_rope(qkv, cos, sin, pos, k_cache, v_cache, q_heads, kv_heads, out | None)
PyObject* py_attention_rope(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  if (na != 9) return general();
  const at::Tensor* t[6];
  for (int i = 0; i < 6; ++i)
    if (!(t[i] = plain(a[i])) || !t[i]->is_cuda() || !t[i]->is_contiguous()) return general();
  const at::Tensor &qkv = *t[0], &cosv = *t[1], &sinv = *t[2], &pos = *t[3], &kc = *t[4], &vc = *t[5];
  const int dev = qkv.get_device();
  if (!PyLong_Check(a[6]) || !PyLong_Check(a[7])) return general();
  const long hq = PyLong_AsLong(a[6]), hkv = PyLong_AsLong(a[7]);
  if ((hq == -1 || hkv == -1) && PyErr_Occurred()) {
    PyErr_Clear();
    return general();
  }
  if (!dense_half(qkv, dev) || !ordinary(dev) || qkv.dim() != 4 || qkv.size(1) != 1 || qkv.size(2) != hq + 2 * hkv)
    return general();
  if (pos.scalar_type() != at::kLong || pos.numel() != 1 || cosv.scalar_type() != at::kHalf || sinv.scalar_type() != at::kHalf)
    return general();
  const int64_t B = qkv.size(0), hd = qkv.size(3);
  if (kc.dim() != 4 || vc.sizes() != kc.sizes() || kc.size(0) != B || kc.size(1) != hkv || kc.size(3) != hd) return general();
  const int64_t shape[2] = {B, hq * hd};
  at::Tensor y;
  if (!out_tensor(a[8], shape, dev, &y)) return general();
  void* st = stream_of(dev);
  void *kp = kc.data_ptr(), *vp = vc.data_ptr(), *yp = y.mutable_data_ptr();
  const void *qp = qkv.data_ptr(), *cp = cosv.data_ptr(), *sp = sinv.data_ptr(), *pp = pos.data_ptr();
  const int max_len = (int)kc.size(2);
  int status;
  {
    WithoutGil released;
    status = abi.attention_rope(qp, cp, sp, pp, kp, vp, yp, (int)B, (int)hq, (int)hkv, (int)hd, max_len, st);
  }
  return give(status, a[8], y);
  END_HANDLE_TH_ERRORS
}

// bind(addresses: dict, nn.Module's __call__, ((class, forward, _call_impl), ...), global_hooks: tuple, hook_keys: tuple,
//      the function mode of a default device)
PyObject* py_bind(PyObject*, PyObject* args) {
  PyObject *addr, *mc, *types, *globals, *keys, *devctx;
  if (!PyArg_ParseTuple(args, "O!OO!O!O!O", &PyDict_Type, &addr, &mc, &PyTuple_Type, &types, &PyTuple_Type, &globals,
                        &PyTuple_Type, &keys, &devctx))
    return nullptr;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(types); ++i)
    if (!PyTuple_Check(PyTuple_GET_ITEM(types, i)) || PyTuple_GET_SIZE(PyTuple_GET_ITEM(types, i)) != 3) {
      PyErr_SetString(PyExc_ValueError, "a served class comes with its forward and its _call_impl");
      return nullptr;
    }
  auto at_name = [&](const char* n) -> void* {
    PyObject* v = PyDict_GetItemString(addr, n);
    return v ? PyLong_AsVoidPtr(v) : nullptr;
  };
  abi.linear = reinterpret_cast<linear_fn>(at_name("qfb_linear_forward"));
  abi.linear_silu_mul = reinterpret_cast<linear_fn>(at_name("qfb_linear_silu_mul_forward"));
  abi.rmsnorm = reinterpret_cast<rmsnorm_fn>(at_name("qfb_rmsnorm"));
  abi.add_rmsnorm = reinterpret_cast<add_rmsnorm_fn>(at_name("qfb_add_rmsnorm"));
  abi.silu_mul = reinterpret_cast<silu_mul_fn>(at_name("qfb_silu_mul"));
  abi.attention_rope = reinterpret_cast<attention_rope_fn>(at_name("qfb_decode_attention_rope"));
  if (!abi.linear || !abi.linear_silu_mul || !abi.rmsnorm || !abi.add_rmsnorm || !abi.silu_mul || !abi.attention_rope) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "an entry point is missing");
    return nullptr;
  }
  for (PyObject* o : {mc, types, globals, keys, devctx}) Py_INCREF(o);
  Py_XSETREF(plain_call, mc);
  Py_XSETREF(served, types);
  Py_XSETREF(global_hooks, globals);
  Py_XSETREF(hook_keys, keys);
  Py_XSETREF(device_context_type, devctx);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, "addresses of the C ABI and the state of torch.nn.Module's call"},
    {"call_layer", reinterpret_cast<PyCFunction>(call_layer), METH_FASTCALL | METH_KEYWORDS, "__call__ of the layers"},
    {"rmsnorm", reinterpret_cast<PyCFunction>(py_rmsnorm), METH_FASTCALL, "rmsnorm(x, weight, eps, out)"},
    {"add_rmsnorm", reinterpret_cast<PyCFunction>(py_add_rmsnorm), METH_FASTCALL, "add_rmsnorm(x, residual, weight, eps, out)"},
    {"silu_mul", reinterpret_cast<PyCFunction>(py_silu_mul), METH_FASTCALL, "silu_mul(gate_up, out)"},
    {"decode_attention_rope", reinterpret_cast<PyCFunction>(py_attention_rope), METH_FASTCALL,
     "decode_attention_rope(qkv, cos, sin, pos, k_cache, v_cache, q_heads, kv_heads, out)"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_qfb_torch", "native call path of the quantized layers", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__qfb_torch(void) {
  LayerType.tp_name = "_qfb_torch.LayerCall";
  LayerType.tp_basicsize = sizeof(LayerCall);
  LayerType.tp_flags = Py_TPFLAGS_DEFAULT;
  LayerType.tp_new = PyType_GenericNew;
  LayerType.tp_init = layer_init;
  LayerType.tp_dealloc = layer_dealloc;
  LayerType.tp_methods = layer_methods;
  LayerType.tp_members = layer_members;
  if (PyType_Ready(&LayerType) < 0) return nullptr;
  key_native = PyUnicode_InternFromString("_native_call");
  key_forward = PyUnicode_InternFromString("forward");
  key_call = PyUnicode_InternFromString("__call__");
  key_call_impl = PyUnicode_InternFromString("_call_impl");
  PyObject* m = PyModule_Create(&module_def);
  if (!m || !key_native || !key_forward || !key_call || !key_call_impl) return nullptr;
  PyObject* call = PyObject_GetAttrString(m, "call_layer");
  PyObject* method = call ? PyInstanceMethod_New(call) : nullptr;  // binds to the instance as a Python function would
  Py_XDECREF(call);
  layer_call_method = Py_XNewRef(method);
  Py_INCREF(&LayerType);
  if (!method || PyModule_AddObject(m, "layer_call_method", method) < 0 ||
      PyModule_AddObject(m, "LayerCall", reinterpret_cast<PyObject*>(&LayerType)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
