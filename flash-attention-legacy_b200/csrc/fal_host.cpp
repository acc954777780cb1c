// The host side of the calls that a generation loop makes for every token or short prompt -- flash_attention without
// gradients, a decode step -- as a small Python extension: checks, output allocation, argument block and call in one
// native function.  In Python the same took longer than the kernels of a short call; us a call, Python -> this, with the
// kernels' share: 2 x 8 x 128 forward 24.6 -> 8.2 (5.3), 2 x 8 x 1 024 24.7 -> 12.3 (10.7), decode of one entry of 1 999
// positions 25.6 -> 10.3 (8).
//
// It takes ordinary calls only and answers None for everything else (tensor subclasses, function transforms, modes,
// tracing, gradients, tangents, tensors that need a copy, wrong shapes or types, an error of the library): the caller
// then goes its general way, which copies, records or refuses as it did.  Nothing is kept between calls but what the
// binding hands over: the library's entry points, the status words and the dictionary of decode workspaces.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/PythonDispatcherTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/csrc/utils/pybind.h>

#include <cmath>
#include <optional>

#include "../../include/fal_b200.h"

namespace {

constexpr int kMaxDevices = 64;

struct Calls {
  PyObject_HEAD
  int (*fwd_run)(const fal_fwd_args*);
  int (*decode_run)(const fal_decode_args*);
  size_t (*decode_workspace_bytes)(int, int, int, int);
  PyObject* workspaces;       // {(device, stream): uint8 tensor}
  size_t workspace_min;
  int* status[kMaxDevices];   // device status words, null until the binding has made one
};

using c10::DispatchKey;
using c10::DispatchKeySet;

bool within(DispatchKeySet keys, DispatchKeySet allowed) { return (keys.raw_repr() & ~allowed.raw_repr()) == 0; }

// No mode, transform or tracer that would see, or change, what the general way does.
bool ordinary_call() {
  if (at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
      c10::impl::PythonDispatcherTLS::get_state() != nullptr || torch::jit::tracer::isTracing())
    return false;
  static const DispatchKeySet usual = DispatchKeySet({DispatchKey::BackendSelect, DispatchKey::ADInplaceOrView});
  return within(c10::impl::tls_local_dispatch_key_set().included_, usual);
}

// A dense CUDA tensor of the given type and rank, of torch.Tensor itself and without a wrapper around it, whose last
// dimension is contiguous; null if it is anything else.
const at::Tensor* plain(PyObject* obj, at::ScalarType type, int64_t ndim) {
  if (!THPVariable_CheckExact(obj)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(obj);
  static const DispatchKeySet usual = DispatchKeySet(
      {DispatchKey::CUDA, DispatchKey::ADInplaceOrView, DispatchKey::AutogradCUDA, DispatchKey::AutocastCUDA});
  if (!t.defined() || !within(t.key_set(), usual) || !t.is_cuda()) return nullptr;
  if (t.scalar_type() != type || t.dim() != ndim || t.stride(ndim - 1) != 1) return nullptr;
  return &t;
}

// What reads through strides without a copy: the general way's rule.
bool kernel_ready(const at::Tensor& t) {
  if (t.is_contiguous()) return true;
  if (reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) return false;
  for (int64_t i = 0; i + 1 < t.dim(); ++i)
    if (t.stride(i) % 8 != 0 || (t.stride(i) <= 0 && t.size(i) != 1)) return false;
  return true;
}

bool tracked(const at::Tensor& t) {
  if (t.unsafeGetTensorImpl()->autograd_meta() == nullptr) return false;
  return (c10::GradMode::is_enabled() && t.requires_grad()) || t._fw_grad(/*level=*/0).defined();
}

bool supported_head_dim(int64_t d) { return d == 32 || d == 64 || d == 96 || d == 128 || d == 256; }

// None: 1 / sqrt(d).  Anything but a float is the general way's to convert.
bool scale_of(PyObject* obj, int64_t d, float& scale) {
  if (obj == Py_None) scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(d)));
  else if (PyFloat_CheckExact(obj)) scale = static_cast<float>(PyFloat_AS_DOUBLE(obj));
  else return false;
  return true;
}

// One of two layout names: 0, 1, or -1.
int layout_of(PyObject* obj, const char* first, const char* second) {
  if (!PyUnicode_CheckExact(obj)) return -1;
  if (PyUnicode_CompareWithASCIIString(obj, first) == 0) return 0;
  return PyUnicode_CompareWithASCIIString(obj, second) == 0 ? 1 : -1;
}

fal_strides strides3(const at::Tensor& t) { return {t.stride(0), t.stride(1), t.stride(2)}; }

bool fits_int(std::initializer_list<int64_t> sizes) {
  for (int64_t s : sizes)
    if (s <= 0 || s > INT32_MAX) return false;
  return true;
}

// forward(q, k, v, softmax_scale, is_causal, out_layout) -> o, or None
PyObject* calls_forward(PyObject* self_obj, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Calls* self = reinterpret_cast<Calls*>(self_obj);
  if (nargs != 6 || !PyBool_Check(args[4])) Py_RETURN_NONE;
  if (!THPVariable_CheckExact(args[0]) || (c10::GradMode::is_enabled() && THPVariable_Unpack(args[0]).requires_grad()))
    Py_RETURN_NONE;  // (a training step is sent on at once)
  if (!ordinary_call()) Py_RETURN_NONE;
  const at::Tensor* in[3];
  for (int i = 0; i < 3; ++i) {
    in[i] = plain(args[i], at::kHalf, 4);
    if (in[i] == nullptr || !kernel_ready(*in[i]) || tracked(*in[i])) Py_RETURN_NONE;
  }
  const at::Tensor &q = *in[0], &k = *in[1], &v = *in[2];
  const int64_t b = q.size(0), h = q.size(1), n = q.size(2), d = q.size(3), hk = k.size(1);
  const int layout = layout_of(args[5], "bhnd", "bnhd");
  fal_fwd_args a{};
  if (layout < 0 || !supported_head_dim(d) || !fits_int({b, h, n, hk}) || h % hk != 0 || !scale_of(args[3], d, a.softmax_scale) ||
      k.size(0) != b || k.size(2) != n || k.size(3) != d || k.sizes() != v.sizes())
    Py_RETURN_NONE;
  const auto dev = q.get_device();
  if (k.get_device() != dev || v.get_device() != dev || dev >= kMaxDevices || self->status[dev] == nullptr ||
      c10::cuda::current_device() != dev)
    Py_RETURN_NONE;
  a.status = self->status[dev];
  at::Tensor o;
  int rc;
  {
    pybind11::gil_scoped_release no_gil;
    o = layout == 0 ? at::empty({b, h, n, d}, q.options()) : at::empty_strided({b, h, n, d}, {n * h * d, d, h * d, 1}, q.options());
    const at::Tensor lse = at::empty({b, h, n}, q.options().dtype(at::kFloat));
    a.q = q.const_data_ptr();
    a.k = k.const_data_ptr();
    a.v = v.const_data_ptr();
    a.o = o.data_ptr();
    a.lse = lse.mutable_data_ptr<float>();
    a.batch = static_cast<int>(b);
    a.heads_q = static_cast<int>(h);
    a.heads_kv = static_cast<int>(hk);
    a.seqlen_q = a.seqlen_k = static_cast<int>(n);
    a.head_dim = static_cast<int>(d);
    a.q_strides = strides3(q);
    a.k_strides = strides3(k);
    a.v_strides = strides3(v);
    a.o_strides = strides3(o);
    a.is_causal = args[4] == Py_True ? 1 : 0;
    a.stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    rc = self->fwd_run(&a);
  }
  if (rc != 0) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// decode(q, k_cache, v_cache, k, v, cache_seqlens, softmax_scale, cache_layout) -> out [B,1,Hq,d], or None
PyObject* calls_decode(PyObject* self_obj, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Calls* self = reinterpret_cast<Calls*>(self_obj);
  if (nargs != 8) Py_RETURN_NONE;
  const at::Tensor* q = plain(args[0], at::kHalf, 4);
  if (q == nullptr || q->size(1) != 1 || !ordinary_call()) Py_RETURN_NONE;  // (a chunk is sent on at once)
  const at::Tensor* kc = plain(args[1], at::kHalf, 4);
  const at::Tensor* vc = plain(args[2], at::kHalf, 4);
  const at::Tensor* lens = plain(args[5], at::kInt, 1);
  if (!kc || !vc || !lens || !q->is_contiguous() || kc->sizes() != vc->sizes()) Py_RETURN_NONE;
  const int layout = layout_of(args[7], "bshd", "bhsd");
  const int64_t b = q->size(0), h = q->size(2), d = q->size(3);
  fal_decode_args a{};
  if (layout < 0 || !supported_head_dim(d) || !scale_of(args[6], d, a.softmax_scale) || kc->size(0) != b || kc->size(3) != d ||
      lens->size(0) != b)
    Py_RETURN_NONE;
  const int seq = layout == 0 ? 1 : 2, head = 3 - seq;
  const int64_t cap = kc->size(seq), hk = kc->size(head);
  if (!fits_int({b, h, cap, hk}) || h % hk != 0) Py_RETURN_NONE;
  const at::Tensor *k = nullptr, *v = nullptr;
  if (args[3] != Py_None || args[4] != Py_None) {
    k = plain(args[3], at::kHalf, 4);
    v = plain(args[4], at::kHalf, 4);
    if (!k || !v || !k->is_contiguous() || !v->is_contiguous() || k->sizes() != v->sizes() || k->size(0) != b ||
        k->size(1) != 1 || k->size(2) != hk || k->size(3) != d)
      Py_RETURN_NONE;
  }
  const auto dev = q->get_device();
  for (const at::Tensor* t : {kc, vc, lens, k, v})
    if (t != nullptr && t->get_device() != dev) Py_RETURN_NONE;
  if (dev >= kMaxDevices || self->status[dev] == nullptr || c10::cuda::current_device() != dev) Py_RETURN_NONE;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  size_t bytes = self->decode_workspace_bytes(static_cast<int>(b), static_cast<int>(h), static_cast<int>(cap), static_cast<int>(d));
  if (bytes < self->workspace_min) bytes = self->workspace_min;
  THPObjectPtr key(Py_BuildValue("(iK)", static_cast<int>(dev), static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream))));
  if (!key) return nullptr;
  PyObject* ws_obj = PyDict_GetItemWithError(self->workspaces, key.get());  // (borrowed)
  if (ws_obj == nullptr || !THPVariable_Check(ws_obj)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const at::Tensor ws = THPVariable_Unpack(ws_obj);  // (kept alive while it is in use)
  if (static_cast<size_t>(ws.numel()) < bytes) Py_RETURN_NONE;
  a.status = self->status[dev];
  at::Tensor o;
  int rc;
  {
    pybind11::gil_scoped_release no_gil;
    o = at::empty({b, 1, h, d}, q->options());
    a.q = q->const_data_ptr();
    a.k_cache = kc->data_ptr();
    a.v_cache = vc->data_ptr();
    a.cache_seqlens = lens->const_data_ptr<int32_t>();
    a.k_new = k != nullptr ? k->const_data_ptr() : nullptr;
    a.v_new = v != nullptr ? v->const_data_ptr() : nullptr;
    a.o = o.data_ptr();
    a.batch = static_cast<int>(b);
    a.heads_q = static_cast<int>(h);
    a.heads_kv = static_cast<int>(hk);
    a.capacity = static_cast<int>(cap);
    a.head_dim = static_cast<int>(d);
    a.k_strides = {kc->stride(0), kc->stride(head), kc->stride(seq)};
    a.v_strides = {vc->stride(0), vc->stride(head), vc->stride(seq)};
    a.workspace = ws.data_ptr();
    a.workspace_bytes = bytes;
    a.stream = stream;
    rc = self->decode_run(&a);
  }
  if (rc != 0) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// set_status(device index, address of its status word)
PyObject* calls_set_status(PyObject* self_obj, PyObject* const* args, Py_ssize_t nargs) {
  const long dev = nargs == 2 ? PyLong_AsLong(args[0]) : -1;
  const unsigned long long ptr = nargs == 2 ? PyLong_AsUnsignedLongLong(args[1]) : 0;
  if (PyErr_Occurred()) return nullptr;
  if (dev >= 0 && dev < kMaxDevices) reinterpret_cast<Calls*>(self_obj)->status[dev] = reinterpret_cast<int*>(ptr);
  Py_RETURN_NONE;
}

// Calls(address of fal_fwd_args_run, of fal_decode_args_run, of fal_decode_workspace_bytes, workspaces, least bytes)
PyObject* calls_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long fwd, dec, bytes_fn, least;
  PyObject* workspaces;
  if (!PyArg_ParseTuple(args, "KKKO!K", &fwd, &dec, &bytes_fn, &PyDict_Type, &workspaces, &least)) return nullptr;
  Calls* self = reinterpret_cast<Calls*>(type->tp_alloc(type, 0));  // (zeroed)
  if (self == nullptr) return nullptr;
  self->fwd_run = reinterpret_cast<decltype(self->fwd_run)>(fwd);
  self->decode_run = reinterpret_cast<decltype(self->decode_run)>(dec);
  self->decode_workspace_bytes = reinterpret_cast<decltype(self->decode_workspace_bytes)>(bytes_fn);
  self->workspaces = Py_NewRef(workspaces);
  self->workspace_min = least;
  return reinterpret_cast<PyObject*>(self);
}

void calls_dealloc(PyObject* self_obj) {
  Py_XDECREF(reinterpret_cast<Calls*>(self_obj)->workspaces);
  Py_TYPE(self_obj)->tp_free(self_obj);
}

template <class F>
PyCFunction fastcall(F f) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

PyMethodDef calls_methods[] = {
    {"forward", fastcall(calls_forward), METH_FASTCALL, "flash_attention without gradients, or None"},
    {"decode", fastcall(calls_decode), METH_FASTCALL, "one decode step, or None"},
    {"set_status", fastcall(calls_set_status), METH_FASTCALL, "address of a device's status word"},
    {nullptr, nullptr, 0, nullptr}};

PyTypeObject calls_type = {PyVarObject_HEAD_INIT(nullptr, 0)};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_fal_host", "Native host path of flash_attn_legacy.", -1, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fal_host() {
  calls_type.tp_name = "_fal_host.Calls";
  calls_type.tp_basicsize = sizeof(Calls);
  calls_type.tp_flags = Py_TPFLAGS_DEFAULT;
  calls_type.tp_new = calls_new;
  calls_type.tp_dealloc = calls_dealloc;
  calls_type.tp_methods = calls_methods;
  if (PyType_Ready(&calls_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module_def);
  if (m == nullptr) return nullptr;
  // sizes of the argument blocks it was compiled with
  if (PyModule_AddObjectRef(m, "Calls", reinterpret_cast<PyObject*>(&calls_type)) < 0 ||
      PyModule_AddIntConstant(m, "FWD_ARGS_BYTES", sizeof(fal_fwd_args)) < 0 ||
      PyModule_AddIntConstant(m, "DECODE_ARGS_BYTES", sizeof(fal_decode_args)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
