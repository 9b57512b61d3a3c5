// Direct entry points: the attention ops called from Python without torch's dispatcher.
//
// A decode-sized call is a few microseconds of GPU time, and the way through the dispatcher (argument boxing, a heap
// handle per tensor, a shim call per size or stride) cost more than that.  These functions take the Python objects, read
// the tensors in place and call the same checks and the same C entry point (attn_ops.h).  They serve the ordinary case
// only - plain CUDA tensors on the current device, no autograd, no mode, tracer, functional transform or profiler that
// wants to see the op - and answer False to everything else, a failed check included: the caller then goes through the
// dispatcher, whose behaviour and error messages are therefore the ones that count.
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/grad_mode.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <array>

#include "attn_ops.h"
#include "buffers.h"

namespace minfer {
namespace {

struct DirectEnv {
  using Tensor = at::Tensor;
  static int device_of(const Tensor& t) { return t.get_device(); }
  static void* stream(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
  static int32_t* status(const Tensor& like) {
    thread_local std::array<int32_t*, 64> known{};
    const int dev = like.get_device();
    if (dev >= 64) return binding_status(const_cast<Tensor*>(&like));
    if (known[dev] == nullptr) known[dev] = binding_status(const_cast<Tensor*>(&like));
    return known[dev];
  }
  static Scratch scratch(const Tensor& like, void* stream, int64_t purpose, size_t want, size_t least) {
    // the latest buffer of each purpose: buffers are kept for the life of the process, so a remembered one stays valid
    struct Entry { int dev; void* stream; Scratch s; };
    thread_local std::array<Entry, 2> last{Entry{-1, nullptr, {}}, Entry{-1, nullptr, {}}};
    Entry& e = last[purpose & 1];
    if (e.dev != like.get_device() || e.stream != stream || e.s.bytes < want)
      e = Entry{like.get_device(), stream, binding_scratch(const_cast<Tensor*>(&like), stream, purpose, want, least)};
    return e.s;
  }
  static int max_ctas() { return binding_max_ctas(); }
  template <class P>
  static int call(int (*fn)(const P*, void*), const P* p, void* stream) {
    // a launch waits while the stream's queue is full: other Python threads run meanwhile
    PyThreadState* s = PyEval_SaveThread();
    const int rc = fn(p, stream);
    PyEval_RestoreThread(s);
    return rc;
  }
};
using Ops = AttnOps<DirectEnv>;

// Nothing on this thread asks to see the call.
bool thread_is_plain() {
  static const c10::DispatchKeySet usual({c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView});
  return (c10::impl::tls_local_dispatch_key_set().included_ - usual).empty() && !at::impl::torch_function_mode_enabled() &&
         !at::hasCallbacks();
}

// The object as a plain CUDA tensor of device `dev` (-1: takes the tensor's), or null.
at::Tensor* plain_tensor(PyObject* o, int& dev) {
  // (every CUDA tensor carries the autocast key; these ops have no autocast rule, so the dispatcher passes it by as well)
  static const c10::DispatchKeySet usual({c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutogradCUDA,
                                          c10::DispatchKey::AutocastCUDA});
  static const c10::DispatchKeySet inference({c10::DispatchKey::CUDA, c10::DispatchKey::AutocastCUDA});
  if (!THPVariable_CheckExact(o)) return nullptr;
  at::Tensor& t = const_cast<at::Tensor&>(THPVariable_Unpack(o));
  if (!(t.key_set() == usual || t.key_set() == inference)) return nullptr;
  if (dev < 0) dev = t.get_device();
  if (t.get_device() != dev || (t.requires_grad() && at::GradMode::is_enabled())) return nullptr;
  return &t;
}

// N tensors starting at args[first], all plain and on the current device.
template <size_t N>
bool plain_tensors(PyObject* const* args, size_t first, std::array<at::Tensor*, N>& t) {
  int dev = -1;
  for (size_t i = 0; i < N; ++i)
    if ((t[i] = plain_tensor(args[first + i], dev)) == nullptr) return false;
  return dev == c10::cuda::current_device();
}

bool as_int(PyObject* o, int64_t& v) {
  if (!PyLong_Check(o)) return false;
  v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

bool as_double(PyObject* o, double& v) {
  if (!PyFloat_Check(o)) return false;
  v = PyFloat_AS_DOUBLE(o);
  return true;
}

template <class F>
PyObject* attempt(bool ready, F&& f) {
  if (!ready) Py_RETURN_FALSE;
  try {
    f();
  } catch (const std::exception&) {
    Py_RETURN_FALSE;  // the dispatcher's turn: it checks again and raises
  }
  Py_RETURN_TRUE;
}

PyObject* flash_attn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  std::array<at::Tensor*, 5> t;
  int64_t q0, q1, q2;
  const bool ready = n == 8 && thread_is_plain() && as_int(a[0], q0) && as_int(a[1], q1) && as_int(a[2], q2) && plain_tensors(a, 3, t);
  return attempt(ready, [&] { Ops::flash_attn(q0, q1, q2, *t[0], *t[1], *t[2], *t[3], *t[4]); });
}

PyObject* flash_attn_causal(PyObject*, PyObject* const* a, Py_ssize_t n) {
  std::array<at::Tensor*, 4> t;
  const bool ready = n == 4 && thread_is_plain() && plain_tensors(a, 0, t);
  return attempt(ready, [&] { Ops::flash_attn_causal(*t[0], *t[1], *t[2], *t[3]); });
}

PyObject* flash_attn_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  std::array<at::Tensor*, 5> t;
  const bool ready = n == 5 && thread_is_plain() && plain_tensors(a, 0, t);
  return attempt(ready, [&] { Ops::flash_attn_decode(*t[0], *t[1], *t[2], *t[3], *t[4]); });
}

PyObject* flash_attn_decode_q8(PyObject*, PyObject* const* a, Py_ssize_t n) {
  std::array<at::Tensor*, 5> t;
  const bool ready = n == 5 && thread_is_plain() && plain_tensors(a, 0, t);
  return attempt(ready, [&] { Ops::flash_attn_decode_q8(*t[0], *t[1], *t[2], *t[3], *t[4]); });
}

PyObject* flash_attn_decode_paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
  std::array<at::Tensor*, 6> t;
  const bool ready = n == 6 && thread_is_plain() && plain_tensors(a, 0, t);
  return attempt(ready, [&] { Ops::flash_attn_decode_paged(*t[0], *t[1], *t[2], *t[3], *t[4], *t[5]); });
}

PyObject* rope(PyObject* const* a, Py_ssize_t n, void (*op)(int64_t, int64_t, double, at::Tensor&)) {
  std::array<at::Tensor*, 1> t;
  int64_t rot, start;
  double base;
  const bool ready = n == 4 && thread_is_plain() && as_int(a[0], rot) && as_int(a[1], start) && as_double(a[2], base) && plain_tensors(a, 3, t);
  return attempt(ready, [&] { op(rot, start, base, *t[0]); });
}
PyObject* il_rope(PyObject*, PyObject* const* a, Py_ssize_t n) { return rope(a, n, &Ops::il_rope); }
PyObject* neox_rope(PyObject*, PyObject* const* a, Py_ssize_t n) { return rope(a, n, &Ops::neox_rope); }

template <bool Q8>
PyObject* rope_kv_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  std::array<at::Tensor*, 6> t;
  int64_t rot, style;
  double base;
  const bool ready = n == 9 && thread_is_plain() && as_int(a[0], rot) && as_double(a[1], base) && as_int(a[2], style) && plain_tensors(a, 3, t);
  return attempt(ready, [&] { Ops::rope_append(rot, base, style, *t[0], *t[1], *t[2], *t[3], *t[4], nullptr, *t[5], Q8); });
}

PyObject* rope_kv_append_paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
  std::array<at::Tensor*, 7> t;
  int64_t rot, style;
  double base;
  const bool ready = n == 10 && thread_is_plain() && as_int(a[0], rot) && as_double(a[1], base) && as_int(a[2], style) && plain_tensors(a, 3, t);
  return attempt(ready, [&] { Ops::rope_kv_append_paged(rot, base, style, *t[0], *t[1], *t[2], *t[3], *t[4], *t[5], *t[6]); });
}

#define MINFER_DIRECT(name, fn) \
  { name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr }
PyMethodDef methods[] = {
    MINFER_DIRECT("flash_attn", &flash_attn),
    MINFER_DIRECT("flash_attn_causal", &flash_attn_causal),
    MINFER_DIRECT("flash_attn_decode", &flash_attn_decode),
    MINFER_DIRECT("flash_attn_decode_q8", &flash_attn_decode_q8),
    MINFER_DIRECT("flash_attn_decode_paged", &flash_attn_decode_paged),
    MINFER_DIRECT("il_rope", &il_rope),
    MINFER_DIRECT("neox_rope", &neox_rope),
    MINFER_DIRECT("rope_kv_append", &rope_kv_append<false>),
    MINFER_DIRECT("rope_kv_append_q8", &rope_kv_append<true>),
    MINFER_DIRECT("rope_kv_append_paged", &rope_kv_append_paged),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_direct", "attention ops without the dispatcher; each returns whether it served the call", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace minfer

// The tensors are read by the layout of the torch that this file was compiled against: ops.py asks which one that was.
PyMODINIT_FUNC PyInit__direct(void) {
  PyObject* m = PyModule_Create(&minfer::module);
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", MINFER_TORCH_VERSION) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
