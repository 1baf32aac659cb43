// The torch-facing calls of ops.py and quantized.py in the form that programs make in earnest: plain, contiguous CUDA
// tensors of the right types and shapes, all on the current device.  Each function checks its arguments, allocates the result, hands raw pointers and
// the current stream to libqmm.so and returns the result.  What it does not recognise it declines (returns None): the Python
// code behind it then takes the call, with its conversions and its error messages.  A status other than QMM_OK comes back as
// an int.
//
// A call from Python took 6 us of checks, allocation and ctypes in front of a launch of 3 to 5 us, about as long as the
// kernels of a decode-sized matmul; here it takes about 1.5 us.
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/autograd/python_variable.h>

#include <initializer_list>

#include "../../include/qmm.h"

namespace {

decltype(&qmm_w8a32_perchannel) p_w8a32;
decltype(&qmm_w8a16_perchannel) p_w8a16;
decltype(&qmm_i8i8_i32) p_i8i8;
decltype(&qmm_w4a16_g128_workspace_bytes) p_w4_workspace;
decltype(&qmm_w4a16_g128) p_w4a16;
decltype(&qmm_mx_matmul) p_mx;
decltype(&qmm_affine_matmul) p_affine;
bool bound = false;

// The tensor behind `o` if it is one that a kernel may be pointed at: no subclass, no transform's wrapper, dense and contiguous.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  static const c10::DispatchKeySet special({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                            c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize,
                                            c10::DispatchKey::ZeroTensor, c10::DispatchKey::Conjugate,
                                            c10::DispatchKey::Negative});
  if (!t.defined() || !t.is_cuda() || t.layout() != c10::kStrided || t.key_set().has_any(special) || !t.is_contiguous()) return nullptr;
  return &t;
}
// Whether all of them are CUDA device number `current`: the library works with the current device's stream, SMs and status word,
// and another device's memory is nothing that it may be pointed at.
bool all_on(const c10::Device* devices, size_t n, c10::DeviceIndex current) {
  for (size_t i = 0; i < n; ++i)
    if (!devices[i].is_cuda() || devices[i].index() != current) return false;
  return true;
}
constexpr size_t kMaxOperands = 4;
// The tensors behind a[0 .. n), if a kernel may be pointed at all of them.
bool operands(PyObject* const* a, size_t n, const at::Tensor** t) {
  c10::Device devices[kMaxOperands] = {c10::kCPU, c10::kCPU, c10::kCPU, c10::kCPU};
  for (size_t i = 0; i < n; ++i) {
    if (!(t[i] = plain(a[i]))) return false;
    devices[i] = t[i]->device();
  }
  return all_on(devices, n, c10::cuda::current_device());
}
bool is(const at::Tensor* t, c10::ScalarType type, std::initializer_list<int64_t> shape) {
  return t->scalar_type() == type && t->sizes() == c10::IntArrayRef(shape);
}
// No mode is to see the allocation (it would be Python's call otherwise), and the library is there.
bool ready() {
  return bound && !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled();
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
at::Tensor result(const at::Tensor& x, int64_t n, c10::ScalarType type) {
  c10::SmallVector<int64_t, 5> sizes(x.sizes().begin(), x.sizes().end());
  sizes.back() = n;
  return at::empty(sizes, x.options().dtype(type).requires_grad(false));
}
template <typename Fn>
int without_gil(Fn fn) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = fn();
  Py_END_ALLOW_THREADS
  return rc;
}
PyObject* finish(int rc, const at::Tensor& y) { return rc != QMM_OK ? PyLong_FromLong(rc) : THPVariable_Wrap(y); }

// A C++ exception (the allocator's, say) becomes Python's.
template <typename Fn>
PyObject* guarded(Fn fn) {
  HANDLE_TH_ERRORS
  return fn();
  END_HANDLE_TH_ERRORS
}

PyObject* w8a32(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 3 || !ready()) Py_RETURN_NONE;
    const at::Tensor* t[3];
    if (!operands(a, 3, t)) Py_RETURN_NONE;
    const at::Tensor *x = t[0], *w = t[1], *s = t[2];
    if (x->scalar_type() != c10::kFloat || x->dim() < 1 || w->dim() != 2 || x->numel() == 0) Py_RETURN_NONE;
    const int64_t K = x->size(-1), N = w->size(1), M = x->numel() / K;
    if (!is(w, c10::kChar, {K, N}) || !is(s, c10::kFloat, {N})) Py_RETURN_NONE;
    at::Tensor y = result(*x, N, c10::kFloat);
    void* st = stream();
    return finish(without_gil([&] {
      return p_w8a32(x->const_data_ptr<float>(), w->const_data_ptr<int8_t>(), s->const_data_ptr<float>(), y.mutable_data_ptr<float>(), M, N, K, st);
    }), y);
  });
}

PyObject* w8a16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 3 || !ready()) Py_RETURN_NONE;
    const at::Tensor* t[3];
    if (!operands(a, 3, t)) Py_RETURN_NONE;
    const at::Tensor *x = t[0], *w = t[1], *s = t[2];
    if (x->scalar_type() != c10::kBFloat16 || x->dim() != 2 || w->dim() != 2) Py_RETURN_NONE;
    const int64_t M = x->size(0), K = x->size(1), N = w->size(1);
    if (!is(w, c10::kChar, {K, N}) || !is(s, c10::kFloat, {N})) Py_RETURN_NONE;
    at::Tensor y = result(*x, N, c10::kBFloat16);
    void* st = stream();
    return finish(without_gil([&] {
      return p_w8a16(static_cast<const uint16_t*>(x->const_data_ptr()), w->const_data_ptr<int8_t>(), s->const_data_ptr<float>(),
                     static_cast<uint16_t*>(y.mutable_data_ptr()), M, N, K, N, st);
    }), y);
  });
}

// (a, b, row_scale or None, col_scale or None, want_acc) -> (acc or None, out or None)
PyObject* i8_dot(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 5 || !ready()) Py_RETURN_NONE;
    const bool rescale = a[2] != Py_None, want = a[4] == Py_True;
    if ((a[3] != Py_None) != rescale || (!want && a[4] != Py_False) || (!rescale && !want)) Py_RETURN_NONE;
    const at::Tensor* t[4];
    if (!operands(a, rescale ? 4 : 2, t)) Py_RETURN_NONE;
    const at::Tensor *x = t[0], *w = t[1];
    if (x->dim() != 2 || w->dim() != 2) Py_RETURN_NONE;
    const c10::ScalarType tx = x->scalar_type(), tw = w->scalar_type();
    const int64_t M = x->size(0), K = x->size(1), N = w->size(1);
    if ((tx != c10::kChar && tx != c10::kByte) || (tw != c10::kChar && tw != c10::kByte) || w->size(0) != K) Py_RETURN_NONE;
    const float *row = nullptr, *col = nullptr;
    if (rescale) {
      if (!is(t[2], c10::kFloat, {M}) || !is(t[3], c10::kFloat, {N})) Py_RETURN_NONE;
      row = t[2]->const_data_ptr<float>();
      col = t[3]->const_data_ptr<float>();
    }
    at::Tensor acc, out;
    if (want) acc = result(*x, N, c10::kInt);
    if (rescale) out = result(*x, N, c10::kFloat);
    void* st = stream();
    const int rc = without_gil([&] {
      return p_i8i8(x->const_data_ptr(), w->const_data_ptr(), want ? acc.mutable_data_ptr<int32_t>() : nullptr, row, col,
                    rescale ? out.mutable_data_ptr<float>() : nullptr, M, N, K, tx == c10::kByte, tw == c10::kByte, st);
    });
    if (rc != QMM_OK) return PyLong_FromLong(rc);
    PyObject* pair = PyTuple_New(2);
    if (!pair) return nullptr;
    auto item = [](const at::Tensor& t) { return t.defined() ? THPVariable_Wrap(t) : (Py_INCREF(Py_None), Py_None); };
    PyTuple_SET_ITEM(pair, 0, item(acc));
    PyTuple_SET_ITEM(pair, 1, item(out));
    return pair;
  });
}

// (x, wq, scales, zeros, zeros_packed, group, static_weights, {(device index, stream): object whose .buf is the
// stream's workspace})
PyObject* w4a16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 8 || !ready() || !PyLong_CheckExact(a[5]) || !PyDict_CheckExact(a[7])) Py_RETURN_NONE;
    if ((a[4] != Py_True && a[4] != Py_False) || (a[6] != Py_True && a[6] != Py_False)) Py_RETURN_NONE;
    const bool packed = a[4] == Py_True;
    const at::Tensor* op[4];
    if (!operands(a, 4, op)) Py_RETURN_NONE;
    const at::Tensor *x = op[0], *w = op[1], *s = op[2], *z = op[3];
    if (x->scalar_type() != c10::kBFloat16 || x->dim() != 2 || w->dim() != 2) Py_RETURN_NONE;
    const long long group = PyLong_AsLongLong(a[5]);
    const int64_t M = x->size(0), K = x->size(1), N = w->size(1);
    if (group <= 0 || K % group != 0 || K % 2 != 0) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    const int64_t G = K / group;
    if (!is(w, c10::kByte, {K / 2, N}) || !is(s, c10::kBFloat16, {G, N}) || !is(z, c10::kByte, {G, packed ? N / 2 : N})) Py_RETURN_NONE;
    const size_t need = p_w4_workspace(M, N, K);
    at::Tensor ws;
    if (need > 0) {   // the stream's workspace, if it is there and large enough; a captured call has its own
      if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) Py_RETURN_NONE;
      PyObject* key = Py_BuildValue("(iK)", static_cast<int>(x->device().index()),
                                    static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream())));
      PyObject* holder = key ? PyDict_GetItemWithError(a[7], key) : nullptr;   // borrowed
      Py_XDECREF(key);
      if (!holder) {
        if (PyErr_Occurred()) return nullptr;
        Py_RETURN_NONE;
      }
      PyObject* buf = PyObject_GetAttrString(holder, "buf");
      if (!buf) return nullptr;
      const at::Tensor* t = plain(buf);
      if (t) ws = *t;
      Py_DECREF(buf);
      if (!t || t->device() != x->device() || t->scalar_type() != c10::kByte || static_cast<size_t>(ws.numel()) < need) Py_RETURN_NONE;
    }
    at::Tensor y = result(*x, N, c10::kBFloat16);
    void* st = stream();
    return finish(without_gil([&] {
      return p_w4a16(static_cast<const uint16_t*>(x->const_data_ptr()), w->const_data_ptr<uint8_t>(),
                     static_cast<const uint16_t*>(s->const_data_ptr()), z->const_data_ptr<uint8_t>(), packed,
                     static_cast<uint16_t*>(y.mutable_data_ptr()), M, N, K, group, ws.defined() ? ws.mutable_data_ptr() : nullptr,
                     ws.defined() ? static_cast<size_t>(ws.numel()) : 0, a[6] == Py_True ? QMM_W4_STATIC_WEIGHTS : 0, st);
    }), y);
  });
}

// Activations of the operator API: f16 or f32, [..., K].
bool activations(const at::Tensor* x, int64_t K, int* dtype) {
  if (x->dim() < 1 || x->numel() == 0 || x->size(-1) != K) return false;
  *dtype = x->scalar_type() == c10::kFloat ? QMM_F32 : QMM_F16;
  return x->scalar_type() == c10::kFloat || x->scalar_type() == c10::kHalf;
}
bool integers(PyObject* const* a, int from, int to, long long* v) {
  for (int i = from; i < to; ++i) {
    if (!PyLong_CheckExact(a[i])) return false;
    int overflow = 0;
    *v = PyLong_AsLongLongAndOverflow(a[i], &overflow);
    if (overflow != 0 || *v <= 0) return false;
    ++v;
  }
  return true;
}

// (x, packed, scales, bits per element, group, mode + 1, K)
PyObject* mx_matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    long long v[4];   // bits, group, mode + 1, K
    if (n != 7 || !ready() || !integers(a, 3, 7, v) || v[3] % v[1] != 0) Py_RETURN_NONE;
    const at::Tensor* t[3];
    if (!operands(a, 3, t)) Py_RETURN_NONE;
    const at::Tensor *x = t[0], *w = t[1], *s = t[2];
    const int64_t K = v[3];
    int dtype;
    if (!activations(x, K, &dtype) || w->dim() != 2) Py_RETURN_NONE;
    const int64_t N = w->size(0), M = x->numel() / K;
    if (!is(w, c10::kByte, {N, v[0] == 4 ? K / 2 : K}) || !is(s, c10::kByte, {N, K / v[1]})) Py_RETURN_NONE;
    at::Tensor y = result(*x, N, x->scalar_type());
    void* st = stream();
    return finish(without_gil([&] {
      return p_mx(x->const_data_ptr(), w->const_data_ptr<uint8_t>(), s->const_data_ptr<uint8_t>(), y.mutable_data_ptr(), M, N, K,
                  static_cast<int>(v[2] - 1), dtype, st);
    }), y);
  });
}

// (x, packed, scales, biases, bits, group, K)
PyObject* affine_matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    long long v[3];   // bits, group, K
    if (n != 7 || !ready() || !integers(a, 4, 7, v) || (v[0] != 4 && v[0] != 8) || v[2] % v[1] != 0) Py_RETURN_NONE;
    const at::Tensor* t[4];
    if (!operands(a, 4, t)) Py_RETURN_NONE;
    const at::Tensor *x = t[0], *w = t[1], *s = t[2], *b = t[3];
    const int64_t K = v[2];
    int dtype;
    if (!activations(x, K, &dtype) || w->dim() != 2) Py_RETURN_NONE;
    const int64_t N = w->size(0), M = x->numel() / K, G = K / v[1];
    if (!(v[0] == 4 ? is(w, c10::kInt, {N, K / 8}) : is(w, c10::kByte, {N, K})) || !is(s, c10::kFloat, {N, G}) || !is(b, c10::kFloat, {N, G}))
      Py_RETURN_NONE;
    at::Tensor y = result(*x, N, x->scalar_type());
    void* st = stream();
    return finish(without_gil([&] {
      return p_affine(x->const_data_ptr(), w->const_data_ptr(), s->const_data_ptr<float>(), b->const_data_ptr<float>(),
                      y.mutable_data_ptr(), M, N, K, static_cast<int>(v[0]), v[1], dtype, st);
    }), y);
  });
}

// one_device(number of the current device, torch.device, ...): what every call above asks of its operands
PyObject* one_device(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    c10::Device devices[kMaxOperands] = {c10::kCPU, c10::kCPU, c10::kCPU, c10::kCPU};
    if (n < 1 || n > static_cast<Py_ssize_t>(kMaxOperands) + 1) {
      PyErr_SetString(PyExc_TypeError, "one_device() takes a number and up to four devices");
      return nullptr;
    }
    const long current = PyLong_AsLong(a[0]);
    if (current == -1 && PyErr_Occurred()) return nullptr;
    for (Py_ssize_t i = 1; i < n; ++i) {
      if (!THPDevice_Check(a[i])) {
        PyErr_SetString(PyExc_TypeError, "one_device() takes devices");
        return nullptr;
      }
      devices[i - 1] = reinterpret_cast<THPDevice*>(a[i])->device;
    }
    return PyBool_FromLong(all_on(devices, static_cast<size_t>(n - 1), static_cast<c10::DeviceIndex>(current)));
  });
}

// bind(address of qmm_w8a32_perchannel, ...): the entry points of the library that the process has loaded, in the order of kNames
constexpr const char* kNames = "qmm_w8a32_perchannel qmm_w8a16_perchannel qmm_i8i8_i32 qmm_w4a16_g128_workspace_bytes "
                               "qmm_w4a16_g128 qmm_mx_matmul qmm_affine_matmul";
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  void* p[7];
  if (n != 7) {
    PyErr_SetString(PyExc_TypeError, "bind() takes seven addresses");
    return nullptr;
  }
  for (int i = 0; i < 7; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (!p[i]) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind(): null address");
      return nullptr;
    }
  }
  p_w8a32 = reinterpret_cast<decltype(p_w8a32)>(p[0]);
  p_w8a16 = reinterpret_cast<decltype(p_w8a16)>(p[1]);
  p_i8i8 = reinterpret_cast<decltype(p_i8i8)>(p[2]);
  p_w4_workspace = reinterpret_cast<decltype(p_w4_workspace)>(p[3]);
  p_w4a16 = reinterpret_cast<decltype(p_w4a16)>(p[4]);
  p_mx = reinterpret_cast<decltype(p_mx)>(p[5]);
  p_affine = reinterpret_cast<decltype(p_affine)>(p[6]);
  bound = true;
  Py_RETURN_NONE;
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(bind), METHOD(w8a32), METHOD(w8a16), METHOD(i8_dot), METHOD(w4a16), METHOD(mx_matmul),
                         METHOD(affine_matmul), METHOD(one_device), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
  PyObject* m = PyModule_Create(&module);
  // the torch whose headers this was compiled with; another one lays its classes out as it likes
  if (m && (PyModule_AddStringConstant(m, "ENTRY_POINTS", kNames) != 0 || PyModule_AddStringConstant(m, "TORCH", QMM_TORCH_VERSION) != 0))
    Py_CLEAR(m);
  return m;
}
