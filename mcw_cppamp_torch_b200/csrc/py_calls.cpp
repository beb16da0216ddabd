// Calls from Python into libTHC.so without ctypes on the way (module mcw_cppamp_torch_b200._calls).
//
// A ctypes call converts its arguments through per-argument Python-level machinery, and the error check behind it is a
// second foreign call: together about 1.5 us, as much as queueing a small kernel.  Here each C function gets an invoker
// generated from its prototype in THC.h; the function's address and the error accessors come from the library that
// ctypes has loaded, so there is one copy of the library and this file links against nothing.  An argument that an
// invoker does not take (a ctypes array, byref(), a number of the wrong kind) sends the call to the ctypes function
// it stands for, which converts or rejects it as before.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstddef>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

#include "THC.h"

namespace {

const char *(*g_last_error)(void) = nullptr;
void (*g_clear_error)(void) = nullptr;
PyObject *g_error_type = nullptr;
// ctypes types whose instances are one pointer: POINTER(THGPUTensor), POINTER(THGPUStorage)
PyTypeObject *g_tensor_type = nullptr, *g_storage_type = nullptr;

// None, or an instance of exactly this type: a pointer to something else is for ctypes to convert or reject.
bool pointer_of(PyObject *o, PyTypeObject *type, void **out) {
  if (o == Py_None) { *out = nullptr; return true; }
  if (Py_TYPE(o) != type) return false;
  Py_buffer b;
  if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) { PyErr_Clear(); return false; }
  std::memcpy(out, b.buf, sizeof(void *));
  PyBuffer_Release(&b);
  return true;
}

template <class T> bool take(PyObject *o, T &out) {
  typedef typename std::remove_cv<typename std::remove_pointer<T>::type>::type Pointee;
  if constexpr (std::is_same<Pointee, THGPUTensor>::value || std::is_same<Pointee, THGPUStorage>::value) {
    void *p;
    if (!pointer_of(o, std::is_same<Pointee, THGPUTensor>::value ? g_tensor_type : g_storage_type, &p)) return false;
    out = (T)p;
    return true;
  } else if constexpr (std::is_floating_point<T>::value) {
    if (PyFloat_CheckExact(o)) { out = (T)PyFloat_AS_DOUBLE(o); return true; }
    if (!PyLong_Check(o)) return false;
    const double d = PyLong_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    out = (T)d;
    return true;
  } else if constexpr (std::is_same<T, int>::value || std::is_same<T, long>::value) {
    if (!PyLong_Check(o)) return false;
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    out = (T)v;
    return true;
  } else {
    return false;
  }
}

// Turns the library's pending error, if there is one, into a Python exception.
bool raised() {
  const char *e = g_last_error();
  if (!e) return false;
  PyObject *msg = PyUnicode_FromString(e);
  g_clear_error();
  if (msg) { PyErr_SetObject(g_error_type, msg); Py_DECREF(msg); }
  return true;
}

typedef PyObject *(*Invoker)(void *fn, PyObject *const *args, Py_ssize_t n, bool *mismatch);

template <class F> struct Invoke;
template <class R, class... A> struct Invoke<R(A...)> {
  template <std::size_t... I>
  static PyObject *run(void *fn, PyObject *const *args, bool *mismatch, std::index_sequence<I...>) {
    std::tuple<A...> v;
    if (!(true && ... && take(args[I], std::get<I>(v)))) { *mismatch = true; return nullptr; }
    R (*f)(A...) = (R(*)(A...))fn;
    if constexpr (std::is_void<R>::value) {
      Py_BEGIN_ALLOW_THREADS
      f(std::get<I>(v)...);
      Py_END_ALLOW_THREADS
      if (raised()) return nullptr;
      Py_RETURN_NONE;
    } else {
      R r;
      Py_BEGIN_ALLOW_THREADS
      r = f(std::get<I>(v)...);
      Py_END_ALLOW_THREADS
      if (raised()) return nullptr;
      if constexpr (std::is_floating_point<R>::value) return PyFloat_FromDouble((double)r);
      else return PyLong_FromLong((long)r);
    }
  }
  static PyObject *call(void *fn, PyObject *const *args, Py_ssize_t n, bool *mismatch) {
    if (n != (Py_ssize_t)sizeof...(A)) { *mismatch = true; return nullptr; }
    return run(fn, args, mismatch, std::index_sequence_for<A...>());
  }
};

#define UNARY(X) X(log) X(log1p) X(exp) X(cos) X(acos) X(cosh) X(sin) X(asin) X(sinh) X(tan) X(atan) X(tanh) X(sqrt) \
  X(ceil) X(floor) X(abs) X(sign) X(round)
#define COMPARE(X) X(lt) X(gt) X(le) X(ge) X(eq) X(ne)

struct Entry { const char *name; Invoker call; };
#define E(NAME) {#NAME, &Invoke<std::remove_pointer<decltype(&NAME)>::type>::call},
#define EU(NAME) E(THGPUTensor_##NAME)
#define EC(NAME) E(THGPUTensor_##NAME##Value) E(THGPUTensor_##NAME##Tensor)
const Entry kEntries[] = {
  E(THGPUStorage_size) E(THGPUStorage_get) E(THGPUTensor_storageOffset) E(THGPUTensor_nDimension) E(THGPUTensor_size)
  E(THGPUTensor_stride) E(THGPUTensor_resizeAs) E(THGPUTensor_resize1d) E(THGPUTensor_resize2d) E(THGPUTensor_resize3d)
  E(THGPUTensor_resize4d) E(THGPUTensor_resize5d) E(THGPUTensor_set) E(THGPUTensor_isContiguous) E(THGPUTensor_isSameSizeAs)
  E(THGPUTensor_nElement) E(THGPUTensor_get1d) E(THGPUTensor_get2d) E(THGPUTensor_copy) E(THGPUTensor_copyGPU)
  E(THGPUTensor_fill) E(THGPUTensor_zero) E(THGPUTensor_numel) E(THGPUTensor_add) E(THGPUTensor_mul) E(THGPUTensor_div)
  E(THGPUTensor_cadd) E(THGPUTensor_cmul) E(THGPUTensor_cdiv) E(THGPUTensor_dot) E(THGPUTensor_minall) E(THGPUTensor_maxall)
  E(THGPUTensor_sumall) E(THGPUTensor_meanall) E(THGPUTensor_min) E(THGPUTensor_max) E(THGPUTensor_sum) E(THGPUTensor_mean)
  E(THGPUTensor_addmv) E(THGPUTensor_addmm) E(THGPUTensor_addr) E(THGPUTensor_addcmul) E(THGPUTensor_addcdiv)
  E(THGPUTensor_pow) E(THGPUTensor_clamp) E(THGPUTensor_atan2) E(THGPUTensor_varall) E(THGPUTensor_stdall)
  E(THGPUTensor_normall) E(THGPUTensor_dist) E(THGPUTensor_norm) E(THGPUTensor_prodall) E(THGPUTensor_prod)
  E(THGPUTensor_renorm) E(THGPUBlas_setMathMode) E(THGPUBlas_getMathMode) E(THGPUSynchronize) E(THGPUKernelLaunchCount)
  E(THGPUNN_SoftMax_updateOutput) E(THGPUNN_SoftMax_updateGradInput) E(THGPUNN_SpatialAveragePooling_updateOutput)
  E(THGPUNN_SpatialAveragePooling_updateGradInput) E(THGPUNN_SpatialConvolutionMM_updateOutput)
  E(THGPUNN_SpatialConvolutionMM_updateGradInput) E(THGPUNN_SpatialConvolutionMM_accGradParameters)
  E(THGPUNN_SpatialConvolutionMM_backward) E(THGPUNN_SpatialMaxPooling_updateOutput)
  E(THGPUNN_SpatialMaxPooling_updateGradInput) E(THGPUNN_Threshold_updateOutput) E(THGPUNN_Threshold_updateGradInput)
  E(THGPUNN_Threshold_SpatialMaxPooling_updateOutput) E(THGPUNN_Threshold_SpatialMaxPooling_updateGradInput)
  E(THGPUNN_Linear_updateOutput) E(THGPUNN_LogSoftMax_updateOutput) E(THGPUNN_LogSoftMax_updateGradInput) E(THGPUNN_ClassNLLCriterion_updateOutput)
  E(THGPUNN_ClassNLLCriterion_updateGradInput) E(THGPUNN_SGD_update)
  UNARY(EU) COMPARE(EC)
};

// A C function callable from Python.
struct Call {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  Invoker invoke;
  void *fn;
  PyObject *slow;   // the ctypes route
};
PyObject *call_vectorcall(PyObject *self, PyObject *const *args, size_t nargsf, PyObject *kw) {
  Call *c = (Call *)self;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  bool mismatch = kw != nullptr && PyTuple_GET_SIZE(kw) > 0;
  if (!mismatch) {
    PyObject *r = c->invoke(c->fn, args, n, &mismatch);
    if (!mismatch) return r;
  }
  return PyObject_Vectorcall(c->slow, args, nargsf, kw);
}
void call_dealloc(PyObject *self) {
  Py_XDECREF(((Call *)self)->slow);
  Py_TYPE(self)->tp_free(self);
}
PyObject *call_get_slow(PyObject *self, void *) {
  PyObject *s = ((Call *)self)->slow;
  Py_INCREF(s);
  return s;
}
PyGetSetDef call_getset[] = {{"slow", call_get_slow, nullptr, "the ctypes route of this function", nullptr}, {}};
PyTypeObject CallType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// setup(last_error address, clear_error address, error class, tensor pointer type, storage pointer type)
PyObject *setup(PyObject *, PyObject *args) {
  unsigned long long le, ce;
  PyObject *cls, *tensor, *storage;
  if (!PyArg_ParseTuple(args, "KKOO!O!", &le, &ce, &cls, &PyType_Type, &tensor, &PyType_Type, &storage)) return nullptr;
  g_last_error = (const char *(*)(void))le;
  g_clear_error = (void (*)(void))ce;
  Py_INCREF(cls);
  g_error_type = cls;
  Py_INCREF(tensor);
  g_tensor_type = (PyTypeObject *)tensor;
  Py_INCREF(storage);
  g_storage_type = (PyTypeObject *)storage;
  Py_RETURN_NONE;
}
// wrap(name, address, slow) -> callable, or None for a function without an invoker
PyObject *wrap(PyObject *, PyObject *args) {
  const char *name;
  unsigned long long fn;
  PyObject *slow;
  if (!PyArg_ParseTuple(args, "sKO", &name, &fn, &slow)) return nullptr;
  for (const Entry &e : kEntries)
    if (std::strcmp(e.name, name) == 0) {
      Call *c = PyObject_New(Call, &CallType);
      if (!c) return nullptr;
      c->vectorcall = call_vectorcall;
      c->invoke = e.call;
      c->fn = (void *)fn;
      Py_INCREF(slow);
      c->slow = slow;
      return (PyObject *)c;
    }
  Py_RETURN_NONE;
}
// ---- tensor metadata and host arrays, without ctypes structures ----------------------------------------------------
void (*g_set_storage)(THGPUTensor *, THGPUStorage *, long, THLongStorage *, THLongStorage *) = nullptr;
void (*g_copy_float)(THGPUTensor *, THFloatTensor *) = nullptr;
void (*g_float_copy)(THFloatTensor *, THGPUTensor *) = nullptr;
constexpr int kMaxNd = 16;

// functions(setStorage, copyFloat, FloatTensor_copyGPU): addresses
PyObject *functions(PyObject *, PyObject *args) {
  unsigned long long a, b, c;
  if (!PyArg_ParseTuple(args, "KKK", &a, &b, &c)) return nullptr;
  g_set_storage = (decltype(g_set_storage))a;
  g_copy_float = (decltype(g_copy_float))b;
  g_float_copy = (decltype(g_float_copy))c;
  Py_RETURN_NONE;
}
THGPUTensor *tensor_arg(PyObject *o) {
  void *p;
  if (!pointer_of(o, g_tensor_type, &p) || !p) {
    PyErr_SetString(PyExc_TypeError, "pointer to a THGPUTensor expected");
    return nullptr;
  }
  return (THGPUTensor *)p;
}
// sizes(tensor) -> tuple
PyObject *sizes(PyObject *, PyObject *o) {
  THGPUTensor *t = tensor_arg(o);
  if (!t) return nullptr;
  PyObject *r = PyTuple_New(t->nDimension);
  for (int d = 0; r && d < t->nDimension; d++) PyTuple_SET_ITEM(r, d, PyLong_FromLong(t->size[d]));
  return r;
}
// set_view(dst, src, sizes): dst becomes a contiguous view of src's storage from src's offset on
PyObject *set_view(PyObject *, PyObject *const *args, Py_ssize_t n) {
  if (n != 3 || !PyTuple_Check(args[2])) {
    PyErr_SetString(PyExc_TypeError, "set_view(dst, src, tuple of sizes)");
    return nullptr;
  }
  THGPUTensor *dst = tensor_arg(args[0]), *src = dst ? tensor_arg(args[1]) : nullptr;
  if (!src) return nullptr;
  const Py_ssize_t nd = PyTuple_GET_SIZE(args[2]);
  long few[kMaxNd], *v = nd <= kMaxNd ? few : PyMem_New(long, nd);
  if (!v) return PyErr_NoMemory();
  THLongStorage st = {};
  st.data = v; st.size = nd; st.refcount = 1;
  bool ok = true;
  for (long d = 0; ok && d < nd; d++) {
    v[d] = PyLong_AsLong(PyTuple_GET_ITEM(args[2], d));
    ok = !(v[d] == -1 && PyErr_Occurred());
  }
  if (ok) {
    Py_BEGIN_ALLOW_THREADS
    g_set_storage(dst, src->storage, src->storageOffset, &st, nullptr);
    Py_END_ALLOW_THREADS
    ok = !raised();
  }
  if (v != few) PyMem_Free(v);
  if (!ok) return nullptr;
  Py_RETURN_NONE;
}
// A dense float32 array as a TH tensor; false: not one (the caller takes the general route).
struct HostFloat {
  Py_buffer b;
  long size[kMaxNd], stride[kMaxNd];
  THFloatStorage st;
  THFloatTensor t;
  bool open(PyObject *o, bool writable) {
    if (PyObject_GetBuffer(o, &b, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT | (writable ? PyBUF_WRITABLE : 0)) != 0) { PyErr_Clear(); return false; }
    if (b.ndim < 1 || b.ndim > kMaxNd || b.itemsize != 4 || !b.format || std::strcmp(b.format, "f") != 0 || b.len == 0) {
      PyBuffer_Release(&b);
      return false;
    }
    st = {}; t = {};
    st.data = (float *)b.buf; st.size = b.len / 4; st.refcount = 1;
    long z = 1;
    for (int d = b.ndim - 1; d >= 0; d--) { size[d] = b.shape[d]; stride[d] = z; z *= b.shape[d]; }
    t.size = size; t.stride = stride; t.nDimension = b.ndim; t.storage = &st; t.refcount = 1;
    return true;
  }
};
// upload(tensor, array) / download(array, tensor) -> whether the array was one these take
PyObject *upload(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HostFloat h;
  THGPUTensor *t = n == 2 ? tensor_arg(args[0]) : nullptr;
  if (!t) return nullptr;
  if (!h.open(args[1], false)) Py_RETURN_FALSE;
  Py_BEGIN_ALLOW_THREADS
  g_copy_float(t, &h.t);
  Py_END_ALLOW_THREADS
  PyBuffer_Release(&h.b);
  if (raised()) return nullptr;
  Py_RETURN_TRUE;
}
PyObject *download(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HostFloat h;
  THGPUTensor *t = n == 2 ? tensor_arg(args[1]) : nullptr;
  if (!t) return nullptr;
  if (!h.open(args[0], true)) Py_RETURN_FALSE;
  Py_BEGIN_ALLOW_THREADS
  g_float_copy(&h.t, t);
  Py_END_ALLOW_THREADS
  PyBuffer_Release(&h.b);
  if (raised()) return nullptr;
  Py_RETURN_TRUE;
}

PyMethodDef kMethods[] = {{"setup", setup, METH_VARARGS, nullptr}, {"wrap", wrap, METH_VARARGS, nullptr},
                          {"functions", functions, METH_VARARGS, nullptr}, {"sizes", sizes, METH_O, nullptr},
                          {"set_view", (PyCFunction)(void *)set_view, METH_FASTCALL, nullptr},
                          {"upload", (PyCFunction)(void *)upload, METH_FASTCALL, nullptr},
                          {"download", (PyCFunction)(void *)download, METH_FASTCALL, nullptr}, {}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) {
  CallType.tp_name = "mcw_cppamp_torch_b200._calls.Call";
  CallType.tp_basicsize = sizeof(Call);
  CallType.tp_dealloc = call_dealloc;
  CallType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  CallType.tp_vectorcall_offset = offsetof(Call, vectorcall);
  CallType.tp_call = PyVectorcall_Call;
  CallType.tp_getset = call_getset;
  if (PyType_Ready(&CallType) < 0) return nullptr;
  return PyModule_Create(&kModule);
}
