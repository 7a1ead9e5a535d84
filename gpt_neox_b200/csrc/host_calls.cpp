// Python's way into the kernel library for the calls that a program issues so often that the interpreter bounds it: typed
// entries in place of ctypes, and the look over a generation layer's modules.
//
// Generation with 12 layers of 768, batch 4, a prompt of 100 tokens and 16 steps: 17.4 ms when ctypes and Python did this, 12.4 ms
// with these calls (11.4 with the layer's launches made fewer, csrc/layer_infer.cu; a step's kernels, captured as a graph, take
// 0.33 ms).
// The module looks everything up on each call and keeps nothing but the functions' addresses.  Plain CPython, no torch headers:
// tensors are asked through their attributes, so whatever answers to is_cuda and data_ptr() passes as before.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

namespace {

PyObject *s_is_cuda, *s_data_ptr, *s_dtype, *s_is_contiguous, *s_forward, *s_forward_hooks, *s_forward_pre_hooks, *s_parameters,
    *s_modules, *s_buffers, *s_weight, *s_bias, *s_dict, *s_shape, *s_numel;
PyObject* host_tensor = nullptr;      // called with a tensor that is not on the GPU: raises

struct Ref {      // an owned reference
  PyObject* o;
  explicit Ref(PyObject* p) : o(p) {}
  ~Ref() { Py_XDECREF(o); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  explicit operator bool() const { return o != nullptr; }
};

// -1: an exception is set
int truth(PyObject* owner, PyObject* name) {
  Ref v(PyObject_GetAttr(owner, name));
  return v ? PyObject_IsTrue(v.o) : -1;
}
bool address(PyObject* tensor, void*& out) {
  Ref v(PyObject_CallMethodNoArgs(tensor, s_data_ptr));
  if (!v) return false;
  out = PyLong_AsVoidPtr(v.o);
  return out != nullptr || !PyErr_Occurred();
}

// None, an address, bytes, or a tensor on the GPU.
bool convert(PyObject* o, void*& out) {
  if (o == Py_None) {
    out = nullptr;
    return true;
  }
  if (PyLong_Check(o)) {
    out = PyLong_AsVoidPtr(o);
    return out != nullptr || !PyErr_Occurred();
  }
  if (PyBytes_Check(o)) {
    out = PyBytes_AS_STRING(o);
    return true;
  }
  const int on_gpu = truth(o, s_is_cuda);
  if (on_gpu < 0) return false;
  if (on_gpu == 0) {
    Ref r(PyObject_CallOneArg(host_tensor, o));
    if (r) PyErr_SetString(PyExc_TypeError, "a host tensor was passed to a CUDA kernel");
    return false;
  }
  return address(o, out);
}
bool convert(PyObject* o, long long& out) {
  out = PyLong_AsLongLong(o);
  return out != -1 || !PyErr_Occurred();
}
bool convert(PyObject* o, int& out) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) return false;
  if (v < INT32_MIN || v > INT32_MAX) {
    PyErr_SetString(PyExc_OverflowError, "argument does not fit in 32 bits");
    return false;
  }
  out = static_cast<int>(v);
  return true;
}
bool convert(PyObject* o, float& out) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) return false;
  out = static_cast<float>(v);
  return true;
}

template <class... A>
struct Entry {
  using Fn = int (*)(A...);
  template <std::size_t... I>
  static PyObject* call(Fn fn, PyObject* const* args, std::index_sequence<I...>) {
    std::tuple<A...> a;
    if (!(convert(args[I], std::get<I>(a)) && ...)) return nullptr;
    int status;
    Py_BEGIN_ALLOW_THREADS      // (a launch waits when the stream's queue is full)
    status = fn(std::get<I>(a)...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
  }
  static PyObject* entry(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    if (n != static_cast<Py_ssize_t>(sizeof...(A))) {
      PyErr_Format(PyExc_TypeError, "expected %zu arguments, got %zd", sizeof...(A), n);
      return nullptr;
    }
    void* fn = PyCapsule_GetPointer(self, nullptr);
    return fn != nullptr ? call(reinterpret_cast<Fn>(fn), args, std::index_sequence_for<A...>{}) : nullptr;
  }
};

using P = void*;
using L = long long;
using I = int;
using F = float;
template <class T>
constexpr char letter = std::is_same_v<T, P> ? 'P' : std::is_same_v<T, L> ? 'L' : std::is_same_v<T, I> ? 'I' : 'F';
template <class... A>
struct Signature {
  static constexpr char text[] = {letter<A>..., 0};
};
struct Bound {
  PyMethodDef def;
  const char* types;
};
template <class... A>
constexpr Bound bound(const char* name, Entry<A...>*) {
  return {{name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Entry<A...>::entry)), METH_FASTCALL, nullptr},
          Signature<A...>::text};
}
template <class E>
constexpr Bound def(const char* name) { return bound(name, static_cast<E*>(nullptr)); }
// The signatures of the entry points (csrc/*.cu); `name` or `name_f16`.
Bound entries[] = {
    def<Entry<I, P, P, P, P, P, P, P, P, P, L, I, F, P>>("nx_norm_fwd"),
    def<Entry<I, P, P, P, P, P, P, P, P, P, P, P, P, P, P, L, I, I, I, P>>("nx_norm_bwd"),
    def<Entry<P, P, P, I, I, I, L, L, L, I, I, P, P, P, P, L, I, F, P>>("nx_gemm_bf16"),
    def<Entry<P, P, P, I, I, I, L, L, L, I, I, P, P, P, P, L, I, F, P>>("nx_gemm2_bf16"),
    def<Entry<P, P, L, I, I, P>>("nx_gated_act_fwd"),
    def<Entry<P, P>>("nx_layer_infer"),
};

// bind(name, address[, types]) -> the entry point as a callable, or None if its signature is not known here.  `types`: a letter of
// "PILF" (pointer, int, long long, float) per parameter as the caller declares them; a difference is an error.
PyObject* bind(PyObject*, PyObject* args) {
  const char *name, *types = nullptr;
  unsigned long long at;
  if (!PyArg_ParseTuple(args, "sK|z", &name, &at, &types)) return nullptr;
  for (Bound& e : entries) {
    const std::size_t n = std::strlen(e.def.ml_name);
    if (std::strncmp(name, e.def.ml_name, n) != 0 || (name[n] != 0 && std::strcmp(name + n, "_f16") != 0)) continue;
    if (types != nullptr && std::strcmp(types, e.types) != 0) {
      PyErr_Format(PyExc_TypeError, "%s takes (%s) here and is declared as (%s)", name, e.types, types);
      return nullptr;
    }
    Ref capsule(PyCapsule_New(reinterpret_cast<void*>(static_cast<std::uintptr_t>(at)), nullptr, nullptr));
    return capsule ? PyCFunction_New(&e.def, capsule.o) : nullptr;
  }
  Py_RETURN_NONE;
}

// dict[name], borrowed; null without an exception where it is missing
PyObject* item(PyObject* dict, PyObject* name) { return PyDict_GetItemWithError(dict, name); }

// Whether calling `m` runs the class's `forward` as it was defined and nothing else.  -1: exception.
int is_plain(PyObject* m, PyObject* cls, PyObject* forward) {
  if (reinterpret_cast<PyObject*>(Py_TYPE(m)) != cls) return 0;
  Ref f(PyObject_GetAttr(cls, s_forward));
  if (!f) return -1;
  if (f.o != forward) return 0;
  Ref d(PyObject_GetAttr(m, s_dict));
  if (!d) return -1;
  if (!PyDict_Check(d.o)) return 0;
  if (item(d.o, s_forward) != nullptr) return 0;
  for (PyObject* name : {s_forward_hooks, s_forward_pre_hooks}) {
    PyObject* hooks = item(d.o, name);
    if (hooks == nullptr) {
      if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, name);
      return -1;
    }
    const Py_ssize_t n = PyObject_Size(hooks);
    if (n != 0) return n < 0 ? -1 : 0;
  }
  return 1;
}

// A module's parameter (or None): getattr, without the module's __getattr__ where nothing in the instance, whose __dict__ is `d`,
// stands before it.
PyObject* parameter(PyObject* m, PyObject* d, PyObject* name) {
  PyObject* params = item(d, s_parameters);
  if (params != nullptr && PyDict_Check(params) && item(d, name) == nullptr) {
    PyObject* p = item(params, name);
    if (p != nullptr) return Py_NewRef(p);
  }
  return PyErr_Occurred() ? nullptr : PyObject_GetAttr(m, name);
}

// sub(m, name): the same for a submodule or a buffer of a module whose class has no attribute of that name.
PyObject* sub(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "sub(module, name)");
    return nullptr;
  }
  Ref d(PyObject_GetAttr(args[0], s_dict));
  if (!d) return nullptr;
  if (item(d.o, args[1]) == nullptr)
    for (PyObject* kind : {s_modules, s_buffers}) {
      PyObject* held = item(d.o, kind);
      PyObject* m = held != nullptr && PyDict_Check(held) ? item(held, args[1]) : nullptr;
      if (m != nullptr && m != Py_None) return Py_NewRef(m);
    }
  return PyErr_Occurred() ? nullptr : PyObject_GetAttr(args[0], args[1]);
}

// plain(module, class, forward, ...): whether all of them are.
PyObject* plain(PyObject*, PyObject* const* args, Py_ssize_t n) {
  for (Py_ssize_t i = 0; i + 2 < n; i += 3) {
    const int ok = is_plain(args[i], args[i + 1], args[i + 2]);
    if (ok < 0) return nullptr;
    if (ok == 0) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
}

// The addresses of x and of modules' weights and biases (0 for None), if the kernels read them where they are: on the GPU,
// contiguous, 16-byte aligned, of x's type, which is one of `dtypes`.
class Addresses {
 public:
  // 1: taken, 0: not where the kernels read it, -1: exception
  int begin(PyObject* dtypes, PyObject* x) {
    if (!PyTuple_Check(dtypes)) {
      PyErr_SetString(PyExc_TypeError, "the first argument is a tuple of types");
      return -1;
    }
    dtype_ = PyObject_GetAttr(x, s_dtype);
    if (dtype_ == nullptr) return -1;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(dtypes); ++i)
      if (PyTuple_GET_ITEM(dtypes, i) == dtype_) return take(x);
    return 0;
  }
  // [rows, columns]: the extents the weight has to have ([rows] for no columns), and the bias [rows]; null: any.  A negative extent is
  // the width that all weights with one share.
  int module(PyObject* m, const long long* size) {
    Ref d(PyObject_GetAttr(m, s_dict));
    if (!d) return -1;
    long long rows = 0;
    for (PyObject* name : {s_weight, s_bias}) {
      Ref t(parameter(m, d.o, name));
      if (!t) return -1;
      int ok = take(t.o);
      if (ok == 1 && size != nullptr) {
        if (name == s_bias) ok = t.o == Py_None ? 1 : has_elements(t.o, rows);
        else ok = t.o == Py_None ? 0 : has_size(t.o, size, rows);
      }
      if (ok != 1) return ok;
    }
    return 1;
  }
  PyObject* bytes() const {
    if ((bits_ & 15) != 0) Py_RETURN_NONE;
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(out_), count_ * sizeof(out_[0]));
  }
  long long width() const { return width_; }
  static constexpr int MAX = 64;
  Addresses() = default;
  Addresses(const Addresses&) = delete;
  ~Addresses() { Py_XDECREF(dtype_); }

 private:
  int take(PyObject* t) {
    if (t == Py_None) {
      out_[count_++] = 0;
      return 1;
    }
    int ok = truth(t, s_is_cuda);
    if (ok <= 0) return ok;
    Ref dt(PyObject_GetAttr(t, s_dtype));
    if (!dt) return -1;
    if (dt.o != dtype_) return 0;
    Ref c(PyObject_CallMethodNoArgs(t, s_is_contiguous));
    if (!c) return -1;
    ok = PyObject_IsTrue(c.o);
    if (ok <= 0) return ok;
    void* p;
    if (!address(t, p)) return -1;
    out_[count_] = reinterpret_cast<std::uintptr_t>(p);
    bits_ |= out_[count_++];
    return 1;
  }
  static int has_elements(PyObject* t, long long n) {
    Ref v(PyObject_CallMethodNoArgs(t, s_numel));
    long long at;
    if (!v || !convert(v.o, at)) return -1;
    return at == n;
  }
  int is_extent(long long at, long long want) {
    if (want >= 0) return at == want;
    if (width_ < 0) width_ = at;
    return at == width_;
  }
  int has_size(PyObject* t, const long long* size, long long& rows) {
    rows = size[0];
    if (size[1] == 0) return has_elements(t, rows);
    Ref shape(PyObject_GetAttr(t, s_shape));
    if (!shape) return -1;
    if (!PyTuple_Check(shape.o) || PyTuple_GET_SIZE(shape.o) != 2) return 0;
    long long at[2];
    for (int i = 0; i < 2; ++i) {
      if (!convert(PyTuple_GET_ITEM(shape.o, i), at[i])) return -1;
      if (!is_extent(at[i], size[i])) return 0;
    }
    rows = at[0];
    return 1;
  }
  std::uintptr_t out_[MAX], bits_ = 0;
  int count_ = 0;
  long long width_ = -1;
  PyObject* dtype_ = nullptr;
};

// pointers(dtypes, x, module, ...): the addresses as bytes, or None.
PyObject* pointers(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n < 2 || 2 * (n - 2) + 1 > Addresses::MAX) {
    PyErr_SetString(PyExc_TypeError, "pointers(dtypes, x, module, ...)");
    return nullptr;
  }
  Addresses a;
  int ok = a.begin(args[0], args[1]);
  for (Py_ssize_t i = 2; i < n && ok == 1; ++i) ok = a.module(args[i], nullptr);
  if (ok < 0) return nullptr;
  if (ok == 0) Py_RETURN_NONE;
  return a.bytes();
}

// weights(dtypes, x, module, rows, columns, ...): (the addresses as bytes, the width that the negative extents stand for), if every
// weight has the size beside its module; else (None, that width or a negative number).
PyObject* weights(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n < 2 || (n - 2) % 3 != 0 || (n - 2) / 3 * 2 + 1 > Addresses::MAX) {
    PyErr_SetString(PyExc_TypeError, "weights(dtypes, x, module, rows, columns, ...)");
    return nullptr;
  }
  Addresses a;
  int ok = a.begin(args[0], args[1]);
  for (Py_ssize_t i = 2; i < n && ok == 1; i += 3) {
    long long size[2];
    if (!convert(args[i + 1], size[0]) || !convert(args[i + 2], size[1])) return nullptr;
    ok = a.module(args[i], size);
  }
  if (ok < 0) return nullptr;
  Ref bytes(ok == 1 ? a.bytes() : Py_NewRef(Py_None));
  return bytes ? Py_BuildValue("(OL)", bytes.o, a.width()) : nullptr;
}

PyObject* set_host_tensor_error(PyObject*, PyObject* f) {
  Py_XSETREF(host_tensor, Py_NewRef(f));
  Py_RETURN_NONE;
}

template <PyObject* (*FN)(PyObject*, PyObject* const*, Py_ssize_t)>
constexpr PyMethodDef fast(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(FN)), METH_FASTCALL, nullptr};
}
PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, nullptr},
                         {"set_host_tensor_error", set_host_tensor_error, METH_O, nullptr},
                         fast<sub>("sub"), fast<plain>("plain"), fast<pointers>("pointers"), fast<weights>("weights"),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "neox_host_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_neox_host_calls(void) {
  struct {
    PyObject** at;
    const char* name;
  } names[] = {{&s_is_cuda, "is_cuda"}, {&s_data_ptr, "data_ptr"}, {&s_dtype, "dtype"}, {&s_is_contiguous, "is_contiguous"},
               {&s_forward, "forward"}, {&s_forward_hooks, "_forward_hooks"}, {&s_forward_pre_hooks, "_forward_pre_hooks"},
               {&s_parameters, "_parameters"}, {&s_modules, "_modules"}, {&s_buffers, "_buffers"}, {&s_weight, "weight"}, {&s_bias, "bias"},
               {&s_dict, "__dict__"}, {&s_shape, "shape"}, {&s_numel, "numel"}};
  for (auto& n : names)
    if ((*n.at = PyUnicode_InternFromString(n.name)) == nullptr) return nullptr;
  return PyModule_Create(&module_def);
}
