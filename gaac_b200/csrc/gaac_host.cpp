// The calls of a decode step without the binding's cost: the library's functions as functions of a Python module that take tensors, and the objects that hold them, as they are.  A ctypes call
// of 15 to 20 arguments takes 1.5 us, a descriptor built from ten data_ptr() calls 1.0 and torch.empty from Python 1.7, against 3 us for the launch itself, and a
// step of short rows was bound by nothing else.  us, through ctypes -> here: attention over two Pages of 500 tokens 10.7 -> 7.3 (5.8 in a graph), append and attention of 7 rows 30.9 -> 22.8, paged
// store and attention of 5 rows 21.9 -> 16.4, an encode of [8, 1111, 128] 47.4 -> 41 with its copy, three prompts of 4001 tokens 117.7 -> 108.
//
// The module knows the functions' types from the C header and finds their addresses in the library that the package has loaded (bind).  What an argument may be:
//   pointer                  a tensor (its data) or what has a data_ptr(), None, or an address
//   gaac_side                a Page, or a tuple (sm, codes, flags, tile_off, ovf, head_start, base3, base4, tail or None)
//   gaac_store               an object with these fields (kv_cache._Store)
//   gaac_paged               a tuple (buf, raw, mt, stack, top, err, b3k, b4k, b3v, b4v, n_kv, TS, ovf_slot)
//   numbers                  as themselves
// Nothing is kept between calls: every pointer is read from its tensor when the call is made.  The interpreter is let go for the duration of the library call, as ctypes does, and of an
// allocation, as torch.empty does: either may wait for the GPU, whose queue may wait for what another thread has yet to launch.
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <ATen/ATen.h>
#include "../../include/gaac_b200.h"

namespace {

struct Failed {};                                    // a Python error is set

PyObject* attr_name(const char* name) { return PyUnicode_InternFromString(name); }
struct Ref {                                         // an attribute or a result, held while it is read
  PyObject* o;
  explicit Ref(PyObject* made) : o(made) { if (!o) throw Failed{}; }
  Ref(PyObject* of, PyObject* name) : Ref(PyObject_GetAttr(of, name)) {}
  ~Ref() { Py_DECREF(o); }
  Ref(const Ref&) = delete;
};
long long whole(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);          // (takes anything with __index__)
  if (v == -1 && PyErr_Occurred()) throw Failed{};
  return v;
}
// o.name(), for what is no tensor but has a tensor's methods
PyObject* asked(PyObject* o, PyObject* name) { return PyObject_CallMethodNoArgs(o, name); }

void* address(PyObject* o) {
  if (o == Py_None) return nullptr;
  if (THPVariable_Check(o)) return THPVariable_Unpack(o).data_ptr();
  if (PyLong_Check(o)) {
    void* p = PyLong_AsVoidPtr(o);
    if (!p && PyErr_Occurred()) throw Failed{};
    return p;
  }
  static PyObject* const data_ptr = attr_name("data_ptr");
  const Ref p(asked(o, data_ptr));
  void* const at = PyLong_AsVoidPtr(p.o);
  if (!at && PyErr_Occurred()) throw Failed{};
  return at;
}
long long elements(PyObject* o) {
  if (THPVariable_Check(o)) return THPVariable_Unpack(o).numel();
  static PyObject* const numel = attr_name("numel");
  return whole(Ref(asked(o, numel)).o);
}
const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) { PyErr_SetString(PyExc_TypeError, "a tensor expected"); throw Failed{}; }
  return THPVariable_Unpack(o);
}
PyObject* item(PyObject* t, Py_ssize_t i, Py_ssize_t n) {
  if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != n) { PyErr_SetString(PyExc_TypeError, "a tuple of the descriptor's fields expected"); throw Failed{}; }
  return PyTuple_GET_ITEM(t, i);
}
template <class P> P pointer(PyObject* o) { return static_cast<P>(address(o)); }

// ---- arguments.  Arg<T>: made from the Python object, converts to what the function takes.
template <class T, class = void> struct Arg;
template <class T> struct Arg<T, std::enable_if_t<std::is_integral_v<T>>> {
  T v;
  explicit Arg(PyObject* o) : v(static_cast<T>(whole(o))) {
    if (sizeof(T) < 8 && static_cast<long long>(v) != whole(o)) { PyErr_SetString(PyExc_OverflowError, "number too large for the argument"); throw Failed{}; }
  }
  operator T() const { return v; }
};
template <> struct Arg<float> {
  float v;
  explicit Arg(PyObject* o) : v((float)PyFloat_AsDouble(o)) { if (PyErr_Occurred()) throw Failed{}; }
  operator float() const { return v; }
};
template <class T> struct Arg<T*> {
  T* v;
  explicit Arg(PyObject* o) : v(pointer<T*>(const_cast<PyObject*>(o))) {}
  operator T*() const { return v; }
};
template <class T> struct Arg<const T*> {
  const T* v;
  explicit Arg(PyObject* o) : v(static_cast<const T*>(address(o))) {}
  operator const T*() const { return v; }
};
template <> struct Arg<const gaac_side*> {
  gaac_side s{};
  explicit Arg(PyObject* o) {
    if (PyTuple_Check(o)) {
      set(item(o, 0, 9), item(o, 1, 9), item(o, 2, 9), item(o, 3, 9), item(o, 4, 9), item(o, 5, 9), item(o, 6, 9), item(o, 7, 9));
      s.tail = pointer<decltype(s.tail)>(item(o, 8, 9));
      return;
    }
    static PyObject *const n[8] = {attr_name("sm"), attr_name("codes"), attr_name("flags"), attr_name("tile_off"), attr_name("ovf"), attr_name("ovf_head_start"), attr_name("base3"), attr_name("base4")};
    const Ref a(o, n[0]), b(o, n[1]), c(o, n[2]), d(o, n[3]), e(o, n[4]), f(o, n[5]), g(o, n[6]), h(o, n[7]);
    set(a.o, b.o, c.o, d.o, e.o, f.o, g.o, h.o);
  }
  void set(PyObject* sm, PyObject* codes, PyObject* flags, PyObject* tile_off, PyObject* ovf, PyObject* head_start, PyObject* base3, PyObject* base4) {
    s.sm = pointer<decltype(s.sm)>(sm); s.codes = pointer<decltype(s.codes)>(codes); s.flags = pointer<decltype(s.flags)>(flags); s.tile_off = pointer<decltype(s.tile_off)>(tile_off);
    s.ovf = pointer<decltype(s.ovf)>(ovf); s.ovf_bytes = elements(ovf); s.head_start = pointer<decltype(s.head_start)>(head_start);
    s.base3 = pointer<decltype(s.base3)>(base3); s.base4 = pointer<decltype(s.base4)>(base4);
  }
  operator const gaac_side*() const { return &s; }
};
template <> struct Arg<const gaac_store*> {
  gaac_store s{};
  explicit Arg(PyObject* o) {
    static PyObject *const n[9] = {attr_name("sm"), attr_name("codes"), attr_name("flags"), attr_name("tile_off"), attr_name("ovf"), attr_name("ovf_used"), attr_name("tail"), attr_name("base3"), attr_name("base4")};
    const Ref a(o, n[0]), b(o, n[1]), c(o, n[2]), d(o, n[3]), e(o, n[4]), f(o, n[5]), g(o, n[6]), h(o, n[7]), i(o, n[8]);
    s.sm = pointer<decltype(s.sm)>(a.o); s.codes = pointer<decltype(s.codes)>(b.o); s.flags = pointer<decltype(s.flags)>(c.o); s.tile_off = pointer<decltype(s.tile_off)>(d.o);
    s.ovf = pointer<decltype(s.ovf)>(e.o); s.ovf_used = pointer<decltype(s.ovf_used)>(f.o); s.tail = pointer<decltype(s.tail)>(g.o);
    s.base3 = pointer<decltype(s.base3)>(h.o); s.base4 = pointer<decltype(s.base4)>(i.o);
  }
  operator const gaac_store*() const { return &s; }
};
template <> struct Arg<const gaac_paged*> {
  gaac_paged s{};
  explicit Arg(PyObject* o) {
    const auto at = [&](int i) { return item(o, i, 13); };
    s.buf = pointer<decltype(s.buf)>(at(0)); s.raw = pointer<decltype(s.raw)>(at(1)); s.mt = pointer<decltype(s.mt)>(at(2)); s.stack = pointer<decltype(s.stack)>(at(3));
    s.top = pointer<decltype(s.top)>(at(4)); s.err = pointer<decltype(s.err)>(at(5)); s.b3k = pointer<decltype(s.b3k)>(at(6)); s.b4k = pointer<decltype(s.b4k)>(at(7));
    s.b3v = pointer<decltype(s.b3v)>(at(8)); s.b4v = pointer<decltype(s.b4v)>(at(9));
    s.n_kv = Arg<int>(at(10)); s.TS = Arg<int>(at(11)); s.ovf_slot = Arg<int>(at(12));
  }
  operator const gaac_paged*() const { return &s; }
};

struct Released {                                    // the interpreter's lock, let go of, also by way of an exception
  PyThreadState* const state = PyEval_SaveThread();
  Released() = default;
  ~Released() { PyEval_RestoreThread(state); }
  Released(const Released&) = delete;
};

template <class F> PyObject* guarded(const F& f) {
  try { return f(); }
  catch (const Failed&) { return nullptr; }
  catch (...) { torch::translate_exception_to_python(std::current_exception()); return nullptr; }
}

// ---- a library function as one of the module
template <class... A, size_t... I>
PyObject* invoke(int (*fn)(A...), PyObject* const* args, std::index_sequence<I...>) {
  const std::tuple<Arg<A>...> a{Arg<A>(args[I])...};
  const auto run = [&] { const Released released; return fn(std::get<I>(a)...); };
  return PyLong_FromLong(run());
}
template <class... A>
PyObject* call(int (*fn)(A...), const char* name, PyObject* const* args, Py_ssize_t n) {
  if (!fn) return PyErr_Format(PyExc_RuntimeError, "%s: the module is not bound to the library", name);
  if (n != (Py_ssize_t)sizeof...(A)) return PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, not %zd", name, (Py_ssize_t)sizeof...(A), n);
  return guarded([&] { return invoke(fn, args, std::index_sequence_for<A...>{}); });
}

#define GAAC_CALLS(X) X(gaac_decode_attn_pages) X(gaac_decode_attn) X(gaac_decode_attn_balanced) X(gaac_decode_attn_flat) X(gaac_append_kv) X(gaac_paged_decode_attn) \
  X(gaac_paged_decode_attn_balanced) X(gaac_paged_decode_attn_flat) X(gaac_paged_decode_attn256) X(gaac_paged_decode_attn256_flat) X(gaac_paged_store) X(gaac_paged_decode_blocks) \
  X(gaac_encode_queued) X(gaac_decode_page) X(gaac_cache_prefill_own) X(gaac_cache_prefill) X(gaac_cache_calibrate)
#define DEFINE(f) \
  decltype(&f) p_##f = nullptr; \
  PyObject* py_##f(PyObject*, PyObject* const* args, Py_ssize_t n) { return call(p_##f, #f, args, n); }
GAAC_CALLS(DEFINE)

// bind(handle): of the library, as dlopen returned it
PyObject* bind(PyObject*, PyObject* o) {
  void* const lib = PyLong_AsVoidPtr(o);
  if (PyErr_Occurred()) return nullptr;
#define FIND(f) if (!(p_##f = reinterpret_cast<decltype(p_##f)>(dlsym(lib, #f)))) return PyErr_Format(PyExc_RuntimeError, "%s is not in the library", #f);
  GAAC_CALLS(FIND)
  Py_RETURN_NONE;
}

// empty(like, dtype, sizes..): torch.empty on the device of `like`; dtype: 0 uint8, 1 int32, 2 bfloat16, 3 that of `like`
PyObject* empty(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n < 2 || n > 6) { PyErr_SetString(PyExc_TypeError, "empty(like, dtype, sizes..)"); return nullptr; }
    const at::Tensor& like = tensor(args[0]);
    const long long kind = whole(args[1]);
    int64_t size[4];
    for (Py_ssize_t i = 2; i < n; i++) size[i - 2] = whole(args[i]);
    auto options = at::TensorOptions().device(like.device()).dtype(kind == 0 ? at::kByte : kind == 1 ? at::kInt : kind == 2 ? at::kBFloat16 : like.scalar_type());
    const auto make = [&] { const Released released; return at::empty(at::IntArrayRef(size, (size_t)(n - 2)), options); };
    return THPVariable_Wrap(make());
  });
}

PyMethodDef methods[] = {
#define METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##f)), METH_FASTCALL, nullptr},
  GAAC_CALLS(METHOD)
  {"bind", bind, METH_O, nullptr},
  {"empty", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(empty)), METH_FASTCALL, nullptr},
  {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

#define TEXT(x) #x
#define TEXT_OF(x) TEXT(x)
const char built_for[] = "ABI " TEXT_OF(GAAC_ABI_VERSION) ", torch " TEXT_OF(GAAC_TORCH_VERSION);          // (checked before bind)

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  PyObject* const made = PyModule_Create(&module);
  if (made && PyModule_AddStringConstant(made, "built_for", built_for) < 0) { Py_DECREF(made); return nullptr; }
  return made;
}
