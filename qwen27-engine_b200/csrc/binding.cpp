// CPython binding of the entry points that an engine calls once per layer and step.
//
// A decode call behind a short context takes about ten microseconds on the GPU; the same call through ctypes
// takes longer than that on the host (a Python-level check and a ctypes object per tensor argument): prologue and
// decode of one token behind 256, 33.5 us a pass through ctypes, 9.3 through this binding. Here the
// arguments are read natively: same checks, same order, same errors. Anything that is not exactly a torch.Tensor
// or an nn.Parameter (a raw address, None, a subclass) goes through the module's Python-level check. The library
// stays the one that the Python module has loaded: it hands over the addresses of its functions.
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

#include <cstdint>

#include "q27b_attn.h"

namespace {

enum Fn { PREP, DECODE, PREP_PAGED, DECODE_PAGED, PREFILL, N_FN };
// One per module object: the package may be loaded under two names, each with its own library and error class.
struct State {
  void* fn[N_FN];
  PyObject* ptr;    // _ptr(tensor, dtype, optional) -> ctypes.c_void_p
  PyObject* check;  // _check(return code): raises
  PyObject *f32, *i32, *i8;  // torch.float32, int32, int8 as Python objects, for ptr
};
PyObject* dtype_object(const State* st, c10::ScalarType t) {
  return t == c10::kFloat ? st->f32 : t == c10::kInt ? st->i32 : t == c10::kChar ? st->i8 : Py_None;
}

// Device address of one tensor argument. want = Undefined: any dtype.
bool ptr(const State* st, PyObject* o, c10::ScalarType want, bool optional, void** out) {
  if (THPVariable_CheckExact(o)) {
    const at::Tensor& t = THPVariable_Unpack(o);
    if (t.is_cuda() && t.is_contiguous() && (want == c10::ScalarType::Undefined || t.scalar_type() == want)) {
      *out = t.data_ptr();
      return true;
    }
  }
  PyObject* r = PyObject_CallFunctionObjArgs(st->ptr, o, dtype_object(st, want), optional ? Py_True : Py_False, nullptr);
  if (!r) return false;
  PyObject* v = PyObject_GetAttrString(r, "value");
  Py_DECREF(r);
  if (!v) return false;
  *out = v == Py_None ? nullptr : PyLong_AsVoidPtr(v);
  Py_DECREF(v);
  return !PyErr_Occurred();
}

bool num(PyObject* o, int* out) {  // int(o), as ctypes takes it: the low 32 bits
  PyObject* l = PyLong_CheckExact(o) ? Py_NewRef(o) : PyObject_CallOneArg((PyObject*)&PyLong_Type, o);
  if (!l) return false;
  *out = (int)PyLong_AsUnsignedLongMask(l);
  Py_DECREF(l);
  return !PyErr_Occurred();
}
bool flt(PyObject* o, float* out) {
  *out = (float)PyFloat_AsDouble(o);
  return !PyErr_Occurred();
}
bool flag(PyObject* o, int* out) {
  const int t = PyObject_IsTrue(o);
  *out = t;
  return t >= 0;
}

PyObject* done(const State* st, int rc) {
  if (rc == 0) Py_RETURN_NONE;
  return PyObject_CallFunction(st->check, "i", rc);
}

constexpr c10::ScalarType F32 = c10::kFloat, I32 = c10::kInt, I8 = c10::kChar, ANY = c10::ScalarType::Undefined;

// Runs `body`, turning C++ exceptions of torch into Python errors.
template <class B>
PyObject* guarded(PyObject* self, Py_ssize_t n, Py_ssize_t want, B body) {
  const State* st = (const State*)PyModule_GetState(self);
  if (!st || !st->ptr) return PyErr_Format(PyExc_RuntimeError, "q27b_binding is not bound");
  if (n != want) return PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
  try {
    return body(st);
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}
void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }

template <c10::ScalarType T> struct Elem { using type = void; };
template <> struct Elem<F32> { using type = float; };
template <> struct Elem<I32> { using type = int; };
template <> struct Elem<I8> { using type = int8_t; };

#define PTR(i, kind, opt, name)                            \
  void* name##_p;                                          \
  if (!ptr(st, a[i], kind, opt, &name##_p)) return nullptr; \
  Elem<kind>::type* name = static_cast<Elem<kind>::type*>(name##_p)
#define NUM(i, name) \
  int name;          \
  if (!num(a[i], &name)) return nullptr
#define FLT(i, name) \
  float name;        \
  if (!flt(a[i], &name)) return nullptr
#define FLAG(i, name) \
  int name;           \
  if (!flag(a[i], &name)) return nullptr
// The signature is the header's: a parameter added, taken out or of another type there does not compile here.
#define CALL(which, entry, ...)                                        \
  void* s = stream();                                                  \
  int rc;                                                              \
  Py_BEGIN_ALLOW_THREADS                                               \
  rc = reinterpret_cast<decltype(&entry)>(st->fn[which])(__VA_ARGS__); \
  Py_END_ALLOW_THREADS                                                 \
  return done(st, rc)

// qg, k, v, q_norm, k_norm, qn, kcache, vcache, pos0, T, eps, theta_scale, nqh, nkvh, n_ctx, q8, rope3, rdelta
PyObject* attn_prep(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  return guarded(self, n, 18, [&](const State* st) -> PyObject* {
    PTR(0, F32, false, qg); PTR(1, F32, false, k); PTR(2, F32, false, v); PTR(3, F32, false, qw); PTR(4, F32, false, kw);
    PTR(5, F32, false, qn); PTR(6, ANY, false, kc); PTR(7, ANY, false, vc); PTR(8, I32, false, pos0);
    NUM(9, T); FLT(10, eps); FLT(11, theta); NUM(12, nqh); NUM(13, nkvh); NUM(14, n_ctx); FLAG(15, q8);
    PTR(16, I32, true, rope3); PTR(17, I32, true, rdelta);
    CALL(PREP, q27b_attn_prep, qg, k, v, qw, kw, qn, kc, vc, pos0, T, eps, theta, nqh, nkvh, n_ctx, q8, s, rope3, rdelta);
  });
}

// qn, qg, kcache, vcache, o, xq, xd, pos0, T, kq_scale, nqh, nkvh, n_ctx, q8
PyObject* attn_decode(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  return guarded(self, n, 14, [&](const State* st) -> PyObject* {
    PTR(0, F32, false, qn); PTR(1, F32, false, qg); PTR(2, ANY, false, kc); PTR(3, ANY, false, vc); PTR(4, F32, true, o);
    PTR(5, I8, true, xq); PTR(6, F32, true, xd); PTR(7, I32, false, pos0);
    NUM(8, T); FLT(9, scale); NUM(10, nqh); NUM(11, nkvh); NUM(12, n_ctx); FLAG(13, q8);
    CALL(DECODE, q27b_attn_decode, qn, qg, kc, vc, o, xq, xd, pos0, T, scale, nqh, nkvh, n_ctx, q8, s);
  });
}

// qg, k, v, q_norm, k_norm, qn, kpool, vpool, page_table, seq_len, B, T, eps, theta_scale, nqh, nkvh, n_pages, max_pages, rope3, rdelta
PyObject* attn_prep_paged(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  return guarded(self, n, 20, [&](const State* st) -> PyObject* {
    PTR(0, F32, true, qg); PTR(1, F32, false, k); PTR(2, F32, false, v); PTR(3, F32, true, qw); PTR(4, F32, true, kw);
    PTR(5, F32, true, qn); PTR(6, ANY, false, kp); PTR(7, ANY, false, vp); PTR(8, I32, false, table); PTR(9, I32, false, lens);
    NUM(10, B); NUM(11, T); FLT(12, eps); FLT(13, theta); NUM(14, nqh); NUM(15, nkvh); NUM(16, n_pages); NUM(17, max_pages);
    PTR(18, I32, true, rope3); PTR(19, I32, true, rdelta);
    CALL(PREP_PAGED, q27b_attn_prep_paged, qg, k, v, qw, kw, qn, kp, vp, table, lens, B, T, eps, theta, nqh, nkvh, n_pages, max_pages, s, rope3, rdelta);
  });
}

// qn, qg, kpool, vpool, page_table, seq_len, o, B, T, kq_scale, nqh, nkvh, n_pages, max_pages, max_seq_len
PyObject* attn_decode_paged(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  return guarded(self, n, 15, [&](const State* st) -> PyObject* {
    PTR(0, F32, false, qn); PTR(1, F32, false, qg); PTR(2, ANY, false, kp); PTR(3, ANY, false, vp); PTR(4, I32, false, table);
    PTR(5, I32, false, lens); PTR(6, F32, false, o);
    NUM(7, B); NUM(8, T); FLT(9, scale); NUM(10, nqh); NUM(11, nkvh); NUM(12, n_pages); NUM(13, max_pages); NUM(14, max_len);
    CALL(DECODE_PAGED, q27b_attn_decode_paged, qn, qg, kp, vp, table, lens, o, B, T, scale, nqh, nkvh, n_pages, max_pages, max_len, s);
  });
}

// qn, qg, kcache, vcache, o, pos0, M, kq_scale, nqh, nkvh, n_ctx, q8, depth_hint
PyObject* attn_prefill(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  return guarded(self, n, 13, [&](const State* st) -> PyObject* {
    PTR(0, F32, false, qn); PTR(1, F32, false, qg); PTR(2, ANY, false, kc); PTR(3, ANY, false, vc); PTR(4, F32, false, o);
    PTR(5, I32, false, pos0);
    NUM(6, M); FLT(7, scale); NUM(8, nqh); NUM(9, nkvh); NUM(10, n_ctx); FLAG(11, q8); NUM(12, depth);
    CALL(PREFILL, q27b_attn_prefill, qn, qg, kc, vc, o, pos0, M, scale, nqh, nkvh, n_ctx, q8, s, depth);
  });
}

// addresses (tuple of N_FN ints), _ptr, _check, torch.float32, torch.int32, torch.int8
PyObject* bind(PyObject* self, PyObject* args) {
  PyObject *fns, *p, *c, *f32, *i32, *i8;
  if (!PyArg_ParseTuple(args, "O!OOOOO", &PyTuple_Type, &fns, &p, &c, &f32, &i32, &i8)) return nullptr;
  if (PyTuple_GET_SIZE(fns) != N_FN) return PyErr_Format(PyExc_ValueError, "expected %d addresses", (int)N_FN);
  State* st = (State*)PyModule_GetState(self);
  for (int i = 0; i < N_FN; i++) st->fn[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(fns, i));
  if (PyErr_Occurred()) return nullptr;
  Py_XSETREF(st->ptr, Py_NewRef(p)); Py_XSETREF(st->check, Py_NewRef(c));
  Py_XSETREF(st->f32, Py_NewRef(f32)); Py_XSETREF(st->i32, Py_NewRef(i32)); Py_XSETREF(st->i8, Py_NewRef(i8));
  Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {{"bind", bind, METH_VARARGS, nullptr}, FAST(attn_prep), FAST(attn_decode), FAST(attn_prep_paged),
                           FAST(attn_decode_paged), FAST(attn_prefill), {nullptr, nullptr, 0, nullptr}};
// The objects of the state belong to the package that holds this module: a cycle for the collector.
int traverse(PyObject* self, visitproc visit, void* arg) {
  State* st = (State*)PyModule_GetState(self);
  if (!st) return 0;
  Py_VISIT(st->ptr); Py_VISIT(st->check); Py_VISIT(st->f32); Py_VISIT(st->i32); Py_VISIT(st->i8);
  return 0;
}
int clear(PyObject* self) {
  State* st = (State*)PyModule_GetState(self);
  if (!st) return 0;
  Py_CLEAR(st->ptr); Py_CLEAR(st->check); Py_CLEAR(st->f32); Py_CLEAR(st->i32); Py_CLEAR(st->i8);
  return 0;
}
void release(void* self) { clear((PyObject*)self); }

PyModuleDef_Slot g_slots[] = {{0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "q27b_binding", nullptr, sizeof(State), g_methods, g_slots, traverse, clear, release};

}  // namespace

PyMODINIT_FUNC PyInit_q27b_binding(void) { return PyModuleDef_Init(&g_module); }
