/* CPython binding of the entry points that a step calls once per layer (lib/_kpx_py.<abi>.so).
 *
 * A decode step of a short context is two launches of a few microseconds per layer, and calling
 * them through ctypes cost more than running them: about 4.5 us of argument conversion per call
 * (an isinstance / hasattr / data_ptr chain per pointer, ctypes' own conversion, the stream's
 * wrapper object) in front of a 3 us launch.  Here an argument costs one type check and, for a
 * tensor, one data_ptr() call: about 1 us a call.  28 layers of a 512-token fp32 chat (56 calls)
 * took 587 us before and 279 us now, 28 fused steps of 8 short sequences 439 and 273 us.  Conversions accept what the ctypes signatures accept: None, int or
 * an object with data_ptr() / ctypes.data for a pointer, int for an integer (cut to its width), a
 * number for a float, a ctypes scalar of the argument's type for either, a KvLayout for the layout.  The GIL is released around the call.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include "kpx.h"

static PyObject *s_data_ptr, *s_ctypes, *s_data;
static PyObject *get_device, *get_stream; /* callables given to set_stream_source */
static PyObject* layout_type;             /* the type of a layout, given to set_layout_type */
static PyObject* get_number;              /* (kind, object) -> number, given to set_number_source */
enum { KIND_I32, KIND_I64, KIND_F32 };

typedef struct {
  PyObject* const* at; /* next argument */
  int bad;             /* a conversion failed: the Python error is set */
} Args;

static void* mask_ptr(PyObject* o, Args* a) {
  void* p = (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(o);
  if (PyErr_Occurred()) a->bad = 1;
  return p;
}
static void* arg_ptr(Args* a) {
  PyObject *o = *a->at++, *v;
  void* p;
  if (a->bad || o == Py_None) return NULL;
  if (PyLong_Check(o)) return mask_ptr(o, a);
  if (strcmp(Py_TYPE(o)->tp_name, "numpy.ndarray") == 0) { /* (its ctypes attribute takes 2 us to make) */
    Py_buffer view;
    if (PyObject_GetBuffer(o, &view, PyBUF_STRIDED_RO) == 0) {
      p = view.buf;
      PyBuffer_Release(&view);
      return p;
    }
    PyErr_Clear();
  }
  v = PyObject_CallMethodNoArgs(o, s_data_ptr);
  if (!v && PyErr_ExceptionMatches(PyExc_AttributeError)) { /* another array */
    PyObject* c;
    PyErr_Clear();
    c = PyObject_GetAttr(o, s_ctypes);
    if (c) {
      v = PyObject_GetAttr(c, s_data);
      Py_DECREF(c);
    } else if (PyErr_ExceptionMatches(PyExc_AttributeError)) {
      PyErr_Clear();
      PyErr_SetObject(PyExc_TypeError, (PyObject*)Py_TYPE(o));
    }
  }
  if (!v) {
    a->bad = 1;
    return NULL;
  }
  if (!PyLong_Check(v)) {
    PyErr_SetString(PyExc_TypeError, "an address is an int");
    a->bad = 1;
    Py_DECREF(v);
    return NULL;
  }
  p = mask_ptr(v, a);
  Py_DECREF(v);
  return p;
}
/* what is no plain number: a ctypes scalar or an object that stands for one, or a TypeError */
static PyObject* number_of(PyObject* o, int kind, Args* a) {
  PyObject* v = get_number ? PyObject_CallFunction(get_number, "iO", kind, o) : NULL;
  if (!v) {
    if (!PyErr_Occurred()) PyErr_Format(PyExc_TypeError, "a number is expected, not %s", Py_TYPE(o)->tp_name);
    a->bad = 1;
  }
  return v;
}
static int64_t arg_int(Args* a, int kind) {
  PyObject* o = *a->at++;
  int64_t v;
  if (a->bad) return 0;
  if (PyLong_Check(o)) {
    Py_INCREF(o);
  } else if (!(o = number_of(o, kind, a))) {
    return 0;
  }
  v = (int64_t)PyLong_AsUnsignedLongLongMask(o);
  if (PyErr_Occurred()) a->bad = 1;
  Py_DECREF(o);
  return v;
}
static int64_t arg_i64(Args* a) { return arg_int(a, KIND_I64); }
static int32_t arg_i32(Args* a) { return (int32_t)arg_int(a, KIND_I32); }
static float arg_f32(Args* a) {
  PyObject* o = *a->at++;
  double v;
  if (a->bad) return 0.f;
  v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) {
    if (!PyErr_ExceptionMatches(PyExc_TypeError)) {
      a->bad = 1;
      return 0.f;
    }
    PyErr_Clear();
    if (!(o = number_of(o, KIND_F32, a))) return 0.f;
    v = PyFloat_AsDouble(o);
    if (PyErr_Occurred()) a->bad = 1;
    Py_DECREF(o);
  }
  return (float)v;
}
/* the layout is copied: nothing of the caller's is held while the GIL is released */
static kpx_kv_layout arg_layout(Args* a) {
  PyObject* o = *a->at++;
  kpx_kv_layout l = {0};
  Py_buffer view;
  if (a->bad) return l;
  if (!layout_type || !PyObject_TypeCheck(o, (PyTypeObject*)layout_type)) { /* (not any bytes of its size) */
    PyErr_Format(PyExc_TypeError, "a KvLayout is expected, not %s", Py_TYPE(o)->tp_name);
    a->bad = 1;
    return l;
  }
  if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0) {
    a->bad = 1;
    return l;
  }
  if (view.len >= (Py_ssize_t)sizeof l) {
    memcpy(&l, view.buf, sizeof l);
  } else {
    PyErr_SetString(PyExc_TypeError, "a KvLayout is expected");
    a->bad = 1;
  }
  PyBuffer_Release(&view);
  return l;
}
/* None: the current stream of the current device */
static void* arg_stream(Args* a) {
  PyObject *o = *a->at++, *dev, *s;
  void* p;
  if (a->bad) return NULL;
  if (o != Py_None) {
    PyObject* n = PyNumber_Long(o);
    if (!n) {
      a->bad = 1;
      return NULL;
    }
    p = mask_ptr(n, a);
    Py_DECREF(n);
    return p;
  }
  dev = get_device ? PyObject_CallNoArgs(get_device) : NULL;
  s = dev ? PyObject_CallOneArg(get_stream, dev) : NULL;
  Py_XDECREF(dev);
  if (!s) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "no source of the current stream");
    a->bad = 1;
    return NULL;
  }
  p = mask_ptr(s, a);
  Py_DECREF(s);
  return p;
}

/* One entry point: its arguments in order, then the call. */
#define ENTRY(name, count, convert, call)                                                            \
  static PyObject* py_##name(PyObject* self, PyObject* const* argv, Py_ssize_t argc) {               \
    Args a = {argv, 0};                                                                              \
    int rc;                                                                                          \
    (void)self;                                                                                      \
    if (argc != count) {                                                                             \
      PyErr_Format(PyExc_TypeError, #name ": %d arguments expected, not %zd", count, argc);          \
      return NULL;                                                                                   \
    }                                                                                                \
    convert;                                                                                         \
    if (a.bad) return NULL;                                                                          \
    Py_BEGIN_ALLOW_THREADS rc = call;                                                                \
    Py_END_ALLOW_THREADS return PyLong_FromLong(rc);                                                 \
  }
#define P(x) void* x = arg_ptr(&a)
#define I(x) int32_t x = arg_i32(&a)
#define Q(x) int64_t x = arg_i64(&a)
#define F(x) float x = arg_f32(&a)
#define L(x) kpx_kv_layout x = arg_layout(&a)
#define S(x) void* x = arg_stream(&a)

ENTRY(append, 10, P(kp); P(vp); L(lay); P(k); P(v); P(slots); P(pos); I(bias); I(n); S(s),
      kpx_append(kp, vp, &lay, k, v, slots, pos, bias, n, s))
ENTRY(rope_append, 14, P(q); P(k); P(v); I(h); P(pos); I(base); P(sn); P(cs); P(kp); P(vp); L(lay); P(slots); I(n); S(s),
      kpx_rope_append(q, k, v, h, pos, base, sn, cs, kp, vp, &lay, slots, n, s))
ENTRY(norm_rope_append, 17, P(q); P(k); P(v); I(h); P(qw); P(kw); F(eps); P(pos); I(base); P(sn); P(cs); P(kp); P(vp);
      L(lay); P(slots); I(n); S(s),
      kpx_norm_rope_append(q, k, v, h, qw, kw, eps, pos, base, sn, cs, kp, vp, &lay, slots, n, s))
ENTRY(paged_decode, 15, P(out); P(q); P(kp); P(vp); L(lay); P(table); I(width); P(lens); I(bias); I(batch); I(h); F(scale);
      P(ws); Q(wsb); S(s), kpx_paged_decode(out, q, kp, vp, &lay, table, width, lens, bias, batch, h, scale, ws, wsb, s))
ENTRY(paged_decode_overlapped, 15, P(out); P(q); P(kp); P(vp); L(lay); P(table); I(width); P(lens); I(bias); I(batch); I(h);
      F(scale); P(ws); Q(wsb); S(s),
      kpx_paged_decode_overlapped(out, q, kp, vp, &lay, table, width, lens, bias, batch, h, scale, ws, wsb, s))
ENTRY(paged_decode_planned, 17, P(out); P(q); P(kp); P(vp); L(lay); P(table); I(width); P(lens); I(bias); I(batch); I(h);
      F(scale); P(ws); Q(wsb); P(plan); I(flags); S(s),
      kpx_paged_decode_planned(out, q, kp, vp, &lay, table, width, lens, bias, batch, h, scale, ws, wsb, plan, flags, s))
ENTRY(decode_plan, 10, P(plan); Q(bytes); L(lay); P(table); I(width); P(lens); I(bias); I(batch); I(h); S(s),
      kpx_decode_plan(plan, bytes, &lay, table, width, lens, bias, batch, h, s))
ENTRY(rope_append_decode, 19, P(out); P(q); P(k); P(v); P(sn); P(cs); P(kp); P(vp); L(lay); P(table); I(width); P(pos);
      I(batch); I(h); F(scale); P(ws); Q(wsb); I(flags); S(s),
      kpx_rope_append_decode(out, q, k, v, sn, cs, kp, vp, &lay, table, width, pos, batch, h, scale, ws, wsb, flags, s))
ENTRY(paged_prefill, 15, P(out); P(q); P(kp); P(vp); L(lay); P(table); I(width); P(cu); P(start); I(batch); I(h); F(scale);
      P(ws); Q(wsb); S(s), kpx_paged_prefill(out, q, kp, vp, &lay, table, width, cu, start, batch, h, scale, ws, wsb, s))

static PyObject* set_stream_source(PyObject* self, PyObject* args) {
  PyObject *dev, *stream;
  (void)self;
  if (!PyArg_ParseTuple(args, "OO", &dev, &stream)) return NULL;
  Py_XSETREF(get_device, Py_NewRef(dev));
  Py_XSETREF(get_stream, Py_NewRef(stream));
  Py_RETURN_NONE;
}

static PyObject* set_layout_type(PyObject* self, PyObject* type) {
  (void)self;
  if (!PyType_Check(type)) {
    PyErr_SetString(PyExc_TypeError, "a type is expected");
    return NULL;
  }
  Py_XSETREF(layout_type, Py_NewRef(type));
  Py_RETURN_NONE;
}

static PyObject* set_number_source(PyObject* self, PyObject* source) {
  (void)self;
  Py_XSETREF(get_number, Py_NewRef(source));
  Py_RETURN_NONE;
}

#define METHOD(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {METHOD(append), METHOD(rope_append), METHOD(norm_rope_append), METHOD(paged_decode),
                                METHOD(paged_decode_overlapped), METHOD(paged_decode_planned), METHOD(decode_plan),
                                METHOD(rope_append_decode), METHOD(paged_prefill),
                                {"set_stream_source", set_stream_source, METH_VARARGS,
                                 "(current device, raw stream of a device): what a stream of None stands for"},
                                {"set_layout_type", set_layout_type, METH_O, "the type that a layout argument is of"},
                                {"set_number_source", set_number_source, METH_O,
                                 "(0 int32, 1 int64, 2 float; object): the number that the object stands for"},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_kpx_py", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__kpx_py(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_ctypes = PyUnicode_InternFromString("ctypes");
  s_data = PyUnicode_InternFromString("data");
  if (!s_data_ptr || !s_ctypes || !s_data) return NULL;
  return PyModule_Create(&module);
}
