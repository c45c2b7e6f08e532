/* The calls a serving loop makes, as a CPython extension over the C ABI
 * (include/fbgemm_b200/embedding_c_api.h).  ctypes converts every argument
 * through Python objects; with tensor addresses and stream handles that was
 * 8 us of the 12 us a launch took.  Tensors are passed as they are: their
 * address is taken here, after the check that they are contiguous. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "fbgemm_b200/embedding_c_api.h"

static PyObject *s_data_ptr, *s_is_contiguous;

/* Address of a tensor (or an address as an int, or None = null). */
static int address_of(PyObject* x, void** p) {
  if (x == Py_None) {
    *p = NULL;
    return 0;
  }
  PyObject* a;
  if (PyLong_CheckExact(x)) {
    a = Py_NewRef(x);
  } else {
    PyObject* c = PyObject_CallMethodNoArgs(x, s_is_contiguous);
    if (!c) {
      return -1;
    }
    const int contiguous = PyObject_IsTrue(c);
    Py_DECREF(c);
    if (contiguous <= 0) {
      if (contiguous == 0) {
        PyErr_SetString(PyExc_AssertionError, "tensors must be contiguous");
      }
      return -1;
    }
    a = PyObject_CallMethodNoArgs(x, s_data_ptr);
    if (!a) {
      return -1;
    }
  }
  *p = PyLong_AsVoidPtr(a);
  Py_DECREF(a);
  return *p == NULL && PyErr_Occurred() ? -1 : 0;
}

static int addresses(PyObject* const* args, int first, int n, void** p) {
  for (int i = 0; i < n; ++i) {
    if (address_of(args[first + i], &p[i])) {
      return -1;
    }
  }
  return 0;
}

static int integers(PyObject* const* args, int first, int n, int64_t* v) {
  for (int i = 0; i < n; ++i) {
    v[i] = PyLong_AsLongLong(args[first + i]);
    if (v[i] == -1 && PyErr_Occurred()) {
      return -1;
    }
  }
  return 0;
}

static int arity(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) {
    PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, got);
    return -1;
  }
  return 0;
}

/* spmdm_launch(ctx, cfg, output_size, index_size, data_size, input, indices, offsets, weights, out, map, slot, stream) */
static PyObject* spmdm_launch(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void *h[2], *t[6], *stream;
  int64_t size[3], slot;
  if (arity(n, 13) || addresses(args, 0, 2, h) || integers(args, 2, 3, size) || addresses(args, 5, 6, t) ||
      integers(args, 11, 1, &slot) || addresses(args, 12, 1, &stream)) {
    return NULL;
  }
  return PyLong_FromLong(fbgemm_b200_spmdm_launch(h[0], h[1], size[0], size[1], size[2], t[0], t[1], t[2], t[3], t[4], t[5],
                                                  (int)slot, stream));
}

/* spmdm(ctx, cfg, output_size, index_size, data_size, input, indices, offsets, weights, out, map, stream): waits */
static PyObject* spmdm(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void *h[2], *t[6], *stream;
  int64_t size[3];
  if (arity(n, 12) || addresses(args, 0, 2, h) || integers(args, 2, 3, size) || addresses(args, 5, 6, t) ||
      addresses(args, 11, 1, &stream)) {
    return NULL;
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = fbgemm_b200_spmdm(h[0], h[1], size[0], size[1], size[2], t[0], t[1], t[2], t[3], t[4], t[5], stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

/* table_set_forward(set, bags, indices, index_size, offsets, weights, out, slot, stream) */
static PyObject* table_set_forward(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void *set, *indices, *t[3], *stream;
  int64_t bags, index_size, slot;
  if (arity(n, 9) || addresses(args, 0, 1, &set) || integers(args, 1, 1, &bags) || addresses(args, 2, 1, &indices) ||
      integers(args, 3, 1, &index_size) || addresses(args, 4, 3, t) || integers(args, 7, 1, &slot) ||
      addresses(args, 8, 1, &stream)) {
    return NULL;
  }
  return PyLong_FromLong(fbgemm_b200_table_set_forward(set, bags, indices, index_size, t[0], t[1], t[2], (int)slot, stream));
}

static PyMethodDef methods[] = {
    {"spmdm_launch", (PyCFunction)(void (*)(void))spmdm_launch, METH_FASTCALL, "fbgemm_b200_spmdm_launch"},
    {"spmdm", (PyCFunction)(void (*)(void))spmdm, METH_FASTCALL, "fbgemm_b200_spmdm"},
    {"table_set_forward", (PyCFunction)(void (*)(void))table_set_forward, METH_FASTCALL, "fbgemm_b200_table_set_forward"},
    {NULL, NULL, 0, NULL}};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__native_calls(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
  return s_data_ptr && s_is_contiguous ? PyModule_Create(&module) : NULL;
}
