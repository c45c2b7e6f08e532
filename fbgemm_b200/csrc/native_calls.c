/* The calls a serving loop makes, as a CPython extension over the C ABI
 * (include/fbgemm_b200/embedding_c_api.h).  ctypes converts every argument
 * through Python objects; with tensor addresses and stream handles that was
 * 8 us of the 12 us a launch took.  Tensors are passed as they are: their
 * address is taken here, after the check that they are contiguous. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "fbgemm_b200/embedding_c_api.h"

static PyObject *s_data_ptr, *s_is_contiguous;

/* Address of a tensor; None = null.  A number is no tensor.  Other arrays (numpy) go by embedding.page_locked_address. */
static int address_of(PyObject* x, void** p) {
  if (x == Py_None) {
    *p = NULL;
    return 0;
  }
  PyObject* c = PyObject_CallMethodNoArgs(x, s_is_contiguous);
  PyObject* a = NULL;
  if (c) {
    const int contiguous = PyObject_IsTrue(c);
    Py_DECREF(c);
    if (contiguous == 0) {
      PyErr_SetString(PyExc_AssertionError, "tensors must be contiguous");
    }
    if (contiguous <= 0) {
      return -1;
    }
    a = PyObject_CallMethodNoArgs(x, s_data_ptr);
  } else if (PyErr_ExceptionMatches(PyExc_AttributeError)) {
    PyErr_Clear();
    PyObject* m = PyImport_ImportModule("fbgemm_b200.embedding");
    if (m) {
      a = PyObject_CallMethod(m, "page_locked_address", "O", x);
      Py_DECREF(m);
    }
  }
  if (!a) {
    return -1;
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

/* Contexts, configurations, table sets and streams: their addresses as numbers; None = null. */
static int handles(PyObject* const* args, int first, int n, void** p) {
  for (int i = 0; i < n; ++i) {
    PyObject* x = args[first + i];
    p[i] = x == Py_None ? NULL : PyLong_AsVoidPtr(x);
    if (p[i] == NULL && PyErr_Occurred()) {
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

/* Runs CALL, which gives an int, without the interpreter's lock: a launch waits when the stream's queue is full, and lengths
 * mode takes the context's lock and may allocate. */
#define WITHOUT_LOCK(CALL)    \
  int rc;                     \
  Py_BEGIN_ALLOW_THREADS      \
  rc = (CALL);                \
  Py_END_ALLOW_THREADS        \
  return PyLong_FromLong(rc)

/* spmdm_launch(ctx, cfg, output_size, index_size, data_size, input, indices, offsets, weights, out, map, slot, stream) */
static PyObject* spmdm_launch(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void *h[2], *t[6], *stream;
  int64_t size[3], slot;
  if (arity(n, 13) || handles(args, 0, 2, h) || integers(args, 2, 3, size) || addresses(args, 5, 6, t) ||
      integers(args, 11, 1, &slot) || handles(args, 12, 1, &stream)) {
    return NULL;
  }
  WITHOUT_LOCK(fbgemm_b200_spmdm_launch(h[0], h[1], size[0], size[1], size[2], t[0], t[1], t[2], t[3], t[4], t[5], (int)slot,
                                        stream));
}

/* spmdm(ctx, cfg, output_size, index_size, data_size, input, indices, offsets, weights, out, map, stream): waits */
static PyObject* spmdm(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void *h[2], *t[6], *stream;
  int64_t size[3];
  if (arity(n, 12) || handles(args, 0, 2, h) || integers(args, 2, 3, size) || addresses(args, 5, 6, t) ||
      handles(args, 11, 1, &stream)) {
    return NULL;
  }
  WITHOUT_LOCK(fbgemm_b200_spmdm(h[0], h[1], size[0], size[1], size[2], t[0], t[1], t[2], t[3], t[4], t[5], stream));
}

/* table_set_forward(set, bags, indices, index_size, offsets, weights, out, slot, stream) */
static PyObject* table_set_forward(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  void *set, *indices, *t[3], *stream;
  int64_t bags, index_size, slot;
  if (arity(n, 9) || handles(args, 0, 1, &set) || integers(args, 1, 1, &bags) || addresses(args, 2, 1, &indices) ||
      integers(args, 3, 1, &index_size) || addresses(args, 4, 3, t) || integers(args, 7, 1, &slot) ||
      handles(args, 8, 1, &stream)) {
    return NULL;
  }
  WITHOUT_LOCK(fbgemm_b200_table_set_forward(set, bags, indices, index_size, t[0], t[1], t[2], (int)slot, stream));
}

/* quantize(bit_rate, x, rows, cols, out, stream); bit_rate 0: 8-bit rows with fp32 scale and bias */
static PyObject* quantize(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  int64_t bits, size[2];
  void *x, *out, *stream;
  if (arity(n, 6) || integers(args, 0, 1, &bits) || addresses(args, 1, 1, &x) || integers(args, 2, 2, size) ||
      addresses(args, 4, 1, &out) || handles(args, 5, 1, &stream)) {
    return NULL;
  }
  WITHOUT_LOCK(bits == 0
                   ? fbgemm_b200_float_to_fused_8bit_rowwise(x, size[0], (int32_t)size[1], out, stream)
                   : fbgemm_b200_float_to_fused_nbit_rowwise((int32_t)bits, x, size[0], (int32_t)size[1], out, stream));
}

/* pruned_lookup(hashmap, ctx, T, B, indices, offsets, index_bytes, index_size, map, map_bytes, map_offsets, dense, slot,
 * stream) */
static PyObject* pruned_lookup(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  int64_t hashmap, size[2], index[2], map_bytes, slot;
  void *ctx, *in[2], *map, *t[2], *stream;
  if (arity(n, 14) || integers(args, 0, 1, &hashmap) || handles(args, 1, 1, &ctx) || integers(args, 2, 2, size) ||
      addresses(args, 4, 2, in) || integers(args, 6, 2, index) || addresses(args, 8, 1, &map) ||
      integers(args, 9, 1, &map_bytes) || addresses(args, 10, 2, t) || integers(args, 12, 1, &slot) ||
      handles(args, 13, 1, &stream)) {
    return NULL;
  }
  WITHOUT_LOCK((hashmap ? fbgemm_b200_pruned_hashmap_lookup : fbgemm_b200_pruned_array_lookup)(
      ctx, (int32_t)size[0], (int32_t)size[1], in[0], in[1], (int32_t)index[0], index[1], map, (int32_t)map_bytes, t[0], t[1],
      (int32_t)slot, stream));
}

/* sequence_lookup(filled, ctx, weights, tables, T, B, D, indices, offsets, index_bytes, index_size, out, out_dtype,
 * out_row_bytes, scale_bias_last, fp8_exponent_bits, fp8_exponent_bias, slot, stream) */
static PyObject* sequence_lookup(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  (void)self;
  int64_t filled, size[3], index[2], out[6];
  void *ctx, *t[2], *in[2], *rows, *stream;
  if (arity(n, 19) || integers(args, 0, 1, &filled) || handles(args, 1, 1, &ctx) || addresses(args, 2, 2, t) ||
      integers(args, 4, 3, size) || addresses(args, 7, 2, in) || integers(args, 9, 2, index) || addresses(args, 11, 1, &rows) ||
      integers(args, 12, 6, out) || handles(args, 18, 1, &stream)) {
    return NULL;
  }
  WITHOUT_LOCK((filled ? fbgemm_b200_sequence_lookup_filled : fbgemm_b200_sequence_lookup)(
      ctx, t[0], t[1], (int32_t)size[0], (int32_t)size[1], (int32_t)size[2], in[0], in[1], (int32_t)index[0], index[1], rows,
      (int32_t)out[0], out[1], (int32_t)out[2], (int32_t)out[3], (int32_t)out[4], (int32_t)out[5], stream));
}

static PyMethodDef methods[] = {
    {"spmdm_launch", (PyCFunction)(void (*)(void))spmdm_launch, METH_FASTCALL, "fbgemm_b200_spmdm_launch"},
    {"spmdm", (PyCFunction)(void (*)(void))spmdm, METH_FASTCALL, "fbgemm_b200_spmdm"},
    {"table_set_forward", (PyCFunction)(void (*)(void))table_set_forward, METH_FASTCALL, "fbgemm_b200_table_set_forward"},
    {"quantize", (PyCFunction)(void (*)(void))quantize, METH_FASTCALL, "fbgemm_b200_float_to_fused_*_rowwise"},
    {"pruned_lookup", (PyCFunction)(void (*)(void))pruned_lookup, METH_FASTCALL, "fbgemm_b200_pruned_*_lookup"},
    {"sequence_lookup", (PyCFunction)(void (*)(void))sequence_lookup, METH_FASTCALL, "fbgemm_b200_sequence_lookup*"},
    {NULL, NULL, 0, NULL}};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__native_calls(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
  return s_data_ptr && s_is_contiguous ? PyModule_Create(&module) : NULL;
}
