// Host code: whole numbers out of Python lists into one buffer of 32-bit integers, as one native call.
//
// The sampler's inputs of a step (request and draw indices, a window of recent tokens for each row) are lists of Python
// integers.  For a batch of 64 they take 29 us read one by one through the interpreter's own functions, and 72 us flattened
// by the interpreter and packed by `struct`.  Called with the interpreter's lock held (ctypes.PyDLL).
// Only functions of the interpreter's stable interface are used, declared here: its headers are not needed to build.
#include <stdint.h>

#include "common.cuh"

extern "C" {
typedef struct _object PyObject;
intptr_t PyList_Size(PyObject*);
PyObject* PyList_GetItem(PyObject*, intptr_t);    // borrowed
long PyLong_AsLong(PyObject*);
PyObject* PyErr_Occurred(void);
void PyErr_Clear(void);
PyObject* PyObject_Type(PyObject*);               // owned
void Py_DecRef(PyObject*);
extern struct _typeobject PyList_Type;
}

namespace {
// numbers [from, n) of a list; false (and no error left behind) where it is no list or holds anything else
bool numbers(PyObject* list, intptr_t from, intptr_t n, int32_t* out) {
  for (intptr_t i = from; i < n; ++i) {
    PyObject* item = PyList_GetItem(list, i);           // (a conversion may run Python code, which may shorten the list)
    const long v = item != nullptr ? PyLong_AsLong(item) : -1;
    if (item == nullptr || (v == -1 && PyErr_Occurred() != nullptr)) {
      PyErr_Clear();
      return false;
    }
    if (v < INT32_MIN || v > INT32_MAX) return false;
    out[i - from] = (int32_t)v;
  }
  return true;
}
// -1 where it is no list, or one of a class of its own, which may give other numbers when it is iterated
intptr_t size_of(PyObject* o) {
  PyObject* type = PyObject_Type(o);
  if (type != nullptr) Py_DecRef(type);
  const intptr_t n = type == (PyObject*)&PyList_Type ? PyList_Size(o) : -1;
  if (n < 0) PyErr_Clear();
  return n;
}
}  // namespace

// `parts`: a list of lists, one after another; then of each list of `rows` its last `width` numbers, -1 behind a shorter
// one.  1: `out`, of `room` numbers, is filled.  0: not lists of whole numbers of 32 bits, or another count.
DLGO_EXPORT int dlgo_pack_rows(PyObject* parts, PyObject* rows, int width, int32_t* out, long long room) {
  const intptr_t n_parts = size_of(parts), n_rows = size_of(rows);
  if (n_parts < 0 || n_rows < 0 || width < 0) return 0;
  long long at = 0;
  for (intptr_t i = 0; i < n_parts; ++i) {
    PyObject* p = PyList_GetItem(parts, i);
    const intptr_t n = p != nullptr ? size_of(p) : -1;
    if (n < 0 || at + n > room || !numbers(p, 0, n, out + at)) return 0;
    at += n;
  }
  for (intptr_t i = 0; i < n_rows; ++i) {
    PyObject* r = PyList_GetItem(rows, i);
    const intptr_t n = r != nullptr ? size_of(r) : -1, from = n > width ? n - width : 0;
    if (n < 0 || at + width > room || !numbers(r, from, n, out + at)) return 0;
    for (intptr_t j = n - from; j < width; ++j) out[at + j] = -1;
    at += width;
  }
  return at == room ? 1 : 0;
}
