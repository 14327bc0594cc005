/* The hot call of the Python binding without ctypes: one fused linear, its constant arguments in a record.  A call through
 * ctypes converts thirteen arguments, about 3 us of a 9 us call; here it is an array of integers. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

typedef int (*gemm_next_fn)(const void* image, const void* header, const void* x, int64_t ldx, uint32_t m, void* y, int64_t ldy, const void* bias,
                            void* workspace, uint64_t workspace_bytes, uint32_t* status, void* stream, const void* next_image,
                            const void* next_header);

/* Filled by georefine_b200/resident.py (LinearRecord). */
typedef struct {
  gemm_next_fn entry;   /* grb_bxr_gemm_next */
  const void* image;
  const void* header;
  void* workspace;
  uint64_t workspace_bytes;
  uint32_t* status;
  const void* next_image;
  const void* next_header;
} linear_record;

/* gemm(record, x, ldx, m, y, ldy, bias, stream) -> status; addresses as integers, 0 for none. */
static PyObject* gemm(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  uint64_t v[8];
  (void)self;
  if (n != 8) {
    PyErr_SetString(PyExc_TypeError, "gemm takes 8 arguments");
    return NULL;
  }
  for (int i = 0; i < 8; ++i) {
    v[i] = PyLong_AsUnsignedLongLong(args[i]);
    if (v[i] == (uint64_t)-1 && PyErr_Occurred()) return NULL;
  }
  const linear_record* r = (const linear_record*)(uintptr_t)v[0];
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = r->entry(r->image, r->header, (const void*)(uintptr_t)v[1], (int64_t)v[2], (uint32_t)v[3], (void*)(uintptr_t)v[4], (int64_t)v[5],
                    (const void*)(uintptr_t)v[6], r->workspace, r->workspace_bytes, r->status, (void*)(uintptr_t)v[7], r->next_image, r->next_header);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(status);
}

static PyMethodDef methods[] = {{"gemm", (PyCFunction)(void (*)(void))gemm, METH_FASTCALL, "one fused linear"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&module); }
