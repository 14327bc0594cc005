/* The hot call of the Python binding without ctypes: one fused linear.  ctypes converts its arguments one by one through
 * the declared types, about 3 us of a 9 us call; here they are seventeen integers. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

typedef int (*gemm_partials_fn)(const void* image, const void* header, const void* x, int64_t ldx, uint32_t m, void* y, int64_t ldy,
                                const void* bias, void* workspace, uint64_t workspace_bytes, void* partials, uint64_t partials_bytes,
                                uint32_t* status, void* stream, const void* next_image, const void* next_header);

/* gemm_partials(entry, <the arguments of grb_bxr_gemm_partials in their order>) -> status; addresses as integers, 0 for none. */
static PyObject* gemm_partials(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  uint64_t v[17];
  (void)self;
  if (n != 17) {
    PyErr_SetString(PyExc_TypeError, "gemm_partials takes 17 arguments");
    return NULL;
  }
  for (int i = 0; i < 17; ++i) {
    v[i] = PyLong_AsUnsignedLongLong(args[i]);
    if (v[i] == (uint64_t)-1 && PyErr_Occurred()) return NULL;
  }
#define ADDRESS(i) ((void*)(uintptr_t)v[i])
  const gemm_partials_fn entry = (gemm_partials_fn)(uintptr_t)v[0];
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = entry(ADDRESS(1), ADDRESS(2), ADDRESS(3), (int64_t)v[4], (uint32_t)v[5], ADDRESS(6), (int64_t)v[7], ADDRESS(8), ADDRESS(9), v[10],
                 ADDRESS(11), v[12], (uint32_t*)ADDRESS(13), ADDRESS(14), ADDRESS(15), ADDRESS(16));
  Py_END_ALLOW_THREADS
#undef ADDRESS
  return PyLong_FromLong(status);
}

static PyMethodDef methods[] = {{"gemm_partials", (PyCFunction)(void (*)(void))gemm_partials, METH_FASTCALL, "one fused linear"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&module); }
