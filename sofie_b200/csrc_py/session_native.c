/* The call of an emitted Session's infer trampoline on array buffers. infer() of one event takes about ten microseconds on the
 * device; building the pointers with ctypes took three more on the host. No dependency but Python itself. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

typedef long (*infer_fn)(void *session, void **inputs, void *result, long capacity, char *err, int errlen);

/* infer(function address, session, input array, result array, capacity, error buffer address, its length) -> values written, or a
 * negative number with the message in the error buffer. Raises BufferError for an array that is not contiguous. */
static PyObject *session_infer(PyObject *self, PyObject *const *a, Py_ssize_t n)
{
   (void)self;
   if (n != 7) {
      PyErr_SetString(PyExc_TypeError, "7 arguments are expected");
      return NULL;
   }
   infer_fn fn = (infer_fn)PyLong_AsVoidPtr(a[0]);
   void *session = PyLong_AsVoidPtr(a[1]);
   const long capacity = PyLong_AsLong(a[4]);
   char *err = (char *)PyLong_AsVoidPtr(a[5]);
   const long errlen = PyLong_AsLong(a[6]);
   if (PyErr_Occurred()) return NULL;
   Py_buffer x, y;
   if (PyObject_GetBuffer(a[2], &x, PyBUF_C_CONTIGUOUS) != 0) return NULL;
   if (PyObject_GetBuffer(a[3], &y, PyBUF_C_CONTIGUOUS | PyBUF_WRITABLE) != 0) {
      PyBuffer_Release(&x);
      return NULL;
   }
   long r;
   void *inputs[1] = {x.buf};
   Py_BEGIN_ALLOW_THREADS;
   r = fn(session, inputs, y.buf, capacity, err, (int)errlen);
   Py_END_ALLOW_THREADS;
   PyBuffer_Release(&y);
   PyBuffer_Release(&x);
   return PyLong_FromLong(r);
}

static PyMethodDef methods[] = {{"infer", (PyCFunction)(void (*)(void))session_infer, METH_FASTCALL, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_session", "Calls of emitted Sessions", -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__session(void) { return PyModule_Create(&module); }
