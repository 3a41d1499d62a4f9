/* The operator call as a CPython function.  lutamm_amm() on tensors of a few hundred rows takes the GPU less than the
 * host: through ctypes the binding alone (argument conversion, four attribute look-ups and two method calls in Python)
 * cost 3 us of a 10 us call.  Same arguments and checks as LutAmmContext.amm_host; anything but tensors - numpy
 * arrays, raw addresses - answers NotImplemented and takes the ctypes way. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

typedef int (*amm_fn)(void*, int, const float*, float*, uint32_t, uint32_t);

static PyObject *s_is_contiguous, *s_data_ptr, *s_shape;

/* Address of a contiguous tensor; 1 on success, 0 if it is no tensor, -1 with an exception set. */
static int address_of(PyObject* t, void** out) {
    PyObject* ok = PyObject_CallMethodNoArgs(t, s_is_contiguous);
    if (!ok) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return -1;
        PyErr_Clear();
        return 0;
    }
    const int contiguous = PyObject_IsTrue(ok);
    Py_DECREF(ok);
    if (contiguous < 0) return -1;
    if (!contiguous) {
        PyErr_SetString(PyExc_AssertionError, "tensors handed to the C ABI must be contiguous");
        return -1;
    }
    PyObject* a = PyObject_CallMethodNoArgs(t, s_data_ptr);
    if (!a) return -1;
    *out = PyLong_AsVoidPtr(a);
    Py_DECREF(a);
    return PyErr_Occurred() ? -1 : 1;
}

/* amm(function address, context address, layer id, input, output, tokens or None, flags) -> return code */
static PyObject* amm(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    (void)self;
    if (n != 7) {
        PyErr_SetString(PyExc_TypeError, "amm takes 7 arguments");
        return NULL;
    }
    const amm_fn fn = (amm_fn)PyLong_AsVoidPtr(args[0]);
    void* ctx = PyLong_AsVoidPtr(args[1]);
    const long layer = PyLong_AsLong(args[2]);
    void *in = NULL, *out = NULL;
    if (PyErr_Occurred()) return NULL;
    int r = address_of(args[3], &in);
    if (r > 0) r = address_of(args[4], &out);
    if (r < 0) return NULL;
    if (r == 0) Py_RETURN_NOTIMPLEMENTED;
    PyObject* rows = NULL;
    if (args[5] == Py_None) {
        PyObject* shape = PyObject_GetAttr(args[3], s_shape);
        if (!shape) return NULL;
        rows = PySequence_GetItem(shape, 0);
        Py_DECREF(shape);
        if (!rows) return NULL;
    }
    PyObject* count = PyNumber_Long(rows ? rows : args[5]);   /* int() of it, as in amm_host */
    Py_XDECREF(rows);
    if (!count) return NULL;
    const unsigned long tokens = PyLong_AsUnsignedLongMask(count);
    Py_DECREF(count);
    const unsigned long flags = PyLong_AsUnsignedLongMask(args[6]);
    if (PyErr_Occurred()) return NULL;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fn(ctx, (int)layer, (const float*)in, (float*)out, (uint32_t)tokens, (uint32_t)flags);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {{"amm", (PyCFunction)(void (*)(void))amm, METH_FASTCALL, "lutamm_amm on two tensors"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void) {
    s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_shape = PyUnicode_InternFromString("shape");
    return PyModule_Create(&module);
}
