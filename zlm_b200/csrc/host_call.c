/* Calls the library's entry points from Python with plain numbers as arguments.
 *
 * A launch through ctypes costs the host an object per argument and a description of the call made anew each time: about 4 us
 * of the 13 that a launch took, as much as the launch itself.  All entry points are C functions of integers and pointers (one
 * 8-byte place each, whatever their width) and at most 8 floats, and return an int.  The platform's calling convention passes
 * these two kinds in registers of their own, the integers that find no register on the stack in their order; so one function
 * type with enough places of both kinds calls all of them, and places beyond an entry point's own are not looked at.  This
 * holds for the System V convention on x86-64 and for AArch64; elsewhere, or without Python's headers, the package goes
 * through ctypes.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <string.h>

#if !defined(__linux__) || !(defined(__x86_64__) || defined(__aarch64__))
#error "the calling convention is not one of those described above"
#endif

#define MAX_INTS 64
#define MAX_FLOATS 8

typedef long long L;
typedef int (*Entry)(L, L, L, L, L, L, L, L, double, double, double, double, double, double, double, double, L, L, L, L, L, L, L, L,
                     L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L,
                     L, L, L, L, L, L, L, L);

static PyObject *value_name;

/* one argument: None is 0, an int (or bool) a place; an object of ctypes counts as its value, a c_float's in 32 bits; a bare
 * Python float is refused, as ctypes refuses it where an integer belongs */
static int take(PyObject *a, L *ints, int *ni, double *floats, int *nf) {
    if (PyLong_Check(a)) {
        if (*ni == MAX_INTS) { PyErr_SetString(PyExc_TypeError, "too many integer arguments"); return -1; }
        L v = PyLong_AsLongLong(a);
        if (v == -1 && PyErr_Occurred()) {
            PyErr_Clear();
            v = (L)PyLong_AsUnsignedLongLong(a);
            if (PyErr_Occurred()) return -1;
        }
        ints[(*ni)++] = v;
        return 0;
    }
    if (a == Py_None) {
        if (*ni == MAX_INTS) { PyErr_SetString(PyExc_TypeError, "too many integer arguments"); return -1; }
        ints[(*ni)++] = 0;
        return 0;
    }
    PyObject *v = PyIndex_Check(a) ? PyNumber_Index(a) : PyObject_GetAttr(a, value_name);
    if (!v) {
        if (PyErr_ExceptionMatches(PyExc_AttributeError)) PyErr_Format(PyExc_TypeError, "an argument of type %s", Py_TYPE(a)->tp_name);
        return -1;
    }
    int rc = 0;
    if (PyFloat_Check(v)) {                              /* (a c_float's value) */
        if (*nf == MAX_FLOATS) {
            PyErr_SetString(PyExc_TypeError, "too many float arguments");
            rc = -1;
        } else {
            const float f = (float)PyFloat_AS_DOUBLE(v);
            floats[*nf] = 0.0;
            memcpy(&floats[*nf], &f, sizeof f);          /* (a float argument is the low half of its register) */
            ++*nf;
        }
    } else if (PyLong_Check(v) || v == Py_None) {
        rc = take(v, ints, ni, floats, nf);
    } else {
        PyErr_Format(PyExc_TypeError, "an argument of type %s", Py_TYPE(a)->tp_name);
        rc = -1;
    }
    Py_DECREF(v);
    return rc;
}

/* call(address, *arguments) -> int */
static PyObject *call(PyObject *self, PyObject *const *args, Py_ssize_t n) {
    L i[MAX_INTS] = {0};
    double f[MAX_FLOATS] = {0};
    int ni = 0, nf = 0, rc;
    if (n < 1) { PyErr_SetString(PyExc_TypeError, "call(address, *arguments)"); return NULL; }
    const Entry entry = (Entry)PyLong_AsVoidPtr(args[0]);
    if (!entry) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "no function at address 0"); return NULL; }
    for (Py_ssize_t k = 1; k < n; ++k)
        if (take(args[k], i, &ni, f, &nf)) return NULL;
    Py_BEGIN_ALLOW_THREADS
    rc = entry(i[0], i[1], i[2], i[3], i[4], i[5], i[6], i[7], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], i[8], i[9], i[10], i[11],
               i[12], i[13], i[14], i[15], i[16], i[17], i[18], i[19], i[20], i[21], i[22], i[23], i[24], i[25], i[26], i[27], i[28],
               i[29], i[30], i[31], i[32], i[33], i[34], i[35], i[36], i[37], i[38], i[39], i[40], i[41], i[42], i[43], i[44], i[45],
               i[46], i[47], i[48], i[49], i[50], i[51], i[52], i[53], i[54], i[55], i[56], i[57], i[58], i[59], i[60], i[61], i[62],
               i[63]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {
    {"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, "call(address, *arguments) -> int"},
    {NULL, NULL, 0, NULL},
};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "zlm_host_call", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit_zlm_host_call(void) {
    value_name = PyUnicode_InternFromString("value");
    return value_name ? PyModule_Create(&module) : NULL;
}
