/* Calls of the C ABI without ctypes. A ctypes call of nine arguments costs 1.3 us in conversions, a
 * tenth of a small operator's whole call; a bound function here costs 0.1. bind(address, kinds)
 * gives a callable for a function that returns int (size_t where `kinds` starts with ">") and takes,
 * per character of `kinds`, an integer or pointer ("i": int, or None for NULL) or a float ("f"). Integer and floating
 * arguments travel in registers of their own (System V x86-64), so one prototype with all integers
 * in front of all floats calls every signature. The GIL is released during the call. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include "../../include/megcc_b200.h"

#if !defined(__x86_64__) || defined(_WIN32)
#error "the argument passing above is that of System V x86-64"
#endif

#define MAX_INTS 16
#define MAX_FLOATS 8

typedef uint64_t (*any_fn)(
        uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
        uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, float, float, float,
        float, float, float, float, float);

typedef struct {
    any_fn fn;
    int n, wide;
    char kinds[MAX_INTS + MAX_FLOATS];
} bound;

static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    const bound* b = (const bound*)PyBytes_AS_STRING(self);
    uint64_t v[MAX_INTS] = {0};
    float f[MAX_FLOATS] = {0};
    int ni = 0, nf = 0;
    uint64_t r;
    if (n != b->n) {
        PyErr_Format(PyExc_TypeError, "the function takes %d arguments (%zd given)", b->n, n);
        return NULL;
    }
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* a = args[i];
        if (b->kinds[i] == 'f') {
            const double d = PyFloat_AsDouble(a);
            if (d == -1.0 && PyErr_Occurred())
                return NULL;
            f[nf++] = (float)d;
        } else if (a == Py_None) {
            ++ni;
        } else if (PyLong_Check(a)) {
            v[ni] = PyLong_AsUnsignedLongLongMask(a);
            if (v[ni++] == (uint64_t)-1 && PyErr_Occurred())
                return NULL;
        } else {
            PyErr_Format(PyExc_TypeError, "argument %zd must be an int or None, not %s", i + 1,
                         Py_TYPE(a)->tp_name);
            return NULL;
        }
    }
    Py_BEGIN_ALLOW_THREADS
    r = b->fn(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12],
              v[13], v[14], v[15], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
    Py_END_ALLOW_THREADS
    /* (an int leaves the upper half of the register undefined) */
    return b->wide ? PyLong_FromUnsignedLongLong(r) : PyLong_FromLong((long)(int)(uint32_t)r);
}

static PyMethodDef call_def = {"bound", (PyCFunction)(void*)call, METH_FASTCALL, NULL};

static PyObject* bind(PyObject* self, PyObject* args) {
    unsigned long long address;
    const char* kinds;
    bound b;
    int ni = 0, nf = 0;
    (void)self;
    if (!PyArg_ParseTuple(args, "Ks", &address, &kinds))
        return NULL;
    memset(&b, 0, sizeof(b));
    if (*kinds == '>') {
        b.wide = 1;
        ++kinds;
    }
    for (; kinds[b.n]; ++b.n) {
        if (kinds[b.n] == 'f')
            ++nf;
        else
            ++ni;
        if (ni > MAX_INTS || nf > MAX_FLOATS) {
            PyErr_SetString(PyExc_ValueError, "too many arguments");
            return NULL;
        }
        b.kinds[b.n] = kinds[b.n];
    }
    b.fn = (any_fn)(uintptr_t)address;
    PyObject* state = PyBytes_FromStringAndSize((const char*)&b, sizeof(b));
    if (!state)
        return NULL;
    PyObject* fn = PyCFunction_New(&call_def, state);
    Py_DECREF(state);
    return fn;
}

static long floor_div(long a, long b) {
    const long q = a / b;
    return q - (a % b != 0 && (a < 0) != (b < 0));
}

/* (n, oh, ow, oc) of the mb200_conv_param at an address */
static PyObject* conv_shape(PyObject* self, PyObject* at) {
    const unsigned long long address = PyLong_AsUnsignedLongLong(at);
    (void)self;
    if (address == (unsigned long long)-1 && PyErr_Occurred())
        return NULL;
    const mb200_conv_param* p = (const mb200_conv_param*)(uintptr_t)address;
    if (p->stride_h == 0 || p->stride_w == 0) {
        PyErr_SetString(PyExc_ZeroDivisionError, "convolution stride is zero");
        return NULL;
    }
    return Py_BuildValue(
            "illi", p->n,
            floor_div((long)p->ih + 2L * p->pad_h - (long)p->dilate_h * (p->kh - 1) - 1, p->stride_h) + 1,
            floor_div((long)p->iw + 2L * p->pad_w - (long)p->dilate_w * (p->kw - 1) - 1, p->stride_w) + 1,
            p->oc);
}

static PyMethodDef methods[] = {
        {"bind", bind, METH_VARARGS, "bind(address, kinds) -> callable"},
        {"conv_shape", conv_shape, METH_O, "conv_shape(address of a conv_param) -> (n, oh, ow, oc)"},
        {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods,
                                    NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void) {
    return PyModule_Create(&module);
}
