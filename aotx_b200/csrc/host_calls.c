/* The entry points that a decode step calls most, from Python without ctypes: converting twelve arguments there takes
 * 1.6 us, a third of what the host spends on a product; here 0.2.  The caller gives the function's address (the
 * library's, of whichever library is loaded) and its arguments as integers, None for a null pointer and for nothing else;
 * integers are taken modulo their width, as ctypes takes them.  The interpreter's lock is released during the call. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include "../../include/aotx_q8_b200.h"

/* `kinds`: a letter per argument, p a pointer, n a number. */
static int take(PyObject *const *args, Py_ssize_t count, const char *kinds, uint64_t *values)
{
    const Py_ssize_t want = (Py_ssize_t)strlen(kinds);
    if (count != want) {
        PyErr_Format(PyExc_TypeError, "%zd arguments, not %zd", want, count);
        return 0;
    }
    for (Py_ssize_t i = 0; i < count; ++i) {
        if (args[i] == Py_None && kinds[i] == 'p') {
            values[i] = 0;
            continue;
        }
        values[i] = PyLong_AsUnsignedLongLongMask(args[i]);      /* (a TypeError for what is no integer) */
        if (values[i] == (uint64_t)-1 && PyErr_Occurred() != NULL) {
            return 0;
        }
    }
    if (values[0] == 0) {
        PyErr_SetString(PyExc_TypeError, "no function");
        return 0;
    }
    return 1;
}

#define PTR(i) ((void *)(uintptr_t)v[i])

static PyObject *call_matmul(PyObject *self, PyObject *const *args, Py_ssize_t count)
{
    uint64_t v[13];
    int code;
    (void)self;
    if (!take(args, count, "ppppnnnpnnppn", v)) {
        return NULL;
    }
    Py_BEGIN_ALLOW_THREADS
    code = ((__typeof__(&aotx_q8_matmul))PTR(0))(PTR(1), PTR(2), PTR(3), (uint32_t)v[4], (uint32_t)v[5], (uint32_t)v[6], PTR(7),
                                                 (int)v[8], (uint32_t)v[9], PTR(10), PTR(11), (int)v[12]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

static PyObject *call_matmul_fused(PyObject *self, PyObject *const *args, Py_ssize_t count)
{
    uint64_t v[14];
    int code;
    (void)self;
    if (!take(args, count, "ppppnnnpnnppnn", v)) {
        return NULL;
    }
    Py_BEGIN_ALLOW_THREADS
    code = ((__typeof__(&aotx_q8_matmul_fused))PTR(0))(PTR(1), PTR(2), PTR(3), (uint32_t)v[4], (uint32_t)v[5], (uint32_t)v[6], PTR(7),
                                                       (int)v[8], (uint32_t)v[9], PTR(10), PTR(11), (int)v[12], (int)v[13]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

static PyObject *call_dequant(PyObject *self, PyObject *const *args, Py_ssize_t count)
{
    uint64_t v[9];
    int code;
    (void)self;
    if (!take(args, count, "ppppnnnnp", v)) {
        return NULL;
    }
    Py_BEGIN_ALLOW_THREADS
    code = ((__typeof__(&aotx_q8_dequant))PTR(0))(PTR(1), PTR(2), PTR(3), (uint32_t)v[4], (uint32_t)v[5], (uint32_t)v[6],
                                                  (uint32_t)v[7], PTR(8));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

static PyMethodDef methods[] = {
    {"aotx_q8_matmul", (PyCFunction)(void (*)(void))call_matmul, METH_FASTCALL, "address, then aotx_q8_matmul's arguments"},
    {"aotx_q8_matmul_fused", (PyCFunction)(void (*)(void))call_matmul_fused, METH_FASTCALL,
     "address, then aotx_q8_matmul_fused's arguments"},
    {"aotx_q8_dequant", (PyCFunction)(void (*)(void))call_dequant, METH_FASTCALL, "address, then aotx_q8_dequant's arguments"},
    {NULL, NULL, 0, NULL},
};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__host_calls(void)
{
    return PyModule_Create(&module);
}
