/* The entry points that a host with its own forward pass calls for every op of every layer, as functions of a CPython extension module.
 *
 * Through ctypes such a call spends 0.9 us on its way to the library (finding the function, converting six to nine arguments one object at a time), as
 * long as half a kernel launch; here 0.2.  Arguments are taken as ctypes takes them for the declared types: integers modulo 2^32 or 2^64 from anything
 * that is an index; floats from anything that converts; None is a null context.  A call with any other argument (ctypes' own numbers, objects with an
 * _as_parameter_, what nothing takes) goes through ctypes, which takes or refuses it.  The interpreter lock is released during the call, as ctypes does. */

#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#include "yule_cuda.h"

static PyObject *through_ctypes(const char *name, PyObject *const *args, Py_ssize_t n) {
    PyErr_Clear();
    PyObject *module = PyImport_ImportModule("yule_b200._lib"), *lib = module ? PyObject_CallMethod(module, "cuda_lib", NULL) : NULL;
    PyObject *function = lib ? PyObject_GetAttrString(lib, name) : NULL, *rc = function ? PyObject_Vectorcall(function, args, (size_t)n, NULL) : NULL;
    Py_XDECREF(function);
    Py_XDECREF(lib);
    Py_XDECREF(module);
    return rc;
}
static int whole(PyObject *const *args, Py_ssize_t at, uint64_t *to) {
    PyObject *v = args[at], *index = PyLong_Check(v) ? Py_NewRef(v) : PyNumber_Index(v);
    if (!index) return 0;
    *to = PyLong_AsUnsignedLongLongMask(index);
    Py_DECREF(index);
    return 1;
}
static int context(PyObject *const *args, yule_cuda_ctx **to) {
    uint64_t v = 0;
    if (args[0] != Py_None && !whole(args, 0, &v)) return 0;
    *to = (yule_cuda_ctx *)(uintptr_t)v;
    return 1;
}
static int real(PyObject *const *args, Py_ssize_t at, float *to) {
    const double v = PyFloat_AsDouble(args[at]);
    if (v == -1.0 && PyErr_Occurred()) return 0;
    *to = (float)v;
    return 1;
}
static int count(Py_ssize_t got, Py_ssize_t want) {
    if (got == want) return 1;
    PyErr_Format(PyExc_TypeError, "this function takes %zd arguments (%zd given)", want, got);
    return 0;
}

/* `CALL` uses ctx, v[i] (argument i as an integer; FLOAT_AT as f) */
#define ENTRY(NAME, N, FLOAT_AT, CALL)                                            \
    static PyObject *NAME(PyObject *self, PyObject *const *args, Py_ssize_t n) {  \
        yule_cuda_ctx *ctx;                                                       \
        uint64_t v[N] = {0};                                                      \
        float f = 0;                                                              \
        int32_t rc;                                                               \
        (void)self;                                                               \
        if (!count(n, N)) return NULL;                                            \
        int ok = context(args, &ctx);                                             \
        for (Py_ssize_t i = 1; ok && i < N; i++)                                  \
            ok = i == FLOAT_AT ? real(args, i, &f) : whole(args, i, &v[i]);       \
        if (!ok) return through_ctypes("yule_cuda_" #NAME, args, n);              \
        (void)f;                                                                  \
        Py_BEGIN_ALLOW_THREADS rc = CALL;                                         \
        Py_END_ALLOW_THREADS return PyLong_FromLong(rc);                          \
    }
#define U(i) ((uint32_t)v[i])

ENTRY(rms_norm, 6, 5, yule_cuda_rms_norm(ctx, v[1], v[2], v[3], U(4), f))
ENTRY(rope, 8, 5, yule_cuda_rope(ctx, v[1], v[2], U(3), U(4), f, U(6), U(7)))
ENTRY(silu, 4, -1, yule_cuda_silu(ctx, v[1], v[2], U(3)))
ENTRY(element_mul, 5, -1, yule_cuda_element_mul(ctx, v[1], v[2], v[3], U(4)))
ENTRY(add, 5, -1, yule_cuda_add(ctx, v[1], v[2], v[3], U(4)))
ENTRY(copy_buffer, 4, -1, yule_cuda_copy_buffer(ctx, v[1], v[2], (size_t)v[3]))
ENTRY(copy_buffer_offset, 6, -1, yule_cuda_copy_buffer_offset(ctx, v[1], v[2], (size_t)v[3], (size_t)v[4], (size_t)v[5]))
ENTRY(quantized_matmul, 7, -1, yule_cuda_quantized_matmul(ctx, v[1], v[2], v[3], U(4), U(5), U(6)))
ENTRY(quantized_matmul_batched, 10, -1, yule_cuda_quantized_matmul_batched(ctx, v[1], v[2], v[3], U(4), U(5), U(6), U(7), U(8), U(9)))
ENTRY(multihead_attention, 10, -1, yule_cuda_multihead_attention(ctx, v[1], v[2], v[3], v[4], U(5), U(6), U(7), U(8), U(9)))
ENTRY(copy_from_device, 4, -1, yule_cuda_copy_from_device(ctx, v[1], (void *)(uintptr_t)v[2], (size_t)v[3]))

#define METHOD(NAME) {"yule_cuda_" #NAME, (PyCFunction)(void (*)(void))NAME, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {METHOD(rms_norm), METHOD(rope), METHOD(silu), METHOD(element_mul), METHOD(add), METHOD(copy_buffer), METHOD(copy_buffer_offset),
                                METHOD(quantized_matmul), METHOD(quantized_matmul_batched), METHOD(multihead_attention), METHOD(copy_from_device),
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", "Entry points of libyule_cuda.so without ctypes on the way.", -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__calls(void) { return PyModule_Create(&module); }
