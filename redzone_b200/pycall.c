// pycall.c -- one native call for the Context methods whose C functions share the signature
//   int f(rz_ctx*, void* data, int64_t n, uint32_t elem_bytes, const uint32_t* idx, int64_t k,
//         int64_t* new_len, uint32_t flags, rz_stream_t)
// (rz_remove, rz_remove_host_idx, rz_partition, rz_keep). It reads pointers and sizes off the two
// tensors and calls f without the interpreter lock. Through ctypes the same takes 2.6 us more per
// call, as long as a launch (1000 of 65521 rows, a loop that also slices the result: 7.9 us a pass
// through ctypes, 5.2 with this; 2^16 of 2^28 rows: 8.3 and 7.1).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

typedef int (*list_fn)(void*, void*, int64_t, uint32_t, const uint32_t*, int64_t, int64_t*, uint32_t, void*);

static PyObject *s_shape, *s_data_ptr, *s_numel, *s_element_size;
static PyObject *get_device, *get_stream;  // torch's current device and its raw current stream

// A whole number: an int, or what says that it is one (a numpy integer).
static int whole(PyObject* v, unsigned long long* out) {
    if (PyLong_CheckExact(v)) {
        *out = PyLong_AsUnsignedLongLong(v);
    } else {
        PyObject* i = PyNumber_Index(v);
        if (!i) return -1;
        *out = PyLong_AsUnsignedLongLong(i);
        Py_DECREF(i);
    }
    return *out == (unsigned long long)-1 && PyErr_Occurred() ? -1 : 0;
}

// An integer-valued method of a tensor.
static int ask(PyObject* t, PyObject* method, unsigned long long* out) {
    PyObject* v = PyObject_CallMethodNoArgs(t, method);
    if (!v) return -1;
    const int bad = whole(v, out);
    Py_DECREF(v);
    return bad;
}

// Items of a tensor, and elements per item. Its shape is a tuple, or with other owners of device memory any
// sequence.
static int sizes(PyObject* t, unsigned long long* n, unsigned long long* per) {
    PyObject* dims = PyObject_GetAttr(t, s_shape);
    if (dims && !PyTuple_Check(dims)) {
        PyObject* tuple = PySequence_Tuple(dims);
        Py_DECREF(dims);
        dims = tuple;
    }
    if (!dims) return -1;
    const Py_ssize_t axes = PyTuple_GET_SIZE(dims);
    int bad = 0;
    if (axes < 1) {
        PyErr_SetString(PyExc_IndexError, "the list needs a first axis");
        bad = -1;
    } else {
        bad = whole(PyTuple_GET_ITEM(dims, 0), n);
    }
    *per = 1;
    for (Py_ssize_t i = 1; i < axes && !bad; ++i) {
        unsigned long long d;
        bad = whole(PyTuple_GET_ITEM(dims, i), &d);
        if (!bad) *per *= d;
    }
    Py_DECREF(dims);
    return bad;
}

static int address(PyObject* v, void** out) {
    *out = PyLong_AsVoidPtr(v);
    return PyErr_Occurred() ? -1 : 0;
}

// call(function address, context address, data, idx, flags, stream address or None)
// -> the new length, or minus the status.
static PyObject* call(PyObject* self, PyObject* const* a, Py_ssize_t nargs) {
    (void)self;
    if (nargs != 6) return PyErr_Format(PyExc_TypeError, "call takes 6 arguments");
    void *fn, *ctx, *stream = NULL;
    if (address(a[0], &fn) || address(a[1], &ctx)) return NULL;
    unsigned long long n = 0, per = 1, data, idx, k, elem;
    if (sizes(a[2], &n, &per) || ask(a[2], s_element_size, &elem) || ask(a[2], s_data_ptr, &data) ||
        ask(a[3], s_data_ptr, &idx) || ask(a[3], s_numel, &k))
        return NULL;
    const uint32_t flags = (uint32_t)PyLong_AsUnsignedLongMask(a[4]);
    if (PyErr_Occurred()) return NULL;
    if (a[5] != Py_None) {
        if (address(a[5], &stream)) return NULL;
    } else {
        if (!get_stream) return PyErr_Format(PyExc_RuntimeError, "no current stream before bind");
        PyObject* dev = PyObject_CallNoArgs(get_device);
        PyObject* raw = dev ? PyObject_CallOneArg(get_stream, dev) : NULL;
        Py_XDECREF(dev);
        if (!raw) return NULL;
        const int bad = address(raw, &stream);
        Py_DECREF(raw);
        if (bad) return NULL;
    }
    int64_t new_len = 0;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = ((list_fn)fn)(ctx, (void*)(uintptr_t)data, (int64_t)n, (uint32_t)(per * elem), (const uint32_t*)(uintptr_t)idx, (int64_t)k,
                       &new_len, flags, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLongLong(st ? -(long long)st : (long long)new_len);
}

// bind(current device, raw current stream of a device): how a stream of None is looked up.
static PyObject* bind(PyObject* self, PyObject* const* a, Py_ssize_t nargs) {
    (void)self;
    if (nargs != 2) return PyErr_Format(PyExc_TypeError, "bind takes 2 arguments");
    Py_INCREF(a[0]);
    Py_INCREF(a[1]);
    Py_XSETREF(get_device, a[0]);
    Py_XSETREF(get_stream, a[1]);
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {{"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, NULL},
                                {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, NULL},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_rzcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__rzcall(void) {
    s_shape = PyUnicode_InternFromString("shape");
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_numel = PyUnicode_InternFromString("numel");
    s_element_size = PyUnicode_InternFromString("element_size");
    if (!s_shape || !s_data_ptr || !s_numel || !s_element_size) return NULL;
    return PyModule_Create(&module);
}
