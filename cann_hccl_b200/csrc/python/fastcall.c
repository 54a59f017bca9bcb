/* Call path of the Python layer: one METH_FASTCALL function per C API entry that sits on a latency path.  It takes the tensors
 * as they are, asks each for its address, fills the argument structure on the stack and calls the library with the
 * interpreter lock released.  Through ctypes the same call costs several microseconds (argument objects, one pointer array per
 * buffer list), as much as a small collective takes on the GPU.  No PyTorch headers: addresses come from data_ptr(). */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>
#include "hccl/hccl_b200.h"

#define MAX_LOCAL 16

typedef HcclResult (*collective_fn)(HcclComm, const HcclB200Op *, void *const *, void *const *, aclrtStream);
typedef HcclResult (*dispatch_fn)(HcclComm, const HcclB200MoeLayer *, void *const *, void *const *, aclrtStream);
typedef HcclResult (*combine_fn)(HcclComm, const HcclB200MoeLayer *, void *const *, void *const *, void *const *, void *const *, aclrtStream);
static collective_fn g_collective;
static dispatch_fn g_dispatch;
static combine_fn g_combine;
static PyObject *s_data_ptr, *s_ctypes, *s_data, *s_numel, *s_size, *s_dtype;
static PyObject *g_dtypes, *g_get_device, *g_get_stream;  /* {torch / numpy dtype: HcclDataType}, current device, its current raw stream */

/* address of a tensor (data_ptr()) or numpy array (ctypes.data); None is null */
static int address(PyObject *x, void **out)
{
    if (x == Py_None) { *out = NULL; return 0; }
    PyObject *v = PyObject_CallMethodNoArgs(x, s_data_ptr);
    if (!v) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return -1;
        PyErr_Clear();
        PyObject *c = PyObject_GetAttr(x, s_ctypes);
        if (!c) return -1;
        v = PyObject_GetAttr(c, s_data);
        Py_DECREF(c);
        if (!v) return -1;
    }
    *out = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    return *out == NULL && PyErr_Occurred() ? -1 : 0;
}

/* one address per local rank, from a list, a tuple or any other sequence (a stacked tensor gives one row per rank); a rank that is
 * alone may pass its buffer without a list */
static int addresses(PyObject *x, Py_ssize_t nlocal, void **out)
{
    if (!PyList_Check(x) && !PyTuple_Check(x) && nlocal == 1) return address(x, out);
    const Py_ssize_t n = PyObject_Size(x);  /* before a long tensor is taken apart */
    if (n < 0) return -1;
    if (n != nlocal) { PyErr_SetString(PyExc_AssertionError, "need one buffer per local rank"); return -1; }
    PyObject *seq = PySequence_Fast(x, "need one buffer per local rank");
    if (!seq) return -1;
    int rc = 0;
    for (Py_ssize_t i = 0; i < nlocal && !rc; ++i) {
        if (i >= PySequence_Fast_GET_SIZE(seq)) { PyErr_SetString(PyExc_AssertionError, "need one buffer per local rank"); rc = -1; break; }
        PyObject *item = Py_NewRef(PySequence_Fast_GET_ITEM(seq, i));  /* asking it for its address runs Python code */
        rc = address(item, out + i);
        Py_DECREF(item);
    }
    Py_DECREF(seq);
    return rc;
}

/* the same where every rank has a buffer: None is refused */
static int all_addresses(PyObject *x, Py_ssize_t nlocal, void **out)
{
    if (addresses(x, nlocal, out)) return -1;
    for (Py_ssize_t i = 0; i < nlocal; ++i)
        if (!out[i]) { PyErr_SetString(PyExc_TypeError, "every rank needs a buffer, got None or one without memory"); return -1; }
    return 0;
}

/* the caller has made these contiguous arrays of 64-bit unsigned integers */
static int words(PyObject *x, Py_buffer *view, const uint64_t **out)
{
    if (PyObject_GetBuffer(x, view, PyBUF_SIMPLE)) return -1;
    *out = (const uint64_t *)view->buf;
    return 0;
}

/* bind(addresses of HcclB200Collective, HcclB200MoeDispatchLocal, HcclB200MoeCombineLocal) */
static PyObject *bind(PyObject *self, PyObject *const *a, Py_ssize_t n)
{
    if (n != 3) { PyErr_SetString(PyExc_TypeError, "bind() takes 3 addresses"); return NULL; }
    g_collective = (collective_fn)PyLong_AsVoidPtr(a[0]);
    g_dispatch = (dispatch_fn)PyLong_AsVoidPtr(a[1]);
    g_combine = (combine_fn)PyLong_AsVoidPtr(a[2]);
    if (PyErr_Occurred()) return NULL;
    Py_RETURN_NONE;
}

/* setup(dtypes, get_device, get_stream): the tables and accessors that op() uses; the accessors may be None without CUDA */
static PyObject *setup(PyObject *self, PyObject *const *a, Py_ssize_t n)
{
    if (n != 3 || !PyDict_Check(a[0])) { PyErr_SetString(PyExc_TypeError, "setup(dict, get_device, get_stream)"); return NULL; }
    Py_XSETREF(g_dtypes, Py_NewRef(a[0]));
    Py_XSETREF(g_get_device, Py_NewRef(a[1]));
    Py_XSETREF(g_get_stream, Py_NewRef(a[2]));
    Py_RETURN_NONE;
}

/* raw stream handle: an integer as it is, None = torch's current stream of the current device */
static int stream_of(PyObject *x, void **out)
{
    if (x != Py_None) {
        *out = PyLong_AsVoidPtr(x);
        return *out == NULL && PyErr_Occurred() ? -1 : 0;
    }
    if (!g_get_stream || g_get_stream == Py_None) { PyErr_SetString(PyExc_RuntimeError, "no CUDA stream accessor"); return -1; }
    PyObject *d = PyObject_CallNoArgs(g_get_device);
    if (!d) return -1;
    PyObject *s = PyObject_CallOneArg(g_get_stream, d);
    Py_DECREF(d);
    if (!s) return -1;
    *out = PyLong_AsVoidPtr(s);
    Py_DECREF(s);
    return *out == NULL && PyErr_Occurred() ? -1 : 0;
}

/* elements and HcclDataType of a tensor or numpy array */
static int describe_one(PyObject *x, uint64_t *count, int32_t *dtype)
{
    PyObject *n = PyObject_CallMethodNoArgs(x, s_numel);
    if (!n) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return -1;
        PyErr_Clear();
        n = PyObject_GetAttr(x, s_size);
        if (!n) return -1;
    }
    *count = PyLong_AsUnsignedLongLong(n);
    Py_DECREF(n);
    PyObject *d = PyObject_GetAttr(x, s_dtype);
    if (!d) return -1;
    PyObject *code = g_dtypes ? PyDict_GetItemWithError(g_dtypes, d) : NULL;
    if (!code) {
        if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, d);
        Py_DECREF(d);
        return -1;
    }
    Py_DECREF(d);
    *dtype = (int32_t)PyLong_AsLong(code);
    return PyErr_Occurred() ? -1 : 0;
}

/* of the first buffer of a list, a tuple or, where there are several ranks, any other sequence */
static int describe(PyObject *x, Py_ssize_t nlocal, uint64_t *count, int32_t *dtype)
{
    const int list = PyList_Check(x) || PyTuple_Check(x);
    if ((!list && nlocal == 1) || (list && PySequence_Fast_GET_SIZE(x) == 0)) return describe_one(x, count, dtype);
    PyObject *first = PySequence_GetItem(x, 0);
    if (!first) return -1;
    const int rc = describe_one(first, count, dtype);
    Py_DECREF(first);
    return rc;
}

/* op(comm, nlocal, coll, algo, nchan, op, root, send, recv, stream, by_recv, divide) -> result code: a collective whose count and
 * type are those of the send buffer (by_recv: of the receive buffer), the count divided by `divide` */
static PyObject *op(PyObject *self, PyObject *const *a, Py_ssize_t n)
{
    if (n != 12 || !g_collective) { PyErr_SetString(PyExc_TypeError, "op() takes 12 arguments, after bind()"); return NULL; }
    HcclB200Op o;
    memset(&o, 0, sizeof(o));
    void *comm = PyLong_AsVoidPtr(a[0]), *stream = NULL;
    const Py_ssize_t nlocal = PyLong_AsSsize_t(a[1]);
    o.coll = (int32_t)PyLong_AsLong(a[2]); o.algo = (int32_t)PyLong_AsLong(a[3]); o.nchan = (int32_t)PyLong_AsLong(a[4]);
    o.op = (int32_t)PyLong_AsLong(a[5]); o.root = (int32_t)PyLong_AsLong(a[6]);
    const uint64_t divide = PyLong_AsUnsignedLongLong(a[11]);
    if (PyErr_Occurred()) return NULL;
    if (nlocal < 1 || nlocal > MAX_LOCAL || !divide) { PyErr_SetString(PyExc_ValueError, "bad number of local ranks"); return NULL; }
    if (describe(a[10] == Py_True ? a[8] : a[7], nlocal, &o.count, &o.dataType)) return NULL;
    o.count /= divide;
    void *send[MAX_LOCAL], *recv[MAX_LOCAL];
    if (addresses(a[7], nlocal, send) || addresses(a[8], nlocal, recv) || stream_of(a[9], &stream)) return NULL;
    HcclResult rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_collective((HcclComm)comm, &o, send, recv, (aclrtStream)stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong((long)rc);
}

/* collective(comm, nlocal, coll, algo, nchan, dtype, op, root, count, send, recv, stream, tables) -> result code
 * tables: None, (counts, displs) or (sendCounts, sdispls, recvCounts, rdispls) */
static PyObject *collective(PyObject *self, PyObject *const *a, Py_ssize_t n)
{
    if (n != 13 || !g_collective) { PyErr_SetString(PyExc_TypeError, "collective() takes 13 arguments, after bind()"); return NULL; }
    HcclB200Op o;
    memset(&o, 0, sizeof(o));
    void *comm = PyLong_AsVoidPtr(a[0]), *stream = a[11] == Py_None ? NULL : PyLong_AsVoidPtr(a[11]);
    const Py_ssize_t nlocal = PyLong_AsSsize_t(a[1]);
    o.coll = (int32_t)PyLong_AsLong(a[2]); o.algo = (int32_t)PyLong_AsLong(a[3]); o.nchan = (int32_t)PyLong_AsLong(a[4]);
    o.dataType = (int32_t)PyLong_AsLong(a[5]); o.op = (int32_t)PyLong_AsLong(a[6]); o.root = (int32_t)PyLong_AsLong(a[7]);
    o.count = PyLong_AsUnsignedLongLong(a[8]);
    if (PyErr_Occurred()) return NULL;
    if (nlocal < 1 || nlocal > MAX_LOCAL) { PyErr_SetString(PyExc_ValueError, "bad number of local ranks"); return NULL; }
    void *send[MAX_LOCAL], *recv[MAX_LOCAL];
    const int barrier = o.coll == HCCL_B200_BARRIER;
    if (!barrier && (addresses(a[9], nlocal, send) || addresses(a[10], nlocal, recv))) return NULL;
    Py_buffer view[4];
    int nview = 0;
    if (a[12] != Py_None) {
        const uint64_t *w[4] = {NULL, NULL, NULL, NULL};
        const Py_ssize_t m = PyTuple_GET_SIZE(a[12]);
        for (; nview < m && nview < 4; ++nview)
            if (words(PyTuple_GET_ITEM(a[12], nview), &view[nview], &w[nview])) goto fail;
        if (m == 2) { o.counts = w[0]; o.displs = w[1]; }
        else { o.sendCounts = w[0]; o.sdispls = w[1]; o.recvCounts = w[2]; o.rdispls = w[3]; }
    }
    HcclResult rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_collective((HcclComm)comm, &o, barrier ? NULL : send, barrier ? NULL : recv, (aclrtStream)stream);
    Py_END_ALLOW_THREADS
    while (nview) PyBuffer_Release(&view[--nview]);
    return PyLong_FromLong((long)rc);
fail:
    while (nview) PyBuffer_Release(&view[--nview]);
    return NULL;
}

/* moe_dispatch(comm, nlocal, layer, x, topk_idx, stream) -> result code */
static PyObject *moe_dispatch(PyObject *self, PyObject *const *a, Py_ssize_t n)
{
    if (n != 6 || !g_dispatch) { PyErr_SetString(PyExc_TypeError, "moe_dispatch() takes 6 arguments, after bind()"); return NULL; }
    void *comm = PyLong_AsVoidPtr(a[0]), *layer = PyLong_AsVoidPtr(a[2]), *stream = PyLong_AsVoidPtr(a[5]);
    const Py_ssize_t nlocal = PyLong_AsSsize_t(a[1]);
    if (PyErr_Occurred()) return NULL;
    if (nlocal < 1 || nlocal > MAX_LOCAL) { PyErr_SetString(PyExc_ValueError, "bad number of local ranks"); return NULL; }
    void *x[MAX_LOCAL], *idx[MAX_LOCAL];
    if (all_addresses(a[3], nlocal, x) || all_addresses(a[4], nlocal, idx)) return NULL;
    HcclResult rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_dispatch((HcclComm)comm, (const HcclB200MoeLayer *)layer, x, idx, (aclrtStream)stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong((long)rc);
}

/* moe_combine(comm, nlocal, layer, rows (address of a table, 0: the layer's), topk_idx, gates, out, stream) -> result code */
static PyObject *moe_combine(PyObject *self, PyObject *const *a, Py_ssize_t n)
{
    if (n != 8 || !g_combine) { PyErr_SetString(PyExc_TypeError, "moe_combine() takes 8 arguments, after bind()"); return NULL; }
    void *comm = PyLong_AsVoidPtr(a[0]), *layer = PyLong_AsVoidPtr(a[2]), *rows = PyLong_AsVoidPtr(a[3]), *stream = PyLong_AsVoidPtr(a[7]);
    const Py_ssize_t nlocal = PyLong_AsSsize_t(a[1]);
    if (PyErr_Occurred()) return NULL;
    if (nlocal < 1 || nlocal > MAX_LOCAL) { PyErr_SetString(PyExc_ValueError, "bad number of local ranks"); return NULL; }
    void *idx[MAX_LOCAL], *gates[MAX_LOCAL], *out[MAX_LOCAL];
    if (all_addresses(a[4], nlocal, idx) || all_addresses(a[5], nlocal, gates) || all_addresses(a[6], nlocal, out)) return NULL;
    HcclResult rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_combine((HcclComm)comm, (const HcclB200MoeLayer *)layer, (void *const *)rows, idx, gates, out, (aclrtStream)stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong((long)rc);
}

static PyMethodDef methods[] = {{"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, NULL},
                                {"setup", (PyCFunction)(void (*)(void))setup, METH_FASTCALL, NULL},
                                {"op", (PyCFunction)(void (*)(void))op, METH_FASTCALL, NULL},
                                {"moe_dispatch", (PyCFunction)(void (*)(void))moe_dispatch, METH_FASTCALL, NULL},
                                {"moe_combine", (PyCFunction)(void (*)(void))moe_combine, METH_FASTCALL, NULL},
                                {"collective", (PyCFunction)(void (*)(void))collective, METH_FASTCALL, NULL},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void)
{
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_ctypes = PyUnicode_InternFromString("ctypes");
    s_data = PyUnicode_InternFromString("data");
    s_numel = PyUnicode_InternFromString("numel");
    s_size = PyUnicode_InternFromString("size");
    s_dtype = PyUnicode_InternFromString("dtype");
    return PyModule_Create(&module);
}
