/* The call of asp_spmv from Python (the module alphasparse_b200._call).
 *
 * A small SpMV takes the GPU less time than its launch takes the host (2.0 us on the measured machine), and ctypes spends 0.7 us more on
 * converting six arguments. This binding is made once per plan group and converts two: 0.1 us. It holds addresses of what the
 * group and its context hold themselves (the context's handle, the array of plans) and reads them at every call, so a context or a
 * group that has been closed is NULL to asp_spmv, as it is through ctypes. The GIL is released meanwhile: a launch waits where the
 * stream's queue is full. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>

typedef int (*spmv_fn)(void *ctx, void *const *plans, int n_plans, const void *d_x, void *d_y, int zero_y);

typedef struct
{
    PyObject_HEAD
    vectorcallfunc vectorcall;
    spmv_fn fn;
    void **ctx; /* where the handle is */
    void **plans;
    int n;
} Spmv;

/* (d_x, d_y, zero_y as asp_spmv takes it) -> status; TypeError where a pointer is no int */
static PyObject *spmv_call(PyObject *self, PyObject *const *args, size_t nargsf, PyObject *kwnames)
{
    Spmv *s = (Spmv *)self;
    if (PyVectorcall_NARGS(nargsf) != 3 || (kwnames && PyTuple_GET_SIZE(kwnames)) || !PyLong_Check(args[0]) || !PyLong_Check(args[1]) || !PyLong_Check(args[2]))
    {
        PyErr_SetString(PyExc_TypeError, "three ints are wanted");
        return NULL;
    }
    /* as ctypes takes ints for pointers: modulo 2^64 */
    const unsigned long long x = PyLong_AsUnsignedLongLongMask(args[0]), y = PyLong_AsUnsignedLongLongMask(args[1]);
    const long zero_y = PyLong_AsLong(args[2]);
    if (PyErr_Occurred()) return NULL;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = s->fn(*s->ctx, s->plans, s->n, (const void *)(size_t)x, (void *)(size_t)y, (int)zero_y);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
}

static PyObject *spmv_new(PyTypeObject *type, PyObject *args, PyObject *kw)
{
    unsigned long long fn, ctx, plans;
    int n;
    (void)kw;
    if (!PyArg_ParseTuple(args, "KKKi", &fn, &ctx, &plans, &n)) return NULL;
    Spmv *s = (Spmv *)type->tp_alloc(type, 0);
    if (!s) return NULL;
    s->vectorcall = spmv_call;
    s->fn = (spmv_fn)(size_t)fn;
    s->ctx = (void **)(size_t)ctx;
    s->plans = (void **)(size_t)plans;
    s->n = n;
    return (PyObject *)s;
}

static PyTypeObject SpmvType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "alphasparse_b200._call.Spmv",
    .tp_doc = "Spmv(address of asp_spmv, address of the context's handle, address of the plans, number of plans)",
    .tp_basicsize = sizeof(Spmv),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_new = spmv_new,
    .tp_call = PyVectorcall_Call,
    .tp_vectorcall_offset = offsetof(Spmv, vectorcall),
};

static PyModuleDef module = {PyModuleDef_HEAD_INIT, .m_name = "_call", .m_doc = "asp_spmv without ctypes", .m_size = -1};

PyMODINIT_FUNC PyInit__call(void)
{
    if (PyType_Ready(&SpmvType) < 0) return NULL;
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddObjectRef(m, "Spmv", (PyObject *)&SpmvType) < 0)
    {
        Py_DECREF(m);
        return NULL;
    }
    return m;
}
