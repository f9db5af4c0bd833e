/* The three operators on prepared weights, from Python to the C ABI in one native call.
 *
 * A call of a small projection is bound by the host: through ctypes and checks written in Python it
 * takes 9.7 us, of which 3.2 are an object for the current stream, 2.5 the checks of three tensors and 1
 * the conversion of arguments, in front of a kernel of 3.2 us.  The functions here ask the tensors the same
 * questions and call the library, 4.1 us with the launch; where an answer is not the expected one, or an argument is not a plain
 * int or float, they return None and do nothing, and the caller goes through the checks in Python, which
 * say what is wrong.  Nothing is kept from one call for the next.
 *
 * The library's functions are handed over as addresses, so that whichever build of it is loaded is used. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <limits.h>

typedef int (*gemv_fn)(const void*, const void*, void*, int, int, int, void*);
typedef int (*gemv_int8_fn)(const void*, const void*, float, void*, int, int, void*);
typedef int (*gemm_fn)(const void*, const void*, void*, int, int, int, void*);

static gemv_fn f_gemv;
static gemv_int8_fn f_gemv_int8;
static gemm_fn f_gemm;
static PyObject *current_device, *raw_stream;                   /* callables of torch */
static PyObject *d_half, *d_int8, *d_uint8;                     /* its dtypes */
static PyObject *s_is_cuda, *s_dtype, *s_is_contiguous, *s_get_device, *s_numel, *s_data_ptr;

/* Consumes a new reference; 1: it is True, 0: it is not (or an exception, which is dropped). */
static int is_true(PyObject* o)
{
    const int r = o == Py_True;
    if (!o) PyErr_Clear();
    Py_XDECREF(o);
    return r;
}
/* Consumes a new reference; -1 where it is no number of the range 0 .. LLONG_MAX. */
static long long number(PyObject* o)
{
    long long v = -1;
    if (o) v = PyLong_AsLongLong(o);
    if (PyErr_Occurred()) {
        PyErr_Clear();
        v = -1;
    }
    Py_XDECREF(o);
    return v;
}
static PyObject* method(PyObject* t, PyObject* name) { return PyObject_CallMethodNoArgs(t, name); }

/* 1 and the address: a contiguous CUDA tensor of this type on the current device with at least `need` elements. */
static int tensor(PyObject* t, PyObject* dtype, long long device, long long need, void** p)
{
    if (!is_true(PyObject_GetAttr(t, s_is_cuda))) return 0;
    PyObject* d = PyObject_GetAttr(t, s_dtype);
    if (!d) PyErr_Clear();
    Py_XDECREF(d);
    if (d != dtype) return 0;
    if (!is_true(method(t, s_is_contiguous)) || number(method(t, s_get_device)) != device || number(method(t, s_numel)) < need) return 0;
    /* an address is unsigned: above 2^63 number() refuses it and the call takes the other way */
    const long long a = number(method(t, s_data_ptr));
    if (a < 0) return 0;
    *p = (void*)a;
    return 1;
}

/* a plain int of 1 .. INT_MAX, else 0 */
static int positive(PyObject* o)
{
    if (!PyLong_CheckExact(o)) return 0;
    int over = 0;
    const long long v = PyLong_AsLongLongAndOverflow(o, &over);
    return over || v < 1 || v > INT_MAX ? 0 : (int)v;
}

static int where(long long* device, void** stream)
{
    PyObject* dev = PyObject_CallNoArgs(current_device);
    PyObject* st = dev ? PyObject_CallOneArg(raw_stream, dev) : NULL;
    if (!st) PyErr_Clear();
    *device = number(dev);
    const long long s = number(st);
    *stream = (void*)s;
    return f_gemv && *device >= 0 && s >= 0;
}

/* (packed, rows, cols, input, output, batch) */
static PyObject* gemv_packed(PyObject* self, PyObject* const* a, Py_ssize_t n)
{
    long long dev;
    void *w, *x, *y, *stream;
    const int rows = n == 6 ? positive(a[1]) : 0, cols = n == 6 ? positive(a[2]) : 0, batch = n == 6 ? positive(a[5]) : 0;
    if (!rows || !batch || cols < 128 || cols % 128 || !where(&dev, &stream) || !tensor(a[0], d_uint8, dev, 0, &w) ||
        !tensor(a[3], d_half, dev, (long long)batch * cols, &x) || !tensor(a[4], d_half, dev, (long long)batch * rows, &y))
        Py_RETURN_NONE;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = f_gemv(w, x, y, batch, rows, cols, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
}

/* (packed, rows, cols, input, scale, output) */
static PyObject* gemv_int8_packed(PyObject* self, PyObject* const* a, Py_ssize_t n)
{
    long long dev;
    void *w, *x, *y, *stream;
    const int rows = n == 6 ? positive(a[1]) : 0, cols = n == 6 ? positive(a[2]) : 0;
    if (!rows || !cols || !PyFloat_CheckExact(a[4]) || !where(&dev, &stream) || !tensor(a[0], d_uint8, dev, 0, &w) ||
        !tensor(a[3], d_int8, dev, cols, &x) || !tensor(a[5], d_half, dev, rows, &y))
        Py_RETURN_NONE;
    const float scale = (float)PyFloat_AS_DOUBLE(a[4]);
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = f_gemv_int8(w, x, scale, y, rows, cols, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
}

/* (A, packed, rows, cols, C, M) */
static PyObject* gemm_packed(PyObject* self, PyObject* const* a, Py_ssize_t n)
{
    long long dev;
    void *w, *x, *y, *stream;
    const int rows = n == 6 ? positive(a[2]) : 0, cols = n == 6 ? positive(a[3]) : 0, m = n == 6 ? positive(a[5]) : 0;
    if (!rows || !m || cols < 128 || cols % 128 || !where(&dev, &stream) || !tensor(a[0], d_half, dev, (long long)m * cols, &x) ||
        !tensor(a[1], d_uint8, dev, 0, &w) || !tensor(a[4], d_half, dev, (long long)m * rows, &y))
        Py_RETURN_NONE;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = f_gemm(x, w, y, m, rows, cols, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
}

/* (gemv, gemv_int8, gemm addresses, current_device, raw_stream, float16, int8, uint8) */
static PyObject* bind(PyObject* self, PyObject* args)
{
    unsigned long long g, i, m;
    PyObject *o[5], **d[5] = {&current_device, &raw_stream, &d_half, &d_int8, &d_uint8};
    if (!PyArg_ParseTuple(args, "KKKOOOOO", &g, &i, &m, &o[0], &o[1], &o[2], &o[3], &o[4])) return NULL;
    for (int k = 0; k < 5; k++) {
        Py_INCREF(o[k]);
        Py_XSETREF(*d[k], o[k]);
    }
    f_gemv_int8 = (gemv_int8_fn)(uintptr_t)i;
    f_gemm = (gemm_fn)(uintptr_t)m;
    f_gemv = (gemv_fn)(uintptr_t)g;
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"gemv_packed", (PyCFunction)(void*)gemv_packed, METH_FASTCALL, NULL},
    {"gemv_int8_packed", (PyCFunction)(void*)gemv_int8_packed, METH_FASTCALL, NULL},
    {"gemm_packed", (PyCFunction)(void*)gemm_packed, METH_FASTCALL, NULL},
    {"bind", bind, METH_VARARGS, NULL},
    {NULL, NULL, 0, NULL},
};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hostcall", "Operators on prepared weights in one native call.", -1, methods,
                                    NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__hostcall(void)
{
    s_is_cuda = PyUnicode_InternFromString("is_cuda");
    s_dtype = PyUnicode_InternFromString("dtype");
    s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    s_get_device = PyUnicode_InternFromString("get_device");
    s_numel = PyUnicode_InternFromString("numel");
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    if (!s_is_cuda || !s_dtype || !s_is_contiguous || !s_get_device || !s_numel || !s_data_ptr) return NULL;
    return PyModule_Create(&module);
}
