// Calls of the kernel library's C entry points from Python.  ctypes converts every argument through a converter object and
// describes the call to libffi anew each time: 3 us for the two dozen arguments of a product, which a step that is not a
// replayed graph pays some sixty times.  A `Function` here holds an entry point's address and one code an argument (the kernels'
// signatures), reads plain ints, floats and None straight into the argument registers' images and calls.
//
// The call goes through one function type: all integer arguments as 64-bit words, then eight doubles.  In the System V
// calling convention of x86-64 and in that of AArch64, integer and floating-point arguments are counted apart: the words fill
// the integer registers and then the stack in the order in which the callee has its integers, the doubles the first eight
// floating-point registers (a float in the low half).  What is passed beyond the callee's own arguments is not looked at and is
// the caller's to clean up.  An entry point with more than eight floating-point arguments, or on another machine, is not bound
// (ctypes takes it).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#if defined(__x86_64__) && !defined(_WIN32)
#define FX_WORDS_THEN_FLOATS 1
#elif defined(__aarch64__) && defined(__linux__)
#define FX_WORDS_THEN_FLOATS 1
#else
#define FX_WORDS_THEN_FLOATS 0
#endif

#define MAX_WORDS 48
#define MAX_FLOATS 8

typedef int64_t W;
#define W4 W, W, W, W
#define W16 W4, W4, W4, W4
#define D8 double, double, double, double, double, double, double, double
#define A4(i) w[i], w[i + 1], w[i + 2], w[i + 3]
#define A16(i) A4(i), A4(i + 4), A4(i + 8), A4(i + 12)
#define F8 f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]

static int call_words(void* fn, int n, const W* w, const double* f)
{
    if (n <= 16) return ((int (*)(W16, D8))fn)(A16(0), F8);
    if (n <= 32) return ((int (*)(W16, W16, D8))fn)(A16(0), A16(16), F8);
    return ((int (*)(W16, W16, W16, D8))fn)(A16(0), A16(16), A16(32), F8);
}

typedef struct {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    void* fn;
    int n;
    char codes[MAX_WORDS + MAX_FLOATS + 1];
} Function;

// The entry point's return value; NotImplemented where an argument is none of the kinds that are read here.
static PyObject* function_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames)
{
    Function* f = (Function*)self;
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    if (n != f->n || (kwnames && PyTuple_GET_SIZE(kwnames))) {
        PyErr_Format(PyExc_TypeError, "entry point takes %d arguments (%zd given)", f->n, n);
        return NULL;
    }
    W words[MAX_WORDS];
    double floats[MAX_FLOATS];
    memset(floats, 0, sizeof floats);
    int nw = 0, nf = 0;
    for (int i = 0; i < f->n; ++i) {
        PyObject* a = args[i];
        switch (f->codes[i]) {
            case 'P':
                if (a == Py_None) { words[nw++] = 0; break; }
                if (!PyLong_Check(a)) Py_RETURN_NOTIMPLEMENTED;
                words[nw++] = (W)PyLong_AsUnsignedLongLongMask(a);
                break;
            case 'I': case 'L': case 'U':
                if (!PyLong_Check(a)) Py_RETURN_NOTIMPLEMENTED;
                words[nw] = (W)PyLong_AsUnsignedLongLongMask(a);
                if (f->codes[i] == 'I') words[nw] = (W)(int32_t)words[nw];
                ++nw;
                break;
            default: {
                const double v = PyFloat_AsDouble(a);
                if (v == -1.0 && PyErr_Occurred()) return NULL;
                if (f->codes[i] == 'F') {
                    const float s = (float)v;
                    memcpy(&floats[nf++], &s, sizeof s);
                } else {
                    floats[nf++] = v;
                }
            }
        }
        if (PyErr_Occurred()) return NULL;
    }
    for (int i = nw; i < MAX_WORDS; ++i) words[i] = 0;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = call_words(f->fn, nw, words, floats);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static void function_free(PyObject* self) { Py_TYPE(self)->tp_free(self); }

static PyTypeObject FunctionType = {
    PyVarObject_HEAD_INIT(NULL, 0)
    .tp_name = "_fx_fastcall.Function",
    .tp_basicsize = sizeof(Function),
    .tp_dealloc = function_free,
    .tp_vectorcall_offset = offsetof(Function, vectorcall),
    .tp_call = PyVectorcall_Call,
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_doc = "A C entry point with its arguments' codes.",
};

// bind(address, codes) -> Function, or None where the call cannot be made this way
static PyObject* bind(PyObject* module, PyObject* args)
{
    unsigned long long address;
    const char* codes;
    if (!PyArg_ParseTuple(args, "Ks", &address, &codes)) return NULL;
    int words = 0, floats = 0;
    for (const char* c = codes; *c; ++c) {
        if (strchr("PILU", *c)) ++words;
        else if (strchr("FD", *c)) ++floats;
        else { PyErr_Format(PyExc_ValueError, "unknown argument code %c", *c); return NULL; }
    }
    if (!FX_WORDS_THEN_FLOATS || words > MAX_WORDS || floats > MAX_FLOATS) Py_RETURN_NONE;
    Function* f = PyObject_New(Function, &FunctionType);
    if (!f) return NULL;
    f->vectorcall = function_call;
    f->fn = (void*)(uintptr_t)address;
    f->n = words + floats;
    memset(f->codes, 0, sizeof f->codes);
    memcpy(f->codes, codes, (size_t)f->n);
    return (PyObject*)f;
}

// A tensor's address and row stride as the wrappers ask for them some hundreds of times a step, without a Python frame each;
// what is not as expected (no CUDA tensor, other strides) goes to the Python functions that name the error.
static PyObject *slow_ptr, *slow_rows, *s_is_cuda, *s_data_ptr, *s_dim, *s_stride, *zero, *one;

static PyObject* ptr(PyObject* module, PyObject* t)
{
    if (t == Py_None) Py_RETURN_NONE;
    PyObject* cuda = PyObject_GetAttr(t, s_is_cuda);
    if (!cuda) return NULL;
    const int yes = cuda == Py_True;
    Py_DECREF(cuda);
    return yes ? PyObject_CallMethodNoArgs(t, s_data_ptr) : PyObject_CallOneArg(slow_ptr, t);
}

static PyObject* rows(PyObject* module, PyObject* t)
{
    PyObject* dim = PyObject_CallMethodNoArgs(t, s_dim);
    if (!dim) return NULL;
    const long d = PyLong_AsLong(dim);
    Py_DECREF(dim);
    if (d == 2) {
        PyObject* inner = PyObject_CallMethodOneArg(t, s_stride, one);
        if (!inner) return NULL;
        const long s = PyLong_AsLong(inner);
        Py_DECREF(inner);
        if (s == 1) return PyObject_CallMethodOneArg(t, s_stride, zero);
    }
    if (PyErr_Occurred()) return NULL;
    return PyObject_CallOneArg(slow_rows, t);
}

static PyObject* set_slow(PyObject* module, PyObject* args)
{
    PyObject *p, *r;
    if (!PyArg_ParseTuple(args, "OO", &p, &r)) return NULL;
    Py_INCREF(p); Py_INCREF(r);
    Py_XSETREF(slow_ptr, p);
    Py_XSETREF(slow_rows, r);
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"ptr", ptr, METH_O, "A CUDA tensor's address, None for None."},
    {"rows", rows, METH_O, "The row stride of a two-dimensional tensor with contiguous rows."},
    {"set_slow", set_slow, METH_VARARGS, "set_slow(ptr, rows): what takes the arguments that these do not."},
    {"bind", bind, METH_VARARGS, "bind(address, codes): the C entry point there as a callable, or None."},
    {NULL, NULL, 0, NULL},
};
static struct PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_fx_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fx_fastcall(void)
{
    if (PyType_Ready(&FunctionType) < 0) return NULL;
    s_is_cuda = PyUnicode_InternFromString("is_cuda"); s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_dim = PyUnicode_InternFromString("dim"); s_stride = PyUnicode_InternFromString("stride");
    zero = PyLong_FromLong(0); one = PyLong_FromLong(1);
    if (!s_is_cuda || !s_data_ptr || !s_dim || !s_stride || !zero || !one) return NULL;
    return PyModule_Create(&module_def);
}
