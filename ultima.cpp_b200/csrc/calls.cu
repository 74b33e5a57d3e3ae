// Calling the kernels' C entry points from Python with little between: a CPython extension module whose ``bind(address,
// signature)`` gives a callable that turns its arguments into machine words and calls the function.
//
// A prompt's layer is 9 to 29 launches, each an entry point with 15 to 37 arguments; a step that is not a captured graph is
// bound by them until the device has some 500 tokens to work on.  Converting the arguments of a call with 14 of them took
// ctypes 2.0 us; this takes 0.2 us.
//
// One call form serves every signature.  Under the System V convention of x86-64 integers and pointers travel in their own
// sequence of registers and 8-byte stack slots, floats in theirs, each in the order of the parameters, and slots that a
// function has no parameter for are not looked at.  So a function is called with all of its integer arguments first, padded
// to MAX_INTS words, then its floats; entry points have at most MAX_FLOATS floats, which all go in registers.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <string.h>

#if !defined(__x86_64__) || !defined(__linux__)
#error "the call form is that of x86-64 Linux"
#endif

constexpr int MAX_INTS = 48, MAX_FLOATS = 8, MAX_ARGS = MAX_INTS + MAX_FLOATS;

typedef struct {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    void* address;
    int n;
    char sig[MAX_ARGS + 1];
} Call;

#define I8(a, i) a[i], a[i + 1], a[i + 2], a[i + 3], a[i + 4], a[i + 5], a[i + 6], a[i + 7]
#define T8(t) t, t, t, t, t, t, t, t
typedef int (*Entry)(T8(long), T8(long), T8(long), T8(long), T8(long), T8(long), T8(float));

static PyObject* array_type = NULL;        // ctypes.Array
static PyObject* pointer_word = NULL;      // ctypes' own conversion to a pointer, for everything rarer than an address, None or an array

// An integer parameter's word: a Python integer (or anything with __index__).  A pointer's: an integer, None (null), or what
// ctypes takes for a void pointer (an array of ctypes: where its elements lie; a pointer: where it points), and nothing else,
// so that a host array is refused here and not read by a kernel.  The caller keeps that memory alive through the call.
static int word_of(PyObject* o, char code, long* out) {
    PyObject* i;
    if (PyLong_Check(o)) {
        *out = (long)PyLong_AsUnsignedLongLongMask(o);
        return *out == -1 && PyErr_Occurred() ? -1 : 0;
    }
    if (code == 'P') {
        if (o == Py_None) { *out = 0; return 0; }
        if (array_type && PyObject_TypeCheck(o, (PyTypeObject*)array_type)) {
            Py_buffer b;
            if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) return -1;
            *out = (long)b.buf;
            PyBuffer_Release(&b);
            return 0;
        }
        if (!pointer_word) { PyErr_SetString(PyExc_TypeError, "a pointer is an integer or None"); return -1; }
        i = PyObject_CallOneArg(pointer_word, o);
        if (i && !PyLong_Check(i)) { Py_DECREF(i); PyErr_SetString(PyExc_TypeError, "a pointer's word is an integer"); return -1; }
    } else {
        i = PyNumber_Index(o);
    }
    if (!i) return -1;
    *out = (long)PyLong_AsUnsignedLongLongMask(i);
    Py_DECREF(i);
    return *out == -1 && PyErr_Occurred() ? -1 : 0;
}

static PyObject* call_vector(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    Call* c = (Call*)self;
    if (PyVectorcall_NARGS(nargsf) != c->n || (kwnames && PyTuple_GET_SIZE(kwnames))) {
        PyErr_Format(PyExc_TypeError, "this entry point takes %d arguments, got %zd", c->n, PyVectorcall_NARGS(nargsf));
        return NULL;
    }
    long a[MAX_INTS] = {0};
    float f[MAX_FLOATS] = {0};
    int ni = 0, nf = 0;
    for (int i = 0; i < c->n; ++i) {
        if (c->sig[i] == 'F') {
            const double v = PyFloat_AsDouble(args[i]);
            if (v == -1.0 && PyErr_Occurred()) return NULL;
            f[nf++] = (float)v;
        } else {
            if (word_of(args[i], c->sig[i], &a[ni]) != 0) return NULL;
            ++ni;
        }
    }
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = ((Entry)c->address)(I8(a, 0), I8(a, 8), I8(a, 16), I8(a, 24), I8(a, 32), I8(a, 40), I8(f, 0));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static PyMemberDef call_members[] = {
    {"__vectorcalloffset__", Py_T_PYSSIZET, offsetof(Call, vectorcall), Py_READONLY, NULL},
    {NULL, 0, 0, 0, NULL},
};
static void call_free(PyObject* self) {
    PyTypeObject* t = Py_TYPE(self);
    PyObject_Free(self);
    Py_DECREF(t);
}
static PyType_Slot call_slots[] = {
    {Py_tp_call, (void*)PyVectorcall_Call},
    {Py_tp_members, call_members},
    {Py_tp_dealloc, (void*)call_free},
    {0, NULL},
};
static PyType_Spec call_spec = {"ultima_calls.Call", sizeof(Call), 0,
                                Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_DISALLOW_INSTANTIATION, call_slots};
static PyTypeObject* call_type = NULL;

// bind(address, signature): one letter a parameter, F a float, P a pointer, anything else (I, L, U) an integer.
static PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long address;
    const char* sig;
    Py_ssize_t n;
    if (!PyArg_ParseTuple(args, "Ks#", &address, &sig, &n)) return NULL;
    int floats = 0;
    for (Py_ssize_t i = 0; i < n; ++i) floats += sig[i] == 'F';
    if (!address || floats > MAX_FLOATS || n - floats > MAX_INTS) {
        PyErr_SetString(PyExc_ValueError, "no entry point, or more parameters than a call has room for");
        return NULL;
    }
    Call* c = PyObject_New(Call, call_type);
    if (!c) return NULL;
    c->vectorcall = call_vector;
    c->address = (void*)address;
    c->n = (int)n;
    memcpy(c->sig, sig, (size_t)n);
    c->sig[n] = 0;
    return (PyObject*)c;
}

// pointers(array type, conversion): see word_of.
static PyObject* pointers(PyObject*, PyObject* args) {
    PyObject *type, *conversion;
    if (!PyArg_ParseTuple(args, "O!O", &PyType_Type, &type, &conversion)) return NULL;
    Py_INCREF(type);
    Py_INCREF(conversion);
    Py_XSETREF(array_type, type);
    Py_XSETREF(pointer_word, conversion);
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "bind(address, signature) -> callable"},
                                {"pointers", pointers, METH_VARARGS, "pointers(array type, conversion)"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "ultima_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit_ultima_calls(void) {
    call_type = (PyTypeObject*)PyType_FromSpec(&call_spec);
    if (!call_type) return NULL;
    return PyModule_Create(&module);
}
