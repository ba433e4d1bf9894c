/* fastcall.c: calls into libornith_cuda.so from Python without ctypes' conversion of every argument.
 *
 * A step of one chat is a dozen calls of a few microseconds of GPU work each, and a ctypes call with nine arguments costs
 * about 1.5 us of them.  Function(address, kind, arguments) is a callable for one entry point whose arguments are all integers and
 * pointers (no floats, no structs by value), at most 16.  `arguments` has a letter for each: i, an int or what has __index__; p, an
 * int, None (a null pointer), a bytes object (its contents) or an object with a data_ptr() method.  kind 0: the entry point returns
 * int, 1: size_t.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <structmember.h>

#define MAX_ARGS 16
typedef uint64_t word;
typedef word (*entry)(word, word, word, word, word, word, word, word, word, word, word, word, word, word, word, word);

typedef struct {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    entry fn;
    int kind, n;
    char arguments[MAX_ARGS];
} Function;

static PyObject *s_data_ptr;

static int int_word(PyObject *o, word *w) {
    if (!o) return -1;
    *w = (word)PyLong_AsUnsignedLongLongMask(o);
    return *w == (word)-1 && PyErr_Occurred() ? -1 : 0;
}
static int to_word(PyObject *o, char argument, word *w) {
    if (PyLong_Check(o)) return int_word(o, w);
    if (argument == 'p' && o == Py_None) { *w = 0; return 0; }
    if (argument == 'p' && PyBytes_Check(o)) { *w = (word)(uintptr_t)PyBytes_AS_STRING(o); return 0; }
    PyObject *p = argument == 'p' ? PyObject_CallMethodNoArgs(o, s_data_ptr) : PyNumber_Index(o);
    const int r = int_word(p, w);
    Py_XDECREF(p);
    return r;
}

static PyObject *function_call(PyObject *self, PyObject *const *args, size_t nargsf, PyObject *kwnames) {
    Function *f = (Function *)self;
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    word a[MAX_ARGS] = {0}, r;
    if (n != f->n || (kwnames && PyTuple_GET_SIZE(kwnames))) {
        PyErr_Format(PyExc_TypeError, "%d positional arguments expected, %zd given", f->n, n);
        return NULL;
    }
    for (Py_ssize_t i = 0; i < n; i++)
        if (to_word(args[i], f->arguments[i], &a[i])) return NULL;
    /* a launch may wait for room in the stream */
    Py_BEGIN_ALLOW_THREADS
    r = f->fn(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15]);
    Py_END_ALLOW_THREADS
    return f->kind ? PyLong_FromUnsignedLongLong(r) : PyLong_FromLong((int)r);
}

static PyObject *function_new(PyTypeObject *type, PyObject *args, PyObject *kwargs) {
    unsigned long long address;
    int kind;
    const char *arguments;
    Py_ssize_t n;
    (void)kwargs;
    if (!PyArg_ParseTuple(args, "Kis#", &address, &kind, &arguments, &n)) return NULL;
    if (n > MAX_ARGS) { PyErr_SetString(PyExc_ValueError, "at most 16 arguments"); return NULL; }
    Function *f = (Function *)type->tp_alloc(type, 0);
    if (!f) return NULL;
    f->vectorcall = function_call;
    f->fn = (entry)(uintptr_t)address;
    f->kind = kind;
    f->n = (int)n;
    for (Py_ssize_t i = 0; i < n; i++) f->arguments[i] = arguments[i];
    return (PyObject *)f;
}

static PyTypeObject function_type = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "ornithology_b200._fastcall.Function",
    .tp_basicsize = sizeof(Function),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_new = function_new,
    .tp_call = PyVectorcall_Call,
    .tp_vectorcall_offset = offsetof(Function, vectorcall),
};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, .m_name = "_fastcall", .m_size = -1};

PyMODINIT_FUNC PyInit__fastcall(void) {
    if (PyType_Ready(&function_type) < 0) return NULL;
    PyObject *m = PyModule_Create(&module);
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    if (!m || !s_data_ptr) return NULL;
    Py_INCREF(&function_type);
    if (PyModule_AddObject(m, "Function", (PyObject *)&function_type) < 0) return NULL;
    return m;
}
