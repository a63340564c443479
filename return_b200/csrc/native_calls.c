// Calls of the kernel libraries' C entries without a foreign-function layer in between: what a launch costs the host.
//
// A Call holds an entry's address and the kinds of its arguments.  Its arguments are Python integers, floats and None; they are turned
// into machine words and handed over in one call of a fixed form: integers and pointers in the order of the integer registers and the
// stack, floats in that of the vector registers.  Under the C calling conventions of x86-64 and aarch64 Linux the two sequences are
// independent of each other, a callee reads only the words it declares and the caller takes the words off the stack again, so one form
// with more words than any entry has serves them all.  Anything else in an argument list (another type, another number of arguments) goes
// to the ctypes function that the Call was made from.  An entry of 22 arguments: 0.3 us (through ctypes 2.8).
//
// `fill` writes lists of integers into an int32 array, which numpy does at 40 ns a number (a step's pages and tokens: 2,000 of them) and this at 2.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>

#if !defined(__linux__) || !(defined(__x86_64__) || defined(__aarch64__))
#error "the form of the call is that of Linux on x86-64 and aarch64"
#endif

#define WORDS 48
#define FLOATS 8
typedef long long W;
#define W8 W, W, W, W, W, W, W, W
typedef int (*Entry)(W8, W8, W8, W8, W8, W8, float, float, float, float, float, float, float, float);
#define A8(i) w[i], w[i + 1], w[i + 2], w[i + 3], w[i + 4], w[i + 5], w[i + 6], w[i + 7]

typedef struct {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    Entry entry;
    PyObject* general;                      // the ctypes function
    int n;
    char kinds[WORDS + FLOATS];             // p pointer, i integer, f float
} Call;

static PyObject* call_vector(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* names) {
    Call* c = (Call*)self;
    W w[WORDS];
    float f[FLOATS] = {0};
    int nw = 0, nf = 0;
    if (names != NULL || PyVectorcall_NARGS(nargsf) != c->n) goto general;
    for (int i = 0; i < c->n; ++i) {
        PyObject* a = args[i];
        if (c->kinds[i] == 'f') {
            if (!PyFloat_CheckExact(a)) goto general;
            f[nf++] = (float)PyFloat_AS_DOUBLE(a);
        } else if (PyLong_CheckExact(a)) {
            w[nw++] = (W)PyLong_AsUnsignedLongLongMask(a);
        } else if (a == Py_None && c->kinds[i] == 'p') {
            w[nw++] = 0;
        } else {
            goto general;
        }
    }
    while (nw < WORDS) w[nw++] = 0;
    int code;
    Py_BEGIN_ALLOW_THREADS
    code = c->entry(A8(0), A8(8), A8(16), A8(24), A8(32), A8(40), f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
general:
    return PyObject_Vectorcall(c->general, args, nargsf, names);
}

static void call_dealloc(PyObject* self) {
    Py_XDECREF(((Call*)self)->general);
    Py_TYPE(self)->tp_free(self);
}

static PyTypeObject CallType = {
    PyVarObject_HEAD_INIT(NULL, 0)
    .tp_name = "return_b200_native_calls.Call",
    .tp_basicsize = sizeof(Call),
    .tp_dealloc = call_dealloc,
    .tp_vectorcall_offset = offsetof(Call, vectorcall),
    .tp_call = PyVectorcall_Call,
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
};

static PyObject* make(PyObject* module, PyObject* args) {
    unsigned long long address;
    const char* kinds;
    PyObject* general;
    if (!PyArg_ParseTuple(args, "KsO", &address, &kinds, &general)) return NULL;
    int n = 0, floats = 0;
    for (; kinds[n]; ++n) floats += kinds[n] == 'f';
    if (floats > FLOATS || n - floats > WORDS) Py_RETURN_NONE;       // more than the form holds
    Call* c = PyObject_New(Call, &CallType);
    if (c == NULL) return NULL;
    c->vectorcall = call_vector;
    c->entry = (Entry)(uintptr_t)address;
    c->general = Py_NewRef(general);
    c->n = n;
    for (int i = 0; i < n; ++i) c->kinds[i] = kinds[i];
    return (PyObject*)c;
}

// fill(array, places, lists, most): the first `most` numbers of lists[i] to array[places[i]], array[places[i] + 1], ...  False, with any part
// of them written, if something is no list or no plain integer of 32 bits, or lies outside the array: then the caller's own way says what it is.
static PyObject* fill(PyObject* module, PyObject* args) {
    PyObject *array, *places, *lists;
    Py_ssize_t most;
    if (!PyArg_ParseTuple(args, "OO!O!n", &array, &PyList_Type, &places, &PyList_Type, &lists, &most)) return NULL;
    Py_buffer to;
    if (PyObject_GetBuffer(array, &to, PyBUF_CONTIG | PyBUF_FORMAT) < 0) return NULL;
    const Py_ssize_t room = to.len / 4, n = PyList_GET_SIZE(lists);
    int fine = to.itemsize == 4 && to.format != NULL && to.format[0] == 'i' && PyList_GET_SIZE(places) == n;
    int* out = (int*)to.buf;
    for (Py_ssize_t r = 0; fine && r < n; ++r) {
        PyObject *list = PyList_GET_ITEM(lists, r), *place = PyList_GET_ITEM(places, r);
        if (!PyList_CheckExact(list) || !PyLong_CheckExact(place)) { fine = 0; break; }
        const Py_ssize_t at = PyLong_AsSsize_t(place), count = PyList_GET_SIZE(list) < most ? PyList_GET_SIZE(list) : most;
        if (at < 0 || count > room || at > room - count) { PyErr_Clear(); fine = 0; break; }
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject* item = PyList_GET_ITEM(list, i);
            int over = 0;
            const long v = PyLong_CheckExact(item) ? PyLong_AsLongAndOverflow(item, &over) : 0;
            if (!PyLong_CheckExact(item) || over || v < -2147483647L - 1 || v > 2147483647L) { fine = 0; break; }
            out[at + i] = (int)v;
        }
    }
    PyBuffer_Release(&to);
    return PyBool_FromLong(fine);
}

static PyMethodDef methods[] = {{"fill", fill, METH_VARARGS, "fill(int32 array, places, lists, most) -> whether all of it was plain integers"},
                                {"make", make, METH_VARARGS, "make(address, kinds, general) -> Call, or None where the form is too small"}, {NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "return_b200_native_calls", NULL, -1, methods};

PyMODINIT_FUNC PyInit_return_b200_native_calls(void) {
    if (PyType_Ready(&CallType) < 0) return NULL;
    return PyModule_Create(&module);
}
