/* Calls a C entry point of the kernel libraries from Python with the cost of its conversions alone.
 *
 * Issuing a launch through ctypes takes 7 to 10 us of the host for the entry points' 20 to 45 arguments (an object made for every
 * pointer, a lookup for every conversion), which is more than a small kernel runs; outside a captured step that is what a call
 * waits for (a gated feed-forward of 8 tokens, two launches that run 23.5 us: 34.7 -> 24.5 us a call; a layer's attention without a
 * softmax for 64 single tokens, four launches and two library products: 76.8 -> 70.3).  An Entry is the address of a function and a letter for each of its arguments: 'i' any integer or pointer (None: 0),
 * 'f' a float.  System V x86-64 hands integers and floats over in registers and on the stack independently of one another, so one
 * call with sixty-four integers and eight floats reaches every function whose floats fit the registers; what it does not take
 * it does not look at.  The interpreter's lock is given back for the length of the call. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>

#if !defined(__x86_64__) || defined(_WIN32)
#error "written for the System V calling convention of x86-64"
#endif

#define MOST_INTS 64
#define MOST_FLOATS 8

typedef struct {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    void* address;
    int n, ints, floats;
    char kinds[MOST_INTS + MOST_FLOATS];
    int wide;
} Entry;

#define I8(a, k) a[k], a[k + 1], a[k + 2], a[k + 3], a[k + 4], a[k + 5], a[k + 6], a[k + 7]
#define L8 long long, long long, long long, long long, long long, long long, long long, long long
typedef long long (*Any)(L8, L8, L8, L8, L8, L8, L8, L8, float, float, float, float, float, float, float, float);

static int as_integer(PyObject* o, long long* out) {
    if (o == Py_None) {
        *out = 0;
        return 0;
    }
    if (PyLong_Check(o)) {
        int over = 0;
        long long v = PyLong_AsLongLongAndOverflow(o, &over);
        if (over) v = (long long)PyLong_AsUnsignedLongLongMask(o);
        *out = v;
        return PyErr_Occurred() ? -1 : 0;
    }
    PyObject* v = PyObject_GetAttrString(o, "value");      /* a ctypes number */
    if (v == NULL) {
        PyErr_Clear();
        v = PyNumber_Index(o);
        if (v == NULL) return -1;
    }
    int rc = v == Py_None || PyLong_Check(v) ? as_integer(v, out) : -1;
    if (rc < 0 && !PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "an integer or a pointer is expected");
    Py_DECREF(v);
    return rc;
}

static PyObject* entry_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    Entry* e = (Entry*)self;
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    if (n != e->n || kwnames != NULL) return PyErr_Format(PyExc_TypeError, "the entry point takes %d arguments, got %zd", e->n, n);
    long long a[MOST_INTS];
    float f[MOST_FLOATS];
    int ni = 0, nf = 0;
    for (int i = 0; i < e->n; ++i) {
        if (e->kinds[i] == 'f') {
            double v = PyFloat_AsDouble(args[i]);
            if (v == -1.0 && PyErr_Occurred()) return NULL;
            f[nf++] = (float)v;
        } else if (as_integer(args[i], a + ni++) < 0) {
            return NULL;
        }
    }
    for (; ni < MOST_INTS; ++ni) a[ni] = 0;
    for (; nf < MOST_FLOATS; ++nf) f[nf] = 0.f;
    long long r;
    Py_BEGIN_ALLOW_THREADS
    r = ((Any)e->address)(I8(a, 0), I8(a, 8), I8(a, 16), I8(a, 24), I8(a, 32), I8(a, 40), I8(a, 48), I8(a, 56), f[0], f[1], f[2], f[3],
                          f[4], f[5], f[6], f[7]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLongLong(e->wide ? r : (long long)(int)r);
}

static PyObject* entry_new(PyTypeObject* type, PyObject* args, PyObject* kw) {
    unsigned long long address;
    const char* kinds;
    Py_ssize_t n;
    int wide = 0;
    if (!PyArg_ParseTuple(args, "Ks#|p", &address, &kinds, &n, &wide)) return NULL;
    int ints = 0, floats = 0;
    for (Py_ssize_t i = 0; i < n; ++i) kinds[i] == 'f' ? ++floats : ++ints;
    if (ints > MOST_INTS || floats > MOST_FLOATS) {
        PyErr_SetString(PyExc_ValueError, "too many arguments");
        return NULL;
    }
    Entry* e = (Entry*)type->tp_alloc(type, 0);
    if (e == NULL) return NULL;
    e->vectorcall = entry_call;
    e->address = (void*)(size_t)address;
    e->n = (int)n;
    e->ints = ints;
    e->floats = floats;
    for (Py_ssize_t i = 0; i < n; ++i) e->kinds[i] = kinds[i];
    e->wide = wide;
    return (PyObject*)e;
}

static PyMemberDef entry_members[] = {{"__vectorcalloffset__", Py_T_PYSSIZET, offsetof(Entry, vectorcall), Py_READONLY, NULL}, {NULL}};
static PyTypeObject EntryType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "blm_entry.Entry",
    .tp_basicsize = sizeof(Entry),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_vectorcall_offset = offsetof(Entry, vectorcall),
    .tp_call = PyVectorcall_Call,
    .tp_members = entry_members,
    .tp_new = entry_new,
    .tp_doc = "Entry(address, kinds, wide result): a C function that takes integers, pointers and floats",
};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "blm_entry", NULL, -1, NULL};

PyMODINIT_FUNC PyInit_blm_entry(void) {
    if (PyType_Ready(&EntryType) < 0) return NULL;
    PyObject* m = PyModule_Create(&module);
    if (m == NULL) return NULL;
    Py_INCREF(&EntryType);
    if (PyModule_AddObject(m, "Entry", (PyObject*)&EntryType) < 0) return NULL;
    return m;
}
