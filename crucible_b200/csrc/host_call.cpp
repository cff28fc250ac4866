// Calls of the kernels' entry points from Python.  ctypes makes an object for every argument: a launch of 26 cost
// the host 3.3 us that way, 0.34 here, and an eager layer is ten launches.  A `Call` keeps an entry point's address and
// the kinds of its parameters, reads plain numbers and None straight from the interpreter's argument vector, and
// leaves everything else (other types, a wrong number of arguments, and with it the errors) to the ctypes
// function that it was made from.
//
// One function type serves all entry points: integers and addresses travel in the integer registers and then on
// the stack in order, floats in the vector registers (System V calling convention of x86-64), each class by
// itself, so that a callee finds its parameters whatever their order, as long as at most eight are floats and none
// is passed in another way; what it does not have is never read.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#if !defined(__x86_64__) || defined(_WIN32)
#error "the calling convention of x86-64 System V is what this file relies on"
#endif

namespace {

constexpr int MAX_INTS = 56, MAX_FLOATS = 8;

struct Call {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    void* address;
    PyObject* general;              // the ctypes function
    int count;
    char kinds[MAX_INTS + MAX_FLOATS];      // 'p' address or None, 'i' integer, 'f' float
};

#define REP8(X, n) X[n], X[n + 1], X[n + 2], X[n + 3], X[n + 4], X[n + 5], X[n + 6], X[n + 7]
#define L8 long, long, long, long, long, long, long, long
typedef int (*Few)(L8, L8, float, float, float, float, float, float, float, float);
typedef int (*Many)(L8, L8, L8, L8, L8, L8, L8, float, float, float, float, float, float, float, float);

PyObject* call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* names) {
    Call* c = reinterpret_cast<Call*>(self);
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    long ints[MAX_INTS];
    float floats[MAX_FLOATS] = {};
    int ni = 0, nf = 0;
    bool plain = names == nullptr && n == c->count;
    for (Py_ssize_t k = 0; plain && k < n; ++k) {
        PyObject* a = args[k];
        if (c->kinds[k] == 'f') {
            if (PyFloat_Check(a)) floats[nf++] = (float)PyFloat_AS_DOUBLE(a);
            else if (PyLong_Check(a)) floats[nf++] = (float)PyLong_AsDouble(a);
            else plain = false;
        } else if (PyLong_Check(a)) {
            ints[ni++] = (long)PyLong_AsUnsignedLongLongMask(a);
        } else if (a == Py_None && c->kinds[k] == 'p') {
            ints[ni++] = 0;
        } else {
            plain = false;
        }
    }
    if (!plain || PyErr_Occurred()) {
        PyErr_Clear();
        return PyObject_Vectorcall(c->general, args, nargsf, names);
    }
    for (int k = ni; k < (ni <= 16 ? 16 : MAX_INTS); ++k) ints[k] = 0;
    int result;
    Py_BEGIN_ALLOW_THREADS                          // (as ctypes does)
    if (ni <= 16)
        result = reinterpret_cast<Few>(c->address)(REP8(ints, 0), REP8(ints, 8), REP8(floats, 0));
    else
        result = reinterpret_cast<Many>(c->address)(REP8(ints, 0), REP8(ints, 8), REP8(ints, 16), REP8(ints, 24),
                                                    REP8(ints, 32), REP8(ints, 40), REP8(ints, 48), REP8(floats, 0));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(result);
}

void dealloc(PyObject* self) {
    PyTypeObject* type = Py_TYPE(self);
    Py_XDECREF(reinterpret_cast<Call*>(self)->general);
    type->tp_free(self);
    Py_DECREF(type);
}

PyObject* getattro(PyObject* self, PyObject* name) {         // argtypes, restype and the like: the ctypes function's
    PyObject* own = PyObject_GenericGetAttr(self, name);
    if (own != nullptr || !PyErr_ExceptionMatches(PyExc_AttributeError)) return own;
    PyErr_Clear();
    return PyObject_GetAttr(reinterpret_cast<Call*>(self)->general, name);
}

// what is set is the ctypes function's, too (another result type, other parameters), and calls are then left to it
int setattro(PyObject* self, PyObject* name, PyObject* value) {
    Call* c = reinterpret_cast<Call*>(self);
    c->count = -1;
    return PyObject_SetAttr(c->general, name, value);
}

PyMemberDef members[] = {{"__vectorcalloffset__", T_PYSSIZET, offsetof(Call, vectorcall), READONLY, nullptr},
                         {nullptr, 0, 0, 0, nullptr}};
PyType_Slot slots[] = {{Py_tp_dealloc, (void*)dealloc}, {Py_tp_call, (void*)PyVectorcall_Call},
                       {Py_tp_getattro, (void*)getattro}, {Py_tp_setattro, (void*)setattro}, {Py_tp_members, members}, {0, nullptr}};
PyType_Spec spec = {"cb_host_call.Call", sizeof(Call), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL, slots};
PyObject* call_type = nullptr;

// wrap(address, kinds, general): None if the entry point has more parameters than a Call takes
PyObject* wrap(PyObject*, PyObject* args) {
    unsigned long long address;
    const char* kinds;
    Py_ssize_t n;
    PyObject* general;
    if (!PyArg_ParseTuple(args, "Ks#O", &address, &kinds, &n, &general)) return nullptr;
    int ints = 0, floats = 0;
    for (Py_ssize_t k = 0; k < n; ++k) kinds[k] == 'f' ? ++floats : ++ints;
    if (ints > MAX_INTS || floats > MAX_FLOATS) Py_RETURN_NONE;
    Call* c = PyObject_New(Call, reinterpret_cast<PyTypeObject*>(call_type));
    if (c == nullptr) return nullptr;
    c->vectorcall = call;
    c->address = reinterpret_cast<void*>(address);
    c->general = Py_NewRef(general);
    c->count = (int)n;
    for (Py_ssize_t k = 0; k < n; ++k) c->kinds[k] = kinds[k];
    return reinterpret_cast<PyObject*>(c);
}

PyMethodDef methods[] = {{"wrap", wrap, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "cb_host_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_cb_host_call() {
    call_type = PyType_FromSpec(&spec);
    return call_type == nullptr ? nullptr : PyModule_Create(&module);
}
