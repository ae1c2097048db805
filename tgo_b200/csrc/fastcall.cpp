// Calls of the kernel libraries' C entry points from Python, without ctypes: `bind(address)` gives a
// callable that takes plain numbers, hands them to the function at that address and returns its int.
//
// How: on x86-64 and System V, whole numbers and pointers travel in the integer registers and then on
// the stack in their order, single- and double-precision numbers in the vector registers in theirs,
// and a function that is handed more than it declares does not look at the rest. So one signature with room
// for everything serves every entry point of up to FC_INTS whole numbers and FC_REALS others: an int,
// a bool or an address goes to the next integer place, a float to the next vector place (as a single-
// precision number), a one-element tuple to the next vector place as a double.
//
// MEASURED (an entry point of 31 arguments that refuses them): 0.9 us a call, 18 by ctypes with an object an
// argument; on a B200 the host side of a decoding layer of routed experts 174 -> 113 us, of retention 80 -> 60.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#if !defined(__x86_64__)
#error "the call below is the System V x86-64 one"
#endif

#define FC_INTS 48
#define FC_REALS 8

typedef int (*FcFn)(long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long,
                    long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long,
                    long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long,
                    double, double, double, double, double, double, double, double);

static PyObject* fc_call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    FcFn fn = (FcFn)PyCapsule_GetPointer(self, "tgo.entry");
    if (!fn) return nullptr;
    long i[FC_INTS] = {};
    double r[FC_REALS] = {};
    int ni = 0, nr = 0;
    for (Py_ssize_t k = 0; k < n; ++k) {
        PyObject* a = args[k];
        if (PyFloat_Check(a) || PyTuple_Check(a)) {
            if (nr == FC_REALS) { PyErr_SetString(PyExc_TypeError, "too many floating-point arguments"); return nullptr; }
            if (PyFloat_Check(a)) {
                const float f = (float)PyFloat_AS_DOUBLE(a);
                memcpy(&r[nr++], &f, sizeof f);
            } else {
                if (PyTuple_GET_SIZE(a) != 1) { PyErr_SetString(PyExc_TypeError, "a double is a tuple of one"); return nullptr; }
                const double d = PyFloat_AsDouble(PyTuple_GET_ITEM(a, 0));
                if (d == -1.0 && PyErr_Occurred()) return nullptr;
                r[nr++] = d;
            }
            continue;
        }
        if (ni == FC_INTS) { PyErr_SetString(PyExc_TypeError, "too many arguments"); return nullptr; }
        if (!PyLong_Check(a)) {
            PyErr_Format(PyExc_TypeError, "argument %zd: whole numbers, floats and one-element tuples only, not %s", k,
                         Py_TYPE(a)->tp_name);
            return nullptr;
        }
        int over = 0;
        const long long v = PyLong_AsLongLongAndOverflow(a, &over);
        if (over > 0) {                                  // an address with its top bit set
            i[ni++] = (long)PyLong_AsUnsignedLongLong(a);
            if (PyErr_Occurred()) return nullptr;
        } else {
            if (over < 0 || (v == -1 && PyErr_Occurred())) {
                if (!PyErr_Occurred()) PyErr_SetString(PyExc_OverflowError, "argument out of range");
                return nullptr;
            }
            i[ni++] = (long)v;
        }
    }
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fn(i[0], i[1], i[2], i[3], i[4], i[5], i[6], i[7], i[8], i[9], i[10], i[11], i[12], i[13], i[14], i[15], i[16],
            i[17], i[18], i[19], i[20], i[21], i[22], i[23], i[24], i[25], i[26], i[27], i[28], i[29], i[30], i[31], i[32],
            i[33], i[34], i[35], i[36], i[37], i[38], i[39], i[40], i[41], i[42], i[43], i[44], i[45], i[46], i[47],
            r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static PyMethodDef fc_def = {"entry", (PyCFunction)(void (*)(void))fc_call, METH_FASTCALL, "a C entry point"};

static PyObject* fc_bind(PyObject*, PyObject* address) {
    void* p = PyLong_AsVoidPtr(address);
    if (!p) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: a null address");
        return nullptr;
    }
    PyObject* capsule = PyCapsule_New(p, "tgo.entry", nullptr);
    if (!capsule) return nullptr;
    PyObject* f = PyCFunction_New(&fc_def, capsule);
    Py_DECREF(capsule);
    return f;
}

static PyMethodDef fc_methods[] = {{"bind", fc_bind, METH_O, "bind(address) -> callable"}, {nullptr, nullptr, 0, nullptr}};
static PyModuleDef fc_module = {PyModuleDef_HEAD_INIT, "tgo_fastcall", nullptr, -1, fc_methods, nullptr, nullptr, nullptr, nullptr};

PyMODINIT_FUNC PyInit_tgo_fastcall() { return PyModule_Create(&fc_module); }
