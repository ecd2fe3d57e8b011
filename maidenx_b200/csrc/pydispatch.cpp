// maidenx_b200._dispatch: the calls around an op (device.dispatch) as one native call.
//
// What a small workload waits for is the host: a launch is 2.2 us of it, and around each launch the interpreted form of this spent another 2.9 us
// (packing the metadata block, three foreign calls, their argument conversions; add of 10000 floats 5.1 us a call, 2.5 here).  Here the block is packed on the stack,
// the op is called with the arguments as C values, and the interpreter lock is given up for the op alone, as ctypes does.
//
// Only the usual call is taken: a list of whole 64-bit numbers as metadata, plain ints (or None for a pointer) and plain numbers as arguments, as
// many as the op has.  Everything else, and every error in the arguments, goes to the interpreted form, which decides what becomes of it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstddef>
#include <cstdint>

namespace {

constexpr int kMostWords = 64, kMostArgs = 8;

struct Op {
    void* fn;
    int args;       // of the entry point
    int meta;       // which of them is the metadata block
    int scalar_at;  // which of them is a by-value scalar; -1: none
    char scalar;    // its type, as in the struct module
    uint32_t pointers;  // bit i: argument i is a pointer
};

int (*g_begin)(int, const size_t*, size_t, void**) = nullptr;
int (*g_end)(void*) = nullptr;
PyObject *g_ops = nullptr;       // op -> {dtype -> address of its Op}
PyObject *g_general = nullptr;   // the interpreted form
PyObject *g_resolve = nullptr;   // (op, dtype): registers it or raises
PyObject *g_begin_failed = nullptr, *g_op_failed = nullptr;
PyObject *g_kw_device = nullptr, *g_kw_check = nullptr;

const Op* find(PyObject* op, PyObject* dtype) {  // borrowed; null without an exception: not registered
    PyObject* of = PyDict_GetItemWithError(g_ops, op);
    PyObject* at = of ? PyDict_GetItemWithError(of, dtype) : nullptr;
    return at ? static_cast<const Op*>(PyLong_AsVoidPtr(at)) : nullptr;
}

// Every argument of an entry point but a by-value scalar is a size_t or a pointer: one register class, so one function type per count serves all.
typedef uintptr_t W;
bool call_words(const Op& o, const W* v) {
    switch (o.args) {
        case 4: reinterpret_cast<void (*)(W, W, W, W)>(o.fn)(v[0], v[1], v[2], v[3]); return true;
        case 5: reinterpret_cast<void (*)(W, W, W, W, W)>(o.fn)(v[0], v[1], v[2], v[3], v[4]); return true;
        case 6: reinterpret_cast<void (*)(W, W, W, W, W, W)>(o.fn)(v[0], v[1], v[2], v[3], v[4], v[5]); return true;
        case 8: reinterpret_cast<void (*)(W, W, W, W, W, W, W, W)>(o.fn)(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]); return true;
        default: return false;
    }
}
template <class T>
void call_scalar(const Op& o, const W* v, T s) {
    if (o.scalar_at == 4) reinterpret_cast<void (*)(W, W, W, W, T, W)>(o.fn)(v[0], v[1], v[2], v[3], s, v[5]);  // (num_els, num_dims, metadata, in, scalar, out)
    else reinterpret_cast<void (*)(W, W, W, W, W, W, T)>(o.fn)(v[0], v[1], v[2], v[3], v[4], v[5], s);          // padding: the value comes last
}
bool known_shape(const Op& o) {
    if (o.meta < 0 || o.meta >= o.args) return false;
    if (o.scalar_at < 0) return o.args == 4 || o.args == 5 || o.args == 6 || o.args == 8;
    return (o.scalar_at == 4 && o.args == 6) || (o.scalar_at == 6 && o.args == 7);
}

void call(const Op& o, const W* v, double f, uint64_t i) {
    if (o.scalar_at < 0) {
        call_words(o, v);
        return;
    }
    switch (o.scalar) {
        case 'f': call_scalar<float>(o, v, (float)f); break;
        case 'd': call_scalar<double>(o, v, f); break;
        case '?': call_scalar<bool>(o, v, i != 0); break;
        case 'b': call_scalar<int8_t>(o, v, (int8_t)i); break;
        case 'B': call_scalar<uint8_t>(o, v, (uint8_t)i); break;
        case 'h': call_scalar<int16_t>(o, v, (int16_t)i); break;
        case 'H': call_scalar<uint16_t>(o, v, (uint16_t)i); break;
        case 'i': call_scalar<int32_t>(o, v, (int32_t)i); break;
        case 'I': call_scalar<uint32_t>(o, v, (uint32_t)i); break;
        case 'q': call_scalar<int64_t>(o, v, (int64_t)i); break;
        default: call_scalar<uint64_t>(o, v, i); break;
    }
}

bool is_meta(PyObject* a) { return PyUnicode_CheckExact(a) && PyUnicode_CompareWithASCIIString(a, "META") == 0; }

PyObject* dispatch(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
    auto general = [&] { return PyObject_Vectorcall(g_general, args, (size_t)nargs, kwnames); };
    if (nargs < 3 || nargs > 3 + kMostArgs || !PyUnicode_CheckExact(args[0]) || !PyUnicode_CheckExact(args[1]) || !PyList_CheckExact(args[2])) return general();
    long device = 0;
    bool check = true;
    if (kwnames) {
        for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(kwnames); i++) {
            PyObject *name = PyTuple_GET_ITEM(kwnames, i), *value = args[nargs + i];
            if (PyUnicode_Compare(name, g_kw_check) == 0 && PyBool_Check(value)) {
                check = value == Py_True;
            } else if (PyUnicode_Compare(name, g_kw_device) == 0 && PyLong_CheckExact(value)) {
                int over = 0;
                device = PyLong_AsLongAndOverflow(value, &over);
                if (over || device != (int)device) return general();
            } else {
                return general();
            }
        }
    }
    const Op* o = find(args[0], args[1]);
    if (!o) {
        if (PyErr_Occurred()) return nullptr;
        PyObject* r = PyObject_CallFunctionObjArgs(g_resolve, args[0], args[1], nullptr);
        if (!r) return nullptr;
        Py_DECREF(r);
        if (!(o = find(args[0], args[1]))) return PyErr_Occurred() ? nullptr : general();
    }
    const Py_ssize_t words = PyList_GET_SIZE(args[2]);
    if (nargs - 3 != o->args || !words || words > kMostWords) return general();
    size_t meta[kMostWords];
    for (Py_ssize_t i = 0; i < words; i++) {
        PyObject* w = PyList_GET_ITEM(args[2], i);
        if (!PyLong_CheckExact(w)) return general();
        meta[i] = PyLong_AsUnsignedLongLong(w);
        if (meta[i] == (size_t)-1 && PyErr_Occurred()) {
            PyErr_Clear();
            return general();
        }
    }
    W v[kMostArgs] = {0};
    double f = 0.0;
    uint64_t whole = 0;
    for (int i = 0; i < o->args; i++) {
        PyObject* a = args[3 + i];
        if (i == o->meta) {
            if (!is_meta(a)) return general();
        } else if (i == o->scalar_at) {
            const bool real = o->scalar == 'f' || o->scalar == 'd';
            if (real && PyFloat_CheckExact(a)) f = PyFloat_AS_DOUBLE(a);
            else if (real && PyLong_CheckExact(a)) f = PyLong_AsDouble(a);
            else if (!real && (PyLong_CheckExact(a) || (o->scalar == '?' && PyBool_Check(a)))) whole = PyLong_AsUnsignedLongLongMask(a);
            else return general();
            // a bool is any number but zero, also one whose low 64 bits are
            if (o->scalar == '?') whole = PyObject_IsTrue(a) == 1;
        } else if (PyLong_CheckExact(a)) {
            v[i] = PyLong_AsUnsignedLongLongMask(a);
        } else if (a == Py_None && (o->pointers >> i & 1)) {
            v[i] = 0;
        } else {
            return general();
        }
        if (PyErr_Occurred()) {
            PyErr_Clear();
            return general();
        }
    }
    void* block = nullptr;
    int status;
    bool begun = false;
    Py_BEGIN_ALLOW_THREADS
    status = g_begin((int)device, meta, (size_t)words, &block);
    if (status == 0) {
        begun = true;
        v[o->meta] = reinterpret_cast<W>(block);
        call(*o, v, f, whole);
        status = g_end(block);
    }
    Py_END_ALLOW_THREADS
    if (!begun) return PyObject_CallFunction(g_begin_failed, "is", status, "metadata upload");
    if (check && status) return PyObject_CallFunctionObjArgs(g_op_failed, args[0], args[1], nullptr);
    Py_RETURN_NONE;
}

// bind(mx_dispatch_begin, mx_dispatch_end): their addresses
PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long begin = 0, end = 0;
    if (!PyArg_ParseTuple(args, "KK", &begin, &end)) return nullptr;
    g_begin = reinterpret_cast<decltype(g_begin)>((uintptr_t)begin);
    g_end = reinterpret_cast<decltype(g_end)>((uintptr_t)end);
    Py_RETURN_NONE;
}

// register(op, dtype, address, types, meta): `types` is a letter per argument, P for a pointer, S for a size, else a scalar's as in the struct module;
// a form that this module does not call is left to the interpreted one
PyObject* add(PyObject*, PyObject* args) {
    PyObject *op = nullptr, *dtype = nullptr;
    unsigned long long fn = 0;
    const char* types = nullptr;
    int meta = 0;
    if (!PyArg_ParseTuple(args, "UUKsi", &op, &dtype, &fn, &types, &meta)) return nullptr;
    Op o = {reinterpret_cast<void*>((uintptr_t)fn), 0, meta, -1, 0, 0};
    for (const char* t = types; *t; t++, o.args++) {
        if (o.args == kMostArgs) Py_RETURN_FALSE;
        if (*t == 'P') o.pointers |= 1u << o.args;
        else if (*t != 'S') {
            if (o.scalar_at >= 0) Py_RETURN_FALSE;
            o.scalar_at = o.args;
            o.scalar = *t;
        }
    }
    if (!g_begin || !g_end || !known_shape(o)) Py_RETURN_FALSE;
    PyObject* of = PyDict_GetItemWithError(g_ops, op);
    if (!of) {
        if (PyErr_Occurred() || !(of = PyDict_New()) || PyDict_SetItem(g_ops, op, of) < 0) return nullptr;
        Py_DECREF(of);  // the table has it
    }
    PyObject* at = PyLong_FromVoidPtr(new Op(o));  // an entry lives as long as the process, as the library does
    if (!at || PyDict_SetItem(of, dtype, at) < 0) return nullptr;
    Py_DECREF(at);
    Py_RETURN_TRUE;
}

// setup(general, resolve, begin_failed, op_failed)
PyObject* setup(PyObject*, PyObject* args) {
    PyObject *g, *r, *b, *o;
    if (!PyArg_ParseTuple(args, "OOOO", &g, &r, &b, &o)) return nullptr;
    PyObject** const at[4] = {&g_general, &g_resolve, &g_begin_failed, &g_op_failed};
    PyObject* const from[4] = {g, r, b, o};
    for (int i = 0; i < 4; i++) {
        Py_INCREF(from[i]);
        Py_XSETREF(*at[i], from[i]);
    }
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"dispatch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(dispatch)), METH_FASTCALL | METH_KEYWORDS,
     "dispatch($module, op, dtype_name, metadata, *args, device=0, metadata_on_host=False, check=True)\n--\n\n"
     "Call cuda_<op>_<dtype> the way maidenx_core does.  `args` is the op's argument list\n"
     "with the string \"META\" standing where the metadata pointer goes."},
    {"bind", bind, METH_VARARGS, nullptr},
    {"register", add, METH_VARARGS, nullptr},
    {"setup", setup, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_dispatch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dispatch(void) {
    g_ops = PyDict_New();
    g_kw_device = PyUnicode_InternFromString("device");
    g_kw_check = PyUnicode_InternFromString("check");
    return g_ops && g_kw_device && g_kw_check ? PyModule_Create(&module) : nullptr;
}
