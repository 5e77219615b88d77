// launch.cc - the launch path of the Python binding (module paddock_b200._launch).
//
// A decode step is a few microseconds of GPU work per launch, so what the host spends between two
// launches is part of the operator's time.  Measured around the pack's calls (B200 host, one decode
// GEMV): 8.4 us per call through ctypes and Python-level argument conversion, of which 2.4 us is
// the launcher itself; through this file 2.9 us.  It holds no GPU code and computes nothing: it
// converts Python arguments by the entry point's signature string, drops the GIL and calls the
// C function pointer.
//
//   Entry(address, signature, name)      one launcher; signature as in pack.py ('p' pointer, 'u' u32,
//                                        'U' u64, 'f' f32; the trailing stream is implied)
//   Caller(resolve, slow, error)         callable (name, *args, stream=0): error is None -> returns the
//                                        status, else raises error(name, status) when it is not 0
//
// Pointer arguments are None, integers or objects with data_ptr(), numbers Python ints and floats, the
// stream an int or None; anything else (ctypes objects, numpy scalars) sends the call to `slow`, the
// ctypes route, which takes what ctypes takes.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <utility>

namespace {

constexpr Py_ssize_t kMaxArgs = 24;

union Slot {
    void* p;
    uint64_t u;
    float f;
};

// ---- one trampoline per signature: the function pointer is called with exactly its own types
template <size_t N>
struct Sig {
    char s[N];
    constexpr Sig(const char (&str)[N]) {
        for (size_t i = 0; i < N; ++i) s[i] = str[i];
    }
};
template <char C> struct Kind;
template <> struct Kind<'p'> { using type = void*; static type get(const Slot& s) { return s.p; } };
template <> struct Kind<'u'> { using type = uint32_t; static type get(const Slot& s) { return (uint32_t)s.u; } };
template <> struct Kind<'U'> { using type = uint64_t; static type get(const Slot& s) { return s.u; } };
template <> struct Kind<'f'> { using type = float; static type get(const Slot& s) { return s.f; } };

using Trampoline = int (*)(void* fn, const Slot* a, void* stream);

template <Sig S, size_t... I>
int invoke_impl(void* fn, const Slot* a, void* stream, std::index_sequence<I...>) {
    using Fn = int (*)(typename Kind<S.s[I]>::type..., void*);
    return reinterpret_cast<Fn>(fn)(Kind<S.s[I]>::get(a[I])..., stream);
}
template <Sig S>
int invoke(void* fn, const Slot* a, void* stream) {
    return invoke_impl<S>(fn, a, stream, std::make_index_sequence<sizeof(S.s) - 1>{});
}

struct SigRow {
    const char* sig;
    Trampoline fn;
};
#define PDK_SIG(s) {s, &invoke<s>}
const SigRow kSigs[] = {
    PDK_SIG("ppU"), PDK_SIG("ppu"), PDK_SIG("pppU"), PDK_SIG("pppppuu"), PDK_SIG("pppppuuu"), PDK_SIG("pppuu"),
    PDK_SIG("ppppuu"), PDK_SIG("pppppufu"), PDK_SIG("ppppppuffu"), PDK_SIG("pppu"), PDK_SIG("ppppppufu"),
    PDK_SIG("ppppu"), PDK_SIG("ppfpuu"), PDK_SIG("pppppfuu"), PDK_SIG("ppuu"), PDK_SIG("ppppppfuuupU"),
    PDK_SIG("ppuuppu"), PDK_SIG("ppppuuuu"), PDK_SIG("ppppuuuuu"), PDK_SIG("ppuuu"), PDK_SIG("ppUu"),
    PDK_SIG("pppUu"), PDK_SIG("ppppuuu"), PDK_SIG("ppppppuuu"), PDK_SIG("pppppppuuuu"), PDK_SIG("pppuU"),
    PDK_SIG("ppppppppppppuuufff"), PDK_SIG("ppppppppppuuuu"), PDK_SIG("ppppppppppuuuuff"), PDK_SIG("ppppppppuuuu"),
    PDK_SIG("ppppppfuuu"), PDK_SIG("pppppppppppuuuuff"), PDK_SIG("ppppppppppuuuuu"), PDK_SIG("ppppppppppuuuuuu"),
    PDK_SIG("ppppppuuuuuu"), PDK_SIG("puuu"), PDK_SIG("up"), PDK_SIG("uup"), PDK_SIG("pppuuu"),
    PDK_SIG("pppppppuuuuff"), PDK_SIG("pppppppppppuuuuuu"), PDK_SIG("pppppppppppppppppuuuuuuu"),
    PDK_SIG("pppppppuuuufff"), PDK_SIG("ppppppppppppppuuuuufff"), PDK_SIG("ppppppuuuuufff"),
    PDK_SIG("pppppuuuuu"), PDK_SIG("ppppppppuuuuu"),
};
#undef PDK_SIG

PyObject* g_data_ptr = nullptr;   // interned "data_ptr"
PyObject* g_stream = nullptr;     // interned "stream"

// ---- Entry
struct Entry {
    PyObject_HEAD
    void* fn;
    Trampoline call;
    Py_ssize_t n;
    char sig[kMaxArgs + 1];
};

int entry_init(PyObject* self, PyObject* args, PyObject*) {
    auto* e = reinterpret_cast<Entry*>(self);
    unsigned long long addr;
    const char *sig, *name;
    if (!PyArg_ParseTuple(args, "Kss", &addr, &sig, &name)) return -1;
    for (const SigRow& r : kSigs)
        if (std::strcmp(r.sig, sig) == 0) {
            e->fn = reinterpret_cast<void*>(static_cast<uintptr_t>(addr));
            e->call = r.fn;
            e->n = (Py_ssize_t)std::strlen(sig);
            std::memcpy(e->sig, sig, (size_t)e->n + 1);
            return 0;
        }
    PyErr_Format(PyExc_ValueError, "%s: no trampoline for signature '%s'", name, sig);
    return -1;
}

PyTypeObject EntryType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// 0 done, 1 not a plain argument (the slow route takes the call), -1 Python error
int convert(char kind, PyObject* o, Slot* out) {
    switch (kind) {
        case 'p': {
            if (o == Py_None) {
                out->p = nullptr;
                return 0;
            }
            PyObject* addr = o;
            if (!PyLong_Check(o)) {
                addr = PyObject_CallMethodNoArgs(o, g_data_ptr);
                if (addr == nullptr) {
                    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return -1;
                    PyErr_Clear();
                    return 1;
                }
            } else {
                Py_INCREF(addr);
            }
            out->p = reinterpret_cast<void*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(addr)));
            Py_DECREF(addr);
            return PyErr_Occurred() ? -1 : 0;
        }
        case 'f': {
            if (!PyFloat_Check(o) && !PyLong_Check(o)) return 1;
            const double v = PyFloat_AsDouble(o);
            if (v == -1.0 && PyErr_Occurred()) return -1;
            out->f = (float)v;
            return 0;
        }
        default: {
            if (!PyLong_Check(o)) return 1;
            const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
            out->u = kind == 'u' ? (uint32_t)v : v;
            return 0;
        }
    }
}

// ---- Caller
struct Caller {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    PyObject* table;     // name -> Entry
    PyObject* resolve;   // name -> Entry, called once per name
    PyObject* slow;      // (name, *args, stream=) -> status
    PyObject* error;     // None or the exception class
};

PyObject* finish(Caller* c, PyObject* name, long rc) {
    if (c->error == Py_None) return PyLong_FromLong(rc);
    if (rc == 0) Py_RETURN_NONE;
    if (PyObject* exc = PyObject_CallFunction(c->error, "Ol", name, rc)) {
        PyErr_SetObject(reinterpret_cast<PyObject*>(Py_TYPE(exc)), exc);
        Py_DECREF(exc);
    }
    return nullptr;
}

PyObject* caller_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    auto* c = reinterpret_cast<Caller*>(self);
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf), nk = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
    if (n < 1 || nk > 1) {
        PyErr_SetString(PyExc_TypeError, "expected (name, *args, stream=0)");
        return nullptr;
    }
    void* stream = nullptr;
    bool plain = true;      // the stream is an int or None
    if (nk == 1) {
        PyObject* key = PyTuple_GET_ITEM(kwnames, 0);
        if (key != g_stream && PyUnicode_Compare(key, g_stream) != 0) {
            PyErr_Format(PyExc_TypeError, "unexpected keyword argument '%U'", key);
            return nullptr;
        }
        if (PyLong_Check(args[n])) {
            stream = reinterpret_cast<void*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(args[n])));
        } else {
            plain = args[n] == Py_None;
        }
    }
    PyObject* name = args[0];
    PyObject* found = PyDict_GetItemWithError(c->table, name);
    if (found == nullptr) {
        if (PyErr_Occurred()) return nullptr;
        found = PyObject_CallOneArg(c->resolve, name);
        if (found == nullptr) return nullptr;
        const bool ok = Py_IS_TYPE(found, &EntryType) && PyDict_SetItem(c->table, name, found) == 0;
        Py_DECREF(found);   // the table holds it
        if (!ok) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "resolve() must return an Entry");
            return nullptr;
        }
    }
    auto* e = reinterpret_cast<Entry*>(found);
    if (n - 1 != e->n) {
        PyErr_Format(PyExc_TypeError, "%U takes %zd arguments before the stream, got %zd", name, e->n, n - 1);
        return nullptr;
    }
    Slot slots[kMaxArgs];
    for (Py_ssize_t i = 0; i < e->n || !plain; ++i) {
        const int r = plain ? convert(e->sig[i], args[1 + i], &slots[i]) : 1;
        if (r < 0) return nullptr;
        if (r > 0) {
            PyObject* res = PyObject_Vectorcall(c->slow, args, (size_t)n, kwnames);
            if (res == nullptr) return nullptr;
            const long rc = PyLong_AsLong(res);
            Py_DECREF(res);
            if (rc == -1 && PyErr_Occurred()) return nullptr;
            return finish(c, name, rc);
        }
    }
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = e->call(e->fn, slots, stream);
    Py_END_ALLOW_THREADS
    return finish(c, name, rc);
}

int caller_init(PyObject* self, PyObject* args, PyObject*) {
    auto* c = reinterpret_cast<Caller*>(self);
    PyObject *resolve, *slow, *error;
    if (!PyArg_ParseTuple(args, "OOO", &resolve, &slow, &error)) return -1;
    Py_XSETREF(c->table, PyDict_New());
    if (c->table == nullptr) return -1;
    Py_XSETREF(c->resolve, Py_NewRef(resolve));
    Py_XSETREF(c->slow, Py_NewRef(slow));
    Py_XSETREF(c->error, Py_NewRef(error));
    c->vectorcall = caller_call;
    return 0;
}
int caller_traverse(PyObject* self, visitproc visit, void* arg) {
    auto* c = reinterpret_cast<Caller*>(self);
    Py_VISIT(c->table);
    Py_VISIT(c->resolve);
    Py_VISIT(c->slow);
    Py_VISIT(c->error);
    return 0;
}
int caller_clear(PyObject* self) {
    auto* c = reinterpret_cast<Caller*>(self);
    Py_CLEAR(c->table);
    Py_CLEAR(c->resolve);
    Py_CLEAR(c->slow);
    Py_CLEAR(c->error);
    return 0;
}
void caller_dealloc(PyObject* self) {
    PyObject_GC_UnTrack(self);
    caller_clear(self);
    Py_TYPE(self)->tp_free(self);
}

PyTypeObject CallerType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_launch", "Launch path of the kernel-pack binding.", -1, nullptr,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__launch(void) {
    EntryType.tp_name = "paddock_b200._launch.Entry";
    EntryType.tp_basicsize = sizeof(Entry);
    EntryType.tp_flags = Py_TPFLAGS_DEFAULT;
    EntryType.tp_new = PyType_GenericNew;
    EntryType.tp_init = entry_init;
    CallerType.tp_name = "paddock_b200._launch.Caller";
    CallerType.tp_basicsize = sizeof(Caller);
    CallerType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL;
    CallerType.tp_new = PyType_GenericNew;
    CallerType.tp_init = caller_init;
    CallerType.tp_dealloc = caller_dealloc;
    CallerType.tp_traverse = caller_traverse;
    CallerType.tp_clear = caller_clear;
    CallerType.tp_vectorcall_offset = offsetof(Caller, vectorcall);
    CallerType.tp_call = PyVectorcall_Call;
    if (PyType_Ready(&EntryType) < 0 || PyType_Ready(&CallerType) < 0) return nullptr;
    g_data_ptr = PyUnicode_InternFromString("data_ptr");
    g_stream = PyUnicode_InternFromString("stream");
    PyObject* m = PyModule_Create(&kModule);
    if (m == nullptr || g_data_ptr == nullptr || g_stream == nullptr) return nullptr;
    if (PyModule_AddObjectRef(m, "Entry", reinterpret_cast<PyObject*>(&EntryType)) < 0 ||
        PyModule_AddObjectRef(m, "Caller", reinterpret_cast<PyObject*>(&CallerType)) < 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
