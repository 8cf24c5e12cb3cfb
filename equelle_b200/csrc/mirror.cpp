// Native half of the Python runtime mirror (equelle_b200/runtime.py): the
// handle types with their operators, and the runtime methods that a
// program's time loop calls, as CPython types over the C ABI of
// include/eqg.h.  An explicit program makes some 250 runtime calls a time
// step; through ctypes a call cost 2.1 us of interpreter work (a Python
// frame or two, an out-parameter object, argument conversion), of which the
// library's part is 0.2 us: a shallow-water step on 64 x 48 cells took 0.79
// ms, 0.19 ms with these.
//
// The entry points come as addresses from the ctypes library that the
// runtime was given (the device library or the CPU oracle): nothing is
// linked.  The interpreter lock is released around the library calls, as
// ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "eqg.h"

#include <cstddef>
#include <cstring>
#include <initializer_list>

namespace {

// ---- entry points of one library ----------------------------------------------
struct Api {
    decltype(&eqg_last_error) last_error;
    decltype(&eqg_set_builtin) set_builtin;
    decltype(&eqg_set_size) set_size;
    decltype(&eqg_set_release) set_release;
    decltype(&eqg_first_cell) first_cell;
    decltype(&eqg_second_cell) second_cell;
    decltype(&eqg_set_on) set_on;
    decltype(&eqg_set_extend) set_extend;
    decltype(&eqg_set_select) set_select;
    decltype(&eqg_mask_release) mask_release;
    decltype(&eqg_mask_logic) mask_logic;
    decltype(&eqg_coll_constant) coll_constant;
    decltype(&eqg_coll_release) coll_release;
    decltype(&eqg_binary) binary;
    decltype(&eqg_binary_scalar) binary_scalar;
    decltype(&eqg_unary) unary;
    decltype(&eqg_compare) compare;
    decltype(&eqg_compare_scalar) compare_scalar;
    decltype(&eqg_gradient) gradient;
    decltype(&eqg_neg_gradient) neg_gradient;
    decltype(&eqg_divergence) divergence;
    decltype(&eqg_interior_divergence) interior_divergence;
    decltype(&eqg_on) on;
    decltype(&eqg_extend) extend;
    decltype(&eqg_select) select;
    decltype(&eqg_reduce) reduce;
    decltype(&eqg_two_norm) two_norm;
    decltype(&eqg_span_subset) span_subset;
    decltype(&eqg_span_superset) span_superset;
};

struct Entry {
    const char* name;
    size_t offset;
};
#define E(name) {"eqg_" #name, offsetof(Api, name)}
const Entry kEntries[] = {E(last_error), E(set_builtin), E(set_size), E(set_release), E(first_cell), E(second_cell),
                          E(set_on), E(set_extend), E(set_select), E(mask_release), E(mask_logic), E(coll_constant),
                          E(coll_release), E(binary), E(binary_scalar), E(unary), E(compare), E(compare_scalar),
                          E(gradient), E(neg_gradient), E(divergence), E(interior_divergence), E(on), E(extend),
                          E(select), E(reduce), E(two_norm), E(span_subset), E(span_superset)};
#undef E

// Classes of the Python module, set by register_classes(), and the runtime's
// methods that make their objects.
template <class T>
struct Made;
template <>
struct Made<eqg_coll> {
    static inline PyObject* cls = nullptr;
    static constexpr const char* hook = "_coll";
};
template <>
struct Made<eqg_mask> {
    static inline PyObject* cls = nullptr;
    static constexpr const char* hook = "_mask";
};
template <>
struct Made<eqg_set> {
    static inline PyObject* cls = nullptr;
    static constexpr const char* hook = "_set";
};
PyObject* g_error_class = nullptr;

struct RuntimeObject {
    PyObject_HEAD
    Api api;
    eqg_runtime* h;
    bool bound, created;  // has its library's entry points; has been given a handle
    bool hooked;          // its class overrides a method that handles are made through
};

struct HandleObject {
    PyObject_HEAD
    RuntimeObject* rt;  // owned
    void* h;
};

extern PyTypeObject RuntimeBaseType, CollBaseType, MaskBaseType, SetBaseType;

// An object whose __init__ has not run (or not got that far) lacks what it
// sets: an error, as for any Python attribute.
__attribute__((noinline, cold)) void* lacks(PyObject* o, const char* name)
{
    PyErr_Format(PyExc_AttributeError, "'%s' object has no attribute '%s'", Py_TYPE(o)->tp_name, name);
    return nullptr;
}

// The runtime that a method is called on; null (an error) before its __init__.
inline RuntimeObject* rt_of(PyObject* self)
{
    RuntimeObject* rt = (RuntimeObject*)self;
    if (!rt->bound) return (RuntimeObject*)lacks(self, "lib");
    if (!rt->created) return (RuntimeObject*)lacks(self, "h");
    return rt;
}

// The runtime of a handle; null (an error) before the handle's __init__.
inline RuntimeObject* rt_of_handle(PyObject* handle)
{
    RuntimeObject* rt = ((HandleObject*)handle)->rt;
    return rt ? rt_of((PyObject*)rt) : (RuntimeObject*)lacks(handle, "rt");
}

PyObject* raise_status(const Api& api, int status)
{
    const char* msg = api.last_error();
    PyObject* e = PyObject_CallFunction(g_error_class, "is", status, msg ? msg : "");
    if (e) {
        PyErr_SetObject(g_error_class, e);
        Py_DECREF(e);
    }
    return nullptr;
}

// Calls an entry point with the interpreter lock released.
template <class F>
int unlocked(F&& f)
{
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = f();
    Py_END_ALLOW_THREADS
    return st;
}

PyObject* new_handle(PyObject* cls, RuntimeObject* rt, void* h)
{
    PyTypeObject* t = (PyTypeObject*)cls;
    HandleObject* o = (HandleObject*)t->tp_alloc(t, 0);
    if (!o) return nullptr;
    Py_INCREF(rt);
    o->rt = rt;
    o->h = h;
    return (PyObject*)o;
}

PyObject* as_object(int v) { return PyLong_FromLong(v); }
PyObject* as_object(int64_t v) { return PyLong_FromLongLong(v); }
PyObject* as_object(double v) { return PyFloat_FromDouble(v); }
PyObject* as_object(const void* v) { return v ? PyLong_FromVoidPtr((void*)v) : Py_NewRef(Py_None); }

// runtime.<hook>(runtime.lib.<name>, args...)
template <class... A>
__attribute__((noinline, cold)) PyObject* call_hook(RuntimeObject* rt, const char* hook, const char* name, A... args)
{
    constexpr Py_ssize_t N = 1 + sizeof...(A);
    PyObject* lib = PyObject_GetAttrString((PyObject*)rt, "lib");
    PyObject* v[N] = {lib ? PyObject_GetAttrString(lib, name) : nullptr, as_object(args)...};
    Py_XDECREF(lib);
    PyObject* m = PyObject_GetAttrString((PyObject*)rt, hook);
    bool ok = m != nullptr;
    for (PyObject* o : v) ok = ok && o;
    PyObject* r = ok ? PyObject_Vectorcall(m, v, N, nullptr) : nullptr;
    for (PyObject* o : v) Py_XDECREF(o);
    Py_XDECREF(m);
    return r;
}

// Calls an entry point that makes a handle, and makes its Python object; a
// runtime class with methods of its own for that (_coll and the like) makes it
// through them.
template <class T, class F, class... A>
inline __attribute__((always_inline)) PyObject* make(RuntimeObject* rt, F Api::*fn, const char* name, A... args)
{
    if (rt->hooked) return call_hook(rt, Made<T>::hook, name, args...);
    T* out = nullptr;
    const int st = unlocked([&] { return (rt->api.*fn)(rt->h, args..., &out); });
    return st == EQG_OK ? new_handle(Made<T>::cls, rt, out) : raise_status(rt->api, st);
}
#define ENTRY(name) &Api::name, "eqg_" #name

// The handle of an object of a handle type.
inline bool own_handle(PyObject* o, void** h)
{
    *h = ((HandleObject*)o)->h;
    return ((HandleObject*)o)->rt || lacks(o, "h");
}

// The handle inside a Python object: a handle type's own, or the integer in
// its attribute `h`.
bool handle_of(PyObject* o, void** h)
{
    if (PyObject_TypeCheck(o, &CollBaseType) || PyObject_TypeCheck(o, &SetBaseType) ||
        PyObject_TypeCheck(o, &MaskBaseType))
        return own_handle(o, h);
    PyObject* v = PyObject_GetAttrString(o, "h");
    if (!v) return false;
    *h = v == Py_None ? nullptr : PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    return !PyErr_Occurred();
}

bool double_of(PyObject* o, double* v)
{
    if (PyFloat_CheckExact(o)) {
        *v = PyFloat_AS_DOUBLE(o);
        return true;
    }
    PyObject* f = PyNumber_Float(o);  // as float(o)
    if (!f) return false;
    *v = PyFloat_AS_DOUBLE(f);
    Py_DECREF(f);
    return true;
}

// ---- handles ---------------------------------------------------------------------
int handle_init(PyObject* self, PyObject* args, PyObject* kwargs)
{
    static const char* names[] = {"rt", "h", nullptr};
    PyObject *rt, *h;
    if (!PyArg_ParseTupleAndKeywords(args, kwargs, "O!O", (char**)names, &RuntimeBaseType, &rt, &h)) return -1;
    void* p = nullptr;
    if (h != Py_None) {
        p = PyLong_AsVoidPtr(h);
        if (!p && PyErr_Occurred()) return -1;
    }
    HandleObject* o = (HandleObject*)self;
    Py_INCREF(rt);
    Py_XSETREF(o->rt, (RuntimeObject*)rt);
    o->h = p;
    return 0;
}

// Whether there are other threads of the interpreter.  (Thread states are
// deleted with the interpreter lock held, which the caller has.)
bool other_threads()
{
    PyThreadState* head = PyInterpreterState_ThreadHead(PyInterpreterState_Get());
    return head && PyThreadState_Next(head);
}

// Gives the handle back to its library and lets go of the runtime.  Without
// the interpreter lock where another thread may want it: the release of a
// destroyed runtime's last handle waits for its stream.  (Letting the lock go
// takes 65 ns, a fifth of an operation on small collections.)  The object
// holds nothing any more when other threads may run.
template <class Release>
int handle_drop(PyObject* self, Release&& release)
{
    HandleObject* o = (HandleObject*)self;
    void* h = o->h;
    RuntimeObject* rt = o->rt;
    o->h = nullptr;
    o->rt = nullptr;
    if (h && rt && rt->bound) {
        if (other_threads()) {
            Py_BEGIN_ALLOW_THREADS
            release(rt->api, h);
            Py_END_ALLOW_THREADS
        } else {
            release(rt->api, h);
        }
    }
    Py_XDECREF(rt);
    return 0;
}
int coll_clear(PyObject* self)
{
    return handle_drop(self, [](const Api& a, void* h) { a.coll_release((eqg_coll*)h); });
}
int mask_clear(PyObject* self)
{
    return handle_drop(self, [](const Api& a, void* h) { a.mask_release((eqg_mask*)h); });
}
int set_clear(PyObject* self)
{
    return handle_drop(self, [](const Api& a, void* h) { a.set_release((eqg_set*)h); });
}
template <int (*Clear)(PyObject*)>
void handle_dealloc(PyObject* self)
{
    PyObject_GC_UnTrack(self);
    Clear(self);
    Py_TYPE(self)->tp_free(self);
}
int handle_traverse(PyObject* self, visitproc visit, void* arg)
{
    Py_VISIT(((HandleObject*)self)->rt);
    return 0;
}

PyObject* handle_get_rt(PyObject* self, void*)
{
    PyObject* rt = (PyObject*)((HandleObject*)self)->rt;
    return rt ? Py_NewRef(rt) : (PyObject*)lacks(self, "rt");
}
PyObject* handle_get_h(PyObject* self, void*)
{
    void* h = ((HandleObject*)self)->h;
    if (!((HandleObject*)self)->rt) return (PyObject*)lacks(self, "h");
    if (!h) Py_RETURN_NONE;
    return PyLong_FromVoidPtr(h);
}
int handle_set_h(PyObject* self, PyObject* v, void*)
{
    void* p = nullptr;
    if (v && v != Py_None) {
        p = PyLong_AsVoidPtr(v);
        if (!p && PyErr_Occurred()) return -1;
    }
    ((HandleObject*)self)->h = p;
    return 0;
}
PyGetSetDef handle_getset[] = {{"rt", handle_get_rt, nullptr, nullptr, nullptr},
                               {"h", handle_get_h, handle_set_h, nullptr, nullptr},
                               {nullptr, nullptr, nullptr, nullptr, nullptr}};

Py_hash_t identity_hash(PyObject* self) { return (Py_hash_t)((uintptr_t)self >> 4); }

// ---- scalar collections ------------------------------------------------------------
// left op right where at least one is a collection.
PyObject* coll_binary(int op, PyObject* left, PyObject* right)
{
    const bool l = PyObject_TypeCheck(left, &CollBaseType), r = PyObject_TypeCheck(right, &CollBaseType);
    HandleObject* self = (HandleObject*)(l ? left : right);
    RuntimeObject* rt = rt_of_handle((PyObject*)self);
    if (!rt) return nullptr;
    if (l && r) {
        void *a0, *b0;
        if (!own_handle(left, &a0) || !own_handle(right, &b0)) return nullptr;
        const eqg_coll *a = (eqg_coll*)a0, *b = (eqg_coll*)b0;
        return make<eqg_coll>(rt, ENTRY(binary), op, a, b);
    }
    double s;
    if (!double_of(l ? right : left, &s)) return nullptr;
    const eqg_coll* a = (eqg_coll*)self->h;
    return make<eqg_coll>(rt, ENTRY(binary_scalar), op, a, s, l ? 0 : 1);
}
PyObject* coll_add(PyObject* a, PyObject* b) { return coll_binary(EQG_ADD, a, b); }
PyObject* coll_sub(PyObject* a, PyObject* b) { return coll_binary(EQG_SUB, a, b); }
PyObject* coll_mul(PyObject* a, PyObject* b) { return coll_binary(EQG_MUL, a, b); }
PyObject* coll_div(PyObject* a, PyObject* b) { return coll_binary(EQG_DIV, a, b); }

PyObject* unary_of(RuntimeObject* rt, int op, const void* h)
{
    return make<eqg_coll>(rt, ENTRY(unary), op, (const eqg_coll*)h);
}
PyObject* coll_neg(PyObject* self)
{
    RuntimeObject* rt = rt_of_handle(self);
    return rt ? unary_of(rt, EQG_NEG, ((HandleObject*)self)->h) : nullptr;
}

PyObject* coll_compare_op(PyObject* self, int op, PyObject* other)
{
    RuntimeObject* rt = rt_of_handle(self);
    if (!rt) return nullptr;
    const eqg_coll* a = (eqg_coll*)((HandleObject*)self)->h;
    if (PyObject_TypeCheck(other, &CollBaseType)) {
        void* b0;
        if (!own_handle(other, &b0)) return nullptr;
        const eqg_coll* b = (eqg_coll*)b0;
        return make<eqg_mask>(rt, ENTRY(compare), op, a, b);
    }
    double v;
    if (!double_of(other, &v)) return nullptr;
    return make<eqg_mask>(rt, ENTRY(compare_scalar), op, a, v, 0);
}
PyObject* coll_richcompare(PyObject* self, PyObject* other, int op)
{
    switch (op) {
    case Py_LT: return coll_compare_op(self, EQG_LT, other);
    case Py_LE: return coll_compare_op(self, EQG_LE, other);
    case Py_GT: return coll_compare_op(self, EQG_GT, other);
    case Py_GE: return coll_compare_op(self, EQG_GE, other);
    default: Py_RETURN_NOTIMPLEMENTED;  // == and != compare identities
    }
}
PyObject* coll_eq(PyObject* self, PyObject* other) { return coll_compare_op(self, EQG_EQ, other); }
PyObject* coll_ne(PyObject* self, PyObject* other) { return coll_compare_op(self, EQG_NE, other); }

PyMethodDef coll_methods[] = {{"eq", coll_eq, METH_O, nullptr}, {"ne", coll_ne, METH_O, nullptr},
                              {nullptr, nullptr, 0, nullptr}};
PyNumberMethods coll_number = {};

// ---- masks ---------------------------------------------------------------------------
PyObject* mask_logic_op(int op, PyObject* self, PyObject* other)
{
    if (!PyObject_TypeCheck(self, &MaskBaseType)) Py_RETURN_NOTIMPLEMENTED;
    HandleObject* s = (HandleObject*)self;
    RuntimeObject* rt = rt_of_handle(self);
    if (!rt) return nullptr;
    void* b = nullptr;
    if (other && other != Py_None && !handle_of(other, &b)) return nullptr;
    return make<eqg_mask>(rt, ENTRY(mask_logic), op, (const eqg_mask*)s->h, (const eqg_mask*)b);
}
PyObject* mask_and(PyObject* a, PyObject* b) { return mask_logic_op(EQG_AND, a, b); }
PyObject* mask_or(PyObject* a, PyObject* b) { return mask_logic_op(EQG_OR, a, b); }
PyObject* mask_invert(PyObject* a) { return mask_logic_op(EQG_NOT, a, nullptr); }
PyNumberMethods mask_number = {};

// ---- runtime ----------------------------------------------------------------------------
// Positional and keyword arguments into v[0 .. n), of which the first `need`
// are required.
bool take(const char* fn, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames, const char* const* names, int n,
          int need, PyObject** v)
{
    for (int i = 0; i < n; ++i) v[i] = nullptr;
    if (nargs > n) {
        PyErr_Format(PyExc_TypeError, "%s() takes at most %d arguments (%zd given)", fn, n, nargs);
        return false;
    }
    for (Py_ssize_t i = 0; i < nargs; ++i) v[i] = args[i];
    const Py_ssize_t nk = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
    for (Py_ssize_t k = 0; k < nk; ++k) {
        PyObject* name = PyTuple_GET_ITEM(kwnames, k);
        int at = -1;
        for (int i = 0; i < n; ++i)
            if (PyUnicode_CompareWithASCIIString(name, names[i]) == 0) at = i;
        if (at < 0 || v[at]) {
            PyErr_Format(PyExc_TypeError, "%s() got an unexpected or repeated keyword argument '%U'", fn, name);
            return false;
        }
        v[at] = args[nargs + k];
    }
    for (int i = 0; i < need; ++i)
        if (!v[i]) {
            PyErr_Format(PyExc_TypeError, "%s() missing required argument: '%s'", fn, names[i]);
            return false;
        }
    return true;
}

#define METHOD_ARGS PyObject *self, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames

// Methods of one collection argument.
template <class F>
PyObject* coll_method(METHOD_ARGS, const char* name, F Api::*fn, const char* entry)
{
    static const char* const names[] = {"x"};
    PyObject* v[1];
    void* h;
    if (!take(name, args, nargs, kwnames, names, 1, 1, v) || !handle_of(v[0], &h)) return nullptr;
    RuntimeObject* rt = rt_of(self);
    if (!rt) return nullptr;
    return make<eqg_coll>(rt, fn, entry, (const eqg_coll*)h);
}
PyObject* rt_gradient(METHOD_ARGS)
{
    return coll_method(self, args, nargs, kwnames, "gradient", ENTRY(gradient));
}
PyObject* rt_neg_gradient(METHOD_ARGS)
{
    return coll_method(self, args, nargs, kwnames, "negGradient", ENTRY(neg_gradient));
}
PyObject* rt_divergence(METHOD_ARGS)
{
    return coll_method(self, args, nargs, kwnames, "divergence", ENTRY(divergence));
}
PyObject* rt_interior_divergence(METHOD_ARGS)
{
    return coll_method(self, args, nargs, kwnames, "interiorDivergence", ENTRY(interior_divergence));
}
PyObject* rt_sqrt(METHOD_ARGS)
{
    static const char* const names[] = {"x"};
    PyObject* v[1];
    void* h;
    if (!take("sqrt", args, nargs, kwnames, names, 1, 1, v) || !handle_of(v[0], &h)) return nullptr;
    RuntimeObject* rt = rt_of(self);
    return rt ? unary_of(rt, EQG_SQRT, h) : nullptr;
}

PyObject* builtin_set(PyObject* self, int which)
{
    RuntimeObject* rt = rt_of(self);
    if (!rt) return nullptr;
    return make<eqg_set>(rt, ENTRY(set_builtin), which);
}
PyObject* rt_all_cells(PyObject* self, PyObject*) { return builtin_set(self, EQG_ALL_CELLS); }
PyObject* rt_boundary_cells(PyObject* self, PyObject*) { return builtin_set(self, EQG_BOUNDARY_CELLS); }
PyObject* rt_interior_cells(PyObject* self, PyObject*) { return builtin_set(self, EQG_INTERIOR_CELLS); }
PyObject* rt_all_faces(PyObject* self, PyObject*) { return builtin_set(self, EQG_ALL_FACES); }
PyObject* rt_boundary_faces(PyObject* self, PyObject*) { return builtin_set(self, EQG_BOUNDARY_FACES); }
PyObject* rt_interior_faces(PyObject* self, PyObject*) { return builtin_set(self, EQG_INTERIOR_FACES); }

template <class F>
PyObject* set_method(METHOD_ARGS, const char* name, F Api::*fn, const char* entry)
{
    static const char* const names[] = {"faces"};
    PyObject* v[1];
    void* h;
    if (!take(name, args, nargs, kwnames, names, 1, 1, v) || !handle_of(v[0], &h)) return nullptr;
    RuntimeObject* rt = rt_of(self);
    if (!rt) return nullptr;
    return make<eqg_set>(rt, fn, entry, (const eqg_set*)h);
}
PyObject* rt_first_cell(METHOD_ARGS)
{
    return set_method(self, args, nargs, kwnames, "firstCell", ENTRY(first_cell));
}
PyObject* rt_second_cell(METHOD_ARGS)
{
    return set_method(self, args, nargs, kwnames, "secondCell", ENTRY(second_cell));
}

PyObject* constant_of(RuntimeObject* rt, PyObject* value, int64_t n)
{
    if (rt->hooked) return PyObject_CallMethod((PyObject*)rt, "constant", "OL", value, (long long)n);
    double s;
    if (!double_of(value, &s)) return nullptr;
    return make<eqg_coll>(rt, ENTRY(coll_constant), s, n);
}

// operatorExtend(data, a, b=None): a constant over a, or data from a to b.
PyObject* rt_extend(METHOD_ARGS)
{
    static const char* const names[] = {"data", "a", "b"};
    PyObject* v[3];
    if (!take("operatorExtend", args, nargs, kwnames, names, 3, 2, v)) return nullptr;
    RuntimeObject* rt = rt_of(self);
    if (!rt) return nullptr;
    if (!v[2] || v[2] == Py_None) {
        int64_t n = 0;
        if (PyObject_TypeCheck(v[1], &SetBaseType)) {
            RuntimeObject* owner = rt_of_handle(v[1]);
            if (!owner) return nullptr;
            const int st = owner->api.set_size((eqg_set*)((HandleObject*)v[1])->h, &n);
            if (st != EQG_OK) return raise_status(owner->api, st);
        } else {
            n = PyObject_Size(v[1]);
            if (n < 0) return nullptr;
        }
        return constant_of(rt, v[0], n);
    }
    void *d, *a, *b;
    if (!handle_of(v[0], &d) || !handle_of(v[1], &a) || !handle_of(v[2], &b)) return nullptr;
    const eqg_set *from = (eqg_set*)a, *to = (eqg_set*)b;
    if (PyObject_TypeCheck(v[0], &SetBaseType))
        return make<eqg_set>(rt, ENTRY(set_extend), (const eqg_set*)d, from, to);
    return make<eqg_coll>(rt, ENTRY(extend), (const eqg_coll*)d, from, to);
}

PyObject* rt_on(METHOD_ARGS)
{
    static const char* const names[] = {"data", "from_set", "to_set"};
    PyObject* v[3];
    void *d, *a, *b;
    if (!take("operatorOn", args, nargs, kwnames, names, 3, 3, v) || !handle_of(v[0], &d) || !handle_of(v[1], &a) ||
        !handle_of(v[2], &b))
        return nullptr;
    RuntimeObject* rt = rt_of(self);
    if (!rt) return nullptr;
    const eqg_set *from = (eqg_set*)a, *to = (eqg_set*)b;
    if (PyObject_TypeCheck(v[0], &SetBaseType))
        return make<eqg_set>(rt, ENTRY(set_on), (const eqg_set*)d, from, to);
    return make<eqg_coll>(rt, ENTRY(on), (const eqg_coll*)d, from, to);
}

PyObject* rt_trinary_if(METHOD_ARGS)
{
    static const char* const names[] = {"pred", "a", "b"};
    PyObject* v[3];
    void *m, *a, *b;
    if (!take("trinaryIf", args, nargs, kwnames, names, 3, 3, v) || !handle_of(v[0], &m) || !handle_of(v[1], &a) ||
        !handle_of(v[2], &b))
        return nullptr;
    RuntimeObject* rt = rt_of(self);
    if (!rt) return nullptr;
    const eqg_mask* p = (eqg_mask*)m;
    if (PyObject_TypeCheck(v[1], &SetBaseType))
        return make<eqg_set>(rt, ENTRY(set_select), p, (const eqg_set*)a, (const eqg_set*)b);
    return make<eqg_coll>(rt, ENTRY(select), p, (const eqg_coll*)a, (const eqg_coll*)b);
}

PyObject* reduce_of(METHOD_ARGS, const char* name, int op)
{
    static const char* const names[] = {"x"};
    PyObject* v[1];
    void* h;
    if (!take(name, args, nargs, kwnames, names, 1, 1, v) || !handle_of(v[0], &h)) return nullptr;
    RuntimeObject* rt = rt_of(self);
    if (!rt) return nullptr;
    double r = 0.0;
    const int st = unlocked([&] {
        return op < 0 ? rt->api.two_norm(rt->h, (eqg_coll*)h, &r) : rt->api.reduce(rt->h, op, (eqg_coll*)h, &r);
    });
    if (rt->hooked) {
        PyObject* checked = PyObject_CallMethod((PyObject*)rt, "_ok", "i", st);
        if (!checked) return nullptr;
        Py_DECREF(checked);
        return PyFloat_FromDouble(r);
    }
    return st == EQG_OK ? PyFloat_FromDouble(r) : raise_status(rt->api, st);
}
PyObject* rt_min(METHOD_ARGS) { return reduce_of(self, args, nargs, kwnames, "minReduce", EQG_MIN); }
PyObject* rt_max(METHOD_ARGS) { return reduce_of(self, args, nargs, kwnames, "maxReduce", EQG_MAX); }
PyObject* rt_sum(METHOD_ARGS) { return reduce_of(self, args, nargs, kwnames, "sumReduce", EQG_SUM); }
PyObject* rt_prod(METHOD_ARGS) { return reduce_of(self, args, nargs, kwnames, "prodReduce", EQG_PROD); }
PyObject* rt_two_norm(METHOD_ARGS) { return reduce_of(self, args, nargs, kwnames, "twoNorm", -1); }

// spanSubset(u, start, num), spanSuperset(u, start, total)
PyObject* span_of(METHOD_ARGS, bool subset)
{
    static const char* const names[2][3] = {{"u", "start", "total"}, {"u", "start", "num"}};
    PyObject* v[3];
    void* h;
    if (!take(subset ? "spanSubset" : "spanSuperset", args, nargs, kwnames, names[subset ? 1 : 0], 3, 3, v) ||
        !handle_of(v[0], &h))
        return nullptr;
    int64_t n[2];
    for (int i = 0; i < 2; ++i) {
        PyObject* l = PyNumber_Long(v[i + 1]);  // as int(...)
        if (!l) return nullptr;
        n[i] = PyLong_AsLongLong(l);
        Py_DECREF(l);
        if (n[i] == -1 && PyErr_Occurred()) return nullptr;
    }
    RuntimeObject* rt = rt_of(self);
    if (!rt) return nullptr;
    const eqg_coll* x = (const eqg_coll*)h;
    return subset ? make<eqg_coll>(rt, ENTRY(span_subset), x, n[0], n[1])
                  : make<eqg_coll>(rt, ENTRY(span_superset), x, n[0], n[1]);
}
PyObject* rt_span_subset(METHOD_ARGS) { return span_of(self, args, nargs, kwnames, true); }
PyObject* rt_span_superset(METHOD_ARGS) { return span_of(self, args, nargs, kwnames, false); }

// _bind({name: address}, hooked=False): the entry points of the runtime's
// library, and whether handles go through methods that its class overrides.
PyObject* rt_bind(PyObject* self, PyObject* args)
{
    RuntimeObject* rt = (RuntimeObject*)self;
    PyObject* table;
    int hooked = 0;
    if (!PyArg_ParseTuple(args, "O|p", &table, &hooked)) return nullptr;
    for (const Entry& e : kEntries) {
        PyObject* a = PyMapping_GetItemString(table, e.name);
        if (!a) return nullptr;
        void* p = PyLong_AsVoidPtr(a);
        Py_DECREF(a);
        if (!p) {
            if (!PyErr_Occurred()) PyErr_Format(PyExc_ValueError, "no address of %s", e.name);
            return nullptr;
        }
        std::memcpy((char*)&rt->api + e.offset, &p, sizeof(p));
    }
    rt->bound = true;
    rt->hooked = hooked != 0;
    Py_RETURN_NONE;
}

PyObject* rt_get_h(PyObject* self, void*)
{
    eqg_runtime* h = ((RuntimeObject*)self)->h;
    if (!((RuntimeObject*)self)->created) return (PyObject*)lacks(self, "h");
    if (!h) Py_RETURN_NONE;
    return PyLong_FromVoidPtr(h);
}
int rt_set_h(PyObject* self, PyObject* v, void*)
{
    void* p = nullptr;
    if (v && v != Py_None) {
        p = PyLong_AsVoidPtr(v);
        if (!p && PyErr_Occurred()) return -1;
    }
    ((RuntimeObject*)self)->h = (eqg_runtime*)p;
    ((RuntimeObject*)self)->created = true;
    return 0;
}
PyGetSetDef rt_getset[] = {{"h", rt_get_h, rt_set_h, nullptr, nullptr}, {nullptr, nullptr, nullptr, nullptr, nullptr}};

#define FAST(f) (PyCFunction)(void (*)(void))(f), METH_FASTCALL | METH_KEYWORDS, nullptr
PyMethodDef rt_methods[] = {{"_bind", rt_bind, METH_VARARGS, nullptr},
                            {"gradient", FAST(rt_gradient)},
                            {"negGradient", FAST(rt_neg_gradient)},
                            {"divergence", FAST(rt_divergence)},
                            {"interiorDivergence", FAST(rt_interior_divergence)},
                            {"sqrt", FAST(rt_sqrt)},
                            {"allCells", rt_all_cells, METH_NOARGS, nullptr},
                            {"boundaryCells", rt_boundary_cells, METH_NOARGS, nullptr},
                            {"interiorCells", rt_interior_cells, METH_NOARGS, nullptr},
                            {"allFaces", rt_all_faces, METH_NOARGS, nullptr},
                            {"boundaryFaces", rt_boundary_faces, METH_NOARGS, nullptr},
                            {"interiorFaces", rt_interior_faces, METH_NOARGS, nullptr},
                            {"firstCell", FAST(rt_first_cell)},
                            {"secondCell", FAST(rt_second_cell)},
                            {"operatorExtend", FAST(rt_extend)},
                            {"operatorOn", FAST(rt_on)},
                            {"trinaryIf", FAST(rt_trinary_if)},
                            {"minReduce", FAST(rt_min)},
                            {"maxReduce", FAST(rt_max)},
                            {"sumReduce", FAST(rt_sum)},
                            {"prodReduce", FAST(rt_prod)},
                            {"twoNorm", FAST(rt_two_norm)},
                            {"spanSubset", FAST(rt_span_subset)},
                            {"spanSuperset", FAST(rt_span_superset)},
                            {nullptr, nullptr, 0, nullptr}};

PyTypeObject make_type(const char* name, size_t size)
{
    PyTypeObject t = {PyVarObject_HEAD_INIT(nullptr, 0)};
    t.tp_name = name;
    t.tp_basicsize = (Py_ssize_t)size;
    t.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE;
    t.tp_new = PyType_GenericNew;
    return t;
}
PyTypeObject RuntimeBaseType = make_type("equelle_b200._mirror.RuntimeBase", sizeof(RuntimeObject));
PyTypeObject CollBaseType = make_type("equelle_b200._mirror.CollBase", sizeof(HandleObject));
PyTypeObject MaskBaseType = make_type("equelle_b200._mirror.MaskBase", sizeof(HandleObject));
PyTypeObject SetBaseType = make_type("equelle_b200._mirror.SetBase", sizeof(HandleObject));

// register_classes(CollOfScalar, CollOfBool, EntitySet, EqgError)
PyObject* register_classes(PyObject*, PyObject* args)
{
    PyObject *c, *m, *s, *e;
    if (!PyArg_ParseTuple(args, "OOOO", &c, &m, &s, &e)) return nullptr;
    if (!PyType_Check(c) || !PyType_IsSubtype((PyTypeObject*)c, &CollBaseType) || !PyType_Check(m) ||
        !PyType_IsSubtype((PyTypeObject*)m, &MaskBaseType) || !PyType_Check(s) ||
        !PyType_IsSubtype((PyTypeObject*)s, &SetBaseType)) {
        PyErr_SetString(PyExc_TypeError, "the classes must derive from CollBase, MaskBase and SetBase");
        return nullptr;
    }
    Py_XSETREF(Made<eqg_coll>::cls, Py_NewRef(c));
    Py_XSETREF(Made<eqg_mask>::cls, Py_NewRef(m));
    Py_XSETREF(Made<eqg_set>::cls, Py_NewRef(s));
    Py_XSETREF(g_error_class, Py_NewRef(e));
    Py_RETURN_NONE;
}

// entry_points(): the names that RuntimeBase._bind needs addresses of.
PyObject* entry_points(PyObject*, PyObject*)
{
    const Py_ssize_t n = sizeof(kEntries) / sizeof(kEntries[0]);
    PyObject* t = PyTuple_New(n);
    for (Py_ssize_t i = 0; t && i < n; ++i) {
        PyObject* s = PyUnicode_FromString(kEntries[i].name);
        if (!s) {
            Py_DECREF(t);
            return nullptr;
        }
        PyTuple_SET_ITEM(t, i, s);
    }
    return t;
}

PyMethodDef module_methods[] = {{"register_classes", register_classes, METH_VARARGS, nullptr},
                                {"entry_points", entry_points, METH_NOARGS, nullptr},
                                {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_mirror", nullptr, -1, module_methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__mirror(void)
{
    RuntimeBaseType.tp_methods = rt_methods;
    RuntimeBaseType.tp_getset = rt_getset;
    coll_number.nb_add = coll_add;
    coll_number.nb_subtract = coll_sub;
    coll_number.nb_multiply = coll_mul;
    coll_number.nb_true_divide = coll_div;
    coll_number.nb_negative = coll_neg;
    CollBaseType.tp_as_number = &coll_number;
    CollBaseType.tp_richcompare = coll_richcompare;
    CollBaseType.tp_hash = identity_hash;
    CollBaseType.tp_methods = coll_methods;
    CollBaseType.tp_dealloc = handle_dealloc<coll_clear>;
    CollBaseType.tp_clear = coll_clear;
    mask_number.nb_and = mask_and;
    mask_number.nb_or = mask_or;
    mask_number.nb_invert = mask_invert;
    MaskBaseType.tp_as_number = &mask_number;
    MaskBaseType.tp_dealloc = handle_dealloc<mask_clear>;
    MaskBaseType.tp_clear = mask_clear;
    SetBaseType.tp_dealloc = handle_dealloc<set_clear>;
    SetBaseType.tp_clear = set_clear;
    for (PyTypeObject* t : {&CollBaseType, &MaskBaseType, &SetBaseType}) {
        t->tp_flags |= Py_TPFLAGS_HAVE_GC;
        t->tp_traverse = handle_traverse;
        t->tp_getset = handle_getset;
        t->tp_init = handle_init;
    }
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    const struct {
        const char* name;
        PyTypeObject* type;
    } types[] = {{"RuntimeBase", &RuntimeBaseType}, {"CollBase", &CollBaseType}, {"MaskBase", &MaskBaseType},
                 {"SetBase", &SetBaseType}};
    for (const auto& t : types) {
        if (PyType_Ready(t.type) < 0 || PyModule_AddObjectRef(m, t.name, (PyObject*)t.type) < 0) {
            Py_DECREF(m);
            return nullptr;
        }
    }
    return m;
}
