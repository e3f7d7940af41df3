// The calls of the kernels' C ABI that a Python program makes once per launch, without ctypes between: ctypes takes 0.75 us for a
// call with five arguments and 1.3 for seven, as much as half of the launch behind it (2.2 us in the driver), and small calls wait for
// nothing else.  The two launches of a small operand (513 x 1040 to fp8) 7.4 -> 5.7 us, a bandwidth step over short arrays 31 -> 29.
//
// A call takes plain int, float and None arguments, and byref() of a clpk_gemm_args_t.  Whatever else ctypes would accept, convert
// or refuse goes to the ctypes wrapper, which is handed over when the call is bound.  The GIL is released meanwhile, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <limits>
#include <string.h>
#include <tuple>
#include <type_traits>
#include <utility>

#include "clpeak_b200_kernels.h"

namespace {

struct Call {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    void *fn;
    PyObject *slow;              // the ctypes wrapper
    PyObject *failed;            // raises for a status
    PyTypeObject *byref_type, *gemm_args_type;
    Py_ssize_t address_at;       // see where_the_address_lies
};

const void *address_in(PyObject *byref, Py_ssize_t at)
{
    const void *p;
    memcpy(&p, reinterpret_cast<const char *>(byref) + at, sizeof p);
    return p;
}

// Where a byref object keeps the address that it carries.  No interface says so, so it is looked for: the one word that is the
// structure's address plus the offset, for several structures and offsets.  0: no word is, or more than one.
Py_ssize_t where_the_address_lies(PyObject *byref, PyObject *args_type)
{
    Py_ssize_t at = 0;
    for (int round = 0; round < 4; round++) {
        PyObject *args = PyObject_CallNoArgs(args_type), *ref = args ? PyObject_CallFunction(byref, "Oi", args, 24 * round) : nullptr;
        Py_buffer buffer = {};
        Py_ssize_t found = 0;
        if (ref && PyObject_GetBuffer(args, &buffer, PyBUF_SIMPLE) == 0) {
            for (Py_ssize_t i = sizeof(PyObject); i + (Py_ssize_t)sizeof(void *) <= Py_TYPE(ref)->tp_basicsize; i += sizeof(void *))
                if (address_in(ref, i) == static_cast<const char *>(buffer.buf) + 24 * round)
                    found = found == 0 ? i : -1;
            PyBuffer_Release(&buffer);
        }
        Py_XDECREF(ref);
        Py_XDECREF(args);
        PyErr_Clear();
        if (found <= 0 || (at != 0 && found != at))
            return 0;
        at = found;
    }
    return at;
}

// One argument on its way from Python; false: not plain
template <typename T, typename = void> struct Arg {
    static_assert(std::is_integral<T>::value, "integers, floats and pointers");
    T v;
    bool from(const Call *, PyObject *o)
    {
        if (!PyLong_CheckExact(o))
            return false;
        int overflow = 0;
        const long long x = PyLong_AsLongLongAndOverflow(o, &overflow);
        if (overflow > 0 && std::is_same<T, uint64_t>::value) {
            v = (T)PyLong_AsUnsignedLongLong(o);
            if (!PyErr_Occurred())
                return true;
            PyErr_Clear();
            return false;
        }
        if (overflow || (std::is_unsigned<T>::value && x < 0) || (sizeof(T) < 8 && (x < (long long)std::numeric_limits<T>::min() || x > (long long)std::numeric_limits<T>::max())))
            return false;
        v = (T)x;
        return true;
    }
    void done() {}
};

template <> struct Arg<float> {
    float v;
    bool from(const Call *, PyObject *o)
    {
        if (!PyFloat_CheckExact(o))
            return false;
        v = (float)PyFloat_AS_DOUBLE(o);
        return true;
    }
    void done() {}
};

template <typename P> struct Arg<P *, std::enable_if_t<!std::is_same<P, const clpk_gemm_args_t>::value>> {
    P *v;
    bool from(const Call *, PyObject *o)
    {
        if (o == Py_None) {
            v = nullptr;
            return true;
        }
        if (!PyLong_CheckExact(o))
            return false;
        const unsigned long long x = PyLong_AsUnsignedLongLong(o);
        if (x == (unsigned long long)-1 && PyErr_Occurred()) {
            PyErr_Clear();
            return false;
        }
        v = reinterpret_cast<P *>((uintptr_t)x);
        return true;
    }
    void done() {}
};

// byref(args): the structure lies in the buffer of the object that it refers to, unless byref was given an offset: only where the
// address that it carries is the buffer's.
template <> struct Arg<const clpk_gemm_args_t *> {
    const clpk_gemm_args_t *v = nullptr;
    Py_buffer buffer = {};
    bool from(const Call *call, PyObject *o)
    {
        if (Py_TYPE(o) != call->byref_type || call->address_at == 0)
            return false;
        static PyObject *const name = PyUnicode_InternFromString("_obj");
        PyObject *args = PyObject_GetAttr(o, name);
        if (!args) {
            PyErr_Clear();
            return false;
        }
        bool ok = Py_TYPE(args) == call->gemm_args_type;
        if (ok && PyObject_GetBuffer(args, &buffer, PyBUF_SIMPLE) != 0) {
            PyErr_Clear();
            ok = false;
        }
        Py_DECREF(args);                                     // the buffer holds the object
        if (ok && (buffer.len != (Py_ssize_t)sizeof(clpk_gemm_args_t) || address_in(o, call->address_at) != buffer.buf)) {
            done();
            ok = false;
        }
        if (ok)
            v = static_cast<const clpk_gemm_args_t *>(buffer.buf);
        return ok;
    }
    void done() { PyBuffer_Release(&buffer); }
};

template <typename... A, size_t... I>
PyObject *invoke_with(Call *call, PyObject *const *args, std::index_sequence<I...>, size_t nargsf)
{
    std::tuple<Arg<A>...> v;
    size_t taken = 0;
    const bool plain = ((std::get<I>(v).from(call, args[I]) && ++taken) && ...);
    int rc = 0;
    if (plain) {
        Py_BEGIN_ALLOW_THREADS
        rc = reinterpret_cast<int (*)(A...)>(call->fn)(std::get<I>(v).v...);
        Py_END_ALLOW_THREADS
    }
    ((I < taken ? std::get<I>(v).done() : void()), ...);
    if (!plain)
        return PyObject_Vectorcall(call->slow, args, nargsf, nullptr);
    if (rc == CLPK_OK)
        Py_RETURN_NONE;
    return PyObject_CallFunction(call->failed, "i", rc);
}

template <typename... A>
PyObject *invoke(PyObject *self, PyObject *const *args, size_t nargsf, PyObject *names)
{
    Call *call = reinterpret_cast<Call *>(self);
    if (names || PyVectorcall_NARGS(nargsf) != (Py_ssize_t)sizeof...(A))
        return PyObject_Vectorcall(call->slow, args, nargsf, names);
    return invoke_with<A...>(call, args, std::index_sequence_for<A...>(), nargsf);
}

template <typename... A> constexpr vectorcallfunc invoker(int (*)(A...)) { return invoke<A...>; }

// the signatures are the header's
#define CALL(name) {#name, invoker(static_cast<decltype(&name)>(nullptr))}
const struct {
    const char *name;
    vectorcallfunc invoke;
} kCalls[] = {CALL(clpk_fill_f32), CALL(clpk_fill_i8), CALL(clpk_convert_f32), CALL(clpk_absmax_f32), CALL(clpk_quantize_fp4), CALL(clpk_stream_read),
              CALL(clpk_stream_copy), CALL(clpk_stream_triad), CALL(clpk_gemm), CALL(clpk_gemm_pack_scales)};

int call_traverse(PyObject *self, visitproc visit, void *arg)
{
    Call *c = reinterpret_cast<Call *>(self);
    Py_VISIT(c->slow);
    Py_VISIT(c->failed);
    Py_VISIT(c->byref_type);
    Py_VISIT(c->gemm_args_type);
    return 0;
}
int call_clear(PyObject *self)
{
    Call *c = reinterpret_cast<Call *>(self);
    Py_CLEAR(c->slow);
    Py_CLEAR(c->failed);
    Py_CLEAR(c->byref_type);
    Py_CLEAR(c->gemm_args_type);
    return 0;
}
void call_dealloc(PyObject *self)
{
    PyObject_GC_UnTrack(self);
    call_clear(self);
    PyObject_GC_Del(self);
}

PyTypeObject CallType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// bind(name, address, slow, failed, byref, its type, args type): the call, or None for a name that has none here
PyObject *bind(PyObject *, PyObject *args)
{
    const char *name;
    unsigned long long address;
    PyObject *slow, *failed, *byref, *byref_type, *args_type;
    if (!PyArg_ParseTuple(args, "sKOOOO!O!", &name, &address, &slow, &failed, &byref, &PyType_Type, &byref_type, &PyType_Type, &args_type))
        return nullptr;
    for (const auto &c : kCalls)
        if (strcmp(c.name, name) == 0) {
            Call *call = PyObject_GC_New(Call, &CallType);
            if (!call)
                return nullptr;
            call->vectorcall = c.invoke;
            call->fn = reinterpret_cast<void *>((uintptr_t)address);
            call->slow = Py_NewRef(slow);
            call->failed = Py_NewRef(failed);
            call->byref_type = reinterpret_cast<PyTypeObject *>(Py_NewRef(byref_type));
            call->gemm_args_type = reinterpret_cast<PyTypeObject *>(Py_NewRef(args_type));
            call->address_at = where_the_address_lies(byref, args_type);
            PyObject_GC_Track(reinterpret_cast<PyObject *>(call));
            return reinterpret_cast<PyObject *>(call);
        }
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {{"bind", bind, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_clpk_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__clpk_calls(void)
{
    CallType.tp_name = "_clpk_calls.Call";
    CallType.tp_basicsize = sizeof(Call);
    CallType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_HAVE_GC;
    CallType.tp_vectorcall_offset = offsetof(Call, vectorcall);
    CallType.tp_call = PyVectorcall_Call;
    CallType.tp_traverse = call_traverse;
    CallType.tp_clear = call_clear;
    CallType.tp_dealloc = call_dealloc;
    if (PyType_Ready(&CallType) < 0)
        return nullptr;
    return PyModule_Create(&kModule);
}
