// fast_call.cpp — the launcher boundary as a CPython extension (ntransformer_b200/_fast.so): what kernels.py's launch_* do with their arguments, without ctypes.
//
// Bound by the host: a call through ctypes takes 4.6 us, of them 2.5 in the driver's launch, the rest in ctypes' conversions and the checks in Python.  A small matrix
// (Q8_0, 1024 x 4096) times a vector, call after call: 4.64 -> 3.87 us, the GPU's time; a decoder layer's sixteen launches on an idle GPU 112 -> 99 us.
// The library's entries come as addresses from the library that is loaded (bind), so that an override of its path holds here too.  The GIL is let go
// around the launch, as ctypes does.  Only the plain forms of an argument are taken here (a tensor, an int, a float, None, a stream object); a call with any
// other goes to kernels.py's own route through ctypes, which takes and refuses what it always did.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <cstddef>
#include <cstdint>
#include <tuple>
#include <type_traits>
#include <utility>
#include "../../include/nt_b200.h"

namespace {

PyObject *tensor_type, *raw_stream, *current_device, *cuda_init, *other_route, *s_is_cuda, *s_is_contiguous, *s_data_ptr, *s_cuda_stream;

// Each conversion returns false with a Python error set, or false without one: not a plain form.
// a contiguous CUDA tensor's address, a raw address, or None
bool to_pointer(PyObject* o, const void*& p) {
    if (PyObject_TypeCheck(o, reinterpret_cast<PyTypeObject*>(tensor_type))) {
        PyObject* cuda = PyObject_GetAttr(o, s_is_cuda);
        if (!cuda) return false;
        const int on = PyObject_IsTrue(cuda);
        Py_DECREF(cuda);
        if (on < 0) return false;
        int flat = 0;
        if (on) {
            PyObject* c = PyObject_VectorcallMethod(s_is_contiguous, &o, 1, nullptr);
            if (!c) return false;
            flat = PyObject_IsTrue(c);
            Py_DECREF(c);
            if (flat < 0) return false;
        }
        if (!flat) { PyErr_SetString(PyExc_AssertionError, "expected a contiguous CUDA tensor"); return false; }
        PyObject* a = PyObject_VectorcallMethod(s_data_ptr, &o, 1, nullptr);
        if (!a) return false;
        p = PyLong_AsVoidPtr(a);
        Py_DECREF(a);
        return !PyErr_Occurred();
    }
    if (o == Py_None) { p = nullptr; return true; }
    if (!PyLong_Check(o)) return false;
    p = reinterpret_cast<const void*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(o)));
    return !PyErr_Occurred();
}
bool to_int(PyObject* o, int& v) {
    if (!PyLong_Check(o)) return false;
    v = static_cast<int>(PyLong_AsUnsignedLongMask(o));
    return !PyErr_Occurred();
}
// None: the current stream of the current device; a stream object; a raw stream
bool to_stream(PyObject* o, void*& s) {
    if (o == Py_None) {
        if (cuda_init) {
            PyObject* done = PyObject_CallNoArgs(cuda_init);
            if (!done) return false;
            Py_DECREF(done);
            Py_CLEAR(cuda_init);
        }
        PyObject* d = PyObject_CallNoArgs(current_device);
        if (!d) return false;
        PyObject* r = PyObject_CallOneArg(raw_stream, d);
        Py_DECREF(d);
        if (!r) return false;
        s = reinterpret_cast<void*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(r)));
        Py_DECREF(r);
        return !PyErr_Occurred();
    }
    PyObject* r = PyObject_GetAttr(o, s_cuda_stream);
    if (!r) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return false;
        PyErr_Clear();
        if (!PyLong_Check(o)) return false;
        r = Py_NewRef(o);
    }
    s = reinterpret_cast<void*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(r)));
    Py_DECREF(r);
    return !PyErr_Occurred();
}
template <class T> bool convert(PyObject* o, T& v) {
    if constexpr (std::is_pointer_v<T>) {
        const void* p = nullptr;
        if (!to_pointer(o, p)) return false;
        v = static_cast<T>(const_cast<void*>(p));
        return true;
    } else if constexpr (std::is_same_v<T, float>) {
        if (!PyFloat_Check(o) && !PyLong_Check(o)) return false;
        v = static_cast<float>(PyFloat_AsDouble(o));
        return !PyErr_Occurred();
    } else {
        static_assert(std::is_same_v<T, int>);
        return to_int(o, v);
    }
}

template <class F> struct Entry;
template <class... A> struct Entry<void(A...)> {
    static constexpr size_t N = sizeof...(A);
    template <size_t I, class T>
    static bool argument(PyObject* o, T& v) {
        if constexpr (I + 1 == N) return to_stream(o, v);          // the last parameter is the stream
        else return convert(o, v);
    }
    template <size_t... I>
    static PyObject* call(const char* name, void (*fn)(A...), PyObject* const* args, std::index_sequence<I...>) {
        std::tuple<A...> v{};
        const bool ok = (argument<I>(args[I], std::get<I>(v)) && ...);
        if (!ok) {
            if (PyErr_Occurred()) return nullptr;
            PyObject* list = PyTuple_New(N);
            if (!list) return nullptr;
            (PyTuple_SET_ITEM(list, I, Py_NewRef(args[I])), ...);
            PyObject* r = PyObject_CallFunction(other_route, "sO", name, list);
            Py_DECREF(list);
            return r;
        }
        Py_BEGIN_ALLOW_THREADS
        fn(std::get<I>(v)...);
        Py_END_ALLOW_THREADS
        Py_RETURN_NONE;
    }
};

#define NT_ENTRIES(X) \
    X(rmsnorm) X(rmsnorm_f16) X(rope) X(softmax) X(masked_softmax) X(gemv) X(gemv_add) X(gemm_f32) X(silu_mul) X(add_bias) X(attention_decode) X(attention_prefill) X(copy_to_kv_cache) X(add) X(add_inplace) X(copy) X(cosine_similarity)

#define NT_ONE(name)                                                                                                            \
    decltype(nt_b200_##name)* at_##name;                                                                                        \
    PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t n) {                                                       \
        using E = Entry<decltype(nt_b200_##name)>;                                                                              \
        if (n != (Py_ssize_t)E::N) { PyErr_Format(PyExc_TypeError, #name ": %zd arguments, %zu expected", n, E::N); return nullptr; }   \
        if (!at_##name) { PyErr_SetString(PyExc_RuntimeError, #name ": not bound"); return nullptr; }                            \
        return E::call(#name, at_##name, args, std::make_index_sequence<E::N>());                                                       \
    }
NT_ENTRIES(NT_ONE)

// bind(Tensor type, current raw stream of a device, current device, init of CUDA, route of other arguments (name, arguments), {name: address})
PyObject* bind(PyObject*, PyObject* args) {
    PyObject *type, *raw, *device, *init, *other, *table;
    if (!PyArg_ParseTuple(args, "O!OOOOO!", &PyType_Type, &type, &raw, &device, &init, &other, &PyDict_Type, &table)) return nullptr;
#define NT_BIND(name)                                                                                                           \
    {                                                                                                                           \
        PyObject* a = PyDict_GetItemString(table, #name);                                                                       \
        if (!a) { PyErr_SetString(PyExc_KeyError, #name); return nullptr; }                                                      \
        at_##name = reinterpret_cast<decltype(at_##name)>(PyLong_AsVoidPtr(a));                                                  \
        if (PyErr_Occurred()) return nullptr;                                                                                    \
    }
    NT_ENTRIES(NT_BIND)
    Py_XSETREF(tensor_type, Py_NewRef(type));
    Py_XSETREF(raw_stream, Py_NewRef(raw));
    Py_XSETREF(current_device, Py_NewRef(device));
    Py_XSETREF(cuda_init, Py_NewRef(init));
    Py_XSETREF(other_route, Py_NewRef(other));
    Py_RETURN_NONE;
}

#define NT_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr},
#define NT_NAME(name) #name,
PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, nullptr}, NT_ENTRIES(NT_METHOD) {nullptr, nullptr, 0, nullptr}};
const char* const names[] = {NT_ENTRIES(NT_NAME) nullptr};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fast() {
    s_is_cuda = PyUnicode_InternFromString("is_cuda");
    s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    PyObject* m = PyModule_Create(&module);
    if (!m) return nullptr;
    PyObject* all = PyList_New(0);
    for (const char* const* n = names; all && *n; n++) {
        PyObject* s = PyUnicode_FromString(*n);
        if (!s || PyList_Append(all, s)) { Py_XDECREF(s); Py_CLEAR(all); break; }
        Py_DECREF(s);
    }
    if (!all || PyModule_AddObject(m, "ENTRIES", all)) { Py_XDECREF(all); Py_DECREF(m); return nullptr; }
    return m;
}
