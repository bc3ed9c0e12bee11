// The calls of nectarml_b200/_nectarml.py into the reference-shaped entry points of include/nectarml_b200.h, in native code.  Built
// into nectarml_b200/_dropin.so, which needs neither torch nor the CUDA headers.
//
// Why it exists: through ctypes a call with its two dozen converted arguments, two array types and a result cell cost 4 us of Python and
// more, a third of what a small batched product takes in all: 7 x 60 x 32 x 123 in fp32 13.6 -> 9.4 us, the three passes of a 3x3 layer of 256
// -> 3 channels on one 8 x 8 image 71 -> 57.
// Arguments are converted as ctypes converted them: integers of any size, cut to the parameter's width, instances of the parameter's
// ctypes type, objects that stand for one of these by `_as_parameter_`; anything else raises its ArgumentError.  The GIL is released for the call.
#include <Python.h>

#include <exception>
#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

#include "../../include/nectarml_b200.h"

namespace {

PyObject* g_argument_error = nullptr;  // ctypes.ArgumentError
PyObject* g_c_int = nullptr;           // ctypes.c_int
PyObject* g_c_size_t = nullptr;        // ctypes.c_size_t

// The integer that `o` stands for where it is none itself: a new reference, or nullptr with an error (also for what stands for nothing).
PyObject* stands_for(PyObject* o, PyObject* type, Py_ssize_t i) {
    PyObject* v = nullptr;
    const int instance = PyObject_IsInstance(o, type);
    if (instance < 0) return nullptr;
    if (instance) return PyObject_GetAttrString(o, "value");
    PyObject* next = PyObject_GetAttrString(o, "_as_parameter_");
    if (!next) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return nullptr;
        PyErr_Clear();
        PyErr_Format(g_argument_error, "argument %zd: TypeError: '%.200s' object cannot be interpreted as an integer", i + 1, Py_TYPE(o)->tp_name);
        return nullptr;
    }
    if (PyLong_Check(next)) return next;
    if (!Py_EnterRecursiveCall(" while processing _as_parameter_")) {
        v = stands_for(next, type, i);
        Py_LeaveRecursiveCall();
    }
    Py_DECREF(next);
    return v;
}

template <class T>
bool convert(PyObject* o, Py_ssize_t i, T* v) {
    static_assert(std::is_same<T, int>::value || std::is_same<T, size_t>::value, "");
    if (PyLong_Check(o)) {
        *v = static_cast<T>(PyLong_AsUnsignedLongLongMask(o));
        return true;
    }
    PyObject* n = stands_for(o, std::is_same<T, int>::value ? g_c_int : g_c_size_t, i);
    if (!n) return false;
    *v = static_cast<T>(PyLong_AsUnsignedLongLongMask(n));
    Py_DECREF(n);
    return !PyErr_Occurred();
}

PyObject* answer(int status, uintptr_t result) {
    if (status == NML_OK) return PyLong_FromSize_t(result);
    PyErr_Format(PyExc_RuntimeError, "nectarml_b200: %s", nml_status_string(status));
    return nullptr;
}

// fn(args..., &result) -> status
template <class... A, size_t... I>
PyObject* call(int (*fn)(A...), PyObject* const* a, Py_ssize_t n, std::index_sequence<I...>) {
    if (n != static_cast<Py_ssize_t>(sizeof...(I))) {
        PyErr_Format(PyExc_TypeError, "%zu arguments are expected, %zd given", sizeof...(I), n);
        return nullptr;
    }
    std::tuple<A...> v;
    if (!(convert(a[I], I, &std::get<I>(v)) && ...)) return nullptr;
    uintptr_t result = 0;
    std::get<sizeof...(I)>(v) = &result;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = std::apply(fn, v);
    Py_END_ALLOW_THREADS
    return answer(status, result);
}
template <auto kFn>
struct Entry;
template <class... A, int (*kFn)(A...)>
struct Entry<kFn> {
    static PyObject* run(PyObject*, PyObject* const* a, Py_ssize_t n) { return call(kFn, a, n, std::make_index_sequence<sizeof...(A) - 1>()); }
};

// (a copy of the sequence: an item's __int__ may change a list while it is read)
bool shape(PyObject* o, std::vector<int>* dims) {
    if (PyObject_Size(o) < 0) return false;
    PyObject* items = PySequence_Tuple(o);
    if (!items) return false;
    const Py_ssize_t n = PyTuple_GET_SIZE(items);
    bool ok = true;
    try {
        dims->resize(n);
    } catch (const std::exception&) {  // (none may leave a C entry)
        PyErr_NoMemory();
        ok = false;
    }
    for (Py_ssize_t i = 0; ok && i < n; ++i) {
        PyObject* v = PyNumber_Long(PyTuple_GET_ITEM(items, i));
        ok = v != nullptr;
        if (ok) (*dims)[i] = static_cast<int>(PyLong_AsUnsignedLongLongMask(v));
        Py_XDECREF(v);
    }
    Py_DECREF(items);
    return ok;
}

// matmul(a_ptr, b_ptr, a_shape, b_shape, dtype) -> pointer
PyObject* matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 5) {
        PyErr_Format(PyExc_TypeError, "5 arguments are expected, %zd given", n);
        return nullptr;
    }
    size_t pa, pb;
    int dtype;
    std::vector<int> da, db;
    if (!shape(a[2], &da) || !shape(a[3], &db) || !convert(a[0], 0, &pa) || !convert(a[1], 1, &pb) || !convert(a[4], 4, &dtype)) return nullptr;
    uintptr_t result = 0;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = nml_ref_matmul(pa, pb, da.data(), static_cast<int>(da.size()), db.data(), static_cast<int>(db.size()), dtype, &result);
    Py_END_ALLOW_THREADS
    return answer(status, result);
}

// free(ptr)
PyObject* release(PyObject*, PyObject* o) {
    size_t p;
    if (!convert(o, 0, &p)) return nullptr;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = nml_ref_free(p);
    Py_END_ALLOW_THREADS
    if (status != NML_OK) return answer(status, 0);
    Py_RETURN_NONE;
}

#define ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(Entry<&nml_ref_##name>::run)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    ENTRY(conv2d), ENTRY(conv_transpose2d), ENTRY(conv2d_backward_input), ENTRY(conv_transpose2d_backward_input),
    ENTRY(conv2d_backward_weight), ENTRY(conv_transpose2d_backward_weight), ENTRY(conv1d), ENTRY(conv_transpose1d),
    ENTRY(conv1d_backward_input), ENTRY(conv_transpose1d_backward_input), ENTRY(conv1d_backward_weight), ENTRY(conv_transpose1d_backward_weight),
    {"matmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(matmul)), METH_FASTCALL, nullptr},
    {"free", release, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_dropin", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dropin(void) {
    PyObject* ctypes = PyImport_ImportModule("ctypes");
    if (!ctypes) return nullptr;
    g_argument_error = PyObject_GetAttrString(ctypes, "ArgumentError");
    g_c_int = PyObject_GetAttrString(ctypes, "c_int");
    g_c_size_t = PyObject_GetAttrString(ctypes, "c_size_t");
    Py_DECREF(ctypes);
    return g_argument_error && g_c_int && g_c_size_t ? PyModule_Create(&kModule) : nullptr;
}
