// The entry points of the C ABI as native Python callables, for ngraph_b200/lib.py.
//
// A program that issues its launches through ctypes spends about 1 us per call on converting arguments, half of what the
// launch itself takes on the host (an encoder layer on 128 tokens: 40 calls around 130 us of kernels).  The callables here
// take the same arguments - integers, None, c_void_p, ctypes arrays, floats, byref of the ABI's structures - and convert them
// by the types of the declaration in b200_kernels.h.  Whatever they do not recognise (wrong counts or types) goes to the
// ctypes function they stand for, which accepts it or raises.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>
#include <tuple>
#include <type_traits>
#include <utility>
#include "b200_kernels.h"

namespace
{
    PyTypeObject *void_pointer_type, *float_type, *array_type; // ctypes.c_void_p, c_float, Array
    char int64_format[8]; // how the buffer of a c_int64 array names its elements

    // What byref() makes is opaque; where its pointer, its tag and the object it refers to lie is found out at import, against
    // known objects (find_byref_layout).  Where that does not hold, byref arguments go to ctypes.
    struct ByRef
    {
        PyObject_HEAD void* ffi_type;
        char tag;
        alignas(16) void* pointer; // of a union as wide as a long double
        alignas(16) PyObject* object;
    };
    PyTypeObject* byref_type; // null: layout not recognised

    // the ctypes structures of lib.py, by the ABI's
    template <typename T>
    PyTypeObject* structure_type = nullptr;

    template <typename T>
    bool by_reference(PyObject* o, T*& out)
    {
        if (!byref_type || Py_TYPE(o) != byref_type || !structure_type<std::remove_cv_t<T>>)
            return false;
        const ByRef* r = reinterpret_cast<const ByRef*>(o);
        if (r->tag != 'P' || !r->object || Py_TYPE(r->object) != structure_type<std::remove_cv_t<T>>)
            return false;
        out = static_cast<T*>(r->pointer);
        return true;
    }

    bool bytes_of(PyObject* o, void* to, Py_ssize_t n)
    {
        Py_buffer v;
        if (PyObject_GetBuffer(o, &v, PyBUF_SIMPLE) != 0)
        {
            PyErr_Clear();
            return false;
        }
        const bool ok = v.len == n;
        if (ok)
            memcpy(to, v.buf, size_t(n));
        PyBuffer_Release(&v);
        return ok;
    }

    template <typename T>
    bool convert(PyObject* o, T*& out)
    {
        if (PyLong_CheckExact(o))
        {
            out = static_cast<T*>(PyLong_AsVoidPtr(o));
            if (out == nullptr && PyErr_Occurred())
            {
                PyErr_Clear();
                return false;
            }
            // as a ctypes c_void_p parameter; a POINTER parameter does not take integers
            return std::is_void<T>::value || std::is_same<std::remove_cv_t<T>, float>::value || sizeof(std::conditional_t<std::is_void<T>::value, char, T>) <= 4;
        }
        if (o == Py_None)
        {
            out = nullptr;
            return true;
        }
        // lib.py declares int64_t* and the structures as POINTER: of those ctypes takes arrays of the very type (or byref), no
        // c_void_p and no array of another type of the same size
        constexpr bool typed = std::is_same<std::remove_cv_t<T>, int64_t>::value;
        if constexpr (std::is_class<T>::value)
            return by_reference(o, out);
        if (Py_TYPE(o) == void_pointer_type)
            return !typed && bytes_of(o, &out, sizeof(out));
        if (PyObject_TypeCheck(o, array_type))
        {
            Py_buffer v;
            if (PyObject_GetBuffer(o, &v, PyBUF_FORMAT | PyBUF_ND) != 0)
            {
                PyErr_Clear();
                return false;
            }
            out = static_cast<T*>(v.buf);
            const bool ok = !typed || (v.ndim == 1 && v.format && strcmp(v.format, int64_format) == 0);
            PyBuffer_Release(&v); // the caller holds the array
            return ok;
        }
        return false;
    }
    template <typename T>
    std::enable_if_t<std::is_integral<T>::value, bool> convert(PyObject* o, T& out)
    {
        if (!PyLong_Check(o))
            return false;
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred())
        {
            PyErr_Clear();
            return false;
        }
        out = static_cast<T>(v);
        return true;
    }
    bool convert(PyObject* o, float& out)
    {
        if (PyFloat_CheckExact(o))
        {
            out = static_cast<float>(PyFloat_AS_DOUBLE(o));
            return true;
        }
        return Py_TYPE(o) == float_type && bytes_of(o, &out, sizeof(out));
    }

    template <typename F>
    struct Slot;
    template <typename... P>
    struct Slot<int (*)(P...)>
    {
        int (*fn)(P...) = nullptr;
        PyObject* ctypes_fn = nullptr;

        PyObject* call(PyObject* const* a, Py_ssize_t n) const { return call(a, n, std::index_sequence_for<P...>()); }
        template <size_t... I>
        PyObject* call(PyObject* const* a, Py_ssize_t n, std::index_sequence<I...>) const
        {
            std::tuple<P...> v;
            if (n != Py_ssize_t(sizeof...(P)) || !(convert(a[I], std::get<I>(v)) && ...))
                return PyObject_Vectorcall(ctypes_fn, a, size_t(n), nullptr);
            int rc;
            Py_BEGIN_ALLOW_THREADS rc = fn(std::get<I>(v)...);
            Py_END_ALLOW_THREADS return PyLong_FromLong(rc);
        }
    };

#define ENTRY_POINTS(X)                                                                                                                        \
    X(b200_quantize) X(b200_dequantize) X(b200_qgemm) X(b200_qgemm_packed) X(b200_qconv) X(b200_qconv_packed) X(b200_qconv_stem)                \
    X(b200_stem_pack_input) X(b200_stem_pack_input_f32) X(b200_nchw_to_nhwc_u8) X(b200_nhwc_to_nchw_u8) X(b200_nhwc_to_nchw_b32)                \
    X(b200_transpose_u8) X(b200_copy_rows) X(b200_maxpool_nhwc_u8) X(b200_maxpool_nhwc_i8) X(b200_global_avgpool_q_nhwc_u8)                     \
    X(b200_requant_scale) X(b200_f32_binary) X(b200_f32_binary_periodic) X(b200_f32_unary) X(b200_broadcast_b32) X(b200_permute_b32)            \
    X(b200_reduce_f32) X(b200_softmax_rows_f32) X(b200_softmax_rows_scaled_f32) X(b200_layer_norm_rows_f32) X(b200_layer_norm_rows_sum_f32)     \
    X(b200_gelu_f32) X(b200_bmm_f32) X(b200_gather_rows_b32) X(b200_strided_sums)

#define DEFINE(name)                                                                                                                           \
    Slot<decltype(&name)> slot_##name;                                                                                                         \
    PyObject* call_##name(PyObject*, PyObject* const* a, Py_ssize_t n) { return slot_##name.call(a, n); }                                      \
    PyMethodDef def_##name = {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_##name)), METH_FASTCALL, nullptr};
    ENTRY_POINTS(DEFINE)

    // wrap(name, address, ctypes function) -> the native callable, or the ctypes function where there is none
    PyObject* wrap(PyObject*, PyObject* args)
    {
        const char* name;
        PyObject *address, *fallback;
        if (!PyArg_ParseTuple(args, "sOO", &name, &address, &fallback))
            return nullptr;
        void* p = PyLong_AsVoidPtr(address);
        if (!p && PyErr_Occurred())
            return nullptr;
#define TAKE(f)                                                                                                                                \
    if (strcmp(name, #f) == 0)                                                                                                                 \
    {                                                                                                                                          \
        slot_##f.fn = reinterpret_cast<decltype(slot_##f.fn)>(p);                                                                              \
        Py_INCREF(fallback);                                                                                                                   \
        Py_XDECREF(slot_##f.ctypes_fn);                                                                                                        \
        slot_##f.ctypes_fn = fallback;                                                                                                         \
        return PyCFunction_New(&def_##f, nullptr);                                                                                             \
    }
        ENTRY_POINTS(TAKE)
        Py_INCREF(fallback);
        return fallback;
    }

    // structures(epilogue type, convolution parameter type)
    PyObject* structures(PyObject*, PyObject* args)
    {
        PyObject *epilogue, *conv;
        if (!PyArg_ParseTuple(args, "O!O!", &PyType_Type, &epilogue, &PyType_Type, &conv))
            return nullptr;
        Py_INCREF(epilogue);
        Py_INCREF(conv);
        structure_type<b200_epilogue> = reinterpret_cast<PyTypeObject*>(epilogue);
        structure_type<b200_conv_params> = reinterpret_cast<PyTypeObject*>(conv);
        Py_RETURN_NONE;
    }

    // byref objects of a known buffer, one with an offset
    void find_byref_layout(PyObject* ctypes)
    {
        PyObject* buffer = PyObject_CallMethod(ctypes, "create_string_buffer", "i", 16);
        PyObject* address = buffer ? PyObject_CallMethod(ctypes, "addressof", "O", buffer) : nullptr;
        PyObject* plain = address ? PyObject_CallMethod(ctypes, "byref", "O", buffer) : nullptr;
        PyObject* shifted = plain ? PyObject_CallMethod(ctypes, "byref", "Oi", buffer, 8) : nullptr;
        if (shifted && Py_TYPE(plain)->tp_basicsize >= Py_ssize_t(sizeof(ByRef)) && Py_TYPE(plain) == Py_TYPE(shifted))
        {
            const ByRef *p = reinterpret_cast<const ByRef*>(plain), *q = reinterpret_cast<const ByRef*>(shifted);
            char* at = static_cast<char*>(PyLong_AsVoidPtr(address));
            if (p->tag == 'P' && q->tag == 'P' && p->object == buffer && q->object == buffer && p->pointer == at && q->pointer == at + 8)
            {
                byref_type = Py_TYPE(plain);
                Py_INCREF(byref_type);
            }
        }
        PyErr_Clear();
        Py_XDECREF(shifted);
        Py_XDECREF(plain);
        Py_XDECREF(address);
        Py_XDECREF(buffer);
    }

    bool find_int64_format(PyObject* ctypes)
    {
        PyObject* type = PyObject_GetAttrString(ctypes, "c_int64");
        PyObject* value = type ? PyObject_CallNoArgs(type) : nullptr;
        Py_buffer v;
        bool ok = value && PyObject_GetBuffer(value, &v, PyBUF_FORMAT) == 0;
        if (ok)
        {
            ok = v.format && v.itemsize == 8 && strlen(v.format) < sizeof(int64_format);
            if (ok)
                strcpy(int64_format, v.format);
            PyBuffer_Release(&v);
        }
        PyErr_Clear();
        Py_XDECREF(value);
        Py_XDECREF(type);
        return ok;
    }

    PyMethodDef methods[] = {{"structures", structures, METH_VARARGS, nullptr}, {"wrap", wrap, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
    PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
}

PyMODINIT_FUNC PyInit__fastcall(void)
{
    PyObject* ctypes = PyImport_ImportModule("ctypes");
    if (!ctypes)
        return nullptr;
    auto type = [&](const char* name) { return reinterpret_cast<PyTypeObject*>(PyObject_GetAttrString(ctypes, name)); };
    void_pointer_type = type("c_void_p"), float_type = type("c_float"), array_type = type("Array");
    find_byref_layout(ctypes);
    if (!find_int64_format(ctypes))
        PyErr_SetString(PyExc_ImportError, "the buffer of a ctypes c_int64 does not name its type");
    Py_DECREF(ctypes);
    return void_pointer_type && float_type && array_type && !PyErr_Occurred() ? PyModule_Create(&module) : nullptr;
}
