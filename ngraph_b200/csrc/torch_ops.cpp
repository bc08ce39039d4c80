// The torch-facing operators of ngraph_b200/ops.py as native code: argument checks, output allocation and the call into the
// C ABI (include/b200_kernels.h) without an interpreted instruction in between.
//
// A call of a small layer is bound by the host: the same steps in Python with ctypes took 12-17 us per call where the
// kernel takes 2-6 (one image through ResNet-50, 58 calls: 944 us of Python around 324 us of kernels); here they take 1-2 us
// beside the launch itself.  The C ABI is reached through function addresses handed over once by bind(), so the library
// that ngraph_b200/lib.py loaded is the one that runs.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include "b200_kernels.h"

namespace
{
    decltype(&b200_quantize) p_quantize;
    decltype(&b200_dequantize) p_dequantize;
    decltype(&b200_qgemm) p_qgemm;
    decltype(&b200_qconv) p_qconv, p_qconv_packed;
    decltype(&b200_qconv_out_shape) p_qconv_out_shape;
    decltype(&b200_nchw_to_nhwc_u8) p_nchw_to_nhwc, p_nhwc_to_nchw;
    decltype(&b200_transpose_u8) p_transpose;
    decltype(&b200_maxpool_nhwc_u8) p_maxpool;
    decltype(&b200_global_avgpool_q_nhwc_u8) p_avgpool;
    PyObject* p_check; // lib.check(status, what): raises B200Error
    PyObject* p_conv_params; // the type lib.ConvParams

    // raised as a Python exception that is already set
    struct PyError
    {
    };
    void fail_assert(const char* text)
    {
        PyErr_SetString(PyExc_AssertionError, text);
        throw PyError();
    }
    inline void require(bool ok, const char* text)
    {
        if (!ok)
            fail_assert(text);
    }

    inline const at::Tensor& tensor(PyObject* o)
    {
        if (!THPVariable_Check(o))
        {
            PyErr_SetString(PyExc_TypeError, "b200 ops take torch tensors");
            throw PyError();
        }
        return THPVariable_Unpack(o);
    }
    // a CUDA tensor, contiguous: the caller's own (which the caller holds during the call), a copy where it is not
    using Dev = c10::MaybeOwned<at::Tensor>;
    inline Dev dev(PyObject* o)
    {
        const at::Tensor& t = tensor(o);
        require(t.is_cuda(), "b200 ops take CUDA tensors");
        return t.expect_contiguous();
    }
    inline Dev dev(PyObject* o, at::ScalarType type)
    {
        Dev t = dev(o);
        if (t->scalar_type() != type)
            fail_assert((std::string("tensor of ") + c10::toString(t->scalar_type()) + " where " + c10::toString(type) + " is wanted").c_str());
        return t;
    }
    inline int code(at::ScalarType t)
    {
        switch (t)
        {
        case at::kByte: return B200_U8;
        case at::kChar: return B200_I8;
        case at::kInt: return B200_I32;
        case at::kFloat: return B200_F32;
        default:
            PyErr_Format(PyExc_KeyError, "%s", c10::toString(t)); // as a lookup in the table of supported types
            throw PyError();
        }
    }
    inline at::ScalarType dtype(PyObject* o)
    {
        if (!THPDtype_Check(o))
        {
            PyErr_SetString(PyExc_TypeError, "a torch.dtype is wanted");
            throw PyError();
        }
        return reinterpret_cast<THPDtype*>(o)->scalar_type;
    }
    // int(o), where `exact` is not asked for; with it what is an integer already (sizes: 3.7 is none)
    inline long long integer(PyObject* o, bool exact = false)
    {
        PyObject* i = exact ? PyNumber_Index(o) : PyNumber_Long(o);
        if (!i)
            throw PyError();
        const long long v = PyLong_AsLongLong(i);
        Py_DECREF(i);
        if (v == -1 && PyErr_Occurred())
            throw PyError();
        return v;
    }
    inline bool truth(PyObject* o)
    {
        const int v = PyObject_IsTrue(o);
        if (v < 0)
            throw PyError();
        return v != 0;
    }
    // up to N integers of a sequence
    template <int N>
    inline int integers(PyObject* o, int64_t (&v)[N])
    {
        PyObject* f = PySequence_Fast(o, "a sequence of integers is wanted");
        if (!f)
            throw PyError();
        const Py_ssize_t n = PySequence_Fast_GET_SIZE(f);
        try
        {
            if (n > N)
            {
                PyErr_SetString(PyExc_ValueError, "too many values");
                throw PyError();
            }
            for (Py_ssize_t i = 0; i < n; ++i)
                v[i] = integer(PySequence_Fast_GET_ITEM(f, i));
        }
        catch (...)
        {
            Py_DECREF(f);
            throw;
        }
        Py_DECREF(f);
        return int(n);
    }
    // the first two items of a sequence of sizes
    inline void pair(PyObject* o, int64_t (&v)[2])
    {
        for (Py_ssize_t i = 0; i < 2; ++i)
        {
            PyObject* item = PySequence_GetItem(o, i);
            if (!item)
                throw PyError();
            try
            {
                v[i] = integer(item, true);
            }
            catch (...)
            {
                Py_DECREF(item);
                throw;
            }
            Py_DECREF(item);
        }
    }
    // torch.empty on the device of `like`; on the current device (where `like` shows that CUDA is initialised) without the
    // device guard and the initialisation checks, a fifth of the allocation
    inline at::Tensor empty(at::IntArrayRef shape, at::ScalarType type, const at::Tensor& like)
    {
        if (like.get_device() == c10::cuda::current_device())
            return at::Tensor(at::detail::empty_generic(shape, c10::cuda::CUDACachingAllocator::get(), c10::DispatchKeySet(c10::DispatchKey::CUDA), type, c10::nullopt));
        return at::Tensor(at::detail::empty_cuda(shape, type, like.device(), c10::nullopt));
    }
    inline void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

    inline void check(int status, const char* what)
    {
        if (status == B200_OK)
            return;
        PyObject* r = PyObject_CallFunction(p_check, "is", status, what);
        Py_XDECREF(r);
        if (r) // lib.check raises for every status but 0
            PyErr_Format(PyExc_RuntimeError, "%s failed with status %d", what, status);
        throw PyError();
    }
    // the launch itself runs without the interpreter lock, as a ctypes call would
    template <typename F>
    inline int unlocked(F f)
    {
        int rc;
        Py_BEGIN_ALLOW_THREADS rc = f();
        Py_END_ALLOW_THREADS return rc;
    }

    template <typename F>
    PyObject* guarded(Py_ssize_t given, Py_ssize_t wanted, F body)
    {
        HANDLE_TH_ERRORS
        if (given != wanted)
        {
            PyErr_Format(PyExc_TypeError, "%zd arguments where %zd are wanted", given, wanted);
            return nullptr;
        }
        try
        {
            return body();
        }
        catch (const PyError&)
        {
            return nullptr;
        }
        END_HANDLE_TH_ERRORS
    }

    // (x, scale, zero_point, axes, round_mode, out or None); Dequantize without round_mode
    PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 6, [&]() -> PyObject* {
            const Dev x = dev(a[0], at::kFloat), scale = dev(a[1], at::kFloat), zp = dev(a[2]);
            int64_t axes[B200_MAX_RANK];
            const int n_axes = integers(a[3], axes);
            std::sort(axes, axes + n_axes);
            const int mode = int(integer(a[4])), type = code(zp->scalar_type());
            const at::Tensor out = a[5] == Py_None ? empty(x->sizes(), zp->scalar_type(), *x) : tensor(a[5]);
            void* st = stream();
            check(unlocked([&] {
                      return p_quantize(static_cast<const float*>(x->data_ptr()), static_cast<const float*>(scale->data_ptr()), zp->data_ptr(), out.data_ptr(),
                                        type, x->sizes().data(), int(x->dim()), axes, n_axes, mode, st);
                  }),
                  "b200_quantize");
            return THPVariable_Wrap(out);
        });
    }
    PyObject* dequantize(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 5, [&]() -> PyObject* {
            const Dev x = dev(a[0]), scale = dev(a[1], at::kFloat), zp = dev(a[2]);
            require(zp->scalar_type() == x->scalar_type(), "zero_point has the type of x");
            int64_t axes[B200_MAX_RANK];
            const int n_axes = integers(a[3], axes);
            std::sort(axes, axes + n_axes);
            const int type = code(x->scalar_type());
            const at::Tensor out = a[4] == Py_None ? empty(x->sizes(), at::kFloat, *x) : tensor(a[4]);
            void* st = stream();
            check(unlocked([&] {
                      return p_dequantize(x->data_ptr(), static_cast<const float*>(scale->data_ptr()), zp->data_ptr(), static_cast<float*>(out.data_ptr()), type,
                                          x->sizes().data(), int(x->dim()), axes, n_axes, st);
                  }),
                  "b200_dequantize");
            return THPVariable_Wrap(out);
        });
    }

    // The fused epilogue of the contractions, with the tensors it points at.
    struct EpilogueArgs
    {
        b200_epilogue e{};
        Dev scale, bias, sum_in, sum_scale;
        // a: scale, out_dtype, bias, relu, sum_in, sum_scale, core, out_zp
        explicit EpilogueArgs(PyObject* const* a)
        {
            scale = dev(a[0], at::kFloat);
            e.scale = static_cast<const float*>(scale->data_ptr());
            e.scale_count = scale->numel();
            if (a[2] != Py_None)
            {
                bias = dev(a[2], at::kInt);
                e.bias = static_cast<const int32_t*>(bias->data_ptr());
            }
            if (a[4] != Py_None)
            {
                sum_in = dev(a[4]);
                sum_scale = dev(a[5], at::kFloat);
                e.sum_in = sum_in->data_ptr();
                e.sum_type = code(sum_in->scalar_type());
                e.sum_scale = static_cast<const float*>(sum_scale->data_ptr());
            }
            e.relu = truth(a[3]);
            e.round_half_away = truth(a[6]);
            e.out_zero_point = int32_t(integer(a[7]));
            e.out_type = code(dtype(a[1]));
        }
    };
    inline int operands(const at::Tensor& data, const at::Tensor& weights)
    {
        require(weights.scalar_type() == at::kChar || weights.scalar_type() == at::kByte, "weights are int8 or uint8");
        return code(data.scalar_type()) | (weights.scalar_type() == at::kByte ? B200_WEIGHTS_U8 : 0);
    }

    // (a, w, out or None, scale, out_dtype, bias, relu, sum_in, sum_scale, core, out_zp)
    PyObject* qgemm(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 11, [&]() -> PyObject* {
            const Dev x = dev(a[0]), w = dev(a[1]);
            const int types = operands(*x, *w);
            require(x->dim() == 2 && w->dim() == 2 && x->size(1) == w->size(1), "a is [M,K] and w is [N,K]");
            const EpilogueArgs e(a + 3);
            const int64_t m = x->size(0), k = x->size(1), cols = w->size(0);
            const at::Tensor out = a[2] == Py_None ? empty({m, cols}, dtype(a[4]), *x) : tensor(a[2]);
            void* st = stream();
            check(unlocked([&] { return p_qgemm(x->data_ptr(), types, static_cast<const int8_t*>(w->data_ptr()), out.data_ptr(), m, cols, k, &e.e, st); }),
                  "b200_qgemm");
            return THPVariable_Wrap(out);
        });
    }

    // The bytes of a ctypes ConvParams.
    struct Params
    {
        Py_buffer view{};
        explicit Params(PyObject* o)
        {
            const int is = PyObject_IsInstance(o, p_conv_params);
            if (is == 0)
                PyErr_SetString(PyExc_TypeError, "a ConvParams is wanted");
            if (is != 1)
                throw PyError();
            if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0)
                throw PyError();
            if (view.len != Py_ssize_t(sizeof(b200_conv_params)))
            {
                PyBuffer_Release(&view);
                PyErr_SetString(PyExc_TypeError, "a ConvParams is wanted");
                throw PyError();
            }
        }
        ~Params() { PyBuffer_Release(&view); }
        const b200_conv_params* get() const { return static_cast<const b200_conv_params*>(view.buf); }
    };

    // (data, filters, cp, prepacked, out or None, scale, out_dtype, bias, relu, sum_in, sum_scale, core, out_zp)
    PyObject* qconv(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 13, [&]() -> PyObject* {
            const Dev x = dev(a[0]), f = dev(a[1]);
            const int types = operands(*x, *f);
            const Params cp(a[2]);
            const bool packed = truth(a[3]);
            const EpilogueArgs e(a + 5);
            int64_t p, q;
            check(p_qconv_out_shape(cp.get(), &p, &q), "b200_qconv_out_shape");
            const at::Tensor out = a[4] == Py_None ? empty({cp.get()->N, p, q, cp.get()->K}, dtype(a[6]), *x) : tensor(a[4]);
            void* st = stream();
            check(unlocked([&] {
                      return (packed ? p_qconv_packed : p_qconv)(x->data_ptr(), types, static_cast<const int8_t*>(f->data_ptr()), out.data_ptr(), cp.get(), &e.e,
                                                                 st);
                  }),
                  packed ? "b200_qconv_packed" : "b200_qconv");
            return THPVariable_Wrap(out);
        });
    }

    // (x, channels of the result): NCHW -> NHWC with the channels padded, NHWC -> NCHW with the padding dropped
    PyObject* nchw_to_nhwc(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 2, [&]() -> PyObject* {
            const Dev x = dev(a[0]);
            require(x->element_size() == 1 && x->dim() == 4, "one-byte elements, four dimensions");
            const int64_t N = x->size(0), c = x->size(1), h = x->size(2), w = x->size(3), c_pad = a[1] == Py_None ? c : integer(a[1], true);
            const at::Tensor out = empty({N, h, w, c_pad}, x->scalar_type(), *x);
            void* st = stream();
            check(unlocked([&] { return p_nchw_to_nhwc(x->data_ptr(), out.data_ptr(), N, c, h, w, c_pad, st); }), "b200_nchw_to_nhwc_u8");
            return THPVariable_Wrap(out);
        });
    }
    PyObject* nhwc_to_nchw(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 2, [&]() -> PyObject* {
            const Dev x = dev(a[0]);
            require(x->element_size() == 1 && x->dim() == 4, "one-byte elements, four dimensions");
            const int64_t N = x->size(0), h = x->size(1), w = x->size(2), c_pad = x->size(3), c = a[1] == Py_None ? c_pad : integer(a[1], true);
            const at::Tensor out = empty({N, c, h, w}, x->scalar_type(), *x);
            void* st = stream();
            check(unlocked([&] { return p_nhwc_to_nchw(x->data_ptr(), out.data_ptr(), N, c, h, w, c_pad, st); }), "b200_nhwc_to_nchw_u8");
            return THPVariable_Wrap(out);
        });
    }
    PyObject* transpose(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 1, [&]() -> PyObject* {
            const Dev x = dev(a[0]);
            require(x->element_size() == 1 && x->dim() == 2, "one-byte elements, two dimensions");
            const at::Tensor out = empty({x->size(1), x->size(0)}, x->scalar_type(), *x);
            void* st = stream();
            check(unlocked([&] { return p_transpose(x->data_ptr(), out.data_ptr(), x->size(0), x->size(1), st); }), "b200_transpose_u8");
            return THPVariable_Wrap(out);
        });
    }

    // (x, window, stride, pad_below, pad_above)
    PyObject* maxpool(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 5, [&]() -> PyObject* {
            const Dev x = dev(a[0], at::kByte);
            require(x->dim() == 4, "x is [N,H,W,C]");
            int64_t v[4][2];
            for (int i = 0; i < 4; ++i)
                pair(a[1 + i], v[i]);
            const int64_t N = x->size(0), h = x->size(1), w = x->size(2), c = x->size(3);
            int64_t d[2];
            for (int i = 0; i < 2; ++i)
            {
                if (v[1][i] == 0)
                {
                    PyErr_SetString(PyExc_ZeroDivisionError, "integer division or modulo by zero");
                    throw PyError();
                }
                const int64_t room = (i == 0 ? h : w) + v[2][i] + v[3][i] - v[0][i];
                d[i] = (room >= 0 ? room / v[1][i] : -((-room + v[1][i] - 1) / v[1][i])) + 1;
            }
            const at::Tensor out = empty({N, d[0], d[1], c}, at::kByte, *x);
            void* st = stream();
            check(unlocked([&] {
                      return p_maxpool(x->data_ptr(), out.data_ptr(), N, h, w, c, v[0][0], v[0][1], v[1][0], v[1][1], v[2][0], v[2][1], v[3][0], v[3][1], st);
                  }),
                  "b200_maxpool_nhwc_u8");
            return THPVariable_Wrap(out);
        });
    }
    // (x, scale_in, scale_out)
    PyObject* global_avgpool(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 3, [&]() -> PyObject* {
            const Dev x = dev(a[0], at::kByte), in = dev(a[1], at::kFloat), o = dev(a[2], at::kFloat);
            require(x->dim() == 4, "x is [N,H,W,C]");
            const at::Tensor out = empty({x->size(0), x->size(3)}, at::kByte, *x);
            void* st = stream();
            check(unlocked([&] {
                      return p_avgpool(x->data_ptr(), out.data_ptr(), static_cast<const float*>(in->data_ptr()), static_cast<const float*>(o->data_ptr()), x->size(0),
                                       x->size(1), x->size(2), x->size(3), st);
                  }),
                  "b200_global_avgpool_q_nhwc_u8");
            return THPVariable_Wrap(out);
        });
    }

    // bind(check, {name: address}, type of the convolution parameters)
    PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n)
    {
        return guarded(n, 3, [&]() -> PyObject* {
            auto take = [&](auto& fn, const char* name) {
                PyObject* v = PyDict_GetItemString(a[1], name);
                if (!v)
                {
                    PyErr_SetString(PyExc_KeyError, name);
                    throw PyError();
                }
                fn = reinterpret_cast<std::decay_t<decltype(fn)>>(PyLong_AsVoidPtr(v));
                if (PyErr_Occurred())
                    throw PyError();
            };
            take(p_quantize, "b200_quantize");
            take(p_dequantize, "b200_dequantize");
            take(p_qgemm, "b200_qgemm");
            take(p_qconv, "b200_qconv");
            take(p_qconv_packed, "b200_qconv_packed");
            take(p_qconv_out_shape, "b200_qconv_out_shape");
            take(p_nchw_to_nhwc, "b200_nchw_to_nhwc_u8");
            take(p_nhwc_to_nchw, "b200_nhwc_to_nchw_u8");
            take(p_transpose, "b200_transpose_u8");
            take(p_maxpool, "b200_maxpool_nhwc_u8");
            take(p_avgpool, "b200_global_avgpool_q_nhwc_u8");
            Py_INCREF(a[0]);
            Py_XDECREF(p_check);
            p_check = a[0];
            Py_INCREF(a[2]);
            Py_XDECREF(p_conv_params);
            p_conv_params = a[2];
            Py_RETURN_NONE;
        });
    }

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
    PyMethodDef methods[] = {METHOD(bind),         METHOD(quantize),     METHOD(dequantize), METHOD(qgemm),          METHOD(qconv), METHOD(nchw_to_nhwc),
                             METHOD(nhwc_to_nchw), METHOD(transpose),    METHOD(maxpool),    METHOD(global_avgpool), {nullptr, nullptr, 0, nullptr}};
    PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
}

PyMODINIT_FUNC PyInit__torch_ops(void) { return PyModule_Create(&module); }
