// CPython bindings of the entry points that a host program calls in its inner loop.
//
// ops.py exposes every C entry point through ctypes; a call there costs about 8 us of
// interpreter time (argument loop, ctypes conversion, current stream lookup), more than most
// of the operators take on the GPU.  The functions below convert their arguments in C and cost
// well under a microsecond on top of the launch.  Arguments, results and error behaviour are
// those of the ctypes form: whatever is not one of the plain cases (a torch tensor, an int,
// None or a description structure, in the expected number) is handed to it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "k3_moe_layer.h"
#include "k3_moe_ops.h"

#include <tuple>
#include <type_traits>
#include <utility>

namespace {

PyObject *g_tensor_type, *g_layer_desc_type, *g_latent_desc_type, *g_get_stream, *g_get_device, *g_is_contiguous, *g_data_ptr, *g_stream_kw;

enum class Got { kYes, kFallback, kError };

Got pointer_of(PyObject *o, void **out) {
    if (o == Py_None) {
        *out = nullptr;
        return Got::kYes;
    }
    if (PyLong_CheckExact(o)) {
        *out = PyLong_AsVoidPtr(o);
        if (PyErr_Occurred()) {
            PyErr_Clear();
            return Got::kFallback;
        }
        return Got::kYes;
    }
    if (!PyObject_TypeCheck(o, (PyTypeObject *)g_tensor_type)) return Got::kFallback;
    PyObject *args[1] = {o};
    PyObject *c = PyObject_VectorcallMethod(g_is_contiguous, args, 1 | PY_VECTORCALL_ARGUMENTS_OFFSET, nullptr);
    if (!c) return Got::kError;
    const bool contiguous = c == Py_True;
    Py_DECREF(c);
    if (!contiguous) return Got::kFallback;                // raises there
    PyObject *p = PyObject_VectorcallMethod(g_data_ptr, args, 1 | PY_VECTORCALL_ARGUMENTS_OFFSET, nullptr);
    if (!p) return Got::kError;
    *out = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    return PyErr_Occurred() ? Got::kError : Got::kYes;
}

template <typename T>
struct Arg {                                               // integers
    static_assert(std::is_integral<T>::value, "");
    static Got get(PyObject *o, T *out) {
        if (!PyLong_CheckExact(o)) return Got::kFallback;
        const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
        if (PyErr_Occurred()) {
            PyErr_Clear();
            return Got::kFallback;
        }
        *out = (T)v;
        return Got::kYes;
    }
};
template <>
struct Arg<float> {
    static Got get(PyObject *o, float *out) {
        if (!PyFloat_CheckExact(o)) return Got::kFallback;
        *out = (float)PyFloat_AS_DOUBLE(o);
        return Got::kYes;
    }
};
template <>
struct Arg<void *> {
    static Got get(PyObject *o, void **out) { return pointer_of(o, out); }
};
template <>
struct Arg<const void *> {
    static Got get(PyObject *o, const void **out) { return pointer_of(o, (void **)out); }
};
template <typename T, PyObject **kType>
struct Structure {                                         // the ctypes structure that mirrors T
    static Got get(PyObject *o, const T **out) {
        Py_buffer view;
        if (!PyObject_TypeCheck(o, (PyTypeObject *)*kType)) return Got::kFallback;
        if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0) {
            PyErr_Clear();
            return Got::kFallback;
        }
        *out = (const T *)view.buf;
        const bool fits = view.len == (Py_ssize_t)sizeof(T);
        PyBuffer_Release(&view);                           // `o` outlives the call
        return fits ? Got::kYes : Got::kFallback;
    }
};
template <> struct Arg<const k3_moe_layer_desc *> : Structure<k3_moe_layer_desc, &g_layer_desc_type> {};
template <> struct Arg<const k3_moe_latent_desc *> : Structure<k3_moe_latent_desc, &g_latent_desc_type> {};

Got current_stream(void **out) {
    PyObject *device = PyObject_CallNoArgs(g_get_device);
    if (!device) return Got::kError;
    PyObject *s = PyObject_CallOneArg(g_get_stream, device);
    Py_DECREF(device);
    if (!s) return Got::kError;
    *out = PyLong_AsVoidPtr(s);
    Py_DECREF(s);
    return PyErr_Occurred() ? Got::kError : Got::kYes;
}

inline PyObject *to_python(bool v) { return PyBool_FromLong(v); }

template <typename A, typename... Rest>
struct Last { using type = typename Last<Rest...>::type; };
template <typename A>
struct Last<A> { using type = A; };

// `self` is the ctypes form of the function.  A trailing void * is the stream: optional,
// positional or by keyword, by default torch's current one.
template <auto kFn, typename Fn> struct Call;
template <auto kFn, typename R, typename... A>
struct Call<kFn, R (*)(A...)> {
    static constexpr Py_ssize_t kArgs = sizeof...(A);
    static constexpr bool kStream = std::is_same<typename Last<A...>::type, void *>::value;

    template <size_t... I>
    static PyObject *run(PyObject *self, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames,
                         std::index_sequence<I...>) {
        PyObject *stream = nullptr;
        bool plain = true;
        if (kwnames && PyTuple_GET_SIZE(kwnames)) {
            plain = kStream && PyTuple_GET_SIZE(kwnames) == 1 && nargs == kArgs - 1 &&
                    PyUnicode_Compare(PyTuple_GET_ITEM(kwnames, 0), g_stream_kw) == 0;
            stream = args[nargs];
            if (stream == Py_None) stream = nullptr;
        } else if (kStream && nargs == kArgs) {
            stream = args[kArgs - 1] == Py_None ? nullptr : args[kArgs - 1];
        } else {
            plain = nargs == kArgs - (kStream ? 1 : 0);
        }
        std::tuple<A...> v{};
        Got got = plain ? Got::kYes : Got::kFallback;
        auto one = [&](auto index, auto *slot) {
            constexpr size_t i = decltype(index)::value;
            if (got != Got::kYes) return;
            if constexpr (kStream && i + 1 == sizeof...(A)) {
                got = stream ? pointer_of(stream, slot) : current_stream(slot);
            } else {
                got = Arg<std::remove_pointer_t<decltype(slot)>>::get(args[i], slot);
            }
        };
        (one(std::integral_constant<size_t, I>{}, &std::get<I>(v)), ...);
        if (got == Got::kError) return nullptr;
        if (got == Got::kFallback) return PyObject_Vectorcall(self, args, (size_t)nargs, kwnames);
        R r;
        Py_BEGIN_ALLOW_THREADS
        r = kFn(std::get<I>(v)...);
        Py_END_ALLOW_THREADS
        return to_python(r);
    }
    static PyObject *call(PyObject *self, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
        return run(self, args, nargs, kwnames, std::make_index_sequence<sizeof...(A)>{});
    }
};

#define K3_BIND(fn) \
    {#fn, (PyCFunction)(void (*)(void))&Call<&fn, decltype(&fn)>::call, METH_FASTCALL | METH_KEYWORDS, \
     "Calls " #fn " (see include/ for the contract)."}

PyMethodDef kBound[] = {
    K3_BIND(k3_rocm_situ_bf16),
    K3_BIND(k3_rocm_mxfp4_gemv_bf16),
    K3_BIND(k3_rocm_mxfp4_gemm_bf16),
    K3_BIND(k3_rocm_mxfp4_gemm_tiled_bf16),
    K3_BIND(k3_rocm_bf16_gemv_bf16),
    K3_BIND(k3_rocm_bf16_gemm_tiled_bf16),
    K3_BIND(k3_rocm_bf16_gemm_bf16),
    K3_BIND(k3_rocm_bf16_gemv_f32),
    K3_BIND(k3_rocm_bf16_gemm_f32),
    K3_BIND(k3_rocm_bf16_gemm_tiled_f32),
    K3_BIND(k3_rocm_bf16_quantize_q8_128),
    K3_BIND(k3_rocm_q8_128_dequantize_bf16),
    K3_BIND(k3_rocm_q8_128_gemv_bf16),
    K3_BIND(k3_rocm_q8_128_gemm_bf16),
    K3_BIND(k3_rocm_q8_128_gemm_tiled_bf16),
    K3_BIND(k3_rocm_rms_norm_bf16),
    K3_BIND(k3_rocm_router_topk_f32),
    K3_BIND(k3_rocm_router_topk_f32_batch),
    K3_BIND(k3_rocm_weighted_sum_bf16),
    K3_BIND(k3_rocm_weighted_sum_bf16_batch),
    K3_BIND(k3_rocm_gather_rows_bf16),
    K3_BIND(k3_rocm_scatter_rows_bf16),
    K3_BIND(k3_rocm_add_bf16),
    K3_BIND(k3_moe_activation_bf16),
    K3_BIND(k3_moe_q8_quantize),
    K3_BIND(k3_moe_q8_gemm_bf16),
    K3_BIND(k3_moe_dispatch_build),
    K3_BIND(k3_moe_route),
    K3_BIND(k3_moe_experts_grouped),
    K3_BIND(k3_moe_experts_grouped_ws),
    K3_BIND(k3_moe_experts_token),
    K3_BIND(k3_moe_shared_expert),
    K3_BIND(k3_moe_shared_expert_ws),
    K3_BIND(k3_moe_combine),
    K3_BIND(k3_moe_combine_residual),
    K3_BIND(k3_moe_layer_forward),
    K3_BIND(k3_moe_block_forward),
    K3_BIND(k3_moe_latent_layer_forward),
    {nullptr, nullptr, 0, nullptr},
};

// bind(fallbacks, tensor type, layer and latent description types, raw stream getter, device
// getter) -> {name: function}
PyObject *bind(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 6 || !PyDict_Check(args[0]) || !PyType_Check(args[1]) || !PyType_Check(args[2]) ||
        !PyType_Check(args[3])) {
        PyErr_SetString(PyExc_TypeError, "bind(dict, tensor type, layer type, latent type, stream getter, device getter)");
        return nullptr;
    }
    g_tensor_type = Py_NewRef(args[1]);
    g_layer_desc_type = Py_NewRef(args[2]);
    g_latent_desc_type = Py_NewRef(args[3]);
    g_get_stream = Py_NewRef(args[4]);
    g_get_device = Py_NewRef(args[5]);
    PyObject *out = PyDict_New();
    for (PyMethodDef *d = kBound; out && d->ml_name; d++) {
        PyObject *fallback = PyDict_GetItemString(args[0], d->ml_name);
        if (!fallback) continue;
        PyObject *fn = PyCFunction_NewEx(d, fallback, nullptr);
        if (!fn || PyDict_SetItemString(out, d->ml_name, fn) != 0) Py_CLEAR(out);
        Py_XDECREF(fn);
    }
    return out;
}

PyMethodDef kModuleMethods[] = {
    {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, "Bound forms of the functions in a dict of ctypes forms."},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_k3ops", nullptr, -1, kModuleMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__k3ops(void) {
    g_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    g_data_ptr = PyUnicode_InternFromString("data_ptr");
    g_stream_kw = PyUnicode_InternFromString("stream");
    if (!g_is_contiguous || !g_data_ptr || !g_stream_kw) return nullptr;
    return PyModule_Create(&kModule);
}
