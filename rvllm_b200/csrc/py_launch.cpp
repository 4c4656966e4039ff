// CPython module `rvllm_b200._native`: the launch entry points of the C ABI as plain built-in functions.
//
// A launch through ctypes costs 7-8 us of host time (argument boxing for 10-30 parameters, a second ctypes call that
// validates, stream look-up), several times the kernel at decode sizes; an executor that issues a layer call by call
// is then bound by the interpreter (measured: 98 us for a layer of eight small kernels).  These wrappers are
// METH_FASTCALL functions whose parameter types are deduced from the C prototypes, so a call costs its conversions only.
// Pointers may be None, integers, or any object with a data_ptr() method (a tensor).  Every wrapper returns the C
// function's status; reading the message and raising stays with the Python side.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>

#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/rvllm_b200.h"

namespace {

PyObject* g_data_ptr = nullptr;  // interned "data_ptr"

bool to_pointer(PyObject* o, uintptr_t* out) {
    if (o == Py_None) {
        *out = 0;
        return true;
    }
    if (PyLong_Check(o)) {
        *out = (uintptr_t)PyLong_AsVoidPtr(o);
        return !(*out == 0 && PyErr_Occurred());
    }
    PyObject* r = PyObject_CallMethodNoArgs(o, g_data_ptr);
    if (!r) return false;
    *out = (uintptr_t)PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    return !(*out == 0 && PyErr_Occurred());
}

template <typename T> bool convert(PyObject* o, T* out) {
    if constexpr (std::is_pointer_v<T>) {
        uintptr_t p;
        if (!to_pointer(o, &p)) return false;
        *out = reinterpret_cast<T>(p);
        return true;
    } else if constexpr (std::is_floating_point_v<T>) {
        const double v = PyFloat_AsDouble(o);
        *out = (T)v;
        return !(v == -1.0 && PyErr_Occurred());
    } else {
        // (wider than the parameter: wraps like a C conversion, which is what the ctypes table does)
        const long long v = (long long)PyLong_AsUnsignedLongLongMask(o);
        *out = (T)v;
        return !(v == -1 && PyErr_Occurred());
    }
}

template <auto Fn> struct Wrap;
template <typename... A, int (*Fn)(A...)> struct Wrap<Fn> {
    template <size_t... I> static PyObject* run(PyObject* const* args, std::index_sequence<I...>) {
        std::tuple<A...> v;
        if (!(convert(args[I], &std::get<I>(v)) && ...)) return nullptr;
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = std::apply(Fn, v);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    }
    static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
        if (n != (Py_ssize_t)sizeof...(A)) {
            PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", (Py_ssize_t)sizeof...(A), n);
            return nullptr;
        }
        return run(args, std::index_sequence_for<A...>{});
    }
};

#define ENTRY(fn) {#fn, (PyCFunction)(void (*)(void))Wrap<fn>::call, METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {
    ENTRY(rvllm_fused_rmsnorm_fp8_quant_launch),
    ENTRY(rvllm_fused_add_rmsnorm_fp8_quant_launch),
    ENTRY(rvllm_quantize_fp8_per_token_launch),
    ENTRY(rvllm_fused_act_mul_fp8_quant_launch),
    ENTRY(rvllm_argmax_launch),
    ENTRY(rvllm_rope_fp8kv_launch),
    ENTRY(rvllm_embedding_gather_launch),
    ENTRY(rvllm_fp8_gemm_channelscale),
    ENTRY(rvllm_fp8_gemm_gateup_act_quant),
    ENTRY(rvllm_fp8_gemm_qkv_rope_fp8kv),
    ENTRY(rvllm_paged_decode_fp8),
    ENTRY(rvllm_paged_decode_fp8_quant),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "Launch entry points of librvllm_b200.so.", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    g_data_ptr = PyUnicode_InternFromString("data_ptr");
    return g_data_ptr ? PyModule_Create(&g_module) : nullptr;
}
