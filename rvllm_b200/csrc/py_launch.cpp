// CPython module `rvllm_b200._native`: the launch entry points of the C ABI as plain built-in functions.
//
// A launch through ctypes costs 7-8 us of host time (argument boxing for 10-30 parameters, a second ctypes call that
// validates, stream look-up), several times the kernel at decode sizes; an executor that issues a layer call by call
// is then bound by the interpreter (measured: 98 us for a layer of eight small kernels).  These wrappers are
// METH_FASTCALL functions whose parameter types are deduced from the C prototypes, so a call costs its conversions only.
// Pointers may be None, integers, torch tensors (read in place: the data_ptr() method costs 0.15 us, and a layer passes 70
// of them), or any other object with that method.  Every wrapper returns the C function's status; reading the message and
// raising stays with the Python side.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/rvllm_b200.h"

namespace {

PyObject* g_current = nullptr;   // CURRENT_STREAM: stands for torch's current stream on the current device
PyObject *g_get_device = nullptr, *g_get_stream = nullptr;  // torch's look-ups of those
PyObject* g_data_ptr = nullptr;  // interned "data_ptr"

// The current stream's handle, as torch.cuda.current_stream().cuda_stream would give it, without the Python frames in between
// (0.06 us instead of 0.2 per launch).
bool current_stream(uintptr_t* out) {
    PyObject* device = PyObject_CallNoArgs(g_get_device);
    if (!device) return false;
    PyObject* handle = PyObject_CallOneArg(g_get_stream, device);
    Py_DECREF(device);
    if (!handle) return false;
    *out = (uintptr_t)PyLong_AsVoidPtr(handle);
    Py_DECREF(handle);
    return !(*out == 0 && PyErr_Occurred());
}

// Torch's look-ups, at load.  CURRENT_STREAM is None with a torch that has none: the Python side then passes handles.  False: an error is set.
bool find_current_stream() {
    if (PyObject* c = PyImport_ImportModule("torch._C")) {
        g_get_device = PyObject_GetAttrString(c, "_cuda_getDevice");
        g_get_stream = g_get_device ? PyObject_GetAttrString(c, "_cuda_getCurrentRawStream") : nullptr;
        Py_DECREF(c);
        if (g_get_stream) g_current = PyObject_CallNoArgs((PyObject*)&PyBaseObject_Type);
    }
    if (!PyErr_Occurred()) return true;
    if (!PyErr_ExceptionMatches(PyExc_ImportError) && !PyErr_ExceptionMatches(PyExc_AttributeError)) return false;
    PyErr_Clear();
    return true;
}

bool to_pointer(PyObject* o, uintptr_t* out) {
    if (o == Py_None) {
        *out = 0;
        return true;
    }
    if (THPVariable_Check(o)) {
        try {
            *out = reinterpret_cast<uintptr_t>(THPVariable_Unpack(o).data_ptr());
        } catch (const std::exception& e) {
            PyErr_SetString(PyExc_RuntimeError, e.what());
            return false;
        }
        return true;
    }
    if (PyLong_Check(o)) {
        *out = (uintptr_t)PyLong_AsVoidPtr(o);
        return !(*out == 0 && PyErr_Occurred());
    }
    if (o == g_current) return current_stream(out);
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

// Calls that take their sizes from the tensors.  None instead of a status: an argument is not what this reads (the Python
// side then goes the long way round, which raises what it always raised).
const at::Tensor* as_tensor(PyObject* o, int64_t dims) {
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.dim() == dims ? &t : nullptr;
}
int kind_of(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kHalf: return RVLLM_OUT_F16;
        case at::kBFloat16: return RVLLM_OUT_BF16;
        case at::kFloat: return RVLLM_OUT_F32;
        default: return -1;
    }
}
bool fits_int(int64_t v) { return v >= 0 && v <= INT32_MAX; }

// gemm(out, a_fp8, w_fp8, a_scale, w_scale, residual, impl, workspace, stream)
PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 9) return PyErr_Format(PyExc_TypeError, "expected 9 arguments, got %zd", n);
    const at::Tensor *A = as_tensor(a[1], 2), *W = as_tensor(a[2], 2);
    if (!A || !W || !THPVariable_Check(a[0])) Py_RETURN_NONE;
    const int kind = kind_of(THPVariable_Unpack(a[0]));
    const int64_t M = A->size(0), K = A->size(1), N = W->size(0);
    if (kind < 0 || !fits_int(M) || !fits_int(N) || !fits_int(K)) Py_RETURN_NONE;
    uintptr_t p[6], ws = 0, stream;
    int impl;
    size_t ws_len = 0;
    for (int i = 0; i < 6; i++)
        if (!to_pointer(a[i], &p[i])) return nullptr;
    if (!convert(a[6], &impl) || !to_pointer(a[8], &stream)) return nullptr;
    if (a[7] != Py_None) {
        if (!THPVariable_Check(a[7])) Py_RETURN_NONE;
        if (!to_pointer(a[7], &ws)) return nullptr;
        ws_len = THPVariable_Unpack(a[7]).nbytes();
    }
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = rvllm_fp8_gemm_channelscale((void*)p[0], kind, (const void*)p[1], (const void*)p[2], (const float*)p[3], (const float*)p[4],
                                     (const void*)p[5], (int)M, (int)N, (int)K, impl, (void*)ws, ws_len, (void*)stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

// rope(qkv, heads, kv_heads, head_dim, rotary_dim, cos, sin, positions, slots, q_fp8, q_scale, k_cache, v_cache, k_scale,
//      v_scale, stream): the packed [T, (heads + 2 * kv_heads) * head_dim] row
PyObject* rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 16) return PyErr_Format(PyExc_TypeError, "expected 16 arguments, got %zd", n);
    const at::Tensor *x = as_tensor(a[0], 2), *cos = as_tensor(a[5], 2);
    if (!x || !cos || !THPVariable_Check(a[13])) Py_RETURN_NONE;
    const int dtype = kind_of(*x);
    int heads, kv_heads, head_dim, rotary;
    if (!convert(a[1], &heads) || !convert(a[2], &kv_heads) || !convert(a[3], &head_dim) || !convert(a[4], &rotary)) return nullptr;
    const int64_t T = x->size(0), stride = x->size(1), positions = cos->size(0);
    if ((dtype != RVLLM_F16 && dtype != RVLLM_BF16) || kv_heads <= 0 || !fits_int(T) || !fits_int(stride) || !fits_int(positions))
        Py_RETURN_NONE;
    const int64_t slots = THPVariable_Unpack(a[13]).numel() / kv_heads;
    if (!fits_int(slots)) Py_RETURN_NONE;
    uintptr_t base, p[10], stream;  // cos .. v_scale
    if (!to_pointer(a[0], &base) || !to_pointer(a[15], &stream)) return nullptr;
    for (int i = 0; i < 10; i++)
        if (!to_pointer(a[5 + i], &p[i])) return nullptr;
    const uintptr_t k_in = base + 2ull * heads * head_dim, v_in = k_in + 2ull * kv_heads * head_dim;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = rvllm_rope_fp8kv_launch((const void*)base, (const void*)k_in, (const void*)v_in, (int)stride, (void*)p[4], (void*)p[6],
                                 (void*)p[7], (float*)p[8], (float*)p[9], (float*)p[5], (const void*)p[0], (const void*)p[1],
                                 (const int32_t*)p[2], (const int32_t*)p[3], (int)T, heads, kv_heads, head_dim, rotary,
                                 (int)positions, (int)slots, dtype, (void*)stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

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
    {"gemm", (PyCFunction)(void (*)(void))gemm, METH_FASTCALL, nullptr},
    {"rope", (PyCFunction)(void (*)(void))rope, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "Launch entry points of librvllm_b200.so.", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    g_data_ptr = PyUnicode_InternFromString("data_ptr");
    PyObject* m = g_data_ptr ? PyModule_Create(&g_module) : nullptr;
    // The class layouts inlined above are those of the torch this was compiled against; the Python side refuses another.
    if (m && PyModule_AddStringConstant(m, "torch_version", RVLLM_TORCH_VERSION) != 0) {
        Py_DECREF(m);
        m = nullptr;
    }
    if (m && !find_current_stream()) {
        Py_DECREF(m);
        m = nullptr;
    }
    if (m && PyObject_SetAttrString(m, "CURRENT_STREAM", g_current ? g_current : Py_None) != 0) {
        Py_DECREF(m);
        m = nullptr;
    }
    return m;
}
