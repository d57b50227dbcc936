// _native: the Python side of the kernel ABI without ctypes. A call of a few microseconds on the GPU cost 8-9 us on the host
// (tensor checks in Python, torch.cuda.current_stream(), ctypes' argument conversion); here the checks, the pointers and the
// current stream are read through the C API and the library is called directly (a 512 x 2048 matvec in a loop: 3.8 us a call).
//
// Every function of the table takes its arguments by position, the stream (None = torch's current one) last. What a parameter
// accepts is one letter: P a tensor, F a float32 tensor, H a float16 tensor, I an int32 tensor, N a tensor or None, V a
// number (of the C parameter's own type).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <tuple>
#include <utility>

#include <cuda_runtime.h>

#include "../../include/mnemo_b200.h"

namespace {

struct Names {
    PyObject *is_cuda, *is_contiguous, *data_ptr, *dtype, *cuda_stream;
} names;
PyObject *dtype_f32, *dtype_f16, *dtype_i32, *raw_stream;  // torch.float32 ..., torch._C._cuda_getCurrentRawStream

bool is_true(PyObject *o)  // steals o
{
    const bool v = o && PyObject_IsTrue(o) == 1;
    Py_XDECREF(o);
    return v;
}

bool tensor_ptr(PyObject *t, char kind, void **out)
{
    if (kind == 'N' && t == Py_None) {
        *out = nullptr;
        return true;
    }
    if (kind != 'P' && kind != 'N') {
        PyObject *want = kind == 'F' ? dtype_f32 : kind == 'H' ? dtype_f16 : dtype_i32;
        PyObject *have = PyObject_GetAttr(t, names.dtype);
        if (!have) return false;
        const bool same = have == want;
        if (!same) PyErr_Format(PyExc_TypeError, "%R tensor expected, got %R", want, have);
        Py_DECREF(have);
        if (!same) return false;
    }
    if (!is_true(PyObject_GetAttr(t, names.is_cuda))) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "device tensor expected (the kernels take device pointers)");
        return false;
    }
    if (!is_true(PyObject_CallMethodNoArgs(t, names.is_contiguous))) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "contiguous tensor expected");
        return false;
    }
    PyObject *p = PyObject_CallMethodNoArgs(t, names.data_ptr);
    if (!p) return false;
    *out = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    return !PyErr_Occurred();
}

bool get_stream(PyObject *s, cudaStream_t *out)
{
    PyObject *v = nullptr;
    if (s == Py_None) {
        int dev = 0;
        cudaGetDevice(&dev);
        PyObject *d = PyLong_FromLong(dev);
        v = d ? PyObject_CallOneArg(raw_stream, d) : nullptr;
        Py_XDECREF(d);
    } else if (PyLong_Check(s)) {
        v = Py_NewRef(s);
    } else if (PyObject_HasAttr(s, names.cuda_stream)) {
        v = PyObject_GetAttr(s, names.cuda_stream);
    } else {
        v = PyNumber_Long(s);
    }
    if (!v) return false;
    *out = static_cast<cudaStream_t>(PyLong_AsVoidPtr(v));
    Py_DECREF(v);
    return !PyErr_Occurred();
}

bool convert(PyObject *o, char kind, const void **out)
{
    void *p = nullptr;
    if (!tensor_ptr(o, kind, &p)) return false;
    *out = p;
    return true;
}
template <class T>
bool convert(PyObject *o, char kind, T **out)
{
    void *p = nullptr;
    if (!tensor_ptr(o, kind, &p)) return false;
    *out = static_cast<T *>(p);
    return true;
}
bool convert(PyObject *o, char, int *out)
{
    const long v = PyLong_AsLong(o);
    *out = static_cast<int>(v);
    return !(v == -1 && PyErr_Occurred());
}
bool convert(PyObject *o, char, float *out)
{
    const double v = PyFloat_AsDouble(o);
    *out = static_cast<float>(v);
    return !(v == -1.0 && PyErr_Occurred());
}
bool convert(PyObject *o, char, size_t *out)
{
    *out = PyLong_AsUnsignedLongMask(o);
    return !PyErr_Occurred();
}
bool convert(PyObject *o, char, unsigned long long *out)
{
    *out = PyLong_AsUnsignedLongLongMask(o);
    return !PyErr_Occurred();
}

PyObject *failed(const char *name, int code, bool clear)
{
    const char *where = mb200_last_status_where();
    PyErr_Format(PyExc_RuntimeError, "%s failed with status %d (%s)", name, code, where ? where : "");
    if (clear) mb200_clear_status();
    return nullptr;
}

template <class F>
struct Traits;
template <class R, class... A>
struct Traits<R (*)(A...)> {
    using Result = R;
    using Args = std::tuple<A...>;  // the last one is the stream
    static constexpr size_t n = sizeof...(A);
};

struct Entry {
    const char *name, *kinds;
};

template <auto Fn, const Entry *E>
PyObject *call(PyObject *, PyObject *const *args, Py_ssize_t n_args)
{
    using T = Traits<decltype(Fn)>;
    constexpr size_t n = T::n;
    if (n_args != static_cast<Py_ssize_t>(n)) {
        PyErr_Format(PyExc_TypeError, "%s takes %d arguments, got %d", E->name, static_cast<int>(n), static_cast<int>(n_args));
        return nullptr;
    }
    typename T::Args a{};
    const bool ok = [&]<size_t... I>(std::index_sequence<I...>) {
        return (convert(args[I], E->kinds[I], &std::get<I>(a)) && ...);
    }(std::make_index_sequence<n - 1>());
    if (!ok || !get_stream(args[n - 1], &std::get<n - 1>(a))) return nullptr;
    int code = MB200_OK;
    Py_BEGIN_ALLOW_THREADS
    if constexpr (std::is_void_v<typename T::Result>) {
        std::apply(Fn, a);
        code = mb200_last_status();
    } else {
        code = std::apply(Fn, a);
    }
    Py_END_ALLOW_THREADS
    if (code != MB200_OK) return failed(E->name, code, std::is_void_v<typename T::Result>);
    Py_RETURN_NONE;
}

#define MB200_FUNCTIONS(X)                                     \
    X(cuda_matvec_q4k, "PFFVV")                                \
    X(cuda_matvec_q4k_add, "PFFFVV")                           \
    X(cuda_matvec_q4k_qkv, "PPPFFFFVVV")                       \
    X(cuda_matvec_q4k_dual, "PPFFFVV")                         \
    X(cuda_matvec_q4k_scaled_add, "PFFVVV")                    \
    X(cuda_matvec_q6k, "PFFVV")                                \
    X(cuda_matvec_f32, "FFFVV")                                \
    X(cuda_matvec_q8_0, "PFFVV")                               \
    X(cuda_matvec_q5k, "PFFVV")                                \
    X(cuda_matvec_q3k, "PFFVV")                                \
    X(cuda_topk_softmax, "FIFVV")                              \
    X(cuda_swiglu, "FFFV")                                     \
    X(cuda_scaled_add, "FFVV")                                 \
    X(cuda_rms_norm, "FFFVV")                                  \
    X(cuda_rms_norm_residual, "FFFFVV")                        \
    X(cuda_rms_norm_batched, "FFFVVV")                         \
    X(cuda_rms_norm_qk, "FFFFVVVV")                            \
    X(cuda_rope, "FFVVVVV")                                    \
    X(cuda_f32_to_f16, "FPV")                                  \
    X(cuda_f32_to_f16_dual, "FFPPV")                           \
    X(cuda_attention_f16kv, "FHHFVVVVVV")                      \
    X(cuda_attention_int8kv, "FPPFFFVVVVVV")                   \
    X(cuda_f32_to_int8_kv, "FPFVV")                            \
    X(cuda_f32_to_int8_kv_dual, "FFPPFFVV")                    \
    X(cuda_residual_add, "FFFV")                               \
    X(cuda_embedding_lookup_q4k, "PFVVV")                      \
    X(cuda_embedding_lookup_q3k, "PFVVV")                      \
    X(cuda_sample_token, "FVVVVI")                             \
    X(mb200_matvec_q4k_dual_swiglu, "PPFFVV")                  \
    X(mb200_matvec_q6k_scaled_add, "PFFVVV")                   \
    X(mb200_norm_matvec_q4k, "PFFVFVV")                        \
    X(mb200_norm_matvec_q6k, "PFFVFVV")                        \
    X(mb200_norm_matvec2_q4k, "PFVPFVFFVV")                    \
    X(mb200_norm_matvec_qkv, "PFVPFPFVFNVV")                   \
    X(mb200_router_topk, "FFPPFVVV")                           \
    X(mb200_router_topk_static, "FFPFVVV")                     \
    X(mb200_moe_gate_up, "PVVVPVFFVV")                         \
    X(mb200_moe_down, "PVVVPFVFNFVV")                          \
    X(mb200_moe_gate_up_local, "PVVVPVVVFFVV")                 \
    X(mb200_moe_down_local, "PVVVPFVVVFNFVV")                  \
    X(mb200_moe_block, "FPVVVVVVVVFNFPFFP")                    \
    X(mb200_moe_block_local, "FPVVVVVVVVVVFNFPFFP")            \
    X(mb200_moe_block_norm, "FPVVVVVVVVVVFNVNNFPFFP")          \
    X(mb200_moe_experts_fused, "PVVVVVPFVVVFFNFVVP")           \
    X(mb200_gemm_q4k_f16, "PHFVVV")                            \
    X(mb200_gemm_q6k_f16, "PHFVVV")                            \
    X(mb200_moe_prefill, "PVVVVVVVVHPFNFVVP")

#define MB200_ENTRY(fn, kinds)                                                                  \
    constexpr Entry entry_##fn{#fn, kinds};                                                     \
    static_assert(sizeof(kinds) == Traits<decltype(&fn)>::n, "a letter for every parameter but the stream");
MB200_FUNCTIONS(MB200_ENTRY)

#define MB200_METHOD(fn, kinds) \
    {#fn, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call<&fn, &entry_##fn>)), METH_FASTCALL, nullptr},
PyMethodDef methods[] = {MB200_FUNCTIONS(MB200_METHOD){nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "The kernel ABI over torch tensors (see binding.cpp).", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void)
{
    names = {PyUnicode_InternFromString("is_cuda"), PyUnicode_InternFromString("is_contiguous"), PyUnicode_InternFromString("data_ptr"),
             PyUnicode_InternFromString("dtype"), PyUnicode_InternFromString("cuda_stream")};
    PyObject *torch = PyImport_ImportModule("torch");
    if (!torch) return nullptr;
    dtype_f32 = PyObject_GetAttrString(torch, "float32");
    dtype_f16 = PyObject_GetAttrString(torch, "float16");
    dtype_i32 = PyObject_GetAttrString(torch, "int32");
    PyObject *c = PyObject_GetAttrString(torch, "_C");
    raw_stream = c ? PyObject_GetAttrString(c, "_cuda_getCurrentRawStream") : nullptr;
    Py_XDECREF(c);
    Py_DECREF(torch);
    if (!dtype_f32 || !dtype_f16 || !dtype_i32 || !raw_stream) return nullptr;
    return PyModule_Create(&module);
}
