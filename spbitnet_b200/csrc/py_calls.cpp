// CPython calls of the kernel entry points (spbitnet_b200._calls): tensors, addresses and streams in; a status other than
// SPB_OK goes to the function that bind() was given, which raises.
//
// A small kernel takes the GPU 3 us and a launch the host 2 us, so the host side of a call decides what a program sees that
// drives the kernels from Python.  Through ctypes a call spent 5.4 us on building argument objects and looking up the
// current stream; here an argument is one conversion and the stream two C calls (9.4 -> 3.7 us for a 640 x 2560 GEMV, a decode layer op by op 229 -> 88).
//
// The functions are bound to the addresses of the loaded library (bind()), not linked: there is one copy of its state.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstddef>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/spbitnet_b200.h"

#define SPB_CALLS(X)                                                                                                       \
    X(spb_sparse_ternary_unpack) X(spb_sparse_ternary_gemv) X(spb_sparse_ternary_gemv_batch) X(spb_sparse_ternary_gemv_scaled) \
    X(spb_fused_sparse_bitlinear) X(spb_sparse_bitlinear_q8) X(spb_sparse_ternary_gemm) X(spb_sparse_bitlinear_gemm)       \
    X(spb_prepare_weights) X(spb_prepared_gemv) X(spb_prepared_bitlinear_q8) X(spb_rms_norm) X(spb_absmax_quantize)        \
    X(spb_absmax_reduce) X(spb_dequantize) X(spb_rope) X(spb_scatter_kv) X(spb_attention_scores) X(spb_softmax)            \
    X(spb_attention_output) X(spb_decode_attention) X(spb_decode_attention_split) X(spb_relu2_mul) X(spb_relu2_mul_f32)    \
    X(spb_rms_norm_f32in) X(spb_float_to_half) X(spb_residual_add) X(spb_half_gemv) X(spb_prune_pack_gpu)

namespace {

enum Index {
#define X(name) k_##name,
    SPB_CALLS(X)
#undef X
    kCount
};
void* g_fn[kCount];
PyObject *g_data_ptr, *g_cuda_stream;                      // attribute names
PyObject *g_get_device = nullptr, *g_get_raw_stream = nullptr;  // torch._C._cuda_getDevice, _cuda_getCurrentRawStream
PyObject* g_check = nullptr;  // called with a status other than 0
bool g_cuda_ready = false;

// a tensor's data pointer, an address, or None
bool to_pointer(PyObject* o, void** out) {
    if (o == Py_None) {
        *out = nullptr;
        return true;
    }
    if (PyLong_Check(o)) {
        *out = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(o));
        return !PyErr_Occurred();
    }
    PyObject* r = PyObject_CallMethodNoArgs(o, g_data_ptr);
    if (!r) return false;
    *out = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(r));
    Py_DECREF(r);
    return !PyErr_Occurred();
}

PyObject* attribute(const char* module, const char* name) {
    PyObject* m = PyImport_ImportModule(module);
    if (!m) return nullptr;
    PyObject* a = PyObject_GetAttrString(m, name);
    Py_DECREF(m);
    return a;
}

// At the first call that leaves the stream to torch: also initialises CUDA there, as the first use of a stream does.
bool init_torch_streams() {
    if (!g_get_device) g_get_device = attribute("torch._C", "_cuda_getDevice");
    if (!g_get_device) return false;
    if (!g_get_raw_stream) g_get_raw_stream = attribute("torch._C", "_cuda_getCurrentRawStream");
    if (!g_get_raw_stream) return false;
    PyObject* current = attribute("torch.cuda", "current_stream");
    if (!current) return false;
    PyObject* s = PyObject_CallNoArgs(current);
    Py_DECREF(current);
    if (!s) return false;
    Py_DECREF(s);
    g_cuda_ready = true;
    return true;
}

// None: torch's current stream of the current device; an address; or a stream object
bool to_stream(PyObject* o, void** out) {
    PyObject* r = nullptr;
    if (o == Py_None) {
        if (!g_cuda_ready && !init_torch_streams()) return false;
        PyObject* dev = PyObject_CallNoArgs(g_get_device);
        if (!dev) return false;
        r = PyObject_CallOneArg(g_get_raw_stream, dev);
        Py_DECREF(dev);
    } else if (PyLong_Check(o)) {
        Py_INCREF(o);
        r = o;
    } else {
        r = PyObject_GetAttr(o, g_cuda_stream);
    }
    if (!r) return false;
    *out = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(r));
    Py_DECREF(r);
    return !PyErr_Occurred();
}

template <typename T>
bool convert(PyObject* o, T* out) {
    if constexpr (std::is_pointer_v<T>) {
        void* p;
        if (!to_pointer(o, &p)) return false;
        *out = static_cast<T>(p);
    } else if constexpr (std::is_floating_point_v<T>) {
        *out = static_cast<T>(PyFloat_AsDouble(o));
        if (PyErr_Occurred()) return false;
    } else if constexpr (std::is_same_v<T, size_t>) {
        *out = PyLong_AsSize_t(o);
        if (PyErr_Occurred()) return false;
    } else {
        *out = static_cast<T>(PyLong_AsLong(o));
        if (PyErr_Occurred()) return false;
    }
    return true;
}

template <int I, typename Fn>
struct Call;
template <int I, typename... A>
struct Call<I, int (*)(A...)> {
    static constexpr Py_ssize_t kArgs = sizeof...(A);
    template <size_t... N>
    static bool take(PyObject* const* args, std::tuple<A...>& v, std::index_sequence<N...>) {
        return (convert(args[N], &std::get<N>(v)) && ...) && to_stream(args[kArgs - 1], &std::get<kArgs - 1>(v));
    }
    static PyObject* invoke(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
        if (nargs != kArgs) return PyErr_Format(PyExc_TypeError, "%zd arguments wanted, %zd given", kArgs, nargs);
        if (!g_fn[I]) return PyErr_Format(PyExc_RuntimeError, "the library is not bound");
        std::tuple<A...> v;
        if (!take(args, v, std::make_index_sequence<kArgs - 1>())) return nullptr;
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = std::apply(reinterpret_cast<int (*)(A...)>(g_fn[I]), v);
        Py_END_ALLOW_THREADS
        if (rc == SPB_OK) Py_RETURN_NONE;
        PyObject* status = PyLong_FromLong(rc);
        if (!status) return nullptr;
        PyObject* r = PyObject_CallOneArg(g_check, status);
        Py_DECREF(status);
        return r;
    }
};

// bind({name: address}, check)
PyObject* bind(PyObject*, PyObject* args) {
    PyObject *table, *check;
    if (!PyArg_ParseTuple(args, "OO", &table, &check)) return nullptr;
    Py_INCREF(check);
    Py_XDECREF(g_check);
    g_check = check;
    static const char* const names[] = {
#define X(name) #name,
        SPB_CALLS(X)
#undef X
    };
    for (int i = 0; i < kCount; ++i) {
        PyObject* a = PyMapping_GetItemString(table, names[i]);
        if (!a) return nullptr;
        g_fn[i] = PyLong_AsVoidPtr(a);
        Py_DECREF(a);
        if (PyErr_Occurred()) return nullptr;
    }
    Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
    {"bind", bind, METH_VARARGS, "bind({name: address}, check) attaches the functions of the loaded library"},
#define X(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&Call<k_##name, decltype(&name)>::invoke)), METH_FASTCALL, nullptr},
    SPB_CALLS(X)
#undef X
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_calls", "Kernel entry points of libspbitnet_b200.so", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
    g_data_ptr = PyUnicode_InternFromString("data_ptr");
    g_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    if (!g_data_ptr || !g_cuda_stream) return nullptr;
    return PyModule_Create(&g_module);
}
