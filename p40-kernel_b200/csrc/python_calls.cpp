// python_calls.cpp -- the Python side of the C ABI as native functions: tensors in, device pointers and torch's current
// stream out.
//
// What bounds a small call is the host: a decoded token's attention step is 48 launches, and a ctypes call that checks
// five tensors and asks torch for the stream costs 6 - 8 us of interpreter work before the launch (2 us) begins.  Here
// the checks and the stream are a few loads each (0.3 us).
//
// The library itself is not linked: bind() takes the addresses that the loaded library exports, so that one build of
// this module serves any build of the library.
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

#include <cstdint>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

namespace {

// Kinds of argument beside plain numbers: device memory (a CUDA tensor or None), a handle (an integer or an object with
// an integer `value`, as ctypes makes them), a truth value.
struct Mem { void *p; };
struct Handle { void *p; };
struct Truth { int v; };

// An object that is no torch tensor but has a tensor's is_cuda, is_contiguous() and data_ptr().
bool get_like_tensor(PyObject *o, const char *name, Mem &out) {
    auto truth = [](PyObject *v) {
        const int t = v ? PyObject_IsTrue(v) : -1;
        Py_XDECREF(v);
        return t;
    };
    const int cuda = truth(PyObject_GetAttrString(o, "is_cuda"));
    if (cuda < 0) return false;
    if (!cuda) {
        PyErr_Format(PyExc_RuntimeError, "%s must be a CUDA tensor: this library has no CPU path", name);
        return false;
    }
    const int contiguous = truth(PyObject_CallMethod(o, "is_contiguous", nullptr));
    if (contiguous < 0) return false;
    if (!contiguous) {
        PyErr_Format(PyExc_RuntimeError, "%s must be contiguous", name);
        return false;
    }
    PyObject *p = PyObject_CallMethod(o, "data_ptr", nullptr);
    if (!p) return false;
    out.p = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    return !PyErr_Occurred();
}

bool get(PyObject *o, const char *name, Mem &out) {
    if (o == Py_None) {
        out.p = nullptr;
        return true;
    }
    if (!THPVariable_Check(o)) return get_like_tensor(o, name, out);
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.is_cuda()) {
        PyErr_Format(PyExc_RuntimeError, "%s must be a CUDA tensor: this library has no CPU path", name);
        return false;
    }
    if (!t.is_contiguous()) {
        PyErr_Format(PyExc_RuntimeError, "%s must be contiguous", name);
        return false;
    }
    out.p = t.mutable_data_ptr();           // outputs are written: a tensor that shares its memory until then gets its own, as by data_ptr()
    return true;
}
bool get(PyObject *o, const char *, Handle &out) {
    if (o == Py_None) {
        out.p = nullptr;
        return true;
    }
    if (PyLong_Check(o)) {
        out.p = PyLong_AsVoidPtr(o);
        return !PyErr_Occurred();
    }
    PyObject *v = PyObject_GetAttrString(o, "value");
    if (!v) return false;
    out.p = v == Py_None ? nullptr : PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    return !PyErr_Occurred();
}
bool get(PyObject *o, const char *, Truth &out) {
    out.v = PyObject_IsTrue(o);
    return out.v >= 0;
}
bool get(PyObject *o, const char *, int64_t &out) {
    out = PyLong_AsLongLong(o);
    return !(out == -1 && PyErr_Occurred());
}
bool get(PyObject *o, const char *name, int &out) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) return false;
    if (v != (long)(int)v) {
        PyErr_Format(PyExc_OverflowError, "%s does not fit an int", name);
        return false;
    }
    out = (int)v;
    return true;
}
bool get(PyObject *o, const char *, float &out) {
    const double v = PyFloat_AsDouble(o);
    out = (float)v;
    return !(v == -1.0 && PyErr_Occurred());
}

void *raw(Mem m) { return m.p; }
void *raw(Handle h) { return h.p; }
int raw(Truth t) { return t.v; }
template <typename T> T raw(T v) { return v; }
template <typename T> using Raw = decltype(raw(std::declval<T>()));

constexpr int MAX_ARGS = 12;

// One exported function: its address, filled in by bind(), and the names of its arguments.
template <typename... A>
struct Call {
    using Fn = int (*)(Raw<A>..., void *);
    static constexpr int N = sizeof...(A);
    const char *name;
    const char *args[N];
    Fn fn = nullptr;

    template <size_t... I>
    PyObject *go(PyObject *const *v, std::index_sequence<I...>) {
        std::tuple<A...> a{};
        if (!(get(v[I], args[I], std::get<I>(a)) && ...)) return nullptr;
        void *stream = c10::cuda::getCurrentCUDAStream().stream();
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = fn(raw(std::get<I>(a))..., stream);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    }

    PyObject *call(PyObject *const *v, Py_ssize_t n, PyObject *kw) {
        static_assert(N <= MAX_ARGS, "");
        PyObject *all[MAX_ARGS];
        if (!fn) {
            PyErr_Format(PyExc_RuntimeError, "%s is not bound to a library", name);
            return nullptr;
        }
        if (kw || n != N) {          // named arguments: put them in their places
            const Py_ssize_t nk = kw ? PyTuple_GET_SIZE(kw) : 0;
            if (n + nk != N) {
                PyErr_Format(PyExc_TypeError, "%s() takes %d arguments, got %zd", name, N, n + nk);
                return nullptr;
            }
            for (int i = 0; i < N; ++i) all[i] = i < n ? v[i] : nullptr;
            for (Py_ssize_t k = 0; k < nk; ++k) {
                const char *s = PyUnicode_AsUTF8(PyTuple_GET_ITEM(kw, k));
                if (!s) return nullptr;
                int at = 0;
                while (at < N && std::strcmp(s, args[at])) ++at;
                if (at == N || all[at]) {
                    PyErr_Format(PyExc_TypeError, "%s() got an unexpected or repeated argument '%s'", name, s);
                    return nullptr;
                }
                all[at] = v[n + k];
            }
            v = all;
        }
        try {
            return go(v, std::make_index_sequence<N>{});
        } catch (const std::exception &e) {
            PyErr_SetString(PyExc_RuntimeError, e.what());
            return nullptr;
        }
    }
};

// include/bonsai_p40.h
Call<Mem, Mem, Mem, int64_t, int64_t> gemv{"gemv", {"W", "xq", "y", "n_out", "n_in"}};
Call<Mem, Mem, int64_t> quant_activations{"quant_activations", {"x", "out", "n"}};
Call<Mem, Mem, Mem, int64_t, int64_t, int64_t> gemm{"gemm", {"W", "Xq", "Y", "n_out", "n_in", "n_tok"}};
Call<Mem, Mem, int64_t, int64_t> repack{"repack", {"src", "dst", "n_out", "n_in"}};
Call<Mem, Mem, Mem, int64_t, int64_t> gemv_repack{"gemv_repack", {"W", "x", "y", "n_out", "n_in"}};
Call<Mem, Mem, int64_t> fwht{"fwht", {"x", "signs", "n"}};
Call<Mem, Mem, Mem, int64_t, int64_t, float> rmsnorm{"rmsnorm", {"x", "w", "y", "n_rows", "n", "eps"}};
Call<Mem, Mem, Mem, Mem, Mem, Mem, Mem, int, int, int, int> gdn_step{
    "gdn_step", {"state", "q", "k", "v", "g", "beta", "out", "n_k_heads", "n_v_heads", "K", "V"}};
Call<Mem, Mem, Mem, Mem, int, int, int, int, float> attn{
    "attn", {"q", "k", "v", "out", "n_tok", "n_head", "n_head_kv", "head_dim", "scale"}};
// include/bonsai_b200_ext.h
Call<Mem, Mem, Mem, Mem, int64_t> fwht_quant{"fwht_quant", {"x", "signs", "xq", "x_rot", "n"}};
Call<Mem, Mem, Mem, int64_t> swiglu{"swiglu", {"gate", "up", "y", "n"}};
Call<Mem, Mem, Mem, int64_t, int64_t, Truth> quant_batch{"quant_batch", {"X", "signs", "Xq", "n_in", "n_tok", "rotate"}};
Call<Mem, Mem, Mem, Mem, Mem, int64_t, int64_t> linear{"linear", {"W", "x", "signs", "y", "xq_scratch", "n_out", "n_in"}};
Call<Mem, Mem, Mem, Mem, int64_t, int64_t> linear_static{"linear_static", {"W", "x", "signs", "y", "n_out", "n_in"}};
Call<Handle> chain_run{"chain_run", {"chain"}};
// include/bonsai_kv.h
Call<Handle, int, int, Mem, Mem> kv_append{"kv_append", {"kv", "layer", "pos", "k", "v"}};
Call<Handle, int, int, int, Mem, Mem> kv_append_batch{"kv_append_batch", {"kv", "layer", "pos0", "n_tok", "k", "v"}};
Call<Handle, int, int, Mem, Mem> kv_attn_decode{"kv_attn_decode", {"kv", "layer", "pos", "q", "out"}};

#define EACH_CALL(X)                                                                                                  \
    X(gemv) X(quant_activations) X(gemm) X(repack) X(gemv_repack) X(fwht) X(rmsnorm) X(gdn_step) X(attn)                \
    X(fwht_quant) X(swiglu) X(quant_batch) X(linear) X(linear_static) X(chain_run) X(kv_append) X(kv_append_batch)      \
    X(kv_attn_decode)

#define WRAPPER(f)                                                                                                    \
    PyObject *py_##f(PyObject *, PyObject *const *v, Py_ssize_t n, PyObject *kw) { return f.call(v, n, kw); }
EACH_CALL(WRAPPER)

// bind({name: address}): every function of this module needs an address.
PyObject *bind(PyObject *, PyObject *addresses) {
    if (!PyDict_Check(addresses)) {
        PyErr_SetString(PyExc_TypeError, "bind() takes a dict of addresses");
        return nullptr;
    }
#define BIND(f)                                                                                                       \
    {                                                                                                                 \
        PyObject *a = PyDict_GetItemString(addresses, #f);                                                              \
        void *p = a ? PyLong_AsVoidPtr(a) : nullptr;                                                                    \
        if (!p) {                                                                                                     \
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, #f);                                                 \
            return nullptr;                                                                                           \
        }                                                                                                             \
        f.fn = reinterpret_cast<decltype(f)::Fn>(p);                                                                    \
    }
    EACH_CALL(BIND)
    Py_RETURN_NONE;
}

#define ENTRY(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(py_##f)), METH_FASTCALL | METH_KEYWORDS, nullptr},
PyMethodDef methods[] = {EACH_CALL(ENTRY){"bind", bind, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) { return PyModule_Create(&module); }
