// Python's way to the launch-only entry points: one METH_FASTCALL function per entry point, its conversions generated from
// the prototype in rivoli_kernels.h.
//
// What bounds a small call is the host: ctypes spends 2 - 3 us on the 25 arguments of a decode step and Python as much again
// on taking the addresses of its tensors, against 2.3 us for each kernel launch. Here a call takes the objects as they are:
//   pointer   None (NULL), an integer address, an object with data_ptr() (a tensor), or one with cuda_stream (a stream)
//   geometry  a ctypes structure, through the buffer protocol; None = NULL
//   CompFinish, CompStep   the same, or a tuple of their fields
//   integer, float         as ctypes: wrapped to the parameter's width, rounded to its precision
// The interpreter lock is released around the call, as ctypes does. Host time with the launches: a decode step (25 arguments,
// four launches) 14.7 -> 12.0 us, the three projection operators 18.0 -> 12.0, a V4 prompt's six calls 26.2 -> 18.4 (which is
// what a prompt of 64 tokens takes), an append of a few tokens 5.6 -> 3.9.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <tuple>
#include <utility>

#include "../../../include/rivoli_kernels.h"

namespace {

PyObject *s_data_ptr, *s_cuda_stream;

bool to_word(PyObject* o, unsigned long long* v) {               // an integer, wrapped
    if (PyLong_Check(o)) {
        *v = PyLong_AsUnsignedLongLongMask(o);
    } else {
        PyObject* i = PyNumber_Index(o);
        if (!i) return false;
        *v = PyLong_AsUnsignedLongLongMask(i);
        Py_DECREF(i);
    }
    return !(*v == ~0ull && PyErr_Occurred());
}

bool to_pointer(PyObject* o, void** p) {
    unsigned long long v = 0;
    if (o == Py_None) {
        *p = nullptr;
        return true;
    }
    if (PyLong_Check(o)) {
        if (!to_word(o, &v)) return false;
    } else {
        PyObject* r = PyObject_CallMethodNoArgs(o, s_data_ptr);
        if (!r && PyErr_ExceptionMatches(PyExc_AttributeError)) {
            PyErr_Clear();
            r = PyObject_GetAttr(o, s_cuda_stream);
        }
        if (!r) return false;
        const bool ok = to_word(r, &v);
        Py_DECREF(r);
        if (!ok) return false;
    }
    *p = reinterpret_cast<void*>(static_cast<uintptr_t>(v));
    return true;
}

template <class T>
struct Arg;                                                      // one converted argument

template <class T>
struct Arg<T*> {
    void* v = nullptr;
    bool set(PyObject* o) { return to_pointer(o, &v); }
    T* get() { return static_cast<T*>(v); }
};

template <>
struct Arg<int> {
    unsigned long long v = 0;
    bool set(PyObject* o) { return to_word(o, &v); }
    int get() { return static_cast<int>(static_cast<unsigned>(v)); }
};

template <class T>
struct Real {
    double v = 0;
    bool set(PyObject* o) {
        v = PyFloat_AsDouble(o);
        return !(v == -1.0 && PyErr_Occurred());
    }
    T get() { return static_cast<T>(v); }
};
template <> struct Arg<float> : Real<float> {};
template <> struct Arg<double> : Real<double> {};

template <class T>
struct Struct {                                                  // const T* of a ctypes structure
    Py_buffer b{};
    bool held = false;
    bool set(PyObject* o) {
        if (o == Py_None) return true;
        if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) return false;
        held = true;
        if (b.len >= static_cast<Py_ssize_t>(sizeof(T))) return true;
        PyErr_SetString(PyExc_TypeError, "the structure is smaller than the one that the entry point reads");
        return false;
    }
    const T* get() { return held ? static_cast<const T*>(b.buf) : nullptr; }
    ~Struct() { if (held) PyBuffer_Release(&b); }
};
template <> struct Arg<const DsaGeom*> : Struct<DsaGeom> {};
template <> struct Arg<const V4Geom*> : Struct<V4Geom> {};
template <> struct Arg<const IndexFrontGeom*> : Struct<IndexFrontGeom> {};
template <> struct Arg<const CompGeom*> : Struct<CompGeom> {};

template <class T, class... F>
struct Fields : Struct<T> {                                      // or of a tuple of its fields
    T v{};
    bool tuple = false;
    template <size_t... I>
    bool fill(PyObject* o, std::index_sequence<I...>) {
        std::tuple<Arg<F>...> f;
        if (!(std::get<I>(f).set(PyTuple_GET_ITEM(o, I)) && ...)) return false;
        v = T{std::get<I>(f).get()...};
        return true;
    }
    bool set(PyObject* o) {
        if (!PyTuple_Check(o)) return Struct<T>::set(o);
        if (PyTuple_GET_SIZE(o) != sizeof...(F)) {
            PyErr_SetString(PyExc_TypeError, "wrong number of fields");
            return false;
        }
        tuple = true;
        return fill(o, std::index_sequence_for<F...>{});
    }
    const T* get() { return tuple ? &v : Struct<T>::get(); }
};
template <> struct Arg<const CompFinish*> : Fields<CompFinish, const float*, const float*, float*> {};
template <>
struct Arg<const CompStep*> : Fields<CompStep, const float*, const float*, const float*, float*, float*, const float*, const float*,
                                     uint16_t*, float*, unsigned char*, uint32_t*, int, int, int> {};

template <auto F, class Sig = decltype(F)>
struct Call;
template <auto F, class... A>
struct Call<F, int (*)(A...)> {
    template <size_t... I>
    static PyObject* run(PyObject* const* args, std::index_sequence<I...>) {
        std::tuple<Arg<A>...> a;
        if (!(std::get<I>(a).set(args[I]) && ...)) return nullptr;
        PyThreadState* state = PyEval_SaveThread();
        const int r = F(std::get<I>(a).get()...);
        PyEval_RestoreThread(state);
        return PyLong_FromLong(r);
    }
    static PyObject* fn(PyObject*, PyObject* const* args, Py_ssize_t n) {
        if (n == static_cast<Py_ssize_t>(sizeof...(A))) return run(args, std::index_sequence_for<A...>{});
        return PyErr_Format(PyExc_TypeError, "%zu arguments expected, %zd given", sizeof...(A), n);
    }
};

#define ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Call<&rivoli_##name>::fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    ENTRY(append_kv), ENTRY(gather_rope), ENTRY(index_append), ENTRY(index_score), ENTRY(index_topk), ENTRY(mla_attend),
    ENTRY(gemv_fp8), ENTRY(layernorm), ENTRY(rope_interleave), ENTRY(mla_absorb_fp8), ENTRY(mla_value_fp8),
    ENTRY(kv_append_paged), ENTRY(index_select_paged), ENTRY(dsa_append_attend_paged), ENTRY(dsa_append_select_paged),
    ENTRY(dsa_decode_step_paged), ENTRY(mla_absorb_batched_bf16), ENTRY(mla_value_batched_bf16),
    ENTRY(index_frontend_bf16), ENTRY(act_quant_f4_rotated), ENTRY(act_quant_f8_prefix), ENTRY(kv_compress_deposit),
    ENTRY(kv_compress_prefill), ENTRY(v4_select_blocks_bf16), ENTRY(v4_sparse_attend_bf16), ENTRY(v4_token_step_bf16),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_launch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__launch(void) {
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    return s_data_ptr && s_cuda_stream ? PyModule_Create(&module) : nullptr;
}
