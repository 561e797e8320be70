// CPython view of the launchers: the calls of hipml_b200/api.py that an engine makes once per
// layer and token, as vectorcall functions over the C ABI.
//
// What bounds these calls is host work: through ctypes a decode call of 20 arguments took 12 us
// (a Python stream object, a c_void_p per tensor, argtypes checks) against 9 us of kernel, so 16
// layers of a short-context step were host-bound. Here a tensor argument costs one data_ptr()
// method call and the stream one raw-handle lookup.
//
// Every function takes the C function's arguments in their order without the stream, which is
// the current torch stream of the current device. A pointer argument is None or an object with
// data_ptr(); numbers are converted as ctypes would. Returns the C status.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <tuple>
#include <utility>

#include "../../include/hipml_cuda.h"

namespace {

PyObject *g_data_ptr;      // the method name, interned
PyObject *g_raw_stream;    // torch._C._cuda_getCurrentRawStream(device) -> int
PyObject *g_get_device;    // torch._C._cuda_getDevice() -> int

void *pointer_of(PyObject *o, bool &ok) {
    if (o == Py_None) return nullptr;
    PyObject *r = PyObject_CallMethodNoArgs(o, g_data_ptr);
    if (!r) {
        ok = false;
        return nullptr;
    }
    void *p = PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    if (!p && PyErr_Occurred()) ok = false;
    return p;
}

// One converter per C parameter type.
template <class T>
struct From;
template <class T>
struct From<T *> {
    static T *py(PyObject *o, bool &ok) { return static_cast<T *>(pointer_of(o, ok)); }
};
template <>
struct From<int> {
    static int py(PyObject *o, bool &ok) {
        const unsigned long v = PyLong_AsUnsignedLongMask(o);
        if (v == (unsigned long)-1 && PyErr_Occurred()) ok = false;
        return (int)v;
    }
};
template <>
struct From<long long> {
    static long long py(PyObject *o, bool &ok) {
        const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
        if (v == (unsigned long long)-1 && PyErr_Occurred()) ok = false;
        return (long long)v;
    }
};
template <>
struct From<size_t> {
    static size_t py(PyObject *o, bool &ok) {
        const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
        if (v == (unsigned long long)-1 && PyErr_Occurred()) ok = false;
        return (size_t)v;
    }
};
template <>
struct From<float> {
    static float py(PyObject *o, bool &ok) {
        const double v = PyFloat_AsDouble(o);
        if (v == -1.0 && PyErr_Occurred()) ok = false;
        return (float)v;
    }
};

// A host array of up to four ints (the rest are 0), or None: any sequence of what int() takes.
struct Sections {
    bool given;
    int s[4];
};
template <>
struct From<Sections> {
    static Sections py(PyObject *o, bool &ok) {
        Sections r = {o != Py_None, {0, 0, 0, 0}};
        PyObject *items = r.given ? PySequence_Tuple(o) : nullptr;
        if (!items) {
            ok = ok && !r.given;
            return r;
        }
        const Py_ssize_t n = PyTuple_GET_SIZE(items);
        if (n > 4) {
            PyErr_Format(PyExc_IndexError, "%zd sections given, 4 at most", n);
            ok = false;
        }
        for (Py_ssize_t i = 0; i < n && ok; i++) {
            PyObject *v = PyNumber_Long(PyTuple_GET_ITEM(items, i));
            ok = v != nullptr;
            if (ok) r.s[i] = From<int>::py(v, ok);
            Py_XDECREF(v);
        }
        Py_DECREF(items);
        return r;
    }
};

// Nothing is converted once an argument has failed: Python must not be called with an exception set.
template <class T>
T take(PyObject *o, bool &ok) {
    return ok ? From<T>::py(o, ok) : T();
}

bool current_stream(hipml_stream_t &stream) {
    PyObject *dev = PyObject_CallNoArgs(g_get_device);
    if (!dev) return false;
    PyObject *r = PyObject_CallOneArg(g_raw_stream, dev);
    Py_DECREF(dev);
    if (!r) return false;
    stream = static_cast<hipml_stream_t>(PyLong_AsVoidPtr(r));
    Py_DECREF(r);
    return !(stream == nullptr && PyErr_Occurred());
}

bool count_is(Py_ssize_t got, size_t want) {
    if (got == (Py_ssize_t)want) return true;
    PyErr_Format(PyExc_TypeError, "%zd arguments given, %zu wanted", got, want);
    return false;
}

template <class Fn, Fn fn>
struct Call;
template <class... A, int (*fn)(hipml_stream_t, A...)>
struct Call<int (*)(hipml_stream_t, A...), fn> {
    template <size_t... I>
    static PyObject *go(PyObject *const *args, std::index_sequence<I...>) {
        bool ok = true;
        hipml_stream_t stream = nullptr;
        std::tuple<A...> v{take<A>(args[I], ok)...};   // (braces: in order)
        if (!ok || !current_stream(stream)) return nullptr;
        int rc;
        Py_BEGIN_ALLOW_THREADS;   // (a launch waits when the device's queue is full)
        rc = fn(stream, std::get<I>(v)...);
        Py_END_ALLOW_THREADS;
        return PyLong_FromLong(rc);
    }
    static PyObject *py(PyObject *, PyObject *const *args, Py_ssize_t n) {
        if (!count_is(n, sizeof...(A))) return nullptr;
        return go(args, std::index_sequence_for<A...>{});
    }
};

// hipml_attn_front_append_q8: as above, but argument 14 (`sections`) is a host array.
int front_append(hipml_stream_t stream, const float *qg, const float *k, const float *v, float *q, float *gate,
                 float *k_out, const float *q_norm, const float *k_norm, void *k_cache, void *v_cache, int n_heads,
                 int n_kv, int head_dim, int n_rot, Sections sections, const int *pos, const int *step,
                 int pos0, int tokens, int stride, float theta_base, float eps) {
    return hipml_attn_front_append_q8(stream, qg, k, v, q, gate, k_out, q_norm, k_norm, k_cache, v_cache, n_heads,
                                      n_kv, head_dim, n_rot, sections.given ? sections.s : nullptr, pos, step, pos0,
                                      tokens, stride, theta_base, eps);
}

#define CALL(name, fn) {name, (PyCFunction)(void (*)(void))Call<decltype(&fn), &fn>::py, METH_FASTCALL, nullptr}

PyMethodDef kMethods[] = {
    CALL("kv_encode", hipml_kv_encode),
    CALL("kv_encode_bulk", hipml_kv_encode_bulk),
    CALL("kv_encode_rows", hipml_kv_encode_rows),
    CALL("kv_append_f32", hipml_kv_append_f32),
    CALL("kv_append_chunk_f32", hipml_kv_append_chunk_f32),
    CALL("kv_append_cols_f32", hipml_kv_append_cols_f32),
    CALL("kv_rows_copy", hipml_kv_rows_copy),
    CALL("attn_decode_kv", hipml_attn_decode_kv),
    CALL("attn_decode_kv_gated", hipml_attn_decode_kv_gated),
    CALL("attn_decode_kv_append", hipml_attn_decode_kv_append),
    CALL("attn_decode_kv_static", hipml_attn_decode_kv_static),
    CALL("attn_decode_kv_shard", hipml_attn_decode_kv_shard),
    CALL("attn_decode_combine", hipml_attn_decode_combine),
    CALL("attn_decode_cols", hipml_attn_decode_cols),
    CALL("attn_decode_cols_f32", hipml_attn_decode_cols_f32),
    CALL("attn_decode_rows", hipml_attn_decode_rows),
    CALL("attn_decode_batch", hipml_attn_decode_batch),
    CALL("attn_decode_batch_append", hipml_attn_decode_batch_append),
    CALL("attn_chunk", hipml_attn_chunk),
    CALL("attn_chunk_stage", hipml_attn_chunk_stage),
    CALL("attn_chunk_staged", hipml_attn_chunk_staged),
    CALL("attn_chunk_staged_gated", hipml_attn_chunk_staged_gated),
    CALL("qg_split_chunk", hipml_qg_split_chunk),
    CALL("norm_rope_chunk", hipml_norm_rope_chunk),
    CALL("q_gate", hipml_q_gate),
    CALL("attn_front_append_q8", front_append),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_hipml_calls", nullptr, -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__hipml_calls(void) {
    g_data_ptr = PyUnicode_InternFromString("data_ptr");
    PyObject *c = PyImport_ImportModule("torch._C");
    if (!g_data_ptr || !c) return nullptr;
    g_raw_stream = PyObject_GetAttrString(c, "_cuda_getCurrentRawStream");
    g_get_device = PyObject_GetAttrString(c, "_cuda_getDevice");
    Py_DECREF(c);
    if (!g_raw_stream || !g_get_device) return nullptr;
    return PyModule_Create(&kModule);
}
