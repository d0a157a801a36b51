// Python bindings of the calls that a forward pass makes for every layer: the same functions under the
// same names as the C ABI, called with Python objects.  A call through ctypes spends about as long in
// argument conversion as the launch itself takes (append: 3.4 us, attention: 4.6 us a call); here the
// conversions are compiled from the functions' own signatures.  The C ABI stays the boundary: this
// module links libvfkv.so and knows nothing of its insides.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/vfkv_next.h"

namespace {

PyObject *s_data_ptr, *s_ctypes, *s_data, *s_value, *t_void_p;

bool as_u64(PyObject *o, unsigned long long *out)
{
    if (PyLong_Check(o)) {
        *out = PyLong_AsUnsignedLongLongMask(o);
    } else {
        PyObject *i = PyNumber_Index(o);
        if (!i) return false;
        *out = PyLong_AsUnsignedLongLongMask(i);
        Py_DECREF(i);
    }
    return !(*out == ~0ull && PyErr_Occurred());
}

// The address of None, an int, a tensor (data_ptr), a numpy array (ctypes.data) or a ctypes pointer (value).
bool as_address(PyObject *o, void **out)
{
    unsigned long long a = 0;
    if (o == Py_None) { *out = nullptr; return true; }
    if (PyLong_Check(o)) {
        if (!as_u64(o, &a)) return false;
        *out = reinterpret_cast<void *>(a);
        return true;
    }
    // handles are c_void_p; an attribute that is missing costs an exception, so they are told apart first
    PyObject *v = reinterpret_cast<PyObject *>(Py_TYPE(o)) == t_void_p ? PyObject_GetAttr(o, s_value) : PyObject_CallMethodNoArgs(o, s_data_ptr);
    if (!v) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return false;
        PyErr_Clear();
        if (PyObject *c = PyObject_GetAttr(o, s_ctypes)) {
            v = PyObject_GetAttr(c, s_data);
            Py_DECREF(c);
        } else {
            PyErr_Clear();
            v = PyObject_GetAttr(o, s_value);
        }
        if (!v) {
            PyErr_Format(PyExc_TypeError, "cannot take the address of %R", reinterpret_cast<PyObject *>(Py_TYPE(o)));
            return false;
        }
    }
    const bool ok = v == Py_None || as_u64(v, &a);
    Py_DECREF(v);
    *out = reinterpret_cast<void *>(a);
    return ok;
}

template <typename T> bool convert(PyObject *o, T *out)
{
    if constexpr (std::is_pointer_v<T>) {
        void *p;
        if (!as_address(o, &p)) return false;
        *out = static_cast<T>(p);
    } else if constexpr (std::is_floating_point_v<T>) {
        const double d = PyFloat_AsDouble(o);
        if (d == -1.0 && PyErr_Occurred()) return false;
        *out = T(d);
    } else {
        unsigned long long v;
        if (!as_u64(o, &v)) return false;
        *out = T(v);
    }
    return true;
}

template <auto Fn> struct Call;
template <typename... A, int32_t (*Fn)(A...)> struct Call<Fn> {
    template <size_t... I>
    static PyObject *run(PyObject *const *args, std::index_sequence<I...>)
    {
        std::tuple<A...> a;
        if (!(convert(args[I], &std::get<I>(a)) && ...)) return nullptr;
        int32_t rc;
        Py_BEGIN_ALLOW_THREADS
        rc = Fn(std::get<I>(a)...);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    }
    static PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n)
    {
        if (n != Py_ssize_t(sizeof...(A))) {
            PyErr_Format(PyExc_TypeError, "%zd arguments given, %zd wanted", n, Py_ssize_t(sizeof...(A)));
            return nullptr;
        }
        return run(args, std::index_sequence_for<A...>{});
    }
};

// the RoPE parameters as three arguments instead of a struct
int32_t rope_append(vfkv_cache *cache, uint32_t layer, const float *k, const float *v, uint32_t n_tokens, uint32_t slot,
                    uint32_t base_pos, uint32_t n_dims, float freq_base, float freq_scale, float *k_rot, void *stream)
{
    const vfkv_rope_params r{n_dims, freq_base, freq_scale};
    return vfkv_rope_append(cache, layer, k, v, n_tokens, slot, base_pos, &r, k_rot, stream);
}
int32_t rope_append_batch(vfkv_cache *cache, uint32_t layer, const float *k, const float *v, const uint32_t *slot_ids,
                          const uint32_t *positions, uint32_t n_seqs, uint32_t n_dims, float freq_base, float freq_scale,
                          float *k_rot, void *stream)
{
    const vfkv_rope_params r{n_dims, freq_base, freq_scale};
    return vfkv_rope_append_batch(cache, layer, k, v, slot_ids, positions, n_seqs, &r, k_rot, stream);
}
int32_t rope_neox(vfkv_ctx *ctx, const float *x, float *out, uint32_t n_rows, uint32_t n_heads, uint32_t head_dim,
                  const uint32_t *positions, uint32_t base_pos, uint32_t n_dims, float freq_base, float freq_scale, void *stream)
{
    const vfkv_rope_params r{n_dims, freq_base, freq_scale};
    return vfkv_rope_neox(ctx, x, out, n_rows, n_heads, head_dim, positions, base_pos, &r, stream);
}

#define VFKV_CALL(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Call<&fn>::entry)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    VFKV_CALL("kv_store_fp8", vfkv_kv_store_fp8),
    VFKV_CALL("kv_copy_fp16", vfkv_kv_copy_fp16),
    VFKV_CALL("kv_fp8_to_f16", vfkv_kv_fp8_to_f16),
    VFKV_CALL("append", vfkv_append),
    VFKV_CALL("append_sharded", vfkv_append_sharded),
    VFKV_CALL("append_batch", vfkv_append_batch),
    VFKV_CALL("attend", vfkv_attend),
    VFKV_CALL("attend_batch", vfkv_attend_batch),
    VFKV_CALL("flash_attn", vfkv_flash_attn),
    VFKV_CALL("scalar_attn", vfkv_scalar_attn),
    VFKV_CALL("attend_prefill", vfkv_attend_prefill),
    VFKV_CALL("attend_partial", vfkv_attend_partial),
    VFKV_CALL("attend_exchange", vfkv_attend_exchange),
    VFKV_CALL("decode_step", vfkv_decode_step),
    VFKV_CALL("decode_token", vfkv_decode_token),
    VFKV_CALL("decode_token_host", vfkv_decode_token_host),
    VFKV_CALL("merge_partials", vfkv_merge_partials),
    VFKV_CALL("rope_append", rope_append),
    VFKV_CALL("rope_append_batch", rope_append_batch),
    VFKV_CALL("rope_neox", rope_neox),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "vfkv calls of a forward pass", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native()
{
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_ctypes = PyUnicode_InternFromString("ctypes");
    s_data = PyUnicode_InternFromString("data");
    s_value = PyUnicode_InternFromString("value");
    if (PyObject *c = PyImport_ImportModule("ctypes")) {
        t_void_p = PyObject_GetAttrString(c, "c_void_p");
        Py_DECREF(c);
    }
    return s_data_ptr && s_ctypes && s_data && s_value && t_void_p ? PyModule_Create(&module) : nullptr;
}
