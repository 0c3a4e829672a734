// The library's entry points as Python functions. A ctypes call converts each of its 10 to 31 arguments through Python objects: 3 to 5 us
// beside 2 to 3 of the launch itself, and a step of a small decoder makes a hundred and fifty of them. Here every argument is read by its C type, known
// from the prototype. Arguments are taken as the ctypes signatures of _lib.py take them: None, an address, or a ctypes array, structure or
// pointer for a pointer (nothing else that has a buffer: an array of the host must not reach a kernel), integers cut to their type, any number
// for a float. The interpreter lock is given up meanwhile.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <initializer_list>
#include <tuple>
#include <utility>

#include "../../include/llark_b200.h"

#define LLARK_CALLS(X) \
    X(llark_gemm) X(llark_gemm_ex) X(llark_linear_qkv_rotary) X(llark_splice_scan) X(llark_embed_splice_fwd) X(llark_embed_splice_bwd) \
    X(llark_cast_f32_to_bf16) X(llark_cast_bf16_to_f32) X(llark_rmsnorm_fwd) X(llark_rmsnorm_bwd) X(llark_rope) X(llark_swiglu_fwd) \
    X(llark_swiglu_bwd) X(llark_attn_fwd) X(llark_attn_alibi_fwd) X(llark_attn_alibi_bwd) X(llark_ln_fwd) X(llark_ln_bwd) \
    X(llark_gelu_fwd) X(llark_gelu_bwd) X(llark_gemv) X(llark_attn_decode) X(llark_attn_decode_packed) X(llark_decode_layers) \
    X(llark_attn_bwd) X(llark_attn_bwd_rope) X(llark_colsum) X(llark_ce_fwd) X(llark_ce_bwd) X(llark_grad_sumsq) X(llark_adamw_step) \
    X(llark_jb_conv_down) X(llark_jb_resblock) X(llark_jb_resblocks) X(llark_jb_wave_resblocks) X(llark_jb_conv_k3) \
    X(llark_jb_vq_encode) X(llark_layernorm_fwd) X(llark_jb_embed_tokens) X(llark_jb_sparse_attn) X(llark_jb_sparse_attn_tc) \
    X(llark_quick_gelu) X(llark_add3) X(llark_jb_pool) X(llark_jb_label_cond) X(llark_jb_pool_batched) X(llark_v32_split_tf32) \
    X(llark_v32_embed_splice_fwd) X(llark_v32_rmsnorm_fwd) X(llark_v32_rope) X(llark_v32_swiglu_fwd) X(llark_v32_attn_fwd) \
    X(llark_v32_ce_fwd) X(llark_seq_step_ints) X(llark_seq_embed) X(llark_seq_short_conv) X(llark_seq_add_rmsnorm_conv) \
    X(llark_seq_zero_slot) X(llark_seq_conv_tail) X(llark_seq_add_rmsnorm) X(llark_seq_gated_norm_add) X(llark_seq_rmsnorm_rows) \
    X(llark_seq_relu2) X(llark_seq_layer_norm_add) X(llark_seq_tanh_norm) X(llark_seq_tanh_norm_add) X(llark_linear_rows) \
    X(llark_linear_simt) X(llark_seq_qk_headnorm) X(llark_seq_qkv_headnorm) X(llark_seq_qkv_rotary) X(llark_seq_swa_attn) \
    X(llark_seq_swa_attn_mma) X(llark_seq_kv_ring_write) X(llark_seq_glr_scan) X(llark_seq_glr_combine) X(llark_seq_chunk_plan) \
    X(llark_seq_glr_chunks) X(llark_seq_delta_chunks) X(llark_seq_glr_step) X(llark_seq_head_rmsnorm) X(llark_seq_rotary_table) \
    X(llark_seq_decay_rows) X(llark_seq_decay_chunks) X(llark_seq_decay_combine) X(llark_linear_simt_w32) X(llark_seq_group_rmsnorm) \
    X(llark_seq_residual_combine) X(llark_seq_conv_act) X(llark_seq_delta_prep) X(llark_seq_delta_scan) X(llark_seq_head_norm_gate) \
    X(llark_seq_skip_gate_group_norm) X(llark_seq_post_norm) X(llark_seq_glu_clamped) X(llark_seq_logit_cap) X(llark_seq_latent_prep) \
    X(llark_seq_head_linear) X(llark_seq_tanh) X(llark_gemm_segments) X(llark_seq_moe_route) X(llark_seq_moe_route_bias) \
    X(llark_seq_moe_route_top) X(llark_seq_moe_sort) X(llark_seq_moe_gather) X(llark_seq_silu_mul) X(llark_seq_moe_up) \
    X(llark_seq_moe_down) X(llark_rmsnorm_bwd_workspace) X(llark_ln_bwd_workspace) X(llark_decode_scratch) X(llark_attn_bwd_workspace) \
    X(llark_jb_resblocks_length) X(llark_seq_chunk_block_bytes) X(llark_seq_moe_tile_rows)

namespace {

PyObject *kinds_in_place, *kinds_of_pointer;  // ctypes' arrays and structures; its pointers

template <typename T> bool get(PyObject* o, T*& v) {
    if (o == Py_None) {
        v = nullptr;
        return true;
    }
    if (PyLong_Check(o)) {
        const unsigned long long x = PyLong_AsUnsignedLongLongMask(o);
        v = reinterpret_cast<T*>(x);
        return x != (unsigned long long)-1 || !PyErr_Occurred();
    }
    const int array = PyObject_IsInstance(o, kinds_in_place), pointer = array ? 0 : PyObject_IsInstance(o, kinds_of_pointer);
    if (array < 0 || pointer < 0) return false;
    Py_buffer b;
    if ((!array && !pointer) || PyObject_GetBuffer(o, &b, PyBUF_SIMPLE)) {
        PyErr_Clear();
        PyErr_Format(PyExc_TypeError, "an address, None or a ctypes object expected, not %s", Py_TYPE(o)->tp_name);
        return false;
    }
    v = array ? reinterpret_cast<T*>(b.buf) : *static_cast<T**>(b.buf);  // the caller holds the object
    PyBuffer_Release(&b);
    return true;
}
bool whole(PyObject* o, unsigned long long& x) {
    if (!PyLong_Check(o) && !PyIndex_Check(o)) {
        PyErr_Format(PyExc_TypeError, "an integer expected, not %s", Py_TYPE(o)->tp_name);
        return false;
    }
    x = PyLong_AsUnsignedLongLongMask(o);
    return x != (unsigned long long)-1 || !PyErr_Occurred();
}
bool get(PyObject* o, int& v) {
    unsigned long long x;
    if (!whole(o, x)) return false;
    v = (int)x;
    return true;
}
bool get(PyObject* o, long long& v) {
    unsigned long long x;
    if (!whole(o, x)) return false;
    v = (long long)x;
    return true;
}
bool get(PyObject* o, float& v) {
    const double x = PyFloat_AsDouble(o);
    v = (float)x;
    return x != -1.0 || !PyErr_Occurred();
}

template <typename R, typename... A, size_t... I>
PyObject* invoke(R (*fn)(A...), const char* name, PyObject* const* args, Py_ssize_t n, std::index_sequence<I...>) {
    if (n != (Py_ssize_t)sizeof...(A)) {
        PyErr_Format(PyExc_TypeError, "%s takes %d arguments (%d given)", name, (int)sizeof...(A), (int)n);
        return nullptr;
    }
    if (!fn) {
        PyErr_Format(PyExc_AttributeError, "%s is not in this library", name);
        return nullptr;
    }
    std::tuple<A...> v;
    if (!(get(args[I], std::get<I>(v)) && ...)) return nullptr;
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = fn(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLongLong((long long)r);
}
template <typename R, typename... A>
PyObject* invoke(R (*fn)(A...), const char* name, PyObject* const* args, Py_ssize_t n) {
    return invoke(fn, name, args, n, std::index_sequence_for<A...>{});
}

#define X(N_)                   \
    decltype(&N_) p_##N_;       \
    PyObject* c_##N_(PyObject*, PyObject* const* args, Py_ssize_t n) { return invoke(p_##N_, #N_, args, n); }
LLARK_CALLS(X)
#undef X

PyObject* bind(PyObject*, PyObject* path) {  // the entry points of the (loaded) library at `path`; returns the names that it has
    const char* p = PyUnicode_AsUTF8(path);
    if (!p) return nullptr;
    if (!kinds_in_place) {
        PyObject* m = PyImport_ImportModule("_ctypes");
        PyObject* c = m ? PyImport_ImportModule("ctypes") : nullptr;
        PyObject *array = nullptr, *structure = nullptr, *pointer = nullptr, *address = nullptr;
        if (c && (array = PyObject_GetAttrString(m, "Array")) && (structure = PyObject_GetAttrString(m, "Structure")) &&
            (pointer = PyObject_GetAttrString(m, "_Pointer")) && (address = PyObject_GetAttrString(c, "c_void_p"))) {
            kinds_of_pointer = PyTuple_Pack(2, pointer, address);
            if (kinds_of_pointer) kinds_in_place = PyTuple_Pack(2, array, structure);
        }
        for (PyObject* o : {m, c, array, structure, pointer, address}) Py_XDECREF(o);
        if (!kinds_in_place) return nullptr;
    }
    void* lib = dlopen(p, RTLD_NOW | RTLD_LOCAL);
    if (!lib) {
        PyErr_SetString(PyExc_OSError, dlerror());
        return nullptr;
    }
    PyObject* names = PyList_New(0);
    if (!names) return nullptr;
#define X(N_)                                                      \
    p_##N_ = reinterpret_cast<decltype(&N_)>(dlsym(lib, #N_));     \
    if (p_##N_) {                                                  \
        PyObject* s = PyUnicode_FromString(#N_);                   \
        if (!s || PyList_Append(names, s)) {                       \
            Py_XDECREF(s);                                         \
            Py_DECREF(names);                                      \
            return nullptr;                                        \
        }                                                          \
        Py_DECREF(s);                                              \
    }
    LLARK_CALLS(X)
#undef X
    return names;
}

PyMethodDef methods[] = {
    {"bind", bind, METH_O, "bind(path): take the entry points from the library at path; the names that it has"},
#define X(N_) {#N_, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(c_##N_)), METH_FASTCALL, nullptr},
    LLARK_CALLS(X)
#undef X
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() { return PyModule_Create(&module); }
