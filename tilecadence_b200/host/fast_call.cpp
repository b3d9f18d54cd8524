// The operators' call path in native code: the checks that the Python operator objects make on their tensors, and the
// call of the C ABI with the tensors' addresses, sizes and strides.
//
// Why: a decode step on a short cache takes 6 us on the GPU, while the same checks through tensor attributes and the
// argument conversion of ctypes took 14 to 16 us of host time per call, so that every small call was bound by them.
//
// Each function returns -1 when it does not take the call (a check that fails, an argument of another type than
// expected, a tensor subclass): the Python operator then goes through its own checks and call, which raise what they
// always raised. Otherwise the call has been made, once, and the result is 16 times the status of the C ABI plus what
// the call returns (0, or the number of key splits). Nothing is kept between calls.
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

#include <initializer_list>
#include <type_traits>

#include "tilecadence_b200.h"

namespace {

constexpr int64_t kDim = 128;

// A plain strided CUDA tensor (exactly torch.Tensor, with memory of its own behind it).
bool plain(PyObject* object, const at::Tensor** out) {
    if (!THPVariable_CheckExact(object)) return false;
    const at::Tensor& tensor = THPVariable_Unpack(object);
    if (!tensor.defined() || !tensor.is_cuda() || tensor.layout() != at::kStrided || !tensor.has_storage()) return false;
    *out = &tensor;
    return true;
}

bool shaped(const at::Tensor& tensor, std::initializer_list<int64_t> sizes) { return tensor.sizes() == at::IntArrayRef(sizes); }

// Contiguous, of this device and type, outside of autograd.
bool dense(const at::Tensor& tensor, const at::Tensor& like, at::ScalarType type) {
    return tensor.device() == like.device() && tensor.scalar_type() == type && tensor.is_contiguous() && !tensor.requires_grad();
}

bool whole(PyObject* object, int64_t* out) {
    if (!PyLong_CheckExact(object)) return false;
    *out = PyLong_AsLongLong(object);
    if (*out == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

bool truth(PyObject* object, bool* out) {
    if (!PyBool_Check(object)) return false;
    *out = object == Py_True;
    return true;
}

void* address(const at::Tensor& tensor) { return tensor.numel() ? tensor.data_ptr() : nullptr; }

// As ctypes does for a foreign function: other Python threads may run while the launch is made. Addresses, sizes and
// strides therefore arrive as numbers, read while the GIL was still held: another thread may resize or re-point a tensor
// from here on.
template <class Function, class... Arguments>
int without_gil(Function function, Arguments... arguments) {
    static_assert((... && !std::is_same_v<std::remove_cv_t<std::remove_pointer_t<Arguments>>, at::Tensor>), "no tensors");
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = function(arguments...);
    Py_END_ALLOW_THREADS
    return status * 16;
}

template <class Function>
Function entry(PyObject* object) { return reinterpret_cast<Function>(PyLong_AsVoidPtr(object)); }

// What the decode operators have in common: q, kcache, vcache, knew, vnew, old_lengths, out, lse, workspace_o,
// workspace_lse, num_splits, mapping, append.
struct Decode {
    const at::Tensor *q, *k, *v, *knew, *vnew, *old, *out, *lse, *ws_o, *ws_lse;
    int64_t batch, heads, splits, mapping;
    bool append;
    int device;
    void* stream;

    bool read(PyObject* const* a, int64_t q_heads, bool indexed) {
        const at::Tensor** tensors[10] = {&q, &k, &v, &knew, &vnew, &old, &out, &lse, &ws_o, &ws_lse};
        for (int i = 0; i < 10; ++i)
            if (!plain(a[i], tensors[i])) return false;
        if (!whole(a[10], &splits) || !whole(a[11], &mapping) || !truth(a[12], &append)) return false;
        if (q->dim() != 4 || k->dim() != 4) return false;
        batch = q->size(0);
        heads = q_heads / 4;
        if (batch < 1 || !shaped(*q, {batch, 1, q_heads, kDim}) || k->size(2) != heads || k->size(3) != kDim) return false;
        if (!indexed && (k->size(0) != batch || k->size(1) < 4)) return false;
        for (const at::Tensor* t : {q, k, v, knew, vnew, out})
            if (!dense(*t, *q, at::kBFloat16)) return false;
        for (const at::Tensor* t : {lse, ws_o, ws_lse})
            if (!dense(*t, *q, at::kFloat)) return false;
        if (!dense(*old, *q, at::kInt) || !shaped(*old, {batch})) return false;
        if (v->sizes() != k->sizes() || !shaped(*knew, {batch, 1, heads, kDim}) || !shaped(*vnew, {batch, 1, heads, kDim}) ||
            out->sizes() != q->sizes() || !shaped(*lse, {batch, q_heads, 1}))
            return false;
        if (reinterpret_cast<uintptr_t>(address(*q)) % 16 || reinterpret_cast<uintptr_t>(address(*k)) % 16) return false;
        device = q->device().index();
        stream = c10::cuda::getCurrentCUDAStream(q->device().index()).stream();
        return true;
    }
};

PyObject* done(int status) { return PyLong_FromLong(status); }
constexpr int kNotTaken = -1;

// (address of tc_decode_forward_out_flags, q heads, the 13 arguments, flags)
int decode_call(PyObject* const* a, Py_ssize_t n) {
    Decode d;
    int64_t heads, flags;
    if (n != 16 || !whole(a[1], &heads) || !whole(a[15], &flags) || !d.read(a + 2, heads, false)) return kNotTaken;
    const auto function = entry<decltype(&tc_decode_forward_out_flags)>(a[0]);
    return without_gil(function, d.device, d.stream, address(*d.q), address(*d.k), address(*d.v), address(*d.knew),
                       address(*d.vnew), static_cast<const int32_t*>(address(*d.old)), address(*d.out),
                       static_cast<float*>(address(*d.lse)), static_cast<float*>(address(*d.ws_o)), d.ws_o->numel(),
                       static_cast<float*>(address(*d.ws_lse)), d.ws_lse->numel(), d.batch, d.k->size(1), d.heads,
                       d.splits, d.mapping, d.append, flags);
}

// (address of tc_decode_rope_forward_out, q heads, the 13 arguments, cos, sin)
int rope_call(PyObject* const* a, Py_ssize_t n) {
    Decode d;
    int64_t heads;
    const at::Tensor *cos, *sin;
    if (n != 17 || !whole(a[1], &heads) || !d.read(a + 2, heads, false) || !plain(a[15], &cos) || !plain(a[16], &sin)) return kNotTaken;
    for (const at::Tensor* t : {cos, sin})
        if (t->device() != d.q->device() || t->scalar_type() != at::kFloat || t->dim() != 2 || t->size(1) != 64 ||
            !t->is_contiguous() || t->sizes() != cos->sizes())
            return kNotTaken;
    const auto function = entry<decltype(&tc_decode_rope_forward_out)>(a[0]);
    return without_gil(function, d.device, d.stream, address(*d.q), address(*d.k), address(*d.v), address(*d.knew),
                       address(*d.vnew), static_cast<const int32_t*>(address(*d.old)), address(*d.out),
                       static_cast<float*>(address(*d.lse)), static_cast<float*>(address(*d.ws_o)), d.ws_o->numel(),
                       static_cast<float*>(address(*d.ws_lse)), d.ws_lse->numel(), d.batch, d.k->size(1), d.heads,
                       d.splits, d.mapping, d.append, static_cast<const float*>(address(*cos)),
                       static_cast<const float*>(address(*sin)), cos->size(0));
}

// (address of tc_decode_indexed_forward_out, q heads, the 13 arguments, block_table or None, cache_batch_idx or None)
int indexed_call(PyObject* const* a, Py_ssize_t n) {
    Decode d;
    int64_t heads;
    if (n != 17 || !whole(a[1], &heads) || (a[15] == Py_None) == (a[16] == Py_None) || !d.read(a + 2, heads, true)) return kNotTaken;
    const bool paged = a[15] != Py_None;
    const at::Tensor* index;
    if (!plain(paged ? a[15] : a[16], &index) || index->device() != d.q->device() || index->scalar_type() != at::kInt ||
        index->dim() != (paged ? 2 : 1) || index->size(0) != d.batch || index->stride(-1) != 1)
        return kNotTaken;
    const auto function = entry<decltype(&tc_decode_indexed_forward_out)>(a[0]);
    const int32_t* table = static_cast<const int32_t*>(address(*index));
    return without_gil(function, d.device, d.stream, address(*d.q), address(*d.k), address(*d.v), address(*d.knew),
                       address(*d.vnew), static_cast<const int32_t*>(address(*d.old)), address(*d.out),
                       static_cast<float*>(address(*d.lse)), static_cast<float*>(address(*d.ws_o)), d.ws_o->numel(),
                       static_cast<float*>(address(*d.ws_lse)), d.ws_lse->numel(), d.batch, d.k->size(0), d.k->size(1),
                       d.heads, d.splits, d.mapping, d.append, paged ? table : nullptr, paged ? index->stride(0) : 0,
                       paged ? index->size(1) : 0, paged ? nullptr : table);
}

// q, k, v, out, lse of the prefill operators.
struct Prefill {
    const at::Tensor *q, *k, *v, *out, *lse;
    int64_t batch, tokens, heads, strides[3][3];
    int device;
    void* stream;

    bool read(PyObject* const* a, int64_t q_heads) {
        const at::Tensor** tensors[5] = {&q, &k, &v, &out, &lse};
        for (int i = 0; i < 5; ++i)
            if (!plain(a[i], tensors[i])) return false;
        const at::Tensor* inputs[3] = {q, k, v};
        for (int i = 0; i < 3; ++i) {
            const at::Tensor& t = *inputs[i];
            if (t.dim() != 4 || t.device() != q->device() || t.scalar_type() != at::kBFloat16 || t.requires_grad() ||
                t.stride(3) != 1 || t.size(3) != kDim || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16)
                return false;
            for (int axis = 0; axis < 3; ++axis) {
                strides[i][axis] = t.stride(axis);
                if (t.size(axis) != 1 && (t.stride(axis) < 0 || t.stride(axis) % 8)) return false;
            }
        }
        batch = q->size(0);
        tokens = q->size(1);
        heads = q_heads;
        if (batch < 1 || tokens < 2 || q->size(2) != heads || !shaped(*k, {batch, tokens, heads / 4, kDim}) ||
            v->sizes() != k->sizes())
            return false;
        if (!dense(*out, *q, at::kBFloat16) || out->sizes() != q->sizes() || !dense(*lse, *q, at::kFloat) ||
            !shaped(*lse, {batch, heads, tokens}))
            return false;
        device = q->device().index();
        stream = c10::cuda::getCurrentCUDAStream(q->device().index()).stream();
        return true;
    }
};

// (address of tc_prefill_forward_out, q heads, q, k, v, out, lse, workspace_o, workspace_lse, num_splits, mapping, scale,
// causal)
int prefill_call(PyObject* const* a, Py_ssize_t n) {
    Prefill p;
    int64_t heads, splits, mapping;
    bool causal;
    const at::Tensor *ws_o, *ws_lse;
    if (n != 13 || !whole(a[1], &heads) || !p.read(a + 2, heads) || !plain(a[7], &ws_o) || !plain(a[8], &ws_lse) ||
        ws_o->numel() || ws_lse->numel() || !whole(a[9], &splits) || !whole(a[10], &mapping) || !PyFloat_CheckExact(a[11]) ||
        !truth(a[12], &causal) || !causal)
        return kNotTaken;
    const double scale = PyFloat_AS_DOUBLE(a[11]);
    const auto function = entry<decltype(&tc_prefill_forward_out)>(a[0]);
    return without_gil(function, p.device, p.stream, address(*p.q), p.strides[0], address(*p.k), p.strides[1],
                       address(*p.v), p.strides[2], address(*p.out), static_cast<float*>(address(*p.lse)), 0, 0, p.batch,
                       p.tokens, p.heads, splits, mapping, scale, 1);
}

// (address of tc_prefill_key_split_forward_out, q heads, q, k, v, out, lse, workspace, mapping, scale, key_splits).
// Returns the number of key splits used with the status.
int key_split_call(PyObject* const* a, Py_ssize_t n) {
    Prefill p;
    int64_t heads, mapping, key_splits, used = 0;
    const at::Tensor* workspace;
    if (n != 11 || !whole(a[1], &heads) || !p.read(a + 2, heads) || !plain(a[7], &workspace) ||
        workspace->device() != p.q->device() || workspace->scalar_type() != at::kByte || !workspace->is_contiguous() ||
        !whole(a[8], &mapping) || !PyFloat_CheckExact(a[9]) || !whole(a[10], &key_splits))
        return kNotTaken;
    const double scale = PyFloat_AS_DOUBLE(a[9]);
    const auto function = entry<decltype(&tc_prefill_key_split_forward_out)>(a[0]);
    const int result = without_gil(function, p.device, p.stream, address(*p.q), p.strides[0], address(*p.k), p.strides[1],
                                   address(*p.v), p.strides[2], address(*p.out), static_cast<float*>(address(*p.lse)),
                                   address(*workspace), workspace->numel(), p.batch, p.tokens, p.heads, mapping, scale,
                                   key_splits, &used);
    return result + int(used);
}

// (address of tc_exchange_forward_out, q, k, v, out, lse, causal)
int exchange_call(PyObject* const* a, Py_ssize_t n) {
    const at::Tensor *q, *k, *v, *out, *lse;
    bool causal;
    if (n != 7 || !plain(a[1], &q) || !plain(a[2], &k) || !plain(a[3], &v) || !plain(a[4], &out) || !plain(a[5], &lse) ||
        !truth(a[6], &causal))
        return kNotTaken;
    const at::ScalarType type = q->scalar_type();
    if (q->dim() != 4 || (type != at::kHalf && type != at::kBFloat16)) return kNotTaken;
    const int64_t batch = q->size(0), heads = q->size(2);
    if (batch < 1 || heads < 1 || !shaped(*q, {batch, 64, heads, kDim})) return kNotTaken;
    for (const at::Tensor* t : {q, k, v, out})
        if (!dense(*t, *q, type) || t->sizes() != q->sizes()) return kNotTaken;
    if (lse->device() != q->device() || lse->scalar_type() != at::kFloat || !lse->is_contiguous() || !shaped(*lse, {batch, heads, 64}))
        return kNotTaken;
    const int device = q->device().index();
    void* stream = c10::cuda::getCurrentCUDAStream(q->device().index()).stream();
    const auto function = entry<decltype(&tc_exchange_forward_out)>(a[0]);
    return without_gil(function, device, stream, address(*q), address(*k), address(*v), address(*out),
                       static_cast<float*>(address(*lse)), batch, heads, type == at::kHalf, causal);
}

template <int (*call)(PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject*, PyObject* const* arguments, Py_ssize_t count) {
    int status = kNotTaken;
    try {
        status = call(arguments, count);
    } catch (...) {  // torch's own checks throw; the Python path then says what is wrong
        status = kNotTaken;
    }
    if (PyErr_Occurred()) PyErr_Clear();
    return done(status);
}

template <int (*call)(PyObject* const*, Py_ssize_t)>
PyCFunction method() { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<call>)); }

PyMethodDef methods[] = {
    {"decode", method<decode_call>(), METH_FASTCALL, nullptr},
    {"rope", method<rope_call>(), METH_FASTCALL, nullptr},
    {"indexed", method<indexed_call>(), METH_FASTCALL, nullptr},
    {"prefill", method<prefill_call>(), METH_FASTCALL, nullptr},
    {"key_split", method<key_split_call>(), METH_FASTCALL, nullptr},
    {"exchange", method<exchange_call>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "tc_fast_call", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_tc_fast_call() { return PyModule_Create(&module); }
