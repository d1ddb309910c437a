// Native front ends of the Python operators: argument checks, output allocation and the call into the C ABI of
// libdsv4_prologue.so, in one CPython extension module (flaggems_vllm/_host_calls.so).
//
// Why: decode-sized launches take 2-5 us on the GPU, and a layer issues about nine of them.  Written in Python, the checks,
// two torch.empty, the device guard, the stream look-up and a ctypes call with 15-25 arguments cost 12-27 us of host time
// per operator, so a decode step was bound by the host (185 us for 52 us of GPU work).  Here an operator costs the launch
// (1.6 to 2 us) plus its output allocations.
//
// Contract with the Python wrappers: a function returns its result (True for operators that fill their arguments) or None
// when an argument is not acceptable; the wrapper then runs its own assertions, which name the argument.  The checks below
// are those assertions, one for one (tests/test_host_checks_agree.py compares the two), and a few limits of the C ABI: the text of
// the first check that failed is what _refusal() returns, for arguments that the assertions let pass.  A non-zero code of the C
// ABI is handed to the callable given to bind(), which raises.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdio>

#include "../../include/dsv4_prologue.h"
#include "current_device.h"

namespace {

using at::ScalarType;
using at::Tensor;

PyObject* g_check = nullptr;  // raises for a non-zero code of the C ABI
thread_local char t_refusal[256] = "";  // why the thread's last refused call was refused

// Argument list of one call.  `ok` turns false at the first argument that is not acceptable.
struct Arguments {
    PyObject* const* values;
    Py_ssize_t count;
    bool ok = true;

    void require(bool condition, const char* text) {
        if (ok && !condition) refuse(text);
    }
    __attribute__((noinline, cold)) void refuse(const char* text, Py_ssize_t argument = -1) {
        ok = false;
        if (argument < 0) std::snprintf(t_refusal, sizeof t_refusal, "%s", text);
        else std::snprintf(t_refusal, sizeof t_refusal, "argument %d %s", static_cast<int>(argument), text);
    }

    // A tensor with storage of its own (wrapper subclasses that dispatch to Python have none), or null.
    const Tensor* tensor(Py_ssize_t i) {
        if (!ok) return nullptr;
        if (i < count && THPVariable_Check(values[i])) {
            const Tensor& t = THPVariable_Unpack(values[i]);
            if (t.defined() && !t.unsafeGetTensorImpl()->is_python_dispatch()) return &t;
        }
        refuse("is not a tensor with storage of its own", i);
        return nullptr;
    }
    bool is_none(Py_ssize_t i) const { return i >= count || values[i] == Py_None; }
    // Whatever int() takes.
    int64_t integer_of(Py_ssize_t i) {
        if (!ok) return 0;
        if (i < count) {
            PyObject* number = PyLong_CheckExact(values[i]) ? values[i] : PyNumber_Long(values[i]);
            const long long v = number ? PyLong_AsLongLong(number) : -1;
            if (number != values[i]) Py_XDECREF(number);
            if (v != -1 || !PyErr_Occurred()) return v;
            PyErr_Clear();
        }
        refuse("is not an integer of 64 bits", i);
        return 0;
    }
    // The same without text, for the sizes that the assertions compare or compute with.
    int64_t integer(Py_ssize_t i) {
        if (ok && i < count && !PyLong_CheckExact(values[i]) && (PyUnicode_Check(values[i]) || PyBytes_Check(values[i]) || PyByteArray_Check(values[i])))
            refuse("is not a number", i);
        return integer_of(i);
    }
    float real(Py_ssize_t i) {
        if (!ok) return 0.0f;
        if (i < count) {
            const double v = PyFloat_AsDouble(values[i]);
            if (v != -1.0 || !PyErr_Occurred()) return static_cast<float>(v);
            PyErr_Clear();
        }
        refuse("is not a number", i);
        return 0.0f;
    }
    bool truth(Py_ssize_t i) {
        if (!ok || i >= count) return false;
        const int v = PyObject_IsTrue(values[i]);
        if (v >= 0) return v != 0;
        PyErr_Clear();
        refuse("has no truth value", i);
        return false;
    }
};

#define REQUIRE(...) a.require((__VA_ARGS__), #__VA_ARGS__)

bool is(const Tensor& t, ScalarType type) { return t.scalar_type() == type; }
bool on(const Tensor& t, const Tensor& first) { return t.is_cuda() && t.get_device() == first.get_device(); }

using dsv4::OnDevice;
OnDevice on_device_of(const Tensor& t, OnDevice::Use use = OnDevice::kAllocatesToo) { return OnDevice(static_cast<c10::DeviceIndex>(t.get_device()), use); }

// A contiguous, uninitialised tensor on the device of the call, without the look at torch's set-up and the device guard that empty_cuda()
// takes each time.
Tensor make_empty(at::IntArrayRef sizes, ScalarType type, const OnDevice&) {
    static const bool set_up = (at::globalContext().lazyInitDevice(at::kCUDA), true);
    (void)set_up;
    return Tensor(at::detail::empty_generic(sizes, c10::cuda::CUDACachingAllocator::get(), c10::DispatchKeySet(c10::DispatchKey::CUDA), type, std::nullopt));
}

// Gives a tensor that was just allocated other sizes and strides over the same storage (what a chain of view operators
// would do, without dispatching them).
void set_view(Tensor& t, at::IntArrayRef sizes, at::IntArrayRef strides) {
    t.unsafeGetTensorImpl()->set_sizes_and_strides(sizes, strides);
}

// Runs `launch(stream)` with the device of the call current.  False after a failed launch, with a Python error set.
template <typename Launch>
bool launch_on(const OnDevice& here, Launch&& launch) {
    void* stream = c10::cuda::getCurrentCUDAStream(here.index).stream();
    int code;
    // a launch can block (full launch queue): other Python threads go on meanwhile
    Py_BEGIN_ALLOW_THREADS
    code = launch(stream);
    Py_END_ALLOW_THREADS
    if (code == 0) return true;
    PyObject* r = PyObject_CallFunction(g_check, "i", code);
    if (r) {
        Py_DECREF(r);
        PyErr_SetString(PyExc_RuntimeError, "a kernel launch failed");
    }
    return false;
}

PyObject* wrap(Tensor&& t) { return THPVariable_Wrap(std::move(t)); }

PyObject* pair(Tensor&& a, Tensor&& b) {
    PyObject* first = wrap(std::move(a));
    if (!first) return nullptr;
    PyObject* second = wrap(std::move(b));
    if (!second) {
        Py_DECREF(first);
        return nullptr;
    }
    PyObject* t = PyTuple_New(2);
    if (!t) {
        Py_DECREF(first), Py_DECREF(second);
        return nullptr;
    }
    PyTuple_SET_ITEM(t, 0, first), PyTuple_SET_ITEM(t, 1, second);
    return t;
}

// Turns C++ exceptions (an allocation that fails, for instance) into Python ones.
template <PyObject* (*Body)(Arguments&)>
PyObject* entry(PyObject*, PyObject* const* values, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    Arguments a{values, count};
    return Body(a);
    END_HANDLE_TH_ERRORS
}

// q, kv, k_cache, slot_mapping, position_ids, cos_sin_cache, eps, cache_block_size
PyObject* prologue(Arguments& a) {
    const Tensor *q = a.tensor(0), *kv = a.tensor(1), *cache = a.tensor(2), *slots = a.tensor(3), *pos = a.tensor(4), *cs = a.tensor(5);
    const float eps = a.real(6);
    const int64_t block = a.integer(7);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(q->is_cuda() && q->is_contiguous() && kv->is_contiguous() && q->dim() == 3 && q->size(2) == 512);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t tokens = q->size(0), heads = q->size(1);
    REQUIRE(kv->dim() == 2 && kv->size(0) == tokens && kv->size(1) == 512);
    REQUIRE(is(*q, at::kBFloat16) && is(*kv, at::kBFloat16) && is(*cache, at::kByte));
    REQUIRE(slots->dim() == 1 && is(*slots, at::kLong) && slots->is_contiguous() && slots->size(0) <= tokens);
    REQUIRE(pos->dim() == 1 && is(*pos, at::kLong) && pos->is_contiguous() && pos->size(0) == tokens);
    REQUIRE(cs->dim() == 2 && cs->size(1) == 64 && is(*cs, at::kFloat) && cs->is_contiguous());
    REQUIRE(cache->dim() == 2 && cache->stride(1) == 1 && block > 0 && cache->size(1) / 584 >= block);
    REQUIRE(on(*kv, *q) && on(*cache, *q) && on(*slots, *q) && on(*pos, *q) && on(*cs, *q));
    if (!a.ok) Py_RETURN_NONE;
    if (tokens == 0) Py_RETURN_TRUE;
    if (!launch_on(on_device_of(*q, OnDevice::kLaunchesOnly), [&](void* stream) {
            return dsv4_qnorm_rope_kv_insert(q->data_ptr(), kv->data_ptr(), cache->data_ptr(), static_cast<const int64_t*>(slots->data_ptr()),
                                             static_cast<const int64_t*>(pos->data_ptr()), static_cast<const float*>(cs->data_ptr()), eps,
                                             tokens, heads, slots->size(0), block, cache->stride(0), stream);
        }))
        return nullptr;
    Py_RETURN_TRUE;
}

// The library's code of a row or weight type, -1 for a type it does not take.
int dtype_code(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kBFloat16: return 0;
        case at::kHalf: return 1;
        case at::kFloat: return 2;
        default: return -1;
    }
}

// qr, kv, q_weight, kv_weight, eps -> (qr_out, kv_out)
PyObject* q_kv_rmsnorm(Arguments& a) {
    const Tensor *qr = a.tensor(0), *kv = a.tensor(1), *qw = a.tensor(2), *kw = a.tensor(3);
    const float eps = a.real(4);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(qr->is_cuda() && qr->dim() == 2 && kv->dim() == 2 && qr->size(0) == kv->size(0));
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(qr->stride(1) == 1 && kv->stride(1) == 1 && qw->is_contiguous() && kw->is_contiguous());
    REQUIRE(dtype_code(*qr) >= 0 && dtype_code(*kv) >= 0 && dtype_code(*qw) >= 0 && dtype_code(*kw) >= 0);
    REQUIRE(on(*kv, *qr) && on(*qw, *qr) && on(*kw, *qr));
    REQUIRE(qw->dim() == 1 && qw->size(0) == qr->size(1) && kw->dim() == 1 && kw->size(0) == kv->size(1));
    if (!a.ok) Py_RETURN_NONE;
    const int64_t tokens = qr->size(0);
    const OnDevice here = on_device_of(*qr);
    Tensor qo = make_empty(qr->sizes(), qr->scalar_type(), here), ko = make_empty(kv->sizes(), kv->scalar_type(), here);
    if (tokens > 0 && !launch_on(here, [&](void* stream) {
            return dsv4_fused_q_kv_rmsnorm_dtypes(qr->data_ptr(), qo.data_ptr(), qw->data_ptr(), qr->stride(0), qo.stride(0), qr->size(1),
                                                  dtype_code(*qr), dtype_code(*qw), kv->data_ptr(), ko.data_ptr(), kw->data_ptr(),
                                                  kv->stride(0), ko.stride(0), kv->size(1), dtype_code(*kv), dtype_code(*kw), tokens, eps, stream);
        }))
        return nullptr;
    return pair(std::move(qo), std::move(ko));
}

// x, group_size, eps, column_major_scales, scale_ue8m0 -> (x_q, x_s)
PyObject* group_quant(Arguments& a) {
    const Tensor* x = a.tensor(0);
    const int64_t group = a.integer(1);
    const float eps = a.real(2);
    const bool column_major = a.truth(3), ue8m0 = a.truth(4);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(x->is_cuda() && is(*x, at::kBFloat16) && x->dim() >= 2 && group > 0);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t cols = x->size(-1);
    REQUIRE(cols % group == 0 && x->stride(-1) == 1 && (x->dim() == 2 || (x->is_contiguous() && !column_major)));
    if (!a.ok) Py_RETURN_NONE;
    const int64_t rows = cols > 0 ? x->numel() / cols : 0, groups = cols / group;
    const OnDevice here = on_device_of(*x);
    Tensor xq = make_empty(x->sizes(), at::kFloat8_e4m3fn, here), xs;
    if (column_major) {
        xs = make_empty({groups, x->size(0)}, at::kFloat, here);
        set_view(xs, {x->size(0), groups}, {1, std::max<int64_t>(x->size(0), 1)});
    } else {
        at::DimVector sizes(x->sizes().begin(), x->sizes().end());
        sizes.back() = groups;
        xs = make_empty(sizes, at::kFloat, here);
    }
    const int64_t stride_row = column_major ? 1 : groups, stride_group = column_major ? x->size(0) : 1;
    if (rows > 0 && !launch_on(here, [&](void* stream) {
            return dsv4_per_token_group_quant_fp8(x->data_ptr(), x->dim() == 2 ? x->stride(0) : cols, xq.data_ptr(),
                                                  static_cast<float*>(xs.data_ptr()), stride_row, stride_group, rows, cols, group, eps,
                                                  ue8m0 ? 1 : 0, stream);
        }))
        return nullptr;
    return pair(std::move(xq), std::move(xs));
}

// x, block_size, round_scale -> (y, s)
PyObject* act_quant(Arguments& a) {
    const Tensor* x = a.tensor(0);
    const int64_t block = a.integer(1);
    const bool round_scale = a.truth(2);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(x->is_cuda() && is(*x, at::kBFloat16) && x->dim() >= 1 && x->is_contiguous() && block > 0 && x->size(-1) % block == 0);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t cols = x->size(-1), rows = cols > 0 ? x->numel() / cols : 0;
    const OnDevice here = on_device_of(*x);
    Tensor y = make_empty(x->sizes(), at::kFloat8_e4m3fn, here);
    at::DimVector sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = cols / block;
    Tensor s = make_empty(sizes, at::kFloat, here);
    if (rows > 0 && !launch_on(here, [&](void* stream) {
            return dsv4_act_quant(x->data_ptr(), cols, y.data_ptr(), static_cast<float*>(s.data_ptr()), rows, cols, block, round_scale ? 1 : 0,
                                  stream);
        }))
        return nullptr;
    return pair(std::move(y), std::move(s));
}

// o, positions, cos_sin_cache, n_groups, heads_per_group, nope_dim, rope_dim, quant_group_size, eps, tma_aligned_scales
// -> (o_fp8, o_scale), both views with the token dimension in front of the group dimension of the storage
PyObject* inv_rope_fp8_quant(Arguments& a) {
    const Tensor *o = a.tensor(0), *pos = a.tensor(1), *cs = a.tensor(2);
    const int64_t n_groups = a.integer(3), per_group = a.integer(4), nope = a.integer(5), rope = a.integer(6), group = a.integer(7);
    const float eps = a.real(8);
    const bool packed = a.truth(9);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(o->is_cuda() && o->dim() == 3 && pos->dim() == 1 && cs->dim() == 2 && n_groups > 0 && per_group > 0 && group > 0);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t tokens = o->size(0), heads = o->size(1), head_dim = o->size(2);
    REQUIRE(o->stride(2) == 1 && pos->size(0) == tokens && heads == n_groups * per_group && nope >= 0 && rope >= 0);
    REQUIRE(head_dim == nope + rope && head_dim % group == 0 && nope % group == group - rope && rope % 2 == 0 && group % 2 == 0);
    REQUIRE(cs->size(1) == rope && is(*cs, at::kFloat) && cs->stride(1) == 1);
    REQUIRE(is(*o, at::kBFloat16) && is(*pos, at::kLong) && pos->is_contiguous() && on(*pos, *o) && on(*cs, *o));
    const int64_t per_head = group > 0 ? head_dim / group : 0;
    REQUIRE(!packed || per_head == 4);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t d = per_group * head_dim, padded = (tokens + 3) / 4 * 4;
    const int64_t inner = packed ? (d / group + 3) / 4 : d / group;
    const OnDevice here = on_device_of(*o);
    Tensor fp8 = make_empty({n_groups, tokens, d}, at::kFloat8_e4m3fn, here);
    Tensor scale = make_empty({n_groups * inner * padded}, packed ? at::kInt : at::kFloat, here);
    if (tokens > 0 && !launch_on(here, [&](void* stream) {
            return dsv4_fused_inv_rope_fp8_quant_geometry(
                o->data_ptr(), o->stride(0), o->stride(1), static_cast<const int64_t*>(pos->data_ptr()),
                static_cast<const float*>(cs->data_ptr()), cs->stride(0), fp8.data_ptr(), scale.data_ptr(), inner * padded, tokens, padded,
                n_groups, per_group, nope, rope, group, eps, packed ? 1 : 0, stream);
        }))
        return nullptr;
    set_view(fp8, {tokens, n_groups, d}, {d, std::max<int64_t>(tokens, 1) * d, 1});
    set_view(scale, {tokens, n_groups, inner}, {1, inner * padded, padded});
    return pair(std::move(fp8), std::move(scale));
}

// positions, index_q, cos_sin_cache, weights, softmax_scale, head_scale, use_fp4 -> (q, weights) or ((q, scale), weights)
PyObject* indexer_q_rope_quant(Arguments& a) {
    const Tensor *pos = a.tensor(0), *q = a.tensor(1), *cs = a.tensor(2), *w = a.tensor(3);
    const float softmax_scale = a.real(4), head_scale = a.real(5);
    const bool fp4 = a.truth(6);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(q->is_cuda() && pos->dim() == 1 && q->dim() == 3 && cs->dim() == 2 && w->dim() == 2);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t tokens = pos->size(0), heads = q->size(1), dim = q->size(2), rot = cs->size(1);
    REQUIRE(is(*q, at::kBFloat16) && q->stride(2) == 1 && q->size(0) == tokens && is(*pos, at::kLong) && pos->is_contiguous());
    REQUIRE((is(*cs, at::kFloat) || is(*cs, at::kBFloat16)) && cs->stride(1) == 1);
    REQUIRE(dtype_code(*w) >= 0 && w->size(0) == tokens && w->size(1) == heads && w->stride(1) == 1);
    REQUIRE((dim == 64 || dim == 128 || dim == 256) && rot % 2 == 0 && rot <= dim && (dim - rot) % (dim / 32) == 0);
    REQUIRE(on(*pos, *q) && on(*cs, *q) && on(*w, *q));
    if (!a.ok) Py_RETURN_NONE;
    const OnDevice here = on_device_of(*q);
    Tensor w_out = make_empty({tokens, heads}, at::kFloat, here), q_out, scale;
    void* scale_ptr = nullptr;
    if (fp4) {
        q_out = make_empty({tokens, heads, dim / 2}, at::kByte, here);
        // the four UE8M0 bytes of a head of 128 travel as one int32 (two for 256); a head of 64 keeps its two bytes
        const int64_t words = dim / 128;
        if (words == 1) scale = make_empty({tokens, heads}, at::kInt, here);
        else if (words > 1) scale = make_empty({tokens, heads, words}, at::kInt, here);
        else scale = make_empty({tokens, heads, dim / 32}, at::kByte, here);
        scale_ptr = scale.data_ptr();
    } else if (q->is_contiguous()) {
        q_out = make_empty(q->sizes(), at::kFloat8_e4m3fn, here);
    } else {  // keeps the order of dimensions in memory that a dense, permuted q has
        q_out = at::empty_like(*q, q->options().dtype(at::kFloat8_e4m3fn));
        REQUIRE(q_out.stride(2) == 1);
        if (!a.ok) Py_RETURN_NONE;
    }
    if (tokens > 0 && !launch_on(here, [&](void* stream) {
            return dsv4_fused_indexer_q_rope_quant(
                static_cast<const int64_t*>(pos->data_ptr()), q->data_ptr(), q->stride(0), q->stride(1), cs->data_ptr(), cs->stride(0),
                is(*cs, at::kBFloat16) ? 1 : 0, rot, q_out.data_ptr(), q_out.stride(0), q_out.stride(1), scale_ptr,
                scale_ptr ? heads * (dim / 32) : 0, scale_ptr ? dim / 32 : 0, w->data_ptr(), w->stride(0), dtype_code(*w),
                static_cast<float*>(w_out.data_ptr()), w_out.stride(0), softmax_scale, head_scale, tokens, heads, dim, fp4 ? 1 : 0, stream);
        }))
        return nullptr;
    if (!fp4) return pair(std::move(q_out), std::move(w_out));
    PyObject* quantised = pair(std::move(q_out), std::move(scale));
    if (!quantised) return nullptr;
    PyObject* weights = wrap(std::move(w_out));
    PyObject* result = weights ? PyTuple_New(2) : nullptr;
    if (!result) {
        Py_DECREF(quantised), Py_XDECREF(weights);
        return nullptr;
    }
    PyTuple_SET_ITEM(result, 0, quantised), PyTuple_SET_ITEM(result, 1, weights);
    return result;
}

// k, kv_cache, slot_mapping, quant_block_size, scale_is_ue8m0
PyObject* indexer_k_quant(Arguments& a) {
    const Tensor *k = a.tensor(0), *cache = a.tensor(1), *slots = a.tensor(2);
    const int64_t group = a.integer(3);
    const bool ue8m0 = a.truth(4);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(k->is_cuda() && k->dim() == 2 && cache->dim() == 3 && slots->dim() == 1 && group > 0);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t dim = k->size(1), tokens = slots->size(0), block = cache->size(1), row = cache->size(2);
    REQUIRE(dim % group == 0 && k->stride(1) == 1 && (is(*k, at::kBFloat16) || is(*k, at::kHalf)) && k->size(0) >= tokens);
    REQUIRE(is(*slots, at::kLong) && slots->is_contiguous() && is(*cache, at::kByte));
    REQUIRE(row == dim + 4 * (dim / group) && (cache->is_contiguous() || (cache->stride(2) == 1 && (block == 1 || cache->stride(1) == row))));
    REQUIRE(on(*cache, *k) && on(*slots, *k));
    if (!a.ok) Py_RETURN_NONE;
    if (tokens == 0 || cache->size(0) == 0) Py_RETURN_TRUE;
    if (!launch_on(on_device_of(*k, OnDevice::kLaunchesOnly), [&](void* stream) {
            return dsv4_indexer_k_quant_and_cache(k->data_ptr(), k->stride(0), is(*k, at::kHalf) ? 1 : 0, cache->data_ptr(), cache->stride(0),
                                                  static_cast<const int64_t*>(slots->data_ptr()), tokens, block, dim, group, ue8m0 ? 1 : 0, stream);
        }))
        return nullptr;
    Py_RETURN_TRUE;
}

// k_cache, k_fp8, k_fp8_scale, block_table, cu_seqlen
PyObject* cp_gather_indexer(Arguments& a) {
    const Tensor *cache = a.tensor(0), *k = a.tensor(1), *scale = a.tensor(2), *table = a.tensor(3), *cu = a.tensor(4);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(cache->is_cuda() && cache->dim() == 3 && k->dim() == 2 && scale->dim() == 2 && table->dim() == 2 && cu->dim() == 1);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t tokens = k->size(0), dim = k->size(1), block = cache->size(1), batch = table->size(0);
    const int64_t scale_bytes = scale->size(1) * static_cast<int64_t>(scale->element_size());
    REQUIRE(scale_bytes > 0);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t group = dim * 4 / scale_bytes;
    REQUIRE(group > 0 && dim % group == 0);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t groups = dim / group;
    REQUIRE(is(*cache, at::kByte) && cache->is_contiguous() && cache->size(2) == dim + 4 * groups);
    REQUIRE(k->element_size() == 1 && k->stride(1) == 1 && scale->size(0) >= tokens && scale->stride(1) == 1 && scale_bytes == 4 * groups);
    REQUIRE(is(*table, at::kInt) && table->stride(1) == 1 && is(*cu, at::kInt) && cu->is_contiguous() && cu->size(0) == batch + 1);
    REQUIRE(on(*k, *cache) && on(*scale, *cache) && on(*table, *cache) && on(*cu, *cache));
    if (!a.ok) Py_RETURN_NONE;
    if (tokens == 0 || batch == 0 || cache->size(0) == 0) Py_RETURN_TRUE;
    if (!launch_on(on_device_of(*cache, OnDevice::kLaunchesOnly), [&](void* stream) {
            return dsv4_cp_gather_indexer_k_quant_cache(cache->data_ptr(), cache->stride(0), k->data_ptr(), k->stride(0), scale->data_ptr(),
                                                        scale->stride(0) * static_cast<int64_t>(scale->element_size()),
                                                        static_cast<const int32_t*>(table->data_ptr()), table->stride(0),
                                                        static_cast<const int32_t*>(cu->data_ptr()), batch, tokens, block, dim, groups, stream);
        }))
        return nullptr;
    Py_RETURN_TRUE;
}

// topk_indices, token_to_req_indices, block_table, block_size, is_valid_token or None -> (global_indices, lens)
PyObject* global_topk(Arguments& a) {
    const Tensor *topk = a.tensor(0), *request = a.tensor(1), *table = a.tensor(2);
    const int64_t block = a.integer_of(3);
    const Tensor* valid = a.is_none(4) ? nullptr : a.tensor(4);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(topk->is_cuda() && topk->dim() == 2 && table->dim() == 2 && request->dim() == 1 && block > 0);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t tokens = topk->size(0), width = topk->size(1);
    REQUIRE(is(*topk, at::kInt) && topk->stride(1) == 1 && is(*table, at::kInt) && table->stride(1) == 1);
    REQUIRE(is(*request, at::kInt) && request->is_contiguous() && request->size(0) == tokens);
    REQUIRE(!valid || (is(*valid, at::kInt) && valid->is_contiguous() && valid->dim() == 1 && valid->size(0) == tokens && on(*valid, *topk)));
    REQUIRE(on(*request, *topk) && on(*table, *topk));
    if (!a.ok) Py_RETURN_NONE;
    const OnDevice here = on_device_of(*topk);
    Tensor out = topk->is_contiguous() ? make_empty(topk->sizes(), at::kInt, here) : at::empty_like(*topk);
    Tensor lens = make_empty({tokens}, at::kInt, here);
    if (tokens > 0 && !launch_on(here, [&](void* stream) {
            return dsv4_compute_global_topk_indices_and_lens(
                static_cast<const int32_t*>(topk->data_ptr()), topk->stride(0), static_cast<const int32_t*>(request->data_ptr()),
                static_cast<const int32_t*>(table->data_ptr()), table->stride(0), valid ? static_cast<const int32_t*>(valid->data_ptr()) : nullptr,
                static_cast<int32_t*>(out.data_ptr()), out.stride(0), static_cast<int32_t*>(lens.data_ptr()), tokens, width, block, stream);
        }))
        return nullptr;
    return pair(std::move(out), std::move(lens));
}

// topk_indices, query_start_loc, seq_lens, gather_lens, window_size, compress_ratio, topk, M, N -> (combined, lens)
PyObject* combine_topk_swa(Arguments& a) {
    constexpr int64_t kAlignment = 128;  // of a row of the result, in entries
    const Tensor *topk = a.tensor(0), *start = a.tensor(1), *seq = a.tensor(2), *gather = a.tensor(3);
    const int64_t window = a.integer(4), ratio = a.integer_of(5), k = a.integer(6), m = a.integer_of(7), n = a.integer_of(8);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(topk->is_cuda() && topk->dim() == 2 && start->dim() == 1 && seq->dim() == 1 && gather->dim() == 1);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t tokens = topk->size(0), requests = seq->size(0);
    REQUIRE(is(*topk, at::kInt) && topk->stride(1) == 1 && k <= topk->size(1) && k + window >= 0);
    for (const Tensor* t : {start, seq, gather}) REQUIRE(is(*t, at::kInt) && t->is_contiguous() && on(*t, *topk));
    REQUIRE(start->size(0) >= requests + 1 && gather->size(0) >= requests);
    if (!a.ok) Py_RETURN_NONE;
    const int64_t width = (k + window + kAlignment - 1) / kAlignment * kAlignment;
    const OnDevice here = on_device_of(*topk);
    Tensor combined = make_empty({tokens, width}, at::kInt, here), lens = make_empty({tokens}, at::kInt, here);
    if (tokens > 0 && requests > 0 && !launch_on(here, [&](void* stream) {
            return dsv4_combine_topk_swa_indices(
                static_cast<const int32_t*>(topk->data_ptr()), topk->stride(0), topk->size(1), static_cast<const int32_t*>(start->data_ptr()),
                static_cast<const int32_t*>(seq->data_ptr()), static_cast<const int32_t*>(gather->data_ptr()),
                static_cast<int32_t*>(combined.data_ptr()), combined.stride(0), width, static_cast<int32_t*>(lens.data_ptr()), requests, tokens,
                window, ratio, k, m, n, stream);
        }))
        return nullptr;
    return pair(std::move(combined), std::move(lens));
}

// out, k_cache, seq_lens, gather_lens or None, block_table, block_size, offset, rope_dim, nope_dim, scale_slots
PyObject* dequantize_and_gather(Arguments& a) {
    const Tensor *out = a.tensor(0), *cache = a.tensor(1), *seq = a.tensor(2);
    const Tensor* gather = a.is_none(3) ? nullptr : a.tensor(3);
    const Tensor* table = a.tensor(4);
    const int64_t block = a.integer_of(5), offset = a.integer_of(6), rope = a.integer(7);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(out->is_cuda() && out->dim() == 3 && seq->dim() == 1 && table->dim() == 2);
    // a 3-D cache with gaps between its rows is copied by the wrapper first
    REQUIRE(cache->dim() == 2 || (cache->dim() == 3 && cache->is_contiguous()));
    if (!a.ok) Py_RETURN_NONE;
    const int64_t width = out->size(2), nope = a.is_none(8) ? width - rope : a.integer(8);
    const int64_t slots = a.is_none(9) ? (nope + 63) / 64 + (nope % 64 == 0 ? 1 : 0) : a.integer(9);
    const int64_t requests = seq->size(0);
    REQUIRE(is(*out, at::kBFloat16) && out->stride(2) == 1 && table->size(0) == requests && requests <= out->size(0));
    REQUIRE(nope >= 0 && rope >= 0 && nope + rope <= width && nope <= INT32_MAX && rope <= INT32_MAX && slots <= INT32_MAX);
    REQUIRE(is(*cache, at::kByte) && cache->stride(-1) == 1);
    const ScalarType index = seq->scalar_type();
    REQUIRE((index == at::kInt || index == at::kLong) && is(*table, index) && seq->is_contiguous() && table->is_contiguous());
    REQUIRE(!gather || (is(*gather, index) && gather->is_contiguous() && gather->dim() == 1 && gather->size(0) == requests && on(*gather, *out)));
    REQUIRE(on(*cache, *out) && on(*seq, *out) && on(*table, *out));
    if (!a.ok) Py_RETURN_NONE;
    if (requests == 0 || out->size(1) == 0) Py_RETURN_TRUE;
    const int64_t pitch = cache->dim() == 3 ? cache->size(1) * cache->size(2) : cache->stride(0);
    if (!launch_on(on_device_of(*out, OnDevice::kLaunchesOnly), [&](void* stream) {
            return dsv4_dequantize_and_gather_k_cache(out->data_ptr(), out->stride(0), out->stride(1), out->size(1), cache->data_ptr(),
                                                      seq->data_ptr(), gather ? gather->data_ptr() : nullptr, table->data_ptr(), requests,
                                                      table->size(1), block, pitch, offset, static_cast<int32_t>(nope),
                                                      static_cast<int32_t>(rope), static_cast<int32_t>(slots), index == at::kLong ? 1 : 0, stream);
        }))
        return nullptr;
    Py_RETURN_TRUE;
}

// The arguments all selection operators share.
void require_topk(Arguments& a, const Tensor& logits, const Tensor& indices, int64_t rows, int64_t stride0, int64_t stride1, int64_t k) {
    REQUIRE(logits.is_cuda() && logits.dim() == 2 && is(logits, at::kFloat) && indices.dim() == 2);
    if (!a.ok) return;
    REQUIRE(rows == logits.size(0) && stride0 == logits.stride(0) && stride1 == logits.stride(1));
    REQUIRE(is(indices, at::kInt) && indices.is_contiguous() && indices.size(0) >= rows && indices.size(1) == k && on(indices, logits));
}

// logits, next_n, seq_lens, indices, num_rows, stride0, stride1, top_k
PyObject* top_k_decode(Arguments& a) {
    const Tensor *logits = a.tensor(0), *seq = a.tensor(2), *indices = a.tensor(3);
    const int64_t next_n = a.integer(1), rows = a.integer(4), stride0 = a.integer(5), stride1 = a.integer(6), k = a.integer(7);
    if (!a.ok) Py_RETURN_NONE;
    require_topk(a, *logits, *indices, rows, stride0, stride1, k);
    REQUIRE(is(*seq, at::kInt) && seq->dim() == 1 && seq->is_contiguous() && on(*seq, *logits));
    REQUIRE(next_n >= 1 && next_n < (int64_t{1} << 31));
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(seq->size(0) * next_n >= rows);
    if (!a.ok) Py_RETURN_NONE;
    if (rows == 0 || k == 0) Py_RETURN_TRUE;
    if (!launch_on(on_device_of(*logits, OnDevice::kLaunchesOnly), [&](void* stream) {
            return dsv4_top_k_per_row_decode(static_cast<const float*>(logits->data_ptr()), stride0, stride1, next_n,
                                             static_cast<const int32_t*>(seq->data_ptr()), static_cast<int32_t*>(indices->data_ptr()), rows,
                                             logits->size(1), k, stream);
        }))
        return nullptr;
    Py_RETURN_TRUE;
}

// logits, row_starts, row_ends, indices, num_rows, stride0, stride1, top_k
PyObject* top_k_prefill(Arguments& a) {
    const Tensor *logits = a.tensor(0), *starts = a.tensor(1), *ends = a.tensor(2), *indices = a.tensor(3);
    const int64_t rows = a.integer(4), stride0 = a.integer(5), stride1 = a.integer(6), k = a.integer(7);
    if (!a.ok) Py_RETURN_NONE;
    require_topk(a, *logits, *indices, rows, stride0, stride1, k);
    for (const Tensor* t : {starts, ends})
        REQUIRE(is(*t, at::kInt) && t->dim() == 1 && t->is_contiguous() && t->size(0) >= rows && on(*t, *logits));
    if (!a.ok) Py_RETURN_NONE;
    if (rows == 0 || k == 0) Py_RETURN_TRUE;
    if (!launch_on(on_device_of(*logits, OnDevice::kLaunchesOnly), [&](void* stream) {
            return dsv4_top_k_per_row_prefill(static_cast<const float*>(logits->data_ptr()), stride0, stride1,
                                              static_cast<const int32_t*>(starts->data_ptr()), static_cast<const int32_t*>(ends->data_ptr()),
                                              static_cast<int32_t*>(indices->data_ptr()), rows, logits->size(1), k, stream);
        }))
        return nullptr;
    Py_RETURN_TRUE;
}

// logits, lengths, output, k, max_seq_len or None
PyObject* persistent_topk(Arguments& a) {
    const Tensor *logits = a.tensor(0), *lengths = a.tensor(1), *output = a.tensor(2);
    const int64_t k = a.integer(3), longest = a.is_none(4) ? INT64_MAX : a.integer_of(4);
    if (!a.ok) Py_RETURN_NONE;
    REQUIRE(logits->is_cuda() && logits->dim() == 2 && output->dim() == 2 && (lengths->dim() == 1 || lengths->dim() == 2));
    if (!a.ok) Py_RETURN_NONE;
    const int64_t rows = logits->size(0);
    REQUIRE(is(*logits, at::kFloat) && is(*lengths, at::kInt) && is(*output, at::kInt) && lengths->is_contiguous() && output->is_contiguous());
    REQUIRE(lengths->numel() == rows && output->size(0) == rows && output->size(1) == k && (k == 512 || k == 1024 || k == 2048));
    REQUIRE(on(*lengths, *logits) && on(*output, *logits));
    if (!a.ok) Py_RETURN_NONE;
    if (rows == 0) Py_RETURN_TRUE;
    if (!launch_on(on_device_of(*logits, OnDevice::kLaunchesOnly), [&](void* stream) {
            return dsv4_top_k_per_row_prefill(static_cast<const float*>(logits->data_ptr()), logits->stride(0), logits->stride(1), nullptr,
                                              static_cast<const int32_t*>(lengths->data_ptr()), static_cast<int32_t*>(output->data_ptr()), rows,
                                              std::min(logits->size(1), longest), k, stream);
        }))
        return nullptr;
    Py_RETURN_TRUE;
}

PyObject* bind(PyObject*, PyObject* check) {
    Py_XDECREF(g_check);
    g_check = Py_NewRef(check);
    Py_RETURN_NONE;
}

PyObject* refusal(PyObject*, PyObject*) { return PyUnicode_FromString(t_refusal); }

#define DSV4_ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name>)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    DSV4_ENTRY(prologue),
    DSV4_ENTRY(q_kv_rmsnorm),
    DSV4_ENTRY(group_quant),
    DSV4_ENTRY(act_quant),
    DSV4_ENTRY(inv_rope_fp8_quant),
    DSV4_ENTRY(indexer_q_rope_quant),
    DSV4_ENTRY(indexer_k_quant),
    DSV4_ENTRY(cp_gather_indexer),
    DSV4_ENTRY(global_topk),
    DSV4_ENTRY(combine_topk_swa),
    DSV4_ENTRY(dequantize_and_gather),
    DSV4_ENTRY(top_k_decode),
    DSV4_ENTRY(top_k_prefill),
    DSV4_ENTRY(persistent_topk),
    {"bind", bind, METH_O, nullptr},
    {"_refusal", refusal, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
// The build records in the module's docstring which interpreter and torch it is for, and builds anew where they have changed.
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host_calls", DSV4_BUILT_FOR, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_calls() { return PyModule_Create(&kModule); }
