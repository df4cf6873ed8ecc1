// The operator functions of ops.py in native code, for calls in their plain form.
//
// A Python operator function spends 10 - 14 us on checks, output tensors and a ctypes call, several times what a small
// kernel takes.  Each function here does the same for the form in which such calls come - dense CUDA tensors of the
// accepted types on the current device, shapes in order, no tensor subclass or mode that wants to see the call - with the
// same outputs through the same C-ABI call.  Anything else returns None, and ops.py goes on with its own code, which
// copies, switches devices or raises as ever.  So no message is repeated here, but the rules are: a call that this file
// takes must be one that passes all of ops.py's checks, and a check that is added there is added here.
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <initializer_list>
#include <string>
#include <vector>

#include "../../../include/w8a8ffn.h"

namespace {

using at::Tensor;

int dtype_code(const Tensor& t)
{
    switch (t.scalar_type()) {
    case at::kHalf:
        return W8A8_DT_F16;
    case at::kBFloat16:
        return W8A8_DT_BF16;
    case at::kFloat:
        return W8A8_DT_F32;
    case at::kChar:
        return W8A8_DT_I8;
    case at::kInt:
        return W8A8_DT_I32;
    default:
        return -1;
    }
}

bool is_half(const Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }
bool is_float(const Tensor& t) { return is_half(t) || t.scalar_type() == at::kFloat; }

// The tensor arguments of one call.  `ok` turns false at the first one that is not plain.
class Args {
public:
    bool ok = !at::impl::torch_function_mode_enabled() && !c10::impl::TorchDispatchModeTLS::any_modes_set();

    const Tensor* tensor(PyObject* o)
    {
        constexpr c10::DispatchKeySet PLAIN({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA,
                                             c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutocastCUDA});
        if (!ok || !THPVariable_CheckExact(o)) {
            return fail();
        }
        const Tensor& t = THPVariable_Unpack(o);
        if (!t.defined() || (t.key_set() | PLAIN) != PLAIN || !t.is_contiguous() || t.numel() == 0) {
            return fail();
        }
        if (device_ < 0) {
            device_ = t.device().index();
            ok = device_ == c10::cuda::current_device();
        } else {
            ok = t.device().index() == device_;
        }
        return ok ? &t : nullptr;
    }

    // null where the caller gave None
    const Tensor* optional(PyObject* o) { return o == Py_None ? nullptr : tensor(o); }

    bool integer(PyObject* o, int64_t* v)
    {
        if (!PyLong_CheckExact(o)) {
            return ok = false;
        }
        int overflow = 0;
        *v = PyLong_AsLongLongAndOverflow(o, &overflow);
        return ok = ok && overflow == 0;
    }

    bool truth(PyObject* o, bool* v)
    {
        ok = ok && PyBool_Check(o);
        *v = o == Py_True;
        return ok;
    }

    // a cumulative group list: a list or tuple of ints, or an int64 device tensor
    bool group_list(PyObject* o, int64_t experts, int64_t rows, std::vector<int64_t>* host, const int64_t** list, int* on_device)
    {
        if (!ok) {
            return false;
        }
        if (PyList_CheckExact(o) || PyTuple_CheckExact(o)) {
            const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
            if (n != experts) {
                return ok = false;
            }
            host->resize(static_cast<size_t>(n));
            int64_t before = 0;
            for (Py_ssize_t i = 0; i < n; ++i) {
                int64_t v = 0;
                if (!integer(PySequence_Fast_GET_ITEM(o, i), &v) || v < before) {
                    return ok = false;
                }
                (*host)[static_cast<size_t>(i)] = before = v;
            }
            *list = host->data();
            *on_device = 0;
            return ok = before == rows;
        }
        const Tensor* t = tensor(o);
        if (!ok || t->scalar_type() != at::kLong || t->numel() != experts) {
            return ok = false;
        }
        *list = t->const_data_ptr<int64_t>();
        *on_device = 1;
        return true;
    }

    void* stream() const { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device_)).stream(); }

private:
    const Tensor* fail()
    {
        ok = false;
        return nullptr;
    }
    int device_ = -1;
};

const void* ptr(const Tensor* t) { return t != nullptr ? t->const_data_ptr() : nullptr; }
template <typename T>
const T* in(const Tensor* t)
{
    return static_cast<const T*>(ptr(t));
}
template <typename T>
T* out(const Tensor& t)
{
    return static_cast<T*>(t.mutable_data_ptr());
}

Tensor make(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like)
{
    return at::empty(sizes, like.options().dtype(type));
}

Tensor make_bytes(size_t bytes, const Tensor& like)
{
    return make({static_cast<int64_t>(std::max<size_t>(bytes, 1))}, at::kByte, like);
}

// the results as a Python object; none if the library refused the call (ops.py then says why)
PyObject* results(int status, std::initializer_list<Tensor> outs)
{
    if (status != W8A8_OK) {
        Py_RETURN_NONE;
    }
    if (outs.size() == 1) {
        return THPVariable_Wrap(*outs.begin());
    }
    PyObject* tuple = PyTuple_New(static_cast<Py_ssize_t>(outs.size()));
    Py_ssize_t i = 0;
    for (const Tensor& t : outs) {
        PyTuple_SET_ITEM(tuple, i++, THPVariable_Wrap(t));
    }
    return tuple;
}

// (x, round_direct)
PyObject* dynamic_quant(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    bool direct = false;
    const Tensor* x = args.tensor(a[0]);
    if (!args.truth(a[1], &direct) || x->dim() < 2 || !is_half(*x)) {
        Py_RETURN_NONE;
    }
    Tensor y, scale;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        y = at::empty_like(*x, x->options().dtype(at::kChar));
        scale = make(x->sizes().slice(0, x->dim() - 1), at::kFloat, *x);
        const int64_t n = x->size(-1);
        status = w8a8_dynamic_quant(ptr(x), out<int8_t>(y), out<float>(scale), x->numel() / n, n, dtype_code(*x),
                                    direct ? W8A8_F_ROUND_DIRECT : 0, args.stream());
    }
    return results(status, {y, scale});
    END_HANDLE_TH_ERRORS
}

// (x1, x2, gamma, epsilon, round_direct)
PyObject* add_rms_norm_dynamic_quant(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    bool direct = false;
    const Tensor *x1 = args.tensor(a[0]), *x2 = args.tensor(a[1]), *gamma = args.tensor(a[2]);
    if (!args.truth(a[4], &direct) || !PyFloat_CheckExact(a[3]) || x1->dim() < 1 || !x1->sizes().equals(x2->sizes()) ||
        gamma->dim() != 1 || gamma->size(0) != x1->size(-1) || !is_half(*x1) || x1->scalar_type() != x2->scalar_type() ||
        x1->scalar_type() != gamma->scalar_type() || x1->size(-1) > 16384) {
        Py_RETURN_NONE;
    }
    const float epsilon = static_cast<float>(PyFloat_AS_DOUBLE(a[3]));
    Tensor y, x_out, scale;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        y = at::empty_like(*x1, x1->options().dtype(at::kChar));
        x_out = at::empty_like(*x1);
        scale = make(x1->sizes().slice(0, x1->dim() - 1), at::kFloat, *x1);
        const int64_t n = x1->size(-1);
        status = w8a8_add_rms_norm_dynamic_quant(ptr(x1), ptr(x2), ptr(gamma), out<int8_t>(y), out<void>(x_out),
                                                 out<float>(scale), x1->numel() / n, n, epsilon, dtype_code(*x1),
                                                 direct ? W8A8_F_ROUND_DIRECT : 0, args.stream());
    }
    return results(status, {y, x_out, scale});
    END_HANDLE_TH_ERRORS
}

// (x1, x2, scale, offset, pertoken_scale, bias, output_dtype, transpose_x2)
PyObject* quant_matmul(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    bool transpose = false;
    const Tensor *x1 = args.tensor(a[0]), *x2 = args.tensor(a[1]), *scale = args.tensor(a[2]);
    const Tensor *offset = args.optional(a[3]), *pertoken = args.optional(a[4]), *bias = args.optional(a[5]);
    if (!args.truth(a[7], &transpose) || (a[6] != Py_None && !PyUnicode_CheckExact(a[6])) || x1->scalar_type() != at::kChar ||
        x2->scalar_type() != at::kChar || x1->dim() < 2 || x1->dim() != x2->dim()) {
        Py_RETURN_NONE;
    }
    const int64_t m = x1->size(-2), k = x1->size(-1), n = x2->size(transpose ? -2 : -1);
    const bool scale_bf16 = scale->scalar_type() == at::kBFloat16;
    if (k != x2->size(transpose ? -1 : -2) ||
        !x1->sizes().slice(0, x1->dim() - 2).equals(x2->sizes().slice(0, x2->dim() - 2)) ||
        (!scale_bf16 && scale->scalar_type() != at::kFloat) || (scale->numel() != 1 && scale->numel() != n)) {
        Py_RETURN_NONE;
    }
    const int64_t batch = x1->numel() / (m * k);
    int64_t flags = (scale->numel() > 1 ? W8A8_QM_SCALE_PERCHAN : 0) | (scale_bf16 ? W8A8_QM_SCALE_BF16 : 0) |
                    (batch > 1 ? W8A8_QM_PT_MOD_M : 0);
    if (offset != nullptr) {
        if (offset->scalar_type() != at::kFloat || (offset->numel() != 1 && offset->numel() != n)) {
            Py_RETURN_NONE;
        }
        flags |= W8A8_QM_HAS_OFFSET | (offset->numel() > 1 ? W8A8_QM_OFFSET_PERCHAN : 0);
    }
    if (pertoken != nullptr) {
        if (pertoken->scalar_type() != at::kFloat || pertoken->numel() != m) {
            Py_RETURN_NONE;
        }
        flags |= W8A8_QM_HAS_PT;
    }
    int64_t bias_batch_stride = 0;
    if (bias != nullptr) {
        const int code = dtype_code(*bias);
        const int64_t kind = code == W8A8_DT_I32   ? W8A8_QM_BIAS_I32
                             : code == W8A8_DT_F16  ? W8A8_QM_BIAS_F16
                             : code == W8A8_DT_BF16 ? W8A8_QM_BIAS_BF16
                             : code == W8A8_DT_F32  ? W8A8_QM_BIAS_F32
                                                    : W8A8_QM_BIAS_NONE;
        const bool per_batch =
            batch > 1 && bias->dim() == 3 && bias->size(0) == batch && bias->size(1) == 1 && bias->size(2) == n;
        if (kind == W8A8_QM_BIAS_NONE || (!per_batch && bias->numel() != 1 && bias->numel() != n)) {
            Py_RETURN_NONE;
        }
        bias_batch_stride = per_batch ? n : 0;
        flags |= (kind << W8A8_QM_BIAS_SHIFT) | ((per_batch ? n : bias->numel()) > 1 ? W8A8_QM_BIAS_PERCHAN : 0);
    }
    const bool bf16 = a[6] != Py_None && PyUnicode_CompareWithASCIIString(a[6], "bfloat16") == 0;
    Tensor result;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        c10::SmallVector<int64_t, 4> sizes(x1->sizes().begin(), x1->sizes().end());
        sizes.back() = n;
        result = make(sizes, bf16 ? at::kBFloat16 : at::kHalf, *x1);
        status = w8a8_quant_matmul(in<int8_t>(x1), in<int8_t>(x2), ptr(scale), in<float>(offset), in<float>(pertoken),
                                   ptr(bias), out<void>(result), batch, m, n, k, flags, bf16 ? W8A8_DT_BF16 : W8A8_DT_F16,
                                   transpose ? W8A8_W_NK : W8A8_W_KN, bias_batch_stride, args.stream());
    }
    return results(status, {result});
    END_HANDLE_TH_ERRORS
}

// (x, weight, weight_scale, x_scale, group_list, transpose_weight, round_direct)
PyObject* grouped_matmul_swiglu_quant(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    bool transpose = false, direct = false;
    const Tensor *x = args.tensor(a[0]), *w = args.tensor(a[1]), *ws = args.tensor(a[2]), *xs = args.tensor(a[3]);
    if (!args.truth(a[5], &transpose) || !args.truth(a[6], &direct) || x->dim() != 2 || w->dim() != 3 ||
        x->scalar_type() != at::kChar || w->scalar_type() != at::kChar || ws->scalar_type() != at::kFloat ||
        xs->scalar_type() != at::kFloat) {
        Py_RETURN_NONE;
    }
    const int64_t m = x->size(0), k = x->size(1), e = w->size(0), n = w->size(transpose ? 1 : 2);
    std::vector<int64_t> host;
    const int64_t* list = nullptr;
    int on_device = 0;
    if (n % 2 != 0 || w->size(transpose ? 2 : 1) != k || xs->numel() != m || ws->dim() != 2 || ws->size(0) != e ||
        ws->size(1) != n || !args.group_list(a[4], e, m, &host, &list, &on_device)) {
        Py_RETURN_NONE;
    }
    Tensor y, y_scale;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        y = make({m, n / 2}, at::kChar, *x);
        y_scale = make({m}, at::kFloat, *x);
        const size_t need = w8a8_grouped_matmul_swiglu_quant_workspace_size(m, k, n, e);
        const Tensor workspace = make_bytes(need, *x);
        status = w8a8_grouped_matmul_swiglu_quant(in<int8_t>(x), in<int8_t>(w), in<float>(ws), in<float>(xs), out<int8_t>(y),
                                                  out<float>(y_scale), m, k, n, e, list, on_device,
                                                  transpose ? W8A8_W_NK : W8A8_W_KN, direct ? W8A8_F_ROUND_DIRECT : 0,
                                                  out<void>(workspace), need, args.stream());
    }
    return results(status, {y, y_scale});
    END_HANDLE_TH_ERRORS
}

// (x, weight, group_list, bias, transpose_weight, x_scale, weight_scale); the joined result
PyObject* grouped_matmul(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    bool transpose = false;
    const Tensor *x = args.tensor(a[0]), *w = args.tensor(a[1]), *bias = args.optional(a[3]);
    const Tensor *xs = args.optional(a[5]), *ws = args.optional(a[6]);
    if (!args.truth(a[4], &transpose) || x->dim() != 2 || w->dim() != 3 || x->scalar_type() != w->scalar_type()) {
        Py_RETURN_NONE;
    }
    const int64_t m = x->size(0), k = x->size(1), e = w->size(0), n = w->size(transpose ? 1 : 2);
    const bool quantised = x->scalar_type() == at::kChar;
    std::vector<int64_t> host;
    const int64_t* list = nullptr;
    int on_device = 0;
    if ((!quantised && !is_float(*x)) || quantised != (xs != nullptr) || quantised != (ws != nullptr) ||
        (quantised && (xs->scalar_type() != at::kFloat || xs->numel() != m || ws->scalar_type() != at::kFloat ||
                       ws->numel() != e * n)) ||
        w->size(transpose ? 2 : 1) != k || (bias != nullptr && (bias->numel() != e * n || !is_float(*bias))) ||
        !args.group_list(a[2], e, m, &host, &list, &on_device)) {
        Py_RETURN_NONE;
    }
    Tensor y;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        y = make({m, n}, quantised ? at::kBFloat16 : x->scalar_type(), *x);
        const int code = dtype_code(*x);
        const size_t need = code == W8A8_DT_F32 ? w8a8_grouped_matmul_f32_workspace_size(m, n, k, e)
                                                : w8a8_grouped_matmul_workspace_size(m, n, k, e);
        const Tensor workspace = make_bytes(need, *x);
        status = w8a8_grouped_matmul(ptr(x), ptr(w), ptr(bias), out<void>(y), in<float>(xs), in<float>(ws), m, n, k, e, list,
                                     on_device, code, bias != nullptr ? dtype_code(*bias) : code, dtype_code(y),
                                     transpose ? W8A8_W_NK : W8A8_W_KN, out<void>(workspace), need, args.stream());
    }
    return results(status, {y});
    END_HANDLE_TH_ERRORS
}

// (tokens, expert_token_num_per_rank, per_token_scales)
PyObject* moe_re_routing(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    const Tensor *tokens = args.tensor(a[0]), *counts = args.tensor(a[1]), *scales = args.optional(a[2]);
    if (!args.ok || tokens->dim() != 2 || counts->dim() != 2 || (!is_half(*tokens) && tokens->scalar_type() != at::kChar) ||
        (counts->scalar_type() != at::kInt && counts->scalar_type() != at::kLong) ||
        (scales != nullptr && (scales->scalar_type() != at::kFloat || scales->numel() != tokens->size(0)))) {
        Py_RETURN_NONE;
    }
    const int64_t rows = tokens->size(0), h = tokens->size(1), n = counts->size(0), e = counts->size(1);
    Tensor out_tokens, out_scales, out_index, out_counts;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        out_tokens = at::empty_like(*tokens);
        out_scales = make({rows}, at::kFloat, *tokens);
        out_index = make({rows}, at::kInt, *tokens);
        out_counts = make({e}, counts->scalar_type(), *tokens);
        const size_t need = w8a8_moe_re_routing_workspace_size(rows, n, e);
        const Tensor workspace = make_bytes(need, *tokens);
        status = w8a8_moe_re_routing(ptr(tokens), ptr(counts), in<float>(scales), out<void>(out_tokens), out<float>(out_scales),
                                     out<int32_t>(out_index), out<void>(out_counts), rows,
                                     h * static_cast<int64_t>(tokens->element_size()), n, e,
                                     static_cast<int>(counts->element_size()), out<void>(workspace), need, args.stream());
    }
    return results(status, {out_tokens, out_scales, out_index, out_counts});
    END_HANDLE_TH_ERRORS
}

// (rows, src_to_dst, skip1, skip2, bias, scales, expert_for_source_row, drop_pad_mode)
PyObject* moe_finalize_routing(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    int64_t mode = 0;
    const Tensor *rows = args.tensor(a[0]), *index = args.tensor(a[1]), *skip1 = args.optional(a[2]);
    const Tensor *skip2 = args.optional(a[3]), *bias = args.optional(a[4]), *scales = args.optional(a[5]);
    const Tensor* expert = args.optional(a[6]);
    if (!args.integer(a[7], &mode) || !is_float(*rows) || rows->dim() < 2 || index->scalar_type() != at::kInt ||
        (scales != nullptr && (scales->dim() != 2 || !is_float(*scales)))) {
        Py_RETURN_NONE;
    }
    const int64_t h = rows->size(-1), k = scales != nullptr ? scales->size(1) : 1;
    const bool has_bias = bias != nullptr && expert != nullptr;
    const auto other_type = [&](const Tensor* t) { return t != nullptr && t->scalar_type() != rows->scalar_type(); };
    if (index->numel() % k != 0 || other_type(skip1) || other_type(skip2) ||
        (has_bias && (other_type(bias) || bias->dim() != 2 || bias->size(1) != h)) ||
        (expert != nullptr && expert->scalar_type() != at::kInt)) {
        Py_RETURN_NONE;
    }
    const int64_t num_rows = index->numel() / k;
    const auto too_few = [](const Tensor* t, int64_t elements) { return t != nullptr && t->numel() < elements; };
    if (too_few(skip1, num_rows * h) || too_few(skip2, num_rows * h) || too_few(scales, index->numel()) ||
        (has_bias && too_few(expert, index->numel()))) {
        Py_RETURN_NONE;
    }
    Tensor result;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        result = make({num_rows, h}, rows->scalar_type(), *rows);
        status = w8a8_moe_finalize_routing(ptr(rows), in<int32_t>(index), ptr(skip1), ptr(skip2),
                                           has_bias ? ptr(bias) : nullptr, ptr(scales),
                                           has_bias ? in<int32_t>(expert) : nullptr, out<void>(result), num_rows, h, k,
                                           has_bias ? bias->size(0) : 0, rows->numel() / h,
                                           static_cast<int>(std::clamp<int64_t>(mode, 0, 3)), dtype_code(*rows),
                                           dtype_code(scales != nullptr ? *scales : *rows), args.stream());
    }
    return results(status, {result});
    END_HANDLE_TH_ERRORS
}

// (x, finished, k)
PyObject* moe_gating_top_k_softmax(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    int64_t k = 0;
    const Tensor *x = args.tensor(a[0]), *finished = args.optional(a[1]);
    if (!args.integer(a[2], &k) || !is_float(*x) || x->dim() < 2 || k <= 0 || k > x->size(-1)) {
        Py_RETURN_NONE;
    }
    const int64_t inner = x->size(-1), rows = x->numel() / inner;
    if (finished != nullptr && (finished->scalar_type() != at::kBool || finished->numel() != rows)) {
        Py_RETURN_NONE;
    }
    Tensor y, expert_idx, row_idx;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        c10::SmallVector<int64_t, 4> sizes(x->sizes().begin(), x->sizes().end());
        sizes.back() = k;
        y = make(sizes, x->scalar_type(), *x);
        expert_idx = make(sizes, at::kInt, *x);
        row_idx = make(sizes, at::kInt, *x);
        status = w8a8_moe_gating_top_k_softmax(ptr(x), in<uint8_t>(finished), out<void>(y), out<int32_t>(expert_idx),
                                               out<int32_t>(row_idx), rows, inner, k, dtype_code(*x), args.stream());
    }
    return results(status, {y, expert_idx, row_idx});
    END_HANDLE_TH_ERRORS
}

// (x, weight_scale, activation_scale, quant_scale, activate_left, round_direct)
PyObject* dequant_swiglu_quant(PyObject*, PyObject* const* a, Py_ssize_t)
{
    HANDLE_TH_ERRORS
    Args args;
    bool left = false, direct = false;
    const Tensor *x = args.tensor(a[0]), *ws = args.optional(a[1]), *as = args.optional(a[2]), *qs = args.optional(a[3]);
    if (!args.truth(a[4], &left) || !args.truth(a[5], &direct) || x->dim() != 2 || x->size(1) % 2 != 0) {
        Py_RETURN_NONE;
    }
    const int64_t m = x->size(0), n2 = x->size(1), h = n2 / 2;
    const bool i32 = x->scalar_type() == at::kInt;
    const auto floats = [](const Tensor* t, int64_t count) { return t->scalar_type() == at::kFloat && t->numel() == count; };
    if ((!i32 && !is_half(*x)) || i32 != (ws != nullptr) || i32 != (as != nullptr) ||
        (i32 && (!floats(ws, n2) || !floats(as, m))) || (qs != nullptr && !floats(qs, h))) {
        Py_RETURN_NONE;
    }
    Tensor y, scale;
    int status;
    {
        pybind11::gil_scoped_release no_gil;
        y = make({m, h}, at::kChar, *x);
        scale = make({m}, at::kFloat, *x);
        status = w8a8_dequant_swiglu_quant(ptr(x), in<float>(ws), in<float>(as), in<float>(qs), out<int8_t>(y),
                                           out<float>(scale), m, h, dtype_code(*x), left ? 1 : 0,
                                           direct ? W8A8_F_ROUND_DIRECT : 0, args.stream());
    }
    return results(status, {y, scale});
    END_HANDLE_TH_ERRORS
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t), Py_ssize_t COUNT>
PyObject* counted(PyObject* self, PyObject* const* a, Py_ssize_t n)
{
    if (n != COUNT) {
        PyErr_Format(PyExc_TypeError, "%zd arguments expected, %zd given", COUNT, n);
        return nullptr;
    }
    return F(self, a, n);
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t), Py_ssize_t COUNT>
PyMethodDef method(const char* name)
{
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&counted<F, COUNT>)), METH_FASTCALL, nullptr};
}

}  // namespace

PyMODINIT_FUNC PyInit__calls()
{
    static PyMethodDef methods[] = {
        method<dynamic_quant, 2>("dynamic_quant"),
        method<add_rms_norm_dynamic_quant, 5>("add_rms_norm_dynamic_quant"),
        method<quant_matmul, 8>("quant_matmul"),
        method<grouped_matmul_swiglu_quant, 7>("grouped_matmul_swiglu_quant"),
        method<grouped_matmul, 7>("grouped_matmul"),
        method<moe_re_routing, 3>("moe_re_routing"),
        method<moe_finalize_routing, 8>("moe_finalize_routing"),
        method<moe_gating_top_k_softmax, 3>("moe_gating_top_k_softmax"),
        method<dequant_swiglu_quant, 6>("dequant_swiglu_quant"),
        {nullptr, nullptr, 0, nullptr},
    };
    static PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
    return PyModule_Create(&module);
}
