// Host side of the operator calls.  Each function takes the plain form of a call (contiguous CUDA tensors of one type on
// one device), allocates its results and enqueues the kernels, and returns None when the call is of any other form or the
// library rejects it: the Python operator then takes its general path, which also words the errors.  A small operator's
// time is its host time: in Python with ctypes a norm of 8192 x 128 took 25 us for a 3 us kernel.
#include <Python.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <limits>

#include "module.h"
#include "native.h"

namespace tb200_host {
namespace {

using torch::autograd::AutogradContext;
using torch::autograd::tensor_list;

// -------------------------------------------------------------------------------------------- arguments
bool is_tensor(PyObject* o) { return THPVariable_Check(o); }
const Tensor& tensor(PyObject* o) { return THPVariable_Unpack(o); }
std::optional<Tensor> optional_tensor(PyObject* o) {
    return o == Py_None ? std::nullopt : std::optional<Tensor>(THPVariable_Unpack(o));
}
double number(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
}
int64_t integer(PyObject* o) {   // as int(o) takes it
    if (PyFloat_Check(o)) {
        const double v = PyFloat_AS_DOUBLE(o);
        TORCH_CHECK_VALUE(std::fabs(v) < 9.2e18, "cannot convert ", v, " to an integer");
        return static_cast<int64_t>(v);
    }
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
bool truth(PyObject* o) {   // as `if o:` takes it
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw python_error();
    return v != 0;
}
// a tensor or None?
bool is_optional(PyObject* o) { return o == Py_None || THPVariable_Check(o); }

bool same_device(const Tensor& a, const std::optional<Tensor>& b) { return !b.has_value() || b->device() == a.device(); }

// -------------------------------------------------------------------------------------------- norms
bool norm_backward_supported(const Tensor& x) {
    const int64_t per16 = 16 / static_cast<int64_t>(x.element_size());
    return x.size(-1) % per16 == 0 && x.size(-1) / per16 <= 128;
}

int norm_forward(const Tensor& x, const Tensor& w, const Tensor* b, bool pre_silu, double eps, const Tensor& y) {
    const int64_t cols = x.size(-1), rows = cols > 0 ? x.numel() / cols : 0;
    const int dt = dtype_code(x.scalar_type());
    if (cols > INT32_MAX) return TB200_ERR_SHAPE;
    const auto c = static_cast<int32_t>(cols);
    const auto e = static_cast<float>(eps);
    void* s = stream_of(x);
    if (b == nullptr) return tb200_rmsnorm_fwd(ptr(x), ptr(w), ptr(y), rows, c, e, dt, s);
    return pre_silu ? tb200_layernorm_silu_fwd(ptr(x), ptr(w), ptr(*b), ptr(y), rows, c, e, dt, s)
                    : tb200_layernorm_fwd(ptr(x), ptr(w), ptr(*b), ptr(y), rows, c, e, dt, s);
}

tensor_list norm_backward(const Tensor& x, const Tensor& w, bool layer, double eps, const Tensor& grad) {
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t cols = x.size(-1), rows = x.numel() / cols;
    const Tensor dy = grad.to(x.scalar_type()).contiguous();
    Tensor dx = at::empty_like(x), dw = at::empty_like(w), db = layer ? at::empty_like(w) : Tensor();
    const auto c = static_cast<int32_t>(cols);
    Tensor work = at::empty({tb200_norm_bwd_workspace_bytes(c, layer ? 1 : 0) / 4}, x.options().dtype(at::kFloat));
    const int dt = dtype_code(x.scalar_type());
    auto* ws = static_cast<float*>(ptr(work));
    if (layer)
        check(tb200_layernorm_bwd(ptr(x), ptr(w), ptr(dy), ptr(dx), ptr(dw), ptr(db), ws, rows, c, static_cast<float>(eps), dt, stream_of(x)),
              "cuda layer_norm backward");
    else
        check(tb200_rmsnorm_bwd(ptr(x), ptr(w), ptr(dy), ptr(dx), ptr(dw), ws, rows, c, static_cast<float>(eps), dt, stream_of(x)),
              "cuda rms_norm backward");
    return {dx, dw, db};
}

struct RmsNormFunction : torch::autograd::Function<RmsNormFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
        ctx->save_for_backward({x, w});
        ctx->saved_data["eps"] = eps;
        Tensor y = at::empty_like(x);
        check(norm_forward(x, w, nullptr, false, eps, y), "cuda rms_norm");
        return y;
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
        const auto saved = ctx->get_saved_variables();
        auto g = norm_backward(saved[0], saved[1], false, ctx->saved_data["eps"].toDouble(), grads[0]);
        return {g[0], g[1], Tensor()};
    }
};

struct LayerNormFunction : torch::autograd::Function<LayerNormFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
        ctx->save_for_backward({x, w});
        ctx->saved_data["eps"] = eps;
        Tensor y = at::empty_like(x);
        check(norm_forward(x, w, &b, false, eps, y), "cuda layer_norm");
        return y;
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
        const auto saved = ctx->get_saved_variables();
        auto g = norm_backward(saved[0], saved[1], true, ctx->saved_data["eps"].toDouble(), grads[0]);
        return {g[0], g[1], g[2], Tensor()};
    }
};

// rms_norm(x, weight, eps)
PyObject* py_rms_norm(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    if (!is_tensor(args[0]) || !is_tensor(args[1])) Py_RETURN_NONE;
    const Tensor& x = tensor(args[0]);
    const Tensor& w = tensor(args[1]);
    const double eps = number(args[2]);
    if (x.dim() < 2 || w.dim() != 1 || x.size(-1) != w.size(0) || x.size(-1) < 1 || dtype_code(x.scalar_type()) < 0 || !dense(x, x.scalar_type()) ||
        !dense(w, x.scalar_type()) || x.device() != w.device())
        Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard(x.device());
    if (!tb200_device_ok()) Py_RETURN_NONE;
    if (wants_grad(x) || wants_grad(w)) {
        if (!norm_backward_supported(x)) Py_RETURN_NONE;
        return THPVariable_Wrap(RmsNormFunction::apply(x, w, eps));
    }
    Tensor y = at::empty_like(x);
    if (norm_forward(x, w, nullptr, false, eps, y) != TB200_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// layer_norm(x, weight, bias, eps, pre_silu)
PyObject* py_layer_norm(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    if (!is_tensor(args[0]) || !is_tensor(args[1]) || !is_tensor(args[2])) Py_RETURN_NONE;
    const Tensor& x = tensor(args[0]);
    const Tensor& w = tensor(args[1]);
    const Tensor& b = tensor(args[2]);
    const double eps = number(args[3]);
    const bool pre_silu = truth(args[4]);
    if (x.dim() < 2 || w.dim() != 1 || b.dim() != 1 || x.size(-1) != w.size(0) || x.size(-1) != b.size(0) || x.size(-1) < 1 ||
        dtype_code(x.scalar_type()) < 0 || !dense(x, x.scalar_type()) || !dense(w, x.scalar_type()) || !dense(b, x.scalar_type()) ||
        x.device() != w.device() || x.device() != b.device())
        Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard(x.device());
    if (!tb200_device_ok()) Py_RETURN_NONE;
    if (wants_grad(x) || wants_grad(w) || wants_grad(b)) {
        if (pre_silu || !norm_backward_supported(x)) Py_RETURN_NONE;
        return THPVariable_Wrap(LayerNormFunction::apply(x, w, b, eps));
    }
    Tensor y = at::empty_like(x);
    if (norm_forward(x, w, &b, pre_silu, eps, y) != TB200_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// -------------------------------------------------------------------------------------------- embedding bags
// embedding_bag_mean(weight, ids)
PyObject* py_embedding_bag_mean(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    if (!is_tensor(args[0]) || !is_tensor(args[1])) Py_RETURN_NONE;
    const Tensor& w = tensor(args[0]);
    const Tensor& ids = tensor(args[1]);
    const int dt = dtype_code(w.scalar_type()), it = id_code(ids.scalar_type());
    if (w.dim() != 2 || ids.dim() != 2 || dt < 0 || it < 0 || !dense(w, w.scalar_type()) || !dense(ids, ids.scalar_type()) ||
        w.device() != ids.device() || w.size(1) > INT32_MAX || ids.size(1) > INT32_MAX)
        Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard(w.device());
    if (!tb200_device_ok()) Py_RETURN_NONE;
    Tensor out = at::empty({ids.size(0), w.size(1)}, w.options().requires_grad(false));
    if (tb200_bag_mean_fwd(ptr(w), w.size(0), static_cast<int32_t>(w.size(1)), ptr(ids), it, ids.size(0), static_cast<int32_t>(ids.size(1)),
                           ptr(out), dt, stream_of(w)) != TB200_OK)
        Py_RETURN_NONE;
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// embedding_bag_mean_backward(ids, grad_out, num_embeddings) -> sparse COO gradient
PyObject* py_embedding_bag_mean_backward(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    if (!is_tensor(args[0]) || !is_tensor(args[1])) Py_RETURN_NONE;
    const Tensor& ids = tensor(args[0]);
    const Tensor& grad = tensor(args[1]);
    const int64_t rows = integer(args[2]);
    const int dt = dtype_code(grad.scalar_type()), it = id_code(ids.scalar_type());
    if (ids.dim() != 2 || grad.dim() != 2 || ids.size(0) != grad.size(0) || dt < 0 || it < 0 || !dense(ids, ids.scalar_type()) ||
        !dense(grad, grad.scalar_type()) || ids.device() != grad.device() || grad.size(1) > INT32_MAX || ids.size(1) > INT32_MAX)
        Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard(grad.device());
    if (!tb200_device_ok()) Py_RETURN_NONE;
    const int64_t n = ids.size(0) * ids.size(1);
    Tensor index = at::empty({1, n}, grad.options().dtype(at::kLong).requires_grad(false));
    Tensor values = at::empty({n, grad.size(1)}, grad.options().requires_grad(false));
    if (tb200_bag_mean_bwd(ptr(ids), it, ptr(grad), static_cast<int64_t*>(ptr(index)), ptr(values), ids.size(0),
                           static_cast<int32_t>(ids.size(1)), static_cast<int32_t>(grad.size(1)), rows, dt, stream_of(grad)) != TB200_OK)
        Py_RETURN_NONE;
    // the kernel writes rows inside the table by construction, so nothing is checked again
    return THPVariable_Wrap(at::_sparse_coo_tensor_unsafe(index, values, {rows, grad.size(1)}, values.options().layout(at::kSparse), false));
    END_HANDLE_TH_ERRORS
}

// -------------------------------------------------------------------------------------------- attention
bool rows_aligned(const Tensor& t) {
    if (t.stride(-1) != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) return false;
    const int64_t per16 = 16 / static_cast<int64_t>(t.element_size());
    for (int64_t d = 0; d + 1 < t.dim(); ++d)
        if (t.stride(d) % per16 != 0) return false;
    return true;
}
Tensor aligned_rows(const Tensor& t) { return rows_aligned(t) ? t : t.contiguous(); }

struct Mask {
    std::optional<Tensor> lens;   // int32 [B]
    int64_t ns_start = 0;
    bool causal = false;
    bool self_rows = false;
};

// (B, H, L, D) tensors, or (B, L, H, D) with `token_major`; the result has q's shape.  Undefined when the library rejects it.
Tensor attention_forward(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Mask& mask, double scale, bool token_major, int kernel,
                         const std::optional<Tensor>& status) {
    const Tensor q = aligned_rows(q_in), k = aligned_rows(k_in), v = aligned_rows(v_in);
    Tensor out = at::empty(q.sizes(), q.options().requires_grad(false));
    const int hd = token_major ? 2 : 1, ld = token_major ? 1 : 2;
    int64_t strides[12];
    int i = 0;
    for (const Tensor* t : {&q, &k, &v, static_cast<const Tensor*>(&out)}) {
        strides[i++] = t->stride(0);
        strides[i++] = t->stride(hd);
        strides[i++] = t->stride(ld);
    }
    const int64_t lk = k.size(ld);
    const int code = tb200_attn_fwd(ptr(q), ptr(k), ptr(v), ptr(out), static_cast<int32_t>(q.size(0)), static_cast<int32_t>(q.size(hd)),
                                    static_cast<int32_t>(q.size(ld)), static_cast<int32_t>(lk), static_cast<int32_t>(q.size(3)), strides,
                                    static_cast<int32_t*>(ptr(mask.lens)), nullptr, nullptr, nullptr, static_cast<int32_t>(mask.ns_start),
                                    mask.causal, mask.self_rows, static_cast<float>(scale), dtype_code(q.scalar_type()), kernel, 0,
                                    static_cast<int32_t*>(ptr(status)), stream_of(q));
    return code == TB200_OK ? out : Tensor();
}

tensor_list attention_backward(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& out_in, const Tensor& grad_in,
                               const Mask& mask, double scale) {
    const c10::cuda::CUDAGuard guard(q_in.device());
    const Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous(), out = out_in.contiguous();
    const Tensor grad = grad_in.to(q.scalar_type()).contiguous();
    Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
    const auto b = static_cast<int32_t>(q.size(0)), h = static_cast<int32_t>(q.size(1)), lq = static_cast<int32_t>(q.size(2)),
               lk = static_cast<int32_t>(k.size(2));
    Tensor work = at::empty({std::max<int64_t>(tb200_attn_bwd_workspace_bytes(b, h, lq) / 4, 1)}, q.options().dtype(at::kFloat));
    int64_t strides[12];
    int i = 0;
    for (const Tensor* t : {&q, &k, &v, &out})
        for (int d = 0; d < 3; ++d) strides[i++] = t->stride(d);
    check(tb200_attn_bwd(ptr(q), ptr(k), ptr(v), ptr(out), ptr(grad), ptr(dq), ptr(dk), ptr(dv), ptr(work), b, h, lq, lk,
                         static_cast<int32_t>(q.size(3)), strides, static_cast<int32_t*>(ptr(mask.lens)), nullptr,
                         static_cast<int32_t>(mask.ns_start), mask.causal, mask.self_rows, static_cast<float>(scale),
                         dtype_code(q.scalar_type()), stream_of(q)),
          "cuda attention_backward");
    return {dq, dk, dv};
}

struct AttentionFunction : torch::autograd::Function<AttentionFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& lens,
                          int64_t ns_start, bool causal, bool self_rows, double scale) {
        Mask mask{lens, ns_start, causal, self_rows};
        Tensor out = attention_forward(q, k, v, mask, scale, false, 0, std::nullopt);
        TORCH_CHECK(out.defined(), "cuda flash_attention: no kernel for this call");
        ctx->save_for_backward({q, k, v, out, lens.value_or(Tensor())});
        ctx->saved_data["ns_start"] = ns_start;
        ctx->saved_data["causal"] = causal;
        ctx->saved_data["self_rows"] = self_rows;
        ctx->saved_data["scale"] = scale;
        return out;
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
        const auto s = ctx->get_saved_variables();
        Mask mask{s[4].defined() ? std::optional<Tensor>(s[4]) : std::nullopt, ctx->saved_data["ns_start"].toInt(),
                  ctx->saved_data["causal"].toBool(), ctx->saved_data["self_rows"].toBool()};
        auto g = attention_backward(s[0], s[1], s[2], s[3], grads[0], mask, ctx->saved_data["scale"].toDouble());
        return {g[0], g[1], g[2], Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

bool attention_operands(const Tensor& q, const Tensor& k, const Tensor& v) {
    if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || !q.is_cuda() || k.device() != q.device() || v.device() != q.device()) return false;
    const auto t = q.scalar_type();
    if ((t != at::kBFloat16 && t != at::kHalf) || k.scalar_type() != t || v.scalar_type() != t) return false;
    const int64_t d = q.size(3);
    return (d == 32 || d == 64 || d == 128) && k.sizes() == v.sizes() && k.size(3) == d && q.size(0) == k.size(0) && q.numel() > 0 && k.numel() > 0;
}

// varlen_attention(q, k, v, seq_len or None, ns_start or None, causal, padded_query_self, scale or None, token_major, kernel, status or None)
PyObject* py_varlen_attention(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    if (!is_tensor(args[0]) || !is_tensor(args[1]) || !is_tensor(args[2]) || !is_optional(args[3]) || !is_optional(args[10])) Py_RETURN_NONE;
    const Tensor& q = tensor(args[0]);
    const Tensor& k = tensor(args[1]);
    const Tensor& v = tensor(args[2]);
    const bool token_major = truth(args[8]);
    const int hd = token_major ? 2 : 1, ld = token_major ? 1 : 2;
    if (!attention_operands(q, k, v) || q.size(hd) != k.size(hd)) Py_RETURN_NONE;
    Mask mask;
    mask.lens = optional_tensor(args[3]);
    const auto status = optional_tensor(args[10]);
    if (!same_device(q, mask.lens) || !same_device(q, status)) Py_RETURN_NONE;
    if (mask.lens.has_value() && !dense(*mask.lens, at::kInt)) {
        if (mask.lens->dim() != 1) Py_RETURN_NONE;
        mask.lens = mask.lens->to(at::kInt).contiguous();
    }
    if (status.has_value() && (status->scalar_type() != at::kInt || status->numel() != 1)) Py_RETURN_NONE;
    mask.ns_start = args[4] == Py_None ? k.size(ld) : integer(args[4]);
    mask.causal = truth(args[5]);
    mask.self_rows = truth(args[6]);
    const double scale = args[7] == Py_None ? 1.0 / std::sqrt(static_cast<double>(q.size(3))) : number(args[7]);
    const int kernel = static_cast<int>(integer(args[9]));
    const c10::cuda::CUDAGuard guard(q.device());
    if (!tb200_device_ok()) Py_RETURN_NONE;
    Tensor out = attention_forward(q, k, v, mask, scale, token_major, kernel, status);
    if (!out.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// Describes a bool mask [B, H, Lq, Lk] by lengths (see mask_plan.cu).  One pass over the mask on the device and one
// synchronisation; false: not one of the recognised forms.
bool plan_mask(const Tensor& m, bool is_causal, Mask& mask) {
    const int64_t b = m.size(0), h = m.size(1), lq = m.size(2), lk = m.size(3);
    if (m.stride(3) != 1 || b > INT32_MAX || lq > INT32_MAX || lk > INT32_MAX) return false;
    Tensor lens = at::empty({b}, m.options().dtype(at::kInt));
    Tensor verdict = at::empty({b, 4}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    const auto stream = c10::cuda::getCurrentCUDAStream(m.device().index());
    if (tb200_mask_plan(static_cast<const uint8_t*>(ptr(m)), m.stride(0), m.stride(1), m.stride(2), static_cast<int32_t>(b),
                        static_cast<int32_t>(h), static_cast<int32_t>(lq), static_cast<int32_t>(lk), static_cast<int32_t*>(ptr(lens)),
                        static_cast<int32_t*>(ptr(verdict)), stream.stream()) != TB200_OK)
        return false;
    Py_BEGIN_ALLOW_THREADS
    stream.synchronize();
    Py_END_ALLOW_THREADS
    const int32_t* w = verdict.data_ptr<int32_t>();
    const int form = w[0];
    if (form == 0) return false;
    int suffix = -1;
    bool any_identity = false;
    for (int64_t i = 0; i < b; ++i, w += 4) {
        if (w[0] != form) return false;
        if (w[3] == 1) {   // a sample with padding tells how long the always-valid suffix is; they have to agree
            if (suffix >= 0 && w[2] != suffix) return false;
            suffix = w[2];
        }
        any_identity |= w[3] == 2;
    }
    if (suffix < 0) suffix = 0;
    if (any_identity && suffix > 1) return false;
    mask.lens = lens;
    mask.ns_start = lk - suffix;
    mask.causal = form == 2 || is_causal;
    mask.self_rows = form == 2;
    return true;
}

// flash_attention(q, k, v, attn_mask or None, is_causal): evaluation or training without dropout
PyObject* py_flash_attention(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    if (!is_tensor(args[0]) || !is_tensor(args[1]) || !is_tensor(args[2]) || !is_optional(args[3])) Py_RETURN_NONE;
    const Tensor& q = tensor(args[0]);
    const Tensor& k = tensor(args[1]);
    const Tensor& v = tensor(args[2]);
    if (!attention_operands(q, k, v) || q.size(1) != k.size(1)) Py_RETURN_NONE;
    const auto attn_mask = optional_tensor(args[3]);
    const bool is_causal = truth(args[4]);
    const bool grad = wants_grad(q) || wants_grad(k) || wants_grad(v);
    if (grad && (q.size(2) > 4096 || k.size(2) > 4096 || q.size(1) > 65535)) Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard(q.device());
    if (!tb200_device_ok()) Py_RETURN_NONE;
    Mask mask{std::nullopt, k.size(2), is_causal, false};
    if (attn_mask.has_value()) {
        const Tensor& m = *attn_mask;
        if (m.scalar_type() != at::kBool || m.dim() != 4 || m.device() != q.device() || m.size(0) != q.size(0) || m.size(1) != q.size(1) ||
            m.size(2) != q.size(2) || m.size(3) != k.size(2))
            Py_RETURN_NONE;
        if (!plan_mask(m, is_causal, mask)) Py_RETURN_NONE;
    }
    const double scale = 1.0 / std::sqrt(static_cast<double>(q.size(3)));
    if (grad)
        return THPVariable_Wrap(AttentionFunction::apply(q, k, v, mask.lens, mask.ns_start, mask.causal, mask.self_rows, scale));
    Tensor out = attention_forward(q, k, v, mask, scale, false, 0, std::nullopt);
    if (!out.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// -------------------------------------------------------------------------------------------- FFN
struct FfnOperands {
    Tensor x;                     // [M, d] bf16
    Tensor w_up, s_up, w_down, s_down;
    std::optional<Tensor> b_up, b_down, residual, status;
    int64_t hidden = 0, d_out = 0;
    bool gated = false;
};

// (x, w_up, s_up, b_up or None, w_down, s_down, b_down or None, hidden, gated, residual or None, status or None)
bool ffn_operands(PyObject* const* args, at::ScalarType up_type, FfnOperands& f) {
    for (int i : {0, 1, 2, 4, 5})
        if (!is_tensor(args[i])) return false;
    for (int i : {3, 6, 9, 10})
        if (!is_optional(args[i])) return false;
    const Tensor& x = tensor(args[0]);
    f.w_up = tensor(args[1]);
    f.s_up = tensor(args[2]);
    f.b_up = optional_tensor(args[3]);
    f.w_down = tensor(args[4]);
    f.s_down = tensor(args[5]);
    f.b_down = optional_tensor(args[6]);
    f.hidden = integer(args[7]);
    f.gated = truth(args[8]);
    f.residual = optional_tensor(args[9]);
    f.status = optional_tensor(args[10]);
    if (x.dim() < 1 || !dense(x, at::kBFloat16) || x.size(-1) < 1 || x.numel() == 0) return false;
    const int64_t d = x.size(-1), m = x.numel() / d;
    if (!dense(f.w_up, up_type) || !dense(f.w_down, at::kFloat8_e4m3fn) || f.w_up.dim() != 2 || f.w_down.dim() != 2 || f.w_up.size(1) != d ||
        f.w_up.size(0) != f.hidden * (f.gated ? 2 : 1) || f.w_down.size(1) != f.hidden || m > INT32_MAX)
        return false;
    f.d_out = f.w_down.size(0);
    for (const auto* t : {&f.b_up, &f.b_down})
        if (t->has_value() && !dense(**t, at::kFloat)) return false;
    if (f.residual.has_value() && (!dense(*f.residual, at::kBFloat16) || f.residual->numel() != m * f.d_out)) return false;
    if (f.status.has_value() && (f.status->scalar_type() != at::kInt || f.status->numel() != 1)) return false;
    for (const auto* t : {&f.b_up, &f.b_down, &f.residual, &f.status})
        if (!same_device(x, *t)) return false;
    for (const Tensor* t : {&f.w_up, &f.s_up, &f.w_down, &f.s_down})
        if (t->device() != x.device()) return false;
    if (d % 128 != 0 || f.hidden % 256 != 0 || f.d_out % 256 != 0) return false;
    f.x = x;
    return true;
}

// the scales of an [n, k] weight: one per 128 x 128 block, `atom` > 0: an atom of so many bytes each
bool scales_fit(const Tensor& s, const Tensor& w, int64_t atom) {
    return s.dim() == (atom > 0 ? 3 : 2) && s.size(0) == w.size(0) / 128 && s.size(1) == w.size(1) / 128 && (atom == 0 || s.size(2) == atom);
}

Tensor ffn_result(const FfnOperands& f) {
    auto sizes = f.x.sizes().vec();
    sizes.back() = f.d_out;
    return at::empty(sizes, f.x.options().requires_grad(false));
}

// ffn_fp8(...): quantise, GEMM 1 with (gated) SiLU and re-quantisation, GEMM 2.  With a bf16 up projection (`precise`) GEMM 1
// runs on the bf16 tensor cores and its result is quantised.
PyObject* ffn_fp8(PyObject* const* args, bool precise) {
    FfnOperands f;
    if (!ffn_operands(args, precise ? at::kBFloat16 : at::kFloat8_e4m3fn, f)) Py_RETURN_NONE;
    if (!dense(f.s_down, at::kFloat) || !scales_fit(f.s_down, f.w_down, 0)) Py_RETURN_NONE;
    if (!precise && (!dense(f.s_up, at::kFloat) || !scales_fit(f.s_up, f.w_up, 0))) Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard(f.x.device());
    if (!tb200_device_ok()) Py_RETURN_NONE;
    const int64_t d = f.x.size(-1), m = f.x.numel() / d;
    const auto n_up = static_cast<int32_t>(f.w_up.size(0)), hid = static_cast<int32_t>(f.hidden);
    const auto fp8 = f.x.options().dtype(at::kFloat8_e4m3fn).requires_grad(false);
    const auto f32 = f.x.options().dtype(at::kFloat).requires_grad(false);
    void* s = stream_of(f.x);
    auto* status = static_cast<int32_t*>(ptr(f.status));
    Tensor h = at::empty({m, f.hidden}, fp8), sh = at::empty({m, f.hidden / 128}, f32), out = ffn_result(f);
    int code;
    if (precise) {
        Tensor hb = at::empty({m, f.hidden}, f.x.options().requires_grad(false));
        code = tb200_gemm_bf16_grouped(ptr(f.x), ptr(f.w_up), static_cast<float*>(ptr(f.b_up)), nullptr, ptr(hb), 1, m, n_up,
                                       static_cast<int32_t>(d), f.gated ? 2 : 1, status, s);
        if (code == TB200_OK) code = tb200_quant_act_1x128(ptr(hb), ptr(h), static_cast<float*>(ptr(sh)), m, hid, s);
    } else {
        Tensor xq = at::empty({m, d}, fp8), sx = at::empty({m, d / 128}, f32);
        code = tb200_quant_act_1x128(ptr(f.x), ptr(xq), static_cast<float*>(ptr(sx)), m, static_cast<int32_t>(d), s);
        if (code == TB200_OK)
            code = tb200_fp8_gemm(ptr(xq), static_cast<float*>(ptr(sx)), ptr(f.w_up), static_cast<float*>(ptr(f.s_up)),
                                  static_cast<float*>(ptr(f.b_up)), nullptr, ptr(h), static_cast<float*>(ptr(sh)), m, n_up,
                                  static_cast<int32_t>(d), f.gated ? 0 : 1, status, s);
    }
    if (code == TB200_OK)
        code = tb200_fp8_gemm(ptr(h), static_cast<float*>(ptr(sh)), ptr(f.w_down), static_cast<float*>(ptr(f.s_down)),
                              static_cast<float*>(ptr(f.b_down)), ptr(f.residual), ptr(out), nullptr, m, static_cast<int32_t>(f.d_out), hid, 2,
                              status, s);
    if (code != TB200_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(out);
}
PyObject* py_ffn_fp8(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    return ffn_fp8(args, false);
    END_HANDLE_TH_ERRORS
}
PyObject* py_ffn_fp8_precise(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    return ffn_fp8(args, true);
    END_HANDLE_TH_ERRORS
}

// ffn_mx(...): the same with power-of-two block scales; the scale operands are uint8 atoms
PyObject* py_ffn_mx(PyObject*, PyObject* const* args, Py_ssize_t) {
    HANDLE_TH_ERRORS
    FfnOperands f;
    if (!ffn_operands(args, at::kFloat8_e4m3fn, f) || !dense(f.s_up, at::kByte) || !dense(f.s_down, at::kByte) ||
        !scales_fit(f.s_up, f.w_up, 512) || !scales_fit(f.s_down, f.w_down, 512))
        Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard(f.x.device());
    if (!tb200_device_ok()) Py_RETURN_NONE;
    const int64_t d = f.x.size(-1), m = f.x.numel() / d, tiles = (m + 127) / 128;
    const auto fp8 = f.x.options().dtype(at::kFloat8_e4m3fn).requires_grad(false);
    const auto bytes = f.x.options().dtype(at::kByte).requires_grad(false);
    // the scale atoms of a ragged last tile hold zeros for the rows behind the end
    auto atoms = [&](int64_t k) { return m % 128 == 0 ? at::empty({tiles, k / 128, 512}, bytes) : at::zeros({tiles, k / 128, 512}, bytes); };
    void* s = stream_of(f.x);
    auto* status = static_cast<int32_t*>(ptr(f.status));
    Tensor xq = at::empty({m, d}, fp8), xa = atoms(d), h = at::empty({m, f.hidden}, fp8), ha = atoms(f.hidden), out = ffn_result(f);
    int code = tb200_quant_act_mx(ptr(f.x), ptr(xq), static_cast<uint8_t*>(ptr(xa)), m, static_cast<int32_t>(d), s);
    if (code == TB200_OK)
        code = tb200_mx_gemm(ptr(xq), static_cast<uint8_t*>(ptr(xa)), ptr(f.w_up), static_cast<uint8_t*>(ptr(f.s_up)),
                             static_cast<float*>(ptr(f.b_up)), nullptr, ptr(h), static_cast<uint8_t*>(ptr(ha)), m,
                             static_cast<int32_t>(f.w_up.size(0)), static_cast<int32_t>(d), f.gated ? 0 : 1, status, s);
    if (code == TB200_OK)
        code = tb200_mx_gemm(ptr(h), static_cast<uint8_t*>(ptr(ha)), ptr(f.w_down), static_cast<uint8_t*>(ptr(f.s_down)),
                             static_cast<float*>(ptr(f.b_down)), ptr(f.residual), ptr(out), nullptr, m, static_cast<int32_t>(f.d_out),
                             static_cast<int32_t>(f.hidden), 2, status, s);
    if (code != TB200_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

#define TB200_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    TB200_METHOD(rms_norm),
    TB200_METHOD(layer_norm),
    TB200_METHOD(embedding_bag_mean),
    TB200_METHOD(embedding_bag_mean_backward),
    TB200_METHOD(varlen_attention),
    TB200_METHOD(flash_attention),
    TB200_METHOD(ffn_fp8),
    TB200_METHOD(ffn_fp8_precise),
    TB200_METHOD(ffn_mx),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Host side of the operator calls.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace tb200_host

PyMODINIT_FUNC PyInit__native() {
    HANDLE_TH_ERRORS
    PyObject* m = PyModule_Create(&tb200_host::module);
    if (m != nullptr) tb200_host::bind_engine(m);
    return m;
    END_HANDLE_TH_ERRORS
}
