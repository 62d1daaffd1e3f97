// The engine's launches: each function allocates its result, enqueues the library's kernel on the current stream and, while
// kernel timing is on, brackets the launch with the timing records of the Python operators (same names and fields).
#pragma once
#include <ATen/cuda/EmptyTensor.h>
#include <pybind11/stl.h>
#include <torch/csrc/utils/pybind.h>

#include <cmath>

#include "native.h"

namespace tb200_host {
namespace py = pybind11;
using namespace pybind11::literals;
using OptTensor = std::optional<Tensor>;

// Timing is switched per forward; the records belong to the list installed with `ops.set_kernel_timing`.
struct Timing {
    static bool& on() {
        static thread_local bool flag = false;
        return flag;
    }
};
class Timed {
public:
    Timed(const char* name, const py::dict& meta) : scope_(py::module_::import("taac_2026_b200.ops").attr("timed")(name, **meta)) {
        scope_.attr("__enter__")();
    }
    ~Timed() {   // also while an error of the launch is on its way: nothing may be thrown from here
        try {
            scope_.attr("__exit__")(py::none(), py::none(), py::none());
        } catch (py::error_already_set& e) {
            e.discard_as_unraisable("kernel timing");
        }
    }

private:
    py::object scope_;
};
#define TB200_TIMED(name, ...)   \
    std::optional<Timed> timed_; \
    if (Timing::on()) timed_.emplace(name, py::dict(__VA_ARGS__))

inline Tensor make(at::IntArrayRef sizes, at::ScalarType type, const at::Device& device) {
    return at::detail::empty_cuda(sizes, type, device, std::nullopt);
}
inline Tensor make_like(at::IntArrayRef sizes, const Tensor& t) { return make(sizes, t.scalar_type(), t.device()); }

template <typename P>
P* data(const Tensor& t) { return static_cast<P*>(t.data_ptr()); }
template <typename P>
P* data(const OptTensor& t) { return t.has_value() ? static_cast<P*>(t->data_ptr()) : nullptr; }

inline Tensor gather_rows(const Tensor& table, const Tensor& ids) {   // table [V, d], ids int64 [n]
    const int64_t n = ids.numel(), dim = table.size(1);
    Tensor out = make_like({n, dim}, table);
    TB200_TIMED("gather_rows", "ids"_a = ids, "dim"_a = dim, "esize"_a = table.element_size());
    check(tb200_gather_rows(ptr(table), table.size(0), static_cast<int32_t>(dim), ptr(ids), TB200_I64, n, std::max<int64_t>(n, 1), 0, ptr(out), dim, 0,
                            dtype_code(table.scalar_type()), stream_of(table)), "cuda gather_rows");
    return out;
}
inline void gather_rows_into(const Tensor& table, const int64_t* ids, const Tensor& ids_meta, const Tensor& out, int64_t col0) {
    const int64_t n = out.size(0), dim = table.size(1);
    TB200_TIMED("gather_rows", "ids"_a = ids_meta, "dim"_a = dim, "esize"_a = table.element_size());
    check(tb200_gather_rows(ptr(table), table.size(0), static_cast<int32_t>(dim), ids, TB200_I64, n, std::max<int64_t>(n, 1), 0, ptr(out), out.size(1),
                            static_cast<int32_t>(col0), dtype_code(table.scalar_type()), stream_of(table)), "cuda gather_rows");
}
// dst[ids[i], col0 ..] = src[i] (+ bias[i / rows per bias row]) (+ residual[ids[i]])
inline void scatter_rows(const Tensor& dst, const Tensor& ids, const Tensor& src, const OptTensor& bias = std::nullopt,
                         const OptTensor& residual = std::nullopt) {   // src: [.., dim], rows src.stride(-2) elements apart
    const int64_t n = ids.numel(), dim = src.size(-1);
    const int64_t per_group = bias.has_value() ? std::max<int64_t>(n / (bias->numel() / dim), 1) : 1;
    TB200_TIMED("scatter_rows", "rows"_a = n, "dim"_a = dim, "esize"_a = dst.element_size());
    check(tb200_scatter_rows_strided(ptr(dst), dst.size(0), dst.size(1), 0, data<int64_t>(ids), ptr(src), src.stride(-2), n,
                                     static_cast<int32_t>(dim), ptr(bias), per_group,
                             ptr(residual), residual.has_value() ? residual->size(1) : 0, dtype_code(dst.scalar_type()), stream_of(dst)),
          "cuda scatter_rows");
}
inline Tensor rms_norm(const Tensor& x, const Tensor& w, const OptTensor& in_bias = std::nullopt) {   // [rows, d], eps 1e-6
    const auto cols = static_cast<int32_t>(x.size(-1));
    const int64_t rows = x.numel() / cols;
    Tensor out = make_like(x.sizes(), x);
    const int dt = dtype_code(x.scalar_type());
    TB200_TIMED("rms_norm", "rows"_a = rows, "cols"_a = cols, "esize"_a = x.element_size());
    check(in_bias.has_value() ? tb200_rmsnorm_bias_fwd(ptr(x), ptr(*in_bias), ptr(w), ptr(out), rows, cols, 1e-6f, dt, stream_of(x))
                              : tb200_rmsnorm_fwd(ptr(x), ptr(w), ptr(out), rows, cols, 1e-6f, dt, stream_of(x)), "cuda rms_norm");
    return out;
}

// A weight in the form this library's GEMMs read: as it is in bf16, as three bf16 parts [.., N, 3 K] in fp32
inline bool own_gemm_serves(at::ScalarType type, int64_t n, int64_t k) {
    return type == at::kBFloat16 ? n % 256 == 0 && k % 64 == 0 : (type == at::kFloat && n % 128 == 0 && k % 64 == 0);
}
inline Tensor own_form(const Tensor& w) {
    if (!w.defined() || w.scalar_type() != at::kFloat) return w;
    auto sizes = w.sizes().vec();
    sizes.back() *= 3;
    Tensor out = make(sizes, at::kBFloat16, w.device());
    const Tensor src = w.contiguous();
    check(tb200_split_f32_weights(data<float>(src), ptr(out), src.numel() / src.size(-1), static_cast<int32_t>(src.size(-1)), stream_of(src)),
          "cuda split_f32_weights");
    return out;
}

// One shared layer: weight [N, K] in the compute type and in the form of this library's GEMM (undefined where that does not serve
// it), bias in fp32 for this library's GEMM and in the compute type for the library's
struct Layer {
    Tensor w, own;
    OptTensor b32, b;
};

// out[g] = act(x[g] w[g]^T + b[g]) (+ residual[g]); x [G, M, K] or [M, K], w in the form of own_form; `out` may be the residual
inline Tensor grouped(const Tensor& x, const Tensor& w, const OptTensor& b32, bool silu, const OptTensor& residual, const OptTensor& out_in,
                      const Tensor& status) {
    const int64_t k = x.size(-1), m = x.size(-2), g = x.dim() == 3 ? x.size(0) : 1, n = w.size(-2);
    Tensor out = out_in.has_value() ? *out_in : (x.dim() == 3 ? make_like({g, m, n}, x) : make_like({m, n}, x));
    if (x.scalar_type() == at::kFloat) {
        TB200_TIMED("gemm_f32", "groups"_a = g, "m"_a = m, "n"_a = n, "k"_a = k, "silu"_a = silu, "residual"_a = residual.has_value());
        check(tb200_gemm_f32_grouped(data<float>(x), ptr(w), data<float>(b32), data<float>(residual), data<float>(out), static_cast<int32_t>(g), m,
                                     static_cast<int32_t>(n), static_cast<int32_t>(k), silu ? 1 : 0, data<int32_t>(status), stream_of(x)),
              "cuda gemm_f32");
        return out;
    }
    TB200_TIMED("gemm_bf16", "groups"_a = g, "m"_a = m, "n"_a = n, "k"_a = k, "silu"_a = silu, "residual"_a = residual.has_value());
    check(tb200_gemm_bf16_grouped(ptr(x), ptr(w), data<float>(b32), ptr(residual), ptr(out), static_cast<int32_t>(g), m, static_cast<int32_t>(n),
                                  static_cast<int32_t>(k), silu ? 1 : 0, data<int32_t>(status), stream_of(x)), "cuda grouped_linear");
    return out;
}

// A layer for few rows per group with the options of the small GEMM: one weight for all groups, RMSNorm of the activations on the
// way in.  false: too many rows, nothing was enqueued.
inline bool few_rows(const Tensor& x, const Tensor& w, const OptTensor& b32, bool silu, const OptTensor& residual, const Tensor& out, bool shared_w,
                     const OptTensor& norm_gamma, const OptTensor& norm_bias) {
    const int64_t g = x.size(0), m = x.size(1), k = x.size(2), n = w.size(-2);
    if (m > 32 || x.scalar_type() != at::kBFloat16) return false;
    TB200_TIMED("gemm_bf16", "groups"_a = g, "m"_a = m, "n"_a = n, "k"_a = k, "silu"_a = silu, "residual"_a = residual.has_value());
    const int code = tb200_gemm_bf16_few_rows(ptr(x), ptr(w), data<float>(b32), ptr(residual), ptr(out), static_cast<int32_t>(g), m,
                                              static_cast<int32_t>(n), static_cast<int32_t>(k), silu ? 1 : 0, shared_w, ptr(norm_gamma),
                                              ptr(norm_bias), 1e-6f, stream_of(x));
    if (code == TB200_ERR_UNSUPPORTED) return false;
    check(code, "cuda grouped_linear");
    return true;
}
// act(rmsnorm(x + norm_bias) gamma w[g]^T + b[g]), x [G, M, K]
inline Tensor norm_grouped(const Tensor& x, const Tensor& gamma, const OptTensor& norm_bias, const Tensor& w, const Tensor& b32, bool silu,
                           const Tensor& status) {
    Tensor out = make_like({x.size(0), x.size(1), w.size(-2)}, x);
    if (few_rows(x, w, b32, silu, std::nullopt, out, false, gamma, norm_bias)) return out;
    return grouped(rms_norm(x, gamma, norm_bias), w, b32, silu, std::nullopt, out, status);
}
// x += a w^T with one weight for all groups; x, a [G, M, K]
inline void add_shared_linear(const Tensor& x, const Tensor& a, const Tensor& w, const Tensor& status) {
    if (few_rows(a, w, std::nullopt, false, x, x, true, std::nullopt, std::nullopt)) return;
    const Tensor flat = x.view({-1, x.size(2)});
    grouped(a.view({-1, a.size(2)}), w, std::nullopt, false, flat, flat, status);
}

// x = act(x + bias[group]) in place, act = SiLU or identity; x [groups, rows, cols]
inline Tensor bias_act_rows(const Tensor& x, const Tensor& bias, bool silu) {
    const int64_t cols = x.size(-1), rows = x.numel() / cols, groups = bias.numel() / cols;
    TB200_TIMED("bias_act_rows", "rows"_a = rows, "cols"_a = cols, "esize"_a = x.element_size());
    check(tb200_bias_act_rows(ptr(x), rows, static_cast<int32_t>(cols), ptr(bias), std::max<int64_t>(rows / groups, 1), silu ? 1 : 0,
                              dtype_code(x.scalar_type()), stream_of(x)), "cuda bias_act_rows");
    return x;
}

// Packed attention: q, k, v strided [rows, H, D] views, sample b owns rows [cu[b], cu[b + 1]); with cu_q the queries are the last
// cu_q[b + 1] - cu_q[b] rows of the sample.  Causal.
inline Tensor packed_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, int64_t max_rows, const OptTensor& cu_q,
                               int64_t max_rows_q, int kernel, const Tensor& status) {
    Tensor out = make_like(q.sizes(), q);
    int64_t s[12];
    int i = 0;
    for (const Tensor* t : {&q, &k, &v, static_cast<const Tensor*>(&out)}) {
        s[i++] = 0;
        s[i++] = t->stride(1);
        s[i++] = t->stride(0);
    }
    const auto b = static_cast<int32_t>(cu.size(0) - 1), h = static_cast<int32_t>(q.size(1)), d = static_cast<int32_t>(q.size(2));
    const int64_t lq = cu_q.has_value() ? max_rows_q : max_rows;
    const bool small = lq <= 32 && max_rows <= 32 && d == 64;
    const char* name = small ? "attention_small"
                       : cu_q.has_value() ? (d == 64 ? "attention_fewq" : "attention_mma")
                                          : (d == 64 && q.scalar_type() == at::kBFloat16 && lq >= 128 ? "attention_tc05" : "attention_mma");
    TB200_TIMED(name, "seq_len"_a = py::none(), "cu_rows"_a = cu, "cu_rows_q"_a = cu_q, "key_valid"_a = py::none(), "batch"_a = b, "heads"_a = h,
                "lq"_a = lq, "lk"_a = max_rows, "dim"_a = d, "ns_start"_a = max_rows, "causal"_a = true, "self_rows"_a = false,
                "esize"_a = q.element_size());
    check(tb200_attn_fwd(ptr(q), ptr(k), ptr(v), ptr(out), b, h, static_cast<int32_t>(lq), static_cast<int32_t>(max_rows), d, s, nullptr,
                         data<int32_t>(cu), data<int32_t>(cu_q), nullptr, static_cast<int32_t>(max_rows), 1, 0,
                         static_cast<float>(1.0 / std::sqrt(static_cast<double>(d))), dtype_code(q.scalar_type()), kernel, k.size(0),
                         data<int32_t>(status), stream_of(q)), "cuda varlen_attention");
    return out;
}

}  // namespace tb200_host
