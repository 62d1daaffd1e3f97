// Shared declarations of the host module: C-ABI calls on torch tensors (allocation, current stream, status checks).
#pragma once
#include <ATen/ATen.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <optional>

#include "../../../include/tb200.h"

namespace tb200_host {

using at::Tensor;

// TB200_* element code of a floating type, -1 for the others
inline int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return TB200_F32;
        case at::kHalf: return TB200_F16;
        case at::kBFloat16: return TB200_BF16;
        default: return -1;
    }
}
inline int id_code(at::ScalarType t) { return t == at::kInt ? TB200_I32 : (t == at::kLong ? TB200_I64 : -1); }

inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
inline void* ptr(const Tensor& t) { return t.data_ptr(); }
inline void* ptr(const std::optional<Tensor>& t) { return t.has_value() ? t->data_ptr() : nullptr; }

// contiguous CUDA tensor of the given type
inline bool dense(const Tensor& t, at::ScalarType type) {
    return t.defined() && t.is_cuda() && t.scalar_type() == type && t.is_contiguous();
}
inline bool wants_grad(const Tensor& t) { return t.requires_grad() && c10::GradMode::is_enabled(); }

inline void check(int code, const char* what) {
    TORCH_CHECK(code == 0, what, ": ", tb200_strerror(code), " (status ", code, ")");
}

}  // namespace tb200_host
