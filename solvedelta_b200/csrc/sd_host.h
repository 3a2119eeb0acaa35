// Helpers shared by the C++ host sources: status checks, the current stream, output and workspace tensors.
#pragma once
#include <torch/extension.h>
#include <torch/csrc/autograd/custom_function.h>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "../../include/solvedelta_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<at::Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

inline void check(int status) {
    TORCH_CHECK(status == SD_OK, "solvedelta_b200: ", sd_status_string(status), " (status ", status, ")");
}

inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

inline float* f32(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
inline void* raw(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline const unsigned char* bytes(const Tensor& t) { return static_cast<const unsigned char*>(raw(t)); }
inline Tensor bf16_like(const Tensor& t, at::IntArrayRef shape) { return at::empty(shape, t.options().dtype(at::kBFloat16)); }
inline Tensor f32_like(const Tensor& t, at::IntArrayRef shape) { return at::empty(shape, t.options().dtype(at::kFloat)); }
inline Tensor workspace(const Tensor& t, size_t n) {
    return at::empty({(int64_t)(n < 16 ? 16 : n)}, t.options().dtype(at::kByte));
}
inline Tensor given(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
inline OptTensor optional(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }

inline void value_error(bool bad, const char* text) {
    if (bad) throw py::value_error(text);
}
inline void type_error(bool bad, const char* text) {
    if (bad) throw py::type_error(text);
}
inline bool is_shape(const Tensor& t, at::IntArrayRef shape) { return t.sizes() == shape; }

// [B,T,H,w] (any outer strides, unit inner stride) or [B,T,H] -> C operand
inline sd_operand operand(const Tensor& t) { return sd_operand{t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)}; }

void register_glue(py::module_& m);
