// The quantisers in front of the GEMM (deep_gemm/quant_ops.py holds the same in Python): the reference's
// third-party/tilelang_ops/swiglu_apply_weight_to_fp8.py:411-449 and the plain cast.
#pragma once

#include "common.hpp"
#include "runtime.hpp"

namespace dg_host {

inline std::pair<torch::Tensor, torch::Tensor> quantise_fp8(const torch::Tensor& x, int64_t hidden, bool swiglu,
                                                            const std::optional<torch::Tensor>& topk_weights,
                                                            const std::optional<torch::Tensor>& psum,
                                                            const std::optional<double>& clamp_value, int64_t expert_alignment) {
    const int64_t tokens = x.size(0), cols = (hidden / 32 + 1) / 2;
    auto out = torch::empty({tokens, hidden}, x.options().dtype(torch::kFloat8_e4m3fn));
    auto out_sf = torch::empty_strided({tokens, cols}, {1, std::max<int64_t>(tokens, 1)}, x.options().dtype(torch::kInt16));
    if (tokens != 0) {
        if (topk_weights.has_value())
            host_assert(topk_weights->scalar_type() == torch::kFloat32 && topk_weights->is_contiguous() && topk_weights->numel() == tokens,
                        "topk_weights must be a contiguous float32 tensor with one weight per token");
        if (psum.has_value())
            host_assert(psum->scalar_type() == torch::kInt32 && psum->dim() == 1 && psum->is_contiguous() && psum->device() == x.device(),
                        "psum_num_tokens_per_expert must be a contiguous int32 vector on the device of x");
        check(dg_quant_fp8_launch(x.data_ptr(), (uint64_t)x.stride(0), (uint32_t)tokens, (uint32_t)hidden, swiglu ? 1 : 0,
                                  topk_weights.has_value() ? static_cast<const float*>(topk_weights->data_ptr()) : nullptr,
                                  psum.has_value() ? static_cast<const int32_t*>(psum->data_ptr()) : nullptr,
                                  psum.has_value() ? (uint32_t)psum->numel() : 0u, (uint32_t)expert_alignment,
                                  clamp_value.has_value() ? 1 : 0, (float)clamp_value.value_or(0.0), out.data_ptr(), (uint64_t)out.stride(0),
                                  static_cast<int16_t*>(out_sf.data_ptr()), (uint64_t)tokens, stream_of(x)));
    }
    return {out, out_sf};
}

inline void register_quant_apis(py::module_& m) {
    m.def("swiglu_apply_weight_to_fp8", [](const torch::Tensor& x, const std::optional<torch::Tensor>& topk_weights,
                                           const std::optional<torch::Tensor>& psum, const std::optional<double>& clamp_value,
                                           int64_t expert_alignment) {
        host_assert(x.dim() == 2 && x.is_contiguous() && x.scalar_type() == torch::kBFloat16, "x must be a contiguous 2-D BF16 tensor");
        host_assert(x.size(1) % 256 == 0, "the row length of x must be a multiple of 256");
        return quantise_fp8(x, x.size(1) / 2, true, topk_weights, psum, clamp_value, expert_alignment);
    }, py::arg("x"), py::arg("topk_weights") = std::nullopt, py::arg("psum_num_tokens_per_expert") = std::nullopt,
       py::arg("clamp_value") = std::nullopt, py::arg("expert_alignment") = 128);
    m.def("cast_to_fp8", [](const torch::Tensor& x, const std::optional<torch::Tensor>& psum, int64_t expert_alignment) {
        host_assert(x.dim() == 2 && x.stride(1) == 1 && x.scalar_type() == torch::kBFloat16, "x must be a row-major 2-D BF16 tensor");
        host_assert(x.size(1) % 32 == 0, "the row length of x must be a multiple of 32");
        return quantise_fp8(x, x.size(1), false, std::nullopt, psum, std::nullopt, expert_alignment);
    }, py::arg("x"), py::arg("psum_num_tokens_per_expert") = std::nullopt, py::arg("expert_alignment") = 128);
}

}  // namespace dg_host
