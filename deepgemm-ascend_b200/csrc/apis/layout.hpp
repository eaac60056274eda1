// Scale-factor layout: the counterpart of csrc/apis/layout.hpp:37-128 (check_sf_layout, transform_sf_into_required_layout,
// transform_k_grouped_sf_into_required_layout, get_recipe) and of the launcher csrc/jit_kernels/transform_sf.hpp:15-105.
#pragma once

#include "common.hpp"
#include "runtime.hpp"

namespace dg_host {

using Recipe3 = std::tuple<int, int, int>;
using Recipe2 = std::tuple<int, int>;

// (gran_m, gran_n, gran_k_a, gran_k_b). The reference requires both gran_k to be 32 (csrc/apis/layout.hpp:55,125); here
// each may be 32 or 128 because a per-128 scale is expanded to the per-32 layout by the transform.
inline std::tuple<int, int, int, int> get_recipe(const std::optional<Recipe3>& recipe, const std::optional<Recipe2>& recipe_a,
                                                 const std::optional<Recipe2>& recipe_b) {
    host_assert(!(recipe.has_value() && (recipe_a.has_value() || recipe_b.has_value())),
                "recipe and recipe_a / recipe_b are mutually exclusive");
    if (recipe.has_value()) {
        const auto [gm, gn, gk] = recipe.value();
        return {gm, gn, gk, gk};
    }
    const auto [gm, gka] = recipe_a.value_or(Recipe2{1, 32});
    const auto [gn, gkb] = recipe_b.value_or(Recipe2{1, 32});
    return {gm, gn, gka, gkb};
}

// csrc/apis/layout.hpp:37-65. True when `sf` already is the required layout.
inline bool check_sf_layout(const View& sf, int64_t mn, int64_t k, int gran_mn, int gran_k,
                            const std::optional<int>& num_groups) {
    host_assert(sf.scalar_type() == torch::kFloat32 || sf.scalar_type() == torch::kInt16,
                "SF must be float32 or int16 (packed ue8m0x2)");
    host_assert(sf.dim() == (num_groups.has_value() ? 1 : 0) + 2, "SF has the wrong number of dimensions");
    host_assert(sf.stride(-1) == 1 || sf.stride(-2) == 1 || sf.size(-1) == 1 || sf.size(-2) == 1,
                "SF input must be contiguous in either the last or second-to-last dimension");
    if (num_groups.has_value()) host_assert(sf.size(-3) == num_groups.value());
    host_assert(gran_k == 32 || gran_k == 128, "gran_k must be 32 (or 128, expanded by the transform)");
    const int64_t div_k = sf.scalar_type() == torch::kFloat32 ? gran_k : gran_k * 2;
    if (sf.size(-2) != ceil_div(mn, gran_mn))
        throw std::runtime_error("SF rows: expected " + std::to_string(ceil_div(mn, gran_mn)) + ", got " + std::to_string(sf.size(-2)));
    if (sf.size(-1) != ceil_div(k, div_k))
        throw std::runtime_error("SF columns: expected " + std::to_string(ceil_div(k, div_k)) + ", got " + std::to_string(sf.size(-1)));
    if (sf.scalar_type() == torch::kInt16 && gran_mn == 1 && gran_k == 32 && sf.stride(-2) == 1 && sf.stride(-1) == sf.size(-2))
        return !num_groups.has_value() || sf.stride(-3) == sf.size(-2) * sf.size(-1);
    return false;
}

inline int check_psum_layout(const torch::Tensor& psum_layout, const View& sf) {
    host_assert(psum_layout.device() == sf.device(), "grouped_layout must be on the same device as the SF input");
    host_assert(psum_layout.scalar_type() == torch::kInt32 && psum_layout.dim() == 1 && psum_layout.is_contiguous(),
                "grouped_layout must be a contiguous 1D int32 tensor");
    host_assert(psum_layout.numel() > 0, "grouped_layout must contain at least one group");
    return (int)psum_layout.numel();
}

// csrc/jit_kernels/transform_sf.hpp:15-105. With `tma_aligned` the column stride of the result is rounded up to 8
// elements (what the GEMM's tensor map needs); the public entry point never does that. `psum_layout` pads along MN
// (m-grouped operands), `k_psum_layout` along K (k-grouped operands).
struct SfTransform {
    View out;                              // the result (or the input when it already has the layout)
    torch::Tensor flag;                    // the invalid-scale flag
    dg_transform_sf_desc_t desc{};
    bool pending = false;                  // `out` is still to be written by the launch that `desc` describes
};
inline SfTransform prepare_transform_sf(const View& sf, int64_t mn, int64_t k, int gran_mn, int gran_k,
                                        const std::optional<torch::Tensor>& psum_layout, bool tma_aligned,
                                        const std::optional<torch::Tensor>& k_psum_layout = std::nullopt) {
    const bool flat = sf.dim() == 2;
    if (!flat && sf.dim() != 3) throw std::runtime_error("Transform SF input must have 2 or 3 dimensions, but got " + std::to_string(sf.dim()));
    host_assert(gran_mn >= 1 && gran_mn <= 128 && (gran_mn & (gran_mn - 1)) == 0, "gran_mn only support a power of two in [1, 128]");
    const int64_t batches = flat ? 1 : sf.size(0);
    int num_groups = 0, num_k_groups = 0;
    if (psum_layout.has_value()) {
        host_assert(batches == 1, "Grouped transform SF requires one logical batch and grouped_layout");
        num_groups = check_psum_layout(psum_layout.value(), sf);
    }
    if (k_psum_layout.has_value()) {
        host_assert(batches == 1 && !psum_layout.has_value(), "Grouped transform SF requires one logical batch and grouped_layout");
        host_assert(gran_k == 32, "K-grouped transform SF requires gran_k = 32");
        num_k_groups = check_psum_layout(k_psum_layout.value(), sf);
    }
    const bool is_fp32 = sf.scalar_type() == torch::kFloat32;
    const int64_t k32 = ceil_div(k, 32);
    const int64_t dst_cols = (!is_fp32 && gran_k == 32) ? sf.size(-1) : ceil_div(k32, 2);
    const int64_t col_stride = tma_aligned ? align_up(mn, 8) : mn;
    const auto storage = torch::empty({batches, dst_cols, col_stride}, sf.t.options().dtype(torch::kInt16));
    SfTransform t;
    t.out.t = storage;
    t.out.permuted = true;
    // (the strides are the storage's own: torch counts an empty dimension as one there)
    if (!flat) { t.out.sizes.push_back(batches); t.out.strides.push_back(storage.stride(0)); }
    t.out.sizes.push_back(mn); t.out.strides.push_back(1);
    t.out.sizes.push_back(dst_cols); t.out.strides.push_back(storage.stride(1));
    if (batches * mn * dst_cols != 0 && !runtime().dry_run && !sf.is_meta()) {
        if (is_fp32) t.flag = sf_invalid_flag(sf.device());
        auto& d = t.desc;
        d.src = sf.data_ptr(); d.src_is_fp32 = is_fp32 ? 1 : 0;
        d.src_row_stride = (uint64_t)sf.stride(-2); d.src_col_stride = (uint64_t)sf.stride(-1); d.src_batch_stride = flat ? (uint64_t)(sf.size(0) * sf.stride(0)) : (uint64_t)sf.stride(0);
        d.src_rows = (uint32_t)sf.size(-2); d.src_cols = (uint32_t)sf.size(-1);
        d.dst = static_cast<int16_t*>(storage.data_ptr());
        d.dst_col_stride = (uint64_t)col_stride; d.dst_batch_stride = (uint64_t)(dst_cols * col_stride);
        d.dst_mn = (uint32_t)mn; d.k32_blocks = (uint32_t)k32; d.gran_mn = (uint32_t)gran_mn; d.k_repeat = (uint32_t)(gran_k / 32);
        d.num_batches = (uint32_t)batches;
        d.psum = psum_layout.has_value() ? static_cast<const int32_t*>(psum_layout->data_ptr()) : nullptr;
        d.num_groups = (uint32_t)num_groups;
        d.k_psum = k_psum_layout.has_value() ? static_cast<const int32_t*>(k_psum_layout->data_ptr()) : nullptr;
        d.num_k_groups = (uint32_t)num_k_groups;
        d.alignment = (uint32_t)kMkAlignment;
        d.invalid_flag = t.flag.defined() ? static_cast<int32_t*>(t.flag.data_ptr()) : nullptr;
        t.pending = true;
    }
    return t;
}

inline void check_invalid_scale(const torch::Tensor& flag) {
    if (flag.defined() && runtime().debug && flag.item<int32_t>() != 0) {
        flag.zero_();
        throw std::runtime_error("Float32 SF must be non-negative and can't have non-zero mantissa");
    }
}

inline View launch_transform_sf(const SfTransform& t, void* stream) {
    if (t.pending) {
        const auto& d = t.desc;
        check(dg_transform_sf_launch(d.src, d.src_is_fp32, d.src_row_stride, d.src_col_stride, d.src_batch_stride, d.src_rows, d.src_cols,
                                     d.dst, d.dst_col_stride, d.dst_batch_stride, d.dst_mn, d.k32_blocks, d.gran_mn, d.k_repeat,
                                     d.num_batches, d.psum, d.num_groups, d.alignment, d.invalid_flag, d.k_psum, d.num_k_groups, stream));
        check_invalid_scale(t.flag);
    }
    return t.out;
}

// The scales of both operands of a GEMM: one launch when both need the relayout.
inline std::pair<View, View> launch_transform_sf_pair(const SfTransform& a, const SfTransform& b, void* stream) {
    if (a.pending && b.pending) {
        check(dg_transform_sf_pair_launch(&a.desc, &b.desc, stream));
        check_invalid_scale(a.flag);
        check_invalid_scale(b.flag);
        return {a.out, b.out};
    }
    return {launch_transform_sf(a, stream), launch_transform_sf(b, stream)};
}

inline SfTransform plan_transform_sf(const View& sf, int64_t mn, int64_t k, int gran_mn, int gran_k,
                                     const std::optional<int>& num_groups, bool disable_ue8m0_cast,
                                     const std::optional<torch::Tensor>& psum_layout, bool tma_aligned,
                                     const std::optional<torch::Tensor>& k_psum_layout = std::nullopt) {
    if (check_sf_layout(sf, mn, k, gran_mn, gran_k, num_groups)) {
        if (!tma_aligned || mn % 8 == 0 || sf.is_meta()) {
            SfTransform t;
            t.out = sf;
            return t;
        }
    } else if (sf.scalar_type() == torch::kFloat32) {
        host_assert(!disable_ue8m0_cast, "Float32 SF must be converted into ue8m0, but disable_ue8m0_cast is set true");
    }
    return prepare_transform_sf(sf, mn, k, gran_mn, gran_k, psum_layout, tma_aligned, k_psum_layout);
}

inline torch::Tensor transform_sf(const torch::Tensor& sf, int64_t mn, int64_t k, int gran_mn, int gran_k,
                                  const std::optional<int>& num_groups, bool disable_ue8m0_cast,
                                  const std::optional<torch::Tensor>& psum_layout, bool tma_aligned,
                                  const std::optional<torch::Tensor>& k_psum_layout = std::nullopt) {
    const auto t = plan_transform_sf(sf, mn, k, gran_mn, gran_k, num_groups, disable_ue8m0_cast, psum_layout, tma_aligned, k_psum_layout);
    return (t.pending ? launch_transform_sf(t, stream_of(sf)) : t.out).tensor();
}

// csrc/apis/layout.hpp:68-92. Returns int16 [..., MN, ceil(K/64)], MN-major; returns `sf` itself when it already has
// that layout. `recipe` has three (gran_m, gran_n, gran_k; `is_sfa` selects) or two (gran_mn, gran_k) elements.
inline torch::Tensor transform_sf_into_required_layout(const torch::Tensor& sf, const int& mn, const int& k,
                                                       const std::vector<int>& recipe, const std::optional<int>& num_groups,
                                                       const std::optional<bool>& is_sfa, const bool& disable_ue8m0_cast,
                                                       const std::optional<torch::Tensor>& psum_layout) {
    int gran_mn, gran_k;
    if (recipe.size() == 3) {
        host_assert(is_sfa.has_value(), "is_sfa must be set for a 3-element recipe");
        gran_mn = is_sfa.value() ? recipe[0] : recipe[1];
        gran_k = recipe[2];
    } else {
        host_assert(recipe.size() == 2, "recipe must have 2 or 3 elements");
        gran_mn = recipe[0];
        gran_k = recipe[1];
    }
    return transform_sf(sf, mn, k, gran_mn, gran_k, num_groups, disable_ue8m0_cast, psum_layout, false);
}

// csrc/apis/layout.hpp:94-111: scale factors of a k-grouped operand ([MN, K] with K holding the groups in psum layout):
// same result layout, with every K unit inside a group's padding set to 0.
inline torch::Tensor transform_k_grouped_sf_into_required_layout(const torch::Tensor& sf, const int& mn, const int& k,
                                                                 const std::vector<int>& recipe, const std::optional<bool>& is_sfa,
                                                                 const torch::Tensor& psum_layout) {
    host_assert(is_sfa.has_value(), "is_sfa must be set");
    host_assert(recipe.size() == 3, "recipe must have 3 elements");
    return transform_sf(sf, mn, k, is_sfa.value() ? recipe[0] : recipe[1], recipe[2], std::nullopt, false, std::nullopt, false, psum_layout);
}

inline void register_layout_apis(py::module_& m) {
    m.def("transform_sf_into_required_layout", &transform_sf_into_required_layout,
          py::arg("sf"), py::arg("mn"), py::arg("k"), py::arg("recipe"),
          py::arg("num_groups") = std::nullopt, py::arg("is_sfa") = std::nullopt,
          py::arg("disable_ue8m0_cast") = false, py::arg("psum_layout") = std::nullopt);
    m.def("transform_k_grouped_sf_into_required_layout", &transform_k_grouped_sf_into_required_layout,
          py::arg("sf"), py::arg("mn"), py::arg("k"), py::arg("recipe"), py::arg("is_sfa"), py::arg("psum_layout"));
    m.def("get_recipe", [](const std::optional<Recipe3>& recipe, const std::optional<Recipe2>& recipe_a,
                           const std::optional<Recipe2>& recipe_b) { return get_recipe(recipe, recipe_a, recipe_b); },
          py::arg("recipe"), py::arg("recipe_a"), py::arg("recipe_b"));
}

}  // namespace dg_host
