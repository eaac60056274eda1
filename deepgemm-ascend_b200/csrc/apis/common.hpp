// Helpers shared by the binding headers: host assertions that surface in Python as RuntimeError with the reference's
// message text, tensor unpacking (pointers, majors, strides), the named-axis shape inference of
// csrc/utils/layout.hpp:140-219, the current CUDA stream, and checked calls into the C ABI.
#pragma once

#include <ATen/cuda/CUDAContext.h>
#include <torch/extension.h>

#include <array>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <mutex>
#include <optional>
#include <sstream>
#include <stdexcept>
#include <string>
#include <tuple>
#include <utility>
#include <vector>

#include "../../../include/dg_b200.h"

namespace dg_host {

namespace py = pybind11;

constexpr auto kPackedFp4 = torch::kInt8;          // csrc/utils/dtype.hpp:9
constexpr int kMkAlignment = 256;                   // csrc/jit/jit.hpp:59-73

// (the message is a literal, or made by the caller once the condition has failed: a string for every check of every call is what
// the checks would cost)
inline void host_assert(bool cond, const char* msg = "Assertion failed") {
    if (!cond) throw std::runtime_error(msg);
}

inline void check(int rc) {
    if (rc != DG_OK) {
        const char* msg = dg_last_error();
        throw std::runtime_error(msg != nullptr && msg[0] != 0 ? std::string(msg) : "libdg_b200 error " + std::to_string(rc));
    }
}

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline int64_t align_up(int64_t a, int64_t b) { return ceil_div(a, b) * b; }

// Sizes and strides of a tensor, or of a permutation of its dimensions: what the entry points look at. at::transpose and at::permute make a tensor for
// each operand (about 0.6 us apiece; the per-head projection had five of them in 7.8 us).
struct View {
    torch::Tensor t;
    c10::SmallVector<int64_t, 4> sizes, strides;
    bool permuted = false;

    View() = default;
    View(const torch::Tensor& x) : t(x), sizes(x.sizes().begin(), x.sizes().end()), strides(x.strides().begin(), x.strides().end()) {}
    int64_t dim() const { return (int64_t)sizes.size(); }
    int64_t at(int64_t i) const {
        if (i < -dim() || i >= dim()) (void)t.size(i);            // (raises torch's own message)
        return i < 0 ? i + dim() : i;
    }
    int64_t size(int64_t i) const { return sizes[at(i)]; }
    int64_t stride(int64_t i) const { return strides[at(i)]; }
    int64_t numel() const { return t.numel(); }
    auto scalar_type() const { return t.scalar_type(); }
    auto device() const { return t.device(); }
    bool is_meta() const { return t.is_meta(); }
    void* data_ptr() const { return t.data_ptr(); }
    torch::Tensor tensor() const { return permuted ? t.as_strided(sizes, strides) : t; }
    View transpose(int64_t i, int64_t j) const {
        if (i >= dim() || j >= dim()) (void)t.transpose(i, j);
        View v = *this;
        std::swap(v.sizes[at(i)], v.sizes[at(j)]);
        std::swap(v.strides[at(i)], v.strides[at(j)]);
        v.permuted = true;
        return v;
    }
    View permute(std::initializer_list<int64_t> p) const {
        if ((int64_t)p.size() != dim()) (void)t.permute(p);
        View v = *this;
        int64_t n = 0;
        for (int64_t i : p) { v.sizes[n] = sizes[i]; v.strides[n++] = strides[i]; }
        v.permuted = true;
        return v;
    }
};
using OptView = std::optional<View>;

// Meta tensors (dry run) have no address; validation only needs something 32-byte aligned.
template <class T> inline void* ptr_of(const T& t) { return t.is_meta() ? reinterpret_cast<void*>(0x1000) : t.data_ptr(); }

template <class T> inline void* stream_of(const T& t) {
    return static_cast<void*>(at::cuda::getCurrentCUDAStream(t.device().index()).stream());
}

// ---- process-wide knobs (csrc/jit/jit.hpp:18-76)
struct Runtime {
    std::atomic<bool> dry_run{false}, deterministic{false};
    std::atomic<int> arch{100};
    const bool debug = [] { const char* e = getenv("DG_JIT_DEBUG"); return e != nullptr && e[0] != 0 && std::string(e) != "0"; }();
};
inline Runtime& runtime() { static Runtime r; return r; }

// ---- majors (csrc/utils/layout.hpp:37-52,88-99)
inline void major_check(const View& t) {
    const auto d = t.dim();
    if (t.stride(d - 2) == 1 && t.stride(d - 1) == 1) {
        std::ostringstream os;
        os << "Ambiguous major axis, the tensor has both last two dimensions contiguous, strides=" << at::IntArrayRef(t.strides);
        throw std::runtime_error(os.str());
    }
    host_assert(t.stride(d - 2) == 1 || t.stride(d - 1) == 1);
}
inline int major_ab(const View& t) {
    major_check(t);
    return t.stride(t.dim() - 1) == 1 ? DG_MAJOR_K : DG_MAJOR_MN;
}
inline int64_t outer_stride(const View& t, int major) {
    return major == DG_MAJOR_K ? t.stride(t.dim() - 2) : t.stride(t.dim() - 1);
}

// ---- named-axis shape inference with conflict diagnostics (csrc/utils/layout.hpp:140-219). A packed-FP4 tensor
// counts double along its contiguous axis.
struct ShapeSpec { const char* dims; const View* t; };
inline std::array<int64_t, 4> shape_by_spec(const char* out_dims, std::initializer_list<ShapeSpec> specs) {
    const ShapeSpec* const spec = specs.begin();
    int majors[4] = {};
    for (size_t idx = 0; idx < specs.size(); ++idx) {
        const View& t = *spec[idx].t;
        if (t.dim() != (int64_t)strlen(spec[idx].dims))
            throw std::runtime_error("Shape mismatch: tensor #" + std::to_string(idx) + ", annotation=\"" + spec[idx].dims + "\"");
        int major = -1;
        for (int i = 0; i < t.dim(); ++i)
            if (t.strides[i] == 1) { major = i; break; }
        if (major < 0) {
            std::ostringstream os;
            os << "Tensor #" << idx << " annotation=\"" << spec[idx].dims << "\" doesn't have major axis, strides=" << at::IntArrayRef(t.strides);
            throw std::runtime_error(os.str());
        }
        majors[idx] = major;
    }
    std::array<int64_t, 4> result{};
    for (size_t o = 0; out_dims[o] != 0; ++o) {
        bool found = false;
        int64_t value = 0;
        size_t f_idx = 0;
        int f_axis = 0;
        for (size_t idx = 0; idx < specs.size(); ++idx) {
            const View& t = *spec[idx].t;
            for (int axis = 0; axis < (int)t.dim(); ++axis) {
                if (spec[idx].dims[axis] != out_dims[o]) continue;
                const int64_t v = t.sizes[axis] * ((axis == majors[idx] && t.scalar_type() == kPackedFp4) ? 2 : 1);
                if (!found) {
                    found = true; value = v; f_idx = idx; f_axis = axis;
                } else if (value != v) {
                    std::ostringstream os;
                    os << "Conflicting shape dimension '" << out_dims[o] << "': tensor #" << idx << " annotation=\"" << spec[idx].dims << "\" axis=" << axis
                       << " gives " << v << ", but tensor #" << f_idx << " annotation=\"" << spec[f_idx].dims << "\" axis=" << f_axis
                       << " gives " << value;
                    throw std::runtime_error(os.str());
                }
            }
        }
        result[o] = found ? value : 0;
    }
    return result;
}

template <class T> inline int dtype_code(const T& t) {
    switch (t.scalar_type()) {
        case torch::kFloat8_e4m3fn: return DG_E4M3;
        case torch::kInt8: return DG_E2M1X2;
        case torch::kBFloat16: return DG_BF16;
        case torch::kFloat32: return DG_F32;
        default: throw std::runtime_error("Unsupported operand dtypes");
    }
}

}  // namespace dg_host
