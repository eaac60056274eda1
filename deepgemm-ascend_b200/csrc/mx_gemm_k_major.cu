// Instantiations of the GEMM kernel: E4M3 x E4M3 (or E2M1 B expanded by TMA), both operands K-major.
#include "launch.h"
#include "mx_gemm.cuh"

namespace dg {

// Tiles of up to 256 columns with TMA stores or any epilogue; kOverlap: accumulators that share columns.
template <bool kOverlap>
static KernelFn pick_narrow(const KernelChoice& c) {
    const bool pair = c.cta_group == 2;
    if (c.bias_epi)         // BF16 output plus bias through TMA stores
        return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, true, false, true, false, kOverlap>
                    : mx_gemm_kernel<1, 0, 0, false, false, false, false, false, true, false, true, false, kOverlap>;
    if (c.simple_epi) {     // plain BF16 output through TMA stores
        if (c.wide_epi)
            return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, true, true, false, false, false, kOverlap>
                        : mx_gemm_kernel<1, 0, 0, false, false, false, false, true, true, false, false, false, kOverlap>;
        return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, true, false, false, false, kOverlap>
                    : mx_gemm_kernel<1, 0, 0, false, false, false, false, false, true, false, false, false, kOverlap>;
    }
    if (c.wide_epi)
        return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, true, false, false, false, false, kOverlap>
                    : mx_gemm_kernel<1, 0, 0, false, false, false, false, true, false, false, false, false, kOverlap>;
    return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, false, false, false, false, kOverlap>
                : mx_gemm_kernel<1, 0, 0, false, false, false, false, false, false, false, false, false, kOverlap>;
}

KernelFn pick_k_major_kernel(const KernelChoice& c) {
    const bool pair = c.cta_group == 2;
    if (c.quant_epi) {      // E4M3 output
        if (c.wide_epi)
            return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, true, false, false, false, true>
                        : mx_gemm_kernel<1, 0, 0, false, false, false, false, true, false, false, false, true>;
        return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, false, false, false, true>
                    : mx_gemm_kernel<1, 0, 0, false, false, false, false, false, false, false, false, true>;
    }
    if (c.wide_tile) {      // CTA pair, block_n > 256
        if (c.bias_epi) return mx_gemm_kernel<2, 0, 0, false, false, false, false, false, true, true, true>;
        return c.simple_epi ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, true, true>
                            : mx_gemm_kernel<2, 0, 0, false, false, false, false, false, false, true>;
    }
    if (c.lean) return mx_gemm_kernel<1, 0, 0, false, true>;
    return c.overlap ? pick_narrow<true>(c) : pick_narrow<false>(c);
}

}  // namespace dg
