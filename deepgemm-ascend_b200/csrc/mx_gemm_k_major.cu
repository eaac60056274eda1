// Instantiations of the GEMM kernel: E4M3 x E4M3 (or E2M1 B expanded by TMA), both operands K-major.
#include "launch.h"
#include "mx_gemm.cuh"

namespace dg {

KernelFn pick_k_major_kernel(const KernelChoice& c) {
    const bool pair = c.cta_group == 2;
    if (c.bias_epi)         // BF16 output plus bias through TMA stores
        return c.wide_tile ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, true, true, true>
               : pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, true, false, true>
                      : mx_gemm_kernel<1, 0, 0, false, false, false, false, false, true, false, true>;
    if (c.quant_epi) {      // E4M3 output
        if (c.wide_epi)
            return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, true, false, false, false, true>
                        : mx_gemm_kernel<1, 0, 0, false, false, false, false, true, false, false, false, true>;
        return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, false, false, false, true>
                    : mx_gemm_kernel<1, 0, 0, false, false, false, false, false, false, false, false, true>;
    }
    if (c.wide_tile)        // CTA pair, block_n > 256
        return c.simple_epi ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, true, true>
                            : mx_gemm_kernel<2, 0, 0, false, false, false, false, false, false, true>;
    if (c.simple_epi) {     // plain BF16 output through TMA stores
        if (c.wide_epi)
            return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, true, true> : mx_gemm_kernel<1, 0, 0, false, false, false, false, true, true>;
        return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, false, true> : mx_gemm_kernel<1, 0, 0, false, false, false, false, false, true>;
    }
    if (c.wide_epi)
        return pair ? mx_gemm_kernel<2, 0, 0, false, false, false, false, true> : mx_gemm_kernel<1, 0, 0, false, false, false, false, true>;
    if (c.lean) return mx_gemm_kernel<1, 0, 0, false, true>;
    return pair ? mx_gemm_kernel<2, 0, 0, false> : mx_gemm_kernel<1, 0, 0, false>;
}

}  // namespace dg
