// Instantiations of the GEMM kernel: both operands packed E2M1, K-major (kind::mxf4).
#include "launch.h"
#include "mx_gemm.cuh"

namespace dg {

KernelFn pick_fp4_kernel(const KernelChoice& c) {
    if (c.wide_tile) return mx_gemm_kernel<2, 0, 0, false, false, true, false, false, false, true>;
    if (c.overlap)
        return c.cta_group == 2 ? mx_gemm_kernel<2, 0, 0, false, false, true, false, false, false, false, false, false, true>
                                : mx_gemm_kernel<1, 0, 0, false, false, true, false, false, false, false, false, false, true>;
    return c.cta_group == 2 ? mx_gemm_kernel<2, 0, 0, false, false, true> : mx_gemm_kernel<1, 0, 0, false, false, true>;
}

}  // namespace dg
