// Instantiations of the GEMM kernel: E4M3 x packed E2M1 with the decoder warps (operands TMA cannot expand).
#include "launch.h"
#include "mx_gemm.cuh"

namespace dg {

KernelFn pick_decode_kernel(const KernelChoice& c) {
    if (c.overlap) {       // (K-major A only)
        static const KernelFn overlapping[2][2] = {
            {mx_gemm_kernel<1, 0, 0, true, false, false, false, false, false, false, false, false, true>,
             mx_gemm_kernel<1, 0, 1, true, false, false, false, false, false, false, false, false, true>},
            {mx_gemm_kernel<2, 0, 0, true, false, false, false, false, false, false, false, false, true>,
             mx_gemm_kernel<2, 0, 1, true, false, false, false, false, false, false, false, false, true>},
        };
        return overlapping[c.cta_group - 1][c.major_b];
    }
    static const KernelFn table[2][2][2] = {
        {{mx_gemm_kernel<1, 0, 0, true>, mx_gemm_kernel<1, 0, 1, true>}, {mx_gemm_kernel<1, 1, 0, true>, mx_gemm_kernel<1, 1, 1, true>}},
        {{mx_gemm_kernel<2, 0, 0, true>, mx_gemm_kernel<2, 0, 1, true>}, {mx_gemm_kernel<2, 1, 0, true>, mx_gemm_kernel<2, 1, 1, true>}},
    };
    return table[c.cta_group - 1][c.major_a][c.major_b];
}

}  // namespace dg
