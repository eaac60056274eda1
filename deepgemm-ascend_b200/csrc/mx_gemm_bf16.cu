// Instantiations of the GEMM kernel: BF16 x BF16 (kind::f16, no scale factors).
#include "launch.h"
#include "mx_gemm.cuh"

namespace dg {

KernelFn pick_bf16_kernel(const KernelChoice& c) {
    if (c.wide_tile) return mx_gemm_kernel<2, 0, 0, false, false, false, true, false, false, true>;
    static const KernelFn table[2][2][2] = {
        {{mx_gemm_kernel<1, 0, 0, false, false, false, true>, mx_gemm_kernel<1, 0, 1, false, false, false, true>},
         {mx_gemm_kernel<1, 1, 0, false, false, false, true>, mx_gemm_kernel<1, 1, 1, false, false, false, true>}},
        {{mx_gemm_kernel<2, 0, 0, false, false, false, true>, mx_gemm_kernel<2, 0, 1, false, false, false, true>},
         {mx_gemm_kernel<2, 1, 0, false, false, false, true>, mx_gemm_kernel<2, 1, 1, false, false, false, true>}},
    };
    return table[c.cta_group - 1][c.major_a][c.major_b];
}

}  // namespace dg
