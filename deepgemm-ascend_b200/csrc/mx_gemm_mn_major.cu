// Instantiations of the GEMM kernel: 8-bit operands of which at least one is MN-major.
#include "launch.h"
#include "mx_gemm.cuh"

namespace dg {

KernelFn pick_mn_major_kernel(const KernelChoice& c) {
    if (c.lean) {
        static const KernelFn lean_table[2][2] = {{nullptr, mx_gemm_kernel<1, 0, 1, false, true>},
                                                  {mx_gemm_kernel<1, 1, 0, false, true>, mx_gemm_kernel<1, 1, 1, false, true>}};
        return lean_table[c.major_a][c.major_b];
    }
    static const KernelFn table[2][2][2] = {
        {{nullptr, mx_gemm_kernel<1, 0, 1, false>}, {mx_gemm_kernel<1, 1, 0, false>, mx_gemm_kernel<1, 1, 1, false>}},
        {{nullptr, mx_gemm_kernel<2, 0, 1, false>}, {mx_gemm_kernel<2, 1, 0, false>, mx_gemm_kernel<2, 1, 1, false>}},
    };
    return table[c.cta_group - 1][c.major_a][c.major_b];
}

}  // namespace dg
