// Instantiations of the GEMM kernel: 8-bit operands of which at least one is MN-major.
#include "launch.h"
#include "mx_gemm.cuh"

namespace dg {

template <bool kOverlap, int kMajorA, int kMajorB>
static KernelFn pick_generic(bool pair) {
    return pair ? mx_gemm_kernel<2, kMajorA, kMajorB, false, false, false, false, false, false, false, false, false, kOverlap>
                : mx_gemm_kernel<1, kMajorA, kMajorB, false, false, false, false, false, false, false, false, false, kOverlap>;
}
template <bool kOverlap>
static KernelFn pick_generic(const KernelChoice& c) {
    const bool pair = c.cta_group == 2;
    if (c.major_a == 0) return pick_generic<kOverlap, 0, 1>(pair);
    return c.major_b == 0 ? pick_generic<kOverlap, 1, 0>(pair) : pick_generic<kOverlap, 1, 1>(pair);
}

KernelFn pick_mn_major_kernel(const KernelChoice& c) {
    if (c.lean) {
        static const KernelFn lean_table[2][2] = {{nullptr, mx_gemm_kernel<1, 0, 1, false, true>},
                                                  {mx_gemm_kernel<1, 1, 0, false, true>, mx_gemm_kernel<1, 1, 1, false, true>}};
        return lean_table[c.major_a][c.major_b];
    }
    return c.overlap ? pick_generic<true>(c) : pick_generic<false>(c);
}

}  // namespace dg
