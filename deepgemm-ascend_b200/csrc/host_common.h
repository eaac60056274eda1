// Host-side helpers shared by the translation units of libdg_b200.so: the status codes of the C ABI,
// the per-thread error message, and argument / CUDA checks that return instead of throwing.
#pragma once

#include <cuda_runtime.h>
#include <cstdarg>
#include <cstdio>

#include "../../include/dg_b200.h"

namespace dg {

void set_last_error(const char* fmt, ...);
void count_kernel_launch(unsigned n = 1);
// Are kernels launched with programmatic stream serialisation (see mx_gemm.cu)?
bool overlap_launches_enabled();

// Launch of a kernel that starts with griddepcontrol.wait: it may be scheduled while the kernel in front of it in the stream is
// still draining.
inline int launch_overlapped(const void* fn, dim3 grid, dim3 block, void** params, cudaStream_t stream, uint32_t smem_bytes = 0) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap_launches_enabled() ? 1 : 0;
    const cudaError_t err = cudaLaunchKernelExC(&cfg, fn, params);
    if (err != cudaSuccess) {
        set_last_error("CUDA error %d (%s) at a kernel launch", (int)err, cudaGetErrorString(err));
        return DG_ERR_CUDA;
    }
    count_kernel_launch();
    return DG_OK;
}

}  // namespace dg

#define DG_CHECK_ARG(cond, ...)                      \
    do {                                             \
        if (!(cond)) {                               \
            dg::set_last_error(__VA_ARGS__);         \
            return DG_ERR_INVALID;                   \
        }                                            \
    } while (0)

#define DG_UNSUPPORTED(cond, ...)                    \
    do {                                             \
        if (cond) {                                  \
            dg::set_last_error(__VA_ARGS__);         \
            return DG_ERR_UNSUPPORTED;               \
        }                                            \
    } while (0)

#define DG_CHECK_CUDA(expr)                                                                  \
    do {                                                                                     \
        cudaError_t err__ = (expr);                                                          \
        if (err__ != cudaSuccess) {                                                          \
            dg::set_last_error("CUDA error %d (%s) at %s:%d", (int)err__,                    \
                               cudaGetErrorString(err__), __FILE__, __LINE__);               \
            return DG_ERR_CUDA;                                                              \
        }                                                                                    \
    } while (0)
