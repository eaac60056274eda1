// The step in front of a block-scaled GEMM: BF16 activations -> E4M3 with one UE8M0 scale per 32 channels, the scales
// written straight into the layout the GEMM reads (int16 [tokens, ceil(H/64)], token-major columns), so that no
// scale-factor relayout runs between the producer and the GEMM. Optionally with SwiGLU in front
// (out = silu(x[:, :H]) * x[:, H:] * weight), which is the operator between the two expert GEMMs of an MoE layer.
//
// Follows third-party/tilelang_ops/swiglu_apply_weight_to_fp8.py of the reference: clamp (:156-161), SiLU = x / (1 + e^-x)
// (:162-165; here with the fast exponential and the hardware reciprocal, each within 2 ulp of the exact operation: a value
// on a rounding boundary of E4M3 may land on the neighbouring code, and the exact division cost a third of the run time), scale = 2^ceil(log2(max(amax, 1e-4) / 448)) from the bit pattern (:80-90), values times the
// inverse scale rounded to E4M3 (:250-252), packed scales transposed per group of 32 tokens (:104-125), tokens in
// the padding of a psum layout skipped (:263-268).
//
// HBM-bound: 4 H bytes read and H + H/32 bytes written per token (2 H + H + H/32 without SwiGLU).
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/dg_b200.h"
#include "host_common.h"
#include "ptx.cuh"

namespace dg {

constexpr uint32_t kTokenGroup = 32;         // tokens per CTA: one 64-byte run of every scale column
constexpr uint32_t kQuantThreads = 256;      // 8 warps, 4 tokens each
constexpr uint32_t kTileChannels = 256;      // channels per CTA: eight per lane, eight 32-channel blocks, four scale columns
constexpr uint32_t kWarpTokens = kTokenGroup / (kQuantThreads / 32);

struct QuantArgs {
    const __nv_bfloat16* x; uint64_t x_stride;          // [tokens, (swiglu ? 2 : 1) * hidden], elements
    uint8_t* out; uint64_t out_stride;                  // [tokens, hidden] E4M3
    uint8_t* out_sf; uint64_t sf_col_stride;            // int16 [ceil(hidden/64)][sf_col_stride] seen as bytes, 2 per token
    const float* weights;                               // [tokens] or nullptr
    const int32_t* psum; uint32_t num_experts, alignment;
    uint32_t tokens, hidden;
    float clamp; uint32_t has_clamp, swiglu;
};

// End of the valid tokens of the group [token_base, token_base + 32) in the psum layout (token_base when it is all
// padding). The lanes of a warp look at 32 experts at a time, so the look-up is one round trip and not a binary search's five.
__device__ __forceinline__ uint32_t valid_end_of(const QuantArgs& a, uint32_t token_base, uint32_t end, uint32_t lane) {
    for (uint32_t e0 = 0; e0 < a.num_experts; e0 += 32) {
        const uint32_t p = e0 + lane < a.num_experts ? (uint32_t)max((int32_t)ld_stream_u32(a.psum + e0 + lane), 0) : 0u;
        const uint32_t hit = __ballot_sync(0xffffffffu, (p + a.alignment - 1) / a.alignment * a.alignment > token_base);
        if (hit != 0) return min(end, __shfl_sync(0xffffffffu, p, __ffs(hit) - 1));
    }
    return token_base;
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// One CTA = 32 tokens x 256 channels. A warp takes four tokens and issues the loads of all of them (4 or 8 x 16 bytes per
// lane) before it uses the first. Cutting the channels as well as the tokens is what gives a decoding step its parallelism:
// a CTA that ran through the whole row left 64 tokens x 7168 channels to two CTAs. Bound by HBM for many tokens, by one
// round trip to memory and the launch for few. Measured back to back: 64 x 7168 25.8 -> 1.7 us, 4096 x 7168 31 -> 12.6 us
// (7.1 TB/s), 68495 x 7168 237 -> 214 us (6.9 TB/s); SwiGLU 4096 x 2048 15.0 -> 7.9 us, 68495 x 2048 118 -> 106 us.
template <bool kSwiglu>
__global__ void __launch_bounds__(kQuantThreads) quant_fp8_kernel(const QuantArgs a) {
    __shared__ __align__(8) uint8_t sf_smem[kTokenGroup][kTileChannels / 32];
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t tiles_c = (a.hidden + kTileChannels - 1) / kTileChannels;
    const uint32_t tg = blockIdx.x / tiles_c, c0 = (blockIdx.x - tg * tiles_c) * kTileChannels;
    const uint32_t token_base = tg * kTokenGroup;
    // (may have been scheduled while the kernel that writes x is still running)
    griddep_wait();
    griddep_launch_dependents();
    uint32_t valid_end = min(a.tokens, token_base + kTokenGroup);
    if (a.psum != nullptr) valid_end = max(valid_end_of(a, token_base, valid_end, lane), token_base);
    if (valid_end <= token_base) return;                  // the whole group is padding (uniform over the CTA)

    const uint32_t c = c0 + lane * 8, t0 = token_base + warp * kWarpTokens;
    uint4 left[kWarpTokens], right[kSwiglu ? kWarpTokens : 1];
    float weight[kSwiglu ? kWarpTokens : 1];
    #pragma unroll
    for (uint32_t i = 0; i < kWarpTokens; ++i) {
        left[i] = make_uint4(0u, 0u, 0u, 0u);
        if constexpr (kSwiglu) { right[i] = left[i]; weight[i] = 1.0f; }
        if (t0 + i < valid_end && c < a.hidden) {
            const __nv_bfloat16* row = a.x + (uint64_t)(t0 + i) * a.x_stride + c;
            left[i] = ld_stream_v4(row);
            if constexpr (kSwiglu) {
                right[i] = ld_stream_v4(row + a.hidden);
                if (a.weights) weight[i] = __uint_as_float(ld_stream_u32(a.weights + t0 + i));
            }
        }
    }
    #pragma unroll
    for (uint32_t i = 0; i < kWarpTokens; ++i) {
        const uint32_t lw[4] = {left[i].x, left[i].y, left[i].z, left[i].w};
        float v[8];
        if constexpr (kSwiglu) {
            const uint32_t rw[4] = {right[i].x, right[i].y, right[i].z, right[i].w};
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                float xl[2] = {bf16_lo(lw[j]), bf16_hi(lw[j])}, xr[2] = {bf16_lo(rw[j]), bf16_hi(rw[j])};
                #pragma unroll
                for (int k = 0; k < 2; ++k) {
                    if (a.has_clamp) {
                        xl[k] = fminf(xl[k], a.clamp);
                        xr[k] = fmaxf(fminf(xr[k], a.clamp), -a.clamp);
                    }
                    const float silu = __fdividef(xl[k], 1.0f + __expf(-xl[k]));
                    float y = silu * xr[k];
                    if (a.weights) y *= weight[i];
                    v[j * 2 + k] = y;
                }
            }
        } else {
            #pragma unroll
            for (int j = 0; j < 4; ++j) { v[j * 2] = bf16_lo(lw[j]); v[j * 2 + 1] = bf16_hi(lw[j]); }
        }
        float amax = 0.f;
        #pragma unroll
        for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        // scale = max(amax, 1e-4) * (1/448) rounded up to a power of two; exponent byte from the bit pattern
        const uint32_t bits = __float_as_uint(fmaxf(amax, 1e-4f) * (1.0f / 448.0f));
        const uint32_t e = ((bits - 1u) >> 23) + 1u;
        const float inv = __uint_as_float((254u - e) << 23);
        if (t0 + i < valid_end && c < a.hidden) {
            uint32_t q[2];
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const __nv_fp8x2_storage_t p0 = __nv_cvt_float2_to_fp8x2(make_float2(v[h * 4] * inv, v[h * 4 + 1] * inv), __NV_SATFINITE, __NV_E4M3);
                const __nv_fp8x2_storage_t p1 = __nv_cvt_float2_to_fp8x2(make_float2(v[h * 4 + 2] * inv, v[h * 4 + 3] * inv), __NV_SATFINITE, __NV_E4M3);
                q[h] = (uint32_t)p0 | ((uint32_t)p1 << 16);
            }
            *reinterpret_cast<uint2*>(a.out + (uint64_t)(t0 + i) * a.out_stride + c) = make_uint2(q[0], q[1]);
        }
        // (the second block of a last, half-used scale column is zero)
        if ((lane & 3u) == 0) sf_smem[warp * kWarpTokens + i][lane / 4] = c < a.hidden ? (uint8_t)e : (uint8_t)0;
    }
    __syncthreads();
    // scale column j (int16 = channels [64 j, 64 j + 64)) of the valid tokens: one contiguous run of 2-byte elements
    const uint32_t col = threadIdx.x / kTokenGroup, tl = threadIdx.x % kTokenGroup;
    if (col < kTileChannels / 64 && c0 + col * 64 < a.hidden && tl < valid_end - token_base) {
        const uint16_t pair = *reinterpret_cast<const uint16_t*>(&sf_smem[tl][col * 2]);
        *reinterpret_cast<uint16_t*>(a.out_sf + ((uint64_t)(c0 / 64 + col) * a.sf_col_stride + token_base + tl) * 2) = pair;
    }
}

}  // namespace dg

using namespace dg;

extern "C" int dg_quant_fp8_launch(const void* x, uint64_t x_stride, uint32_t tokens, uint32_t hidden, int swiglu,
                                   const float* topk_weights, const int32_t* psum, uint32_t num_experts, uint32_t alignment,
                                   int has_clamp, float clamp_value, void* out, uint64_t out_stride,
                                   int16_t* out_sf, uint64_t sf_col_stride, void* stream) {
    DG_CHECK_ARG(x != nullptr && out != nullptr && out_sf != nullptr, "quant_fp8: null pointer");
    DG_CHECK_ARG(hidden > 0 && hidden % 32 == 0, "quant_fp8: hidden must be a multiple of 32");
    DG_CHECK_ARG((reinterpret_cast<uintptr_t>(x) & 15) == 0 && x_stride % 8 == 0,
                 "quant_fp8: input rows must start on 16-byte boundaries");
    DG_CHECK_ARG((reinterpret_cast<uintptr_t>(out) & 7) == 0 && out_stride % 8 == 0,
                 "quant_fp8: output rows must start on 8-byte boundaries");
    DG_CHECK_ARG(!swiglu || hidden % 8 == 0, "quant_fp8: hidden must be a multiple of 8");
    DG_CHECK_ARG(sf_col_stride >= tokens, "quant_fp8: scale column stride smaller than the token count");
    DG_CHECK_ARG(psum == nullptr || (num_experts > 0 && alignment > 0 && alignment % kTokenGroup == 0),
                 "quant_fp8: a psum layout needs experts and an alignment that is a multiple of 32");
    if (tokens == 0) return DG_OK;
    QuantArgs a{};
    a.x = static_cast<const __nv_bfloat16*>(x); a.x_stride = x_stride;
    a.out = static_cast<uint8_t*>(out); a.out_stride = out_stride;
    a.out_sf = reinterpret_cast<uint8_t*>(out_sf); a.sf_col_stride = sf_col_stride;
    a.weights = topk_weights; a.psum = psum; a.num_experts = psum ? num_experts : 0; a.alignment = alignment;
    a.tokens = tokens; a.hidden = hidden;
    a.clamp = clamp_value; a.has_clamp = has_clamp ? 1u : 0u; a.swiglu = swiglu ? 1u : 0u;
    const uint64_t tiles = (uint64_t)((tokens + kTokenGroup - 1) / kTokenGroup) * ((hidden + kTileChannels - 1) / kTileChannels);
    DG_CHECK_ARG(tiles <= 0x7fffffffull, "quant_fp8: too many tokens");
    const void* fn = swiglu ? (const void*)quant_fp8_kernel<true> : (const void*)quant_fp8_kernel<false>;
    void* params[] = {&a};
    if (int rc = launch_overlapped(fn, dim3((uint32_t)tiles), dim3(kQuantThreads), params, static_cast<cudaStream_t>(stream))) return rc;
    return DG_OK;
}
