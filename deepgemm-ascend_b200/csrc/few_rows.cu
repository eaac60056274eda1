// Dense FP8 x FP8 / FP8 x FP4 GEMM of a handful of rows (M <= 8) on a matrix B of at most 20 MB (few_rows_size has the rule): a
// decoding step of one or a few sequences through one projection. A CTA takes sixteen rows of B; one CTA has an SM to itself where
// they all fit, two share it where there are more, and the rest of a larger B waits for a free place.
//
// The block-scaled tensor-core kernel computes 128 rows whatever M is; to fill the chip it splits K, which costs an exchange
// of partial sums (or a second kernel), and its tensor maps want the scales of A in columns of 16-byte multiples, which M
// rows do not give, so a relayout runs in front. Here sixteen rows of B take the row side of mma.sync.m16n8k32 (K = 32 is
// exactly one scale block), the rows of A its column side, and each block's product is scaled in FP32 and added to FP32
// sums (by the sum of the two exponents where a scale of the CTA's is far from 1, see scale_by_both). Every scale is read where it lies, in any stride. One launch.
//
// Bound by latency: the launch, one round trip to memory, the bytes of a CTA's rows (115 KB at K = 7168) through one SM's port.
// So every byte of B is requested as early as shared memory allows, in row-wise bulk copies of 1 KB (copies of 256 bytes are
// bound by their number, about 26 cycles each; fragments loaded straight to registers touch eight cache lines an instruction
// and are bound by the tag look-ups), and the eight warps take an eighth of every piece of K each.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <type_traits>

#include "../../include/dg_b200.h"
#include "host_common.h"
#include "launch.h"
#include "mx_gemm.cuh"
#include "ptx.cuh"

namespace dg {

constexpr uint32_t kFewMaxRows = 8;          // rows of A
constexpr uint32_t kFewTileN = 16;           // rows of B per CTA
constexpr uint32_t kFewWarps = 8;            // they split K
constexpr uint32_t kFewPiece = 1024;         // K per slot of the ring: one row's copy is 1 KB (packed E2M1: 512 bytes)
constexpr uint32_t kFewWarpK = kFewPiece / kFewWarps;
constexpr uint32_t kFewMaxDepth = 12;
constexpr uint32_t kFewMaxSmem = 216 * 1024;
constexpr uint32_t kFewThreads = kFewWarps * 32;
constexpr uint32_t kFewMaxK = 8192;

struct FewRowsArgs {
    const uint8_t* a; uint64_t a_stride;
    const uint8_t* b; uint64_t b_stride;
    const uint16_t* sfa; uint64_t sfa_row, sfa_col;      // strides of the scales (elements between rows, between K64 columns)
    const uint16_t* sfb; uint64_t sfb_row, sfb_col;
    void* d; uint64_t d_stride;
    const void* bias;
    float alpha;
    uint32_t has_alpha, d_is_fp32;
    uint32_t m, n, k;                              // k: a multiple of 32
    uint32_t depth, a_pitch;                       // slots of the ring; bytes between rows of A in shared memory
    int32_t* status;
};

// Shared memory: the ring of B, the rows of A, the scales of both. The pitches put the eight-byte (packed E2M1: four-byte)
// fragments of a half warp (a warp) on distinct banks.
template <bool kFp4B> struct FewTile {
    static constexpr uint32_t row_bytes = kFp4B ? kFewPiece / 2 : kFewPiece;
    static constexpr uint32_t pitch = row_bytes + (kFp4B ? 16 : 32);
    static constexpr uint32_t slot = kFewTileN * pitch;
};
static uint32_t few_a_pitch(uint32_t k) { return k + (32u + 128u - k % 128u) % 128u; }
static uint32_t few_smem(bool fp4, uint32_t m, uint32_t k, uint32_t depth) {
    return depth * (fp4 ? FewTile<true>::slot : FewTile<false>::slot) + m * few_a_pitch(k) + (k + 63) / 64 * (kFewTileN + kFewMaxRows) * 2;
}

// Two UE8M0 bytes -> two BF16 powers of two (0 -> 2^-127, 255 -> NaN).
__device__ __forceinline__ uint32_t ue8m0x2_to_bf16x2(uint16_t e) {
    uint32_t v;
    asm("cvt.rn.bf16x2.ue8m0x2 %0, %1;" : "=r"(v) : "h"(e));
    return v;
}
// c = A (16 x 32, E4M3) * B (32 x 8, E4M3). A thread's four bytes of a fragment word are K elements of its choice as long as A
// and B agree: thread q of a quad holds elements 8q .. 8q + 7 of the block.
__device__ __forceinline__ void mma_e4m3_16x8x32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// Where a scale is far from 1: s * 2^(ea + eb - 254) for any two scale bytes (255: NaN), as two multiplications by a half of the exponent each: s is a sum of 32
// products, so the first one leaves the range of FP32 only where the result does.
__device__ __forceinline__ float scale_by_both(float s, uint32_t ea, uint32_t eb) {
    if (ea == 255u || eb == 255u) return __uint_as_float(0x7fffffffu);
    const int32_t e = (int32_t)(ea + eb) - 254, e1 = e >> 1, e2 = e - e1;                  // (both in [-127, 127])
    const auto pow2 = [](int32_t x) { return __uint_as_float(x < -126 ? 0x00400000u : (uint32_t)(x + 127) << 23); };
    return s * pow2(e1) * pow2(e2);
}

// kFp4B: B is packed E2M1 (expanded to E4M3 in registers, exactly).
// kLoads: scales of B a thread loads (half as many of A), 1024 of K each. Fewer for a short K; a branch around the ones it does not need
// would keep the others from being in flight together (2 rows of 1920 x 3200: 6.2 -> 7.0 us).
template <bool kFp4B, uint32_t kLoads>
__global__ void __launch_bounds__(kFewThreads) few_rows_kernel(const FewRowsArgs p) {
    using Tile = FewTile<kFp4B>;
    extern __shared__ __align__(128) uint8_t few_smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kFewMaxDepth + 1];
    __shared__ float partial[kFewWarps][kFewMaxRows][kFewTileN + 1];
    __shared__ uint32_t aborted;
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, q = lane % 4;
    const uint32_t n0 = blockIdx.x * kFewTileN;
    const uint32_t pieces = (p.k + kFewPiece - 1) / kFewPiece, units = (p.k + 63) / 64;
    const AbortFlag ab{&aborted, p.status};
    const uint32_t a_bar = smem_u32(&bars[2 * kFewMaxDepth]);
    const auto full_bar = [&](uint32_t s) { return smem_u32(&bars[s]); };
    const auto empty_bar = [&](uint32_t s) { return smem_u32(&bars[kFewMaxDepth + s]); };
    uint8_t* a_rows = few_smem_raw + p.depth * Tile::slot;
    uint16_t* sfb_smem = reinterpret_cast<uint16_t*>(a_rows + p.m * p.a_pitch);          // [K64 column][16 rows]
    uint16_t* sfa_smem = sfb_smem + units * kFewTileN;                                   // [K64 column][8 rows]
    // sixteen lanes of warp 0 fetch one row's part of a piece each (rows beyond N fetch the last one and are not stored)
    const uint8_t* src_row = p.b + (uint64_t)min(n0 + (lane & 15u), p.n - 1) * p.b_stride;
    const auto fetch = [&](uint32_t i, uint32_t s) {
        const uint32_t len = min(kFewPiece, p.k - i * kFewPiece) / (kFp4B ? 2 : 1);
        if (lane == 0) mbar_arrive_expect_tx(full_bar(s), len * kFewTileN);
        __syncwarp();
        if (lane < kFewTileN) bulk_copy_to_smem(smem_u32(few_smem_raw + s * Tile::slot + lane * Tile::pitch), src_row + (uint64_t)i * Tile::row_bytes, len, full_bar(s));
    };
    if (warp == 0) {
        if (lane == 0) {
            for (uint32_t s = 0; s < p.depth; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), kFewWarps); }
            mbar_init(a_bar, 1);
            aborted = 0;
            fence_mbar_init();
            fence_proxy_async_smem();
        }
        __syncwarp();
        griddep_wait();
        for (uint32_t i = 0; i < p.depth; ++i) {
            fetch(i, i);
            if (i == 0) {
                if (lane == 0) mbar_arrive_expect_tx(a_bar, p.m * p.k);
                __syncwarp();
                if (lane < p.m) bulk_copy_to_smem(smem_u32(a_rows + lane * p.a_pitch), p.a + lane * p.a_stride, p.k, a_bar);
            }
        }
    } else {
        griddep_wait();
    }
    griddep_launch_dependents();
    // The scales meanwhile: every load of both operands is issued before the first is used (one after the other they cost a second round
    // trip to memory, 0.7 us). Scales of rows that do not exist are 1.
    const uint16_t *const sfb = p.sfb + n0 * p.sfb_row, *const sfa = p.sfa;
    const uint32_t rows_b = min(kFewTileN, p.n - n0);
    uint16_t vb[kLoads], va[kLoads / 2];
    const auto load_scales = [&](auto& v, const uint16_t* src, uint64_t row_stride, uint64_t col_stride, uint32_t rows, auto width) {
        #pragma unroll
        for (uint32_t j = 0; j < sizeof(v) / sizeof(v[0]); ++j) {
            const uint32_t i = threadIdx.x + j * kFewThreads, r = i % width.value, col = i / width.value;
            v[j] = 0x7f7f;
            if (col < units && r < rows) v[j] = ld_global_u16(src + r * row_stride + col * col_stride);
        }
    };
    load_scales(vb, sfb, p.sfb_row, p.sfb_col, rows_b, std::integral_constant<uint32_t, kFewTileN>{});
    load_scales(va, sfa, p.sfa_row, p.sfa_col, p.m, std::integral_constant<uint32_t, kFewMaxRows>{});
    // A byte in [64, 191], no farther than 2^64 from 1, has two different top bits: `near` is the AND of that over all bytes. A block's product
    // is between 2^-18 and 2^23, so two such scales can be applied one after the other.
    uint32_t near = 0xffffu;
    const auto store_scales = [&](const auto& v, uint16_t* dst, auto width) {
        #pragma unroll
        for (uint32_t j = 0; j < sizeof(v) / sizeof(v[0]); ++j) {
            const uint32_t i = threadIdx.x + j * kFewThreads;
            // (the second byte of a last, half-used column belongs to no block)
            const uint32_t pair = i < p.k / 64 * width.value ? v[j] : (v[j] & 0xffu) | 0x7f00u;
            near &= pair ^ (pair << 1);
            if (i < units * width.value) dst[i] = v[j];
        }
    };
    store_scales(vb, sfb_smem, std::integral_constant<uint32_t, kFewTileN>{});
    store_scales(va, sfa_smem, std::integral_constant<uint32_t, kFewMaxRows>{});
    const bool any_far = __syncthreads_or((near & 0x8080u) != 0x8080u);

    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    uint32_t fetched = p.depth;                        // pieces requested so far
    bool ok = wait_barrier(a_bar, 0, ab, kStatusTimeoutProducer);
    // (a loop for each way of scaling: a branch between two blocks would keep their products from overlapping, 2112 x 7168 9.6 -> 12.3 us)
    const auto run_pieces = [&](auto far_tag) {
        uint32_t slot = 0, phase = 0;
        for (uint32_t i = 0; ok && i < pieces; ++i) {
            if (!(ok = wait_barrier(full_bar(slot), phase, ab, kStatusTimeoutProducer))) break;
            const uint32_t k0 = i * kFewPiece + warp * kFewWarpK;               // this warp's part of the piece
            const uint8_t* w = few_smem_raw + slot * Tile::slot + g * Tile::pitch + (warp * kFewWarpK + q * 8) / (kFp4B ? 2 : 1);
            const uint8_t* x = a_rows + g * p.a_pitch + k0 + q * 8;
            #pragma unroll
            for (uint32_t u = 0; u < kFewWarpK / 64; ++u) {
                if (k0 + u * 64 >= p.k) continue;                               // (uniform)
                const uint16_t* sw = sfb_smem + (k0 / 64 + u) * kFewTileN + g;
                const uint16_t* sx = sfa_smem + (k0 / 64 + u) * kFewMaxRows + 2 * q;
                const uint32_t fw0 = ue8m0x2_to_bf16x2(sw[0]), fw1 = ue8m0x2_to_bf16x2(sw[8]);
                const uint32_t fx0 = ue8m0x2_to_bf16x2(sx[0]), fx1 = ue8m0x2_to_bf16x2(sx[1]);
                #pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    const uint32_t blk = 2 * u + h;
                    if (k0 + blk * 32 >= p.k) continue;                         // (uniform)
                    const uint2 xv = g < p.m ? *reinterpret_cast<const uint2*>(x + blk * 32) : make_uint2(0u, 0u);
                    float s[4];
                    if constexpr (kFp4B) {
                        const uint32_t lo = *reinterpret_cast<const uint32_t*>(w + blk * 16), hi = *reinterpret_cast<const uint32_t*>(w + 8 * Tile::pitch + blk * 16);
                        mma_e4m3_16x8x32(s, e2m1x4_to_e4m3x4(lo), e2m1x4_to_e4m3x4(hi), e2m1x4_to_e4m3x4(lo >> 16), e2m1x4_to_e4m3x4(hi >> 16), xv.x, xv.y);
                    } else {
                        const uint2 lo = *reinterpret_cast<const uint2*>(w + blk * 32), hi = *reinterpret_cast<const uint2*>(w + 8 * Tile::pitch + blk * 32);
                        mma_e4m3_16x8x32(s, lo.x, hi.x, lo.y, hi.y, xv.x, xv.y);
                    }
                    if constexpr (decltype(far_tag)::value) {
                        const auto byte = [h](uint32_t v) { return (v >> (8 * h)) & 0xffu; };
                        acc[0] += scale_by_both(s[0], byte(sx[0]), byte(sw[0]));
                        acc[1] += scale_by_both(s[1], byte(sx[1]), byte(sw[0]));
                        acc[2] += scale_by_both(s[2], byte(sx[0]), byte(sw[8]));
                        acc[3] += scale_by_both(s[3], byte(sx[1]), byte(sw[8]));
                    } else {
                        const auto half = [h](uint32_t v) { return __uint_as_float(h ? v & 0xffff0000u : v << 16); };
                        acc[0] += (s[0] * half(fx0)) * half(fw0);
                        acc[1] += (s[1] * half(fx1)) * half(fw0);
                        acc[2] += (s[2] * half(fx0)) * half(fw1);
                        acc[3] += (s[3] * half(fx1)) * half(fw1);
                    }
                }
            }
            if (i + p.depth < pieces) {                                          // the slot is needed again
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_bar(slot));
                if (warp == 0) {
                    if (!(ok = wait_barrier(empty_bar(slot), phase, ab, kStatusTimeoutProducer))) break;
                    __syncwarp();
                    fetch(i + p.depth, slot);
                    ++fetched;
                }
            }
            if (++slot == p.depth) { slot = 0; phase ^= 1; }
        }
    };
    if (__builtin_expect(any_far, 0)) run_pieces(std::true_type{});
    else run_pieces(std::false_type{});
    if (warp == 0 && !ok) {
        // A wait gave up: what has been requested must not land in shared memory that belongs to another CTA by then.
        const auto landed = [&](uint32_t bar, uint32_t parity, uint64_t t0) {
            while (!mbar_try_wait(bar, parity)) if (global_timer_ns() - t0 > kWaitTimeoutNs) return;
        };
        const uint64_t t0 = global_timer_ns();
        landed(a_bar, 0, t0);
        for (uint32_t s = 0; s < p.depth; ++s) landed(full_bar(s), ((fetched - s + p.depth - 1) / p.depth - 1) & 1u, t0);
    }
    partial[warp][2 * q][g] = acc[0];
    partial[warp][2 * q + 1][g] = acc[1];
    partial[warp][2 * q][g + 8] = acc[2];
    partial[warp][2 * q + 1][g + 8] = acc[3];
    __syncthreads();
    const uint32_t row = threadIdx.x / kFewTileN, col = threadIdx.x % kFewTileN;
    if (row < p.m && n0 + col < p.n && !ab.raised()) {
        float sum = 0.f;
        #pragma unroll
        for (uint32_t w = 0; w < kFewWarps; ++w) sum += partial[w][row][col];
        if (p.has_alpha) sum *= p.alpha;
        const uint64_t at = (uint64_t)row * p.d_stride + n0 + col;
        if (p.d_is_fp32) {
            if (p.bias != nullptr) sum += __uint_as_float(ld_global_u32(reinterpret_cast<const float*>(p.bias) + n0 + col));
            reinterpret_cast<float*>(p.d)[at] = sum;
        } else {
            if (p.bias != nullptr) sum += __uint_as_float((uint32_t)ld_global_u16(reinterpret_cast<const uint16_t*>(p.bias) + n0 + col) << 16);
            reinterpret_cast<__nv_bfloat16*>(p.d)[at] = __float2bfloat16_rn(sum);
        }
    }
}

// Where this kernel is the faster one: us of this one / of the block-scaled kernel, 1 and 8 rows, packed scales. (Below 8 rows the other
// kernel needs its scales of A relaid, 1.2 us; FP32 scales are relaid in front of either, and lie between the two columns.)
//   E4M3, K <= 4096      512 x 512 2.7 / 5.4, 2.9 / 4.0     4096 x 4096 8.0 / 13.9, 8.3 / 12.1    7168 x 2048 8.2 / 10.1, 7.8 / 8.7
//     many CTAs          9472 x 2048 8.8 / 10.4, 8.4 / 9.5  10240 x 2048 9.3 / 10.9, 11.2 / 9.4   16384 x 1024 8.5 / 9.4, 9.2 / 7.6
//                        9472 x 512 4.3 / 6.1, 4.6 / 5.1    12288 x 512 5.8 / 6.3, 6.6 / 5.0      16384 x 512 7.0 / 6.7, 7.6 / 5.4
//   E4M3, longer K       1024 x 6144 8.1 / 8.8, 8.3 / 8.5   1536 x 7168 9.9 / 10.1, 10.1 / 9.6    1024 x 8192 10.1 / 8.8, 10.4 / 8.7
//                        2112 x 7168 9.9 / 12.5, 10.2 / 10.5                                      2500 x 8192 13.5 / 14.9, 14.2 / 13.8
// An SM takes a CTA's 16 rows of B in no faster however few CTAs there are, and five CTAs share one at most. E2M1: 2368 x 4096 6.8 / 13.1,
// 7.1 / 11.4, and not 7168 x 2048 10.4 / 8.5, 2112 x 7168 10.9 / 10.5: the codes cost this kernel as long as whole bytes and the other
// half as long.
static bool few_rows_size(uint32_t m, uint32_t n, uint32_t k, bool fp4) {
    static_assert(kFewMaxK == 8192, "the rule stays inside it");
    if (few_smem(fp4, m, k, 1) > kFewMaxSmem) return false;
    if (fp4) return k <= 4096 && n <= 148 * kFewTileN;
    if ((uint64_t)n * k > (20ull << 20)) return false;
    if (k > 4096) return k <= 7168 ? n >= 1024 : k <= kFewMaxK && n >= 2048;
    if (m == kFewMaxRows) return n <= 4 * 148 * kFewTileN;         // (four CTAs per SM)
    return n <= (k <= 512 ? 12288 : k <= 1024 ? 16384 : 10240);
}

bool takes_few_rows(const dg_gemm_desc_t& d) {
    return d.gemm_type == DG_GEMM_NORMAL && d.m >= 1 && d.m <= kFewMaxRows && d.n > 0 && d.k > 0 && d.k % 32 == 0 &&
           d.a_dtype == DG_E4M3 && (d.b_dtype == DG_E4M3 || d.b_dtype == DG_E2M1X2) && d.major_a == DG_MAJOR_K && d.major_b == DG_MAJOR_K &&
           (d.d_dtype == DG_BF16 || d.d_dtype == DG_F32) && !d.accumulate &&
           (d.epilogue == DG_EPILOGUE_IDENTITY || d.epilogue == DG_EPILOGUE_ALPHA || d.epilogue == DG_EPILOGUE_BIAS) &&
           few_rows_size(d.m, d.n, d.k, d.b_dtype == DG_E2M1X2);
}

int launch_few_rows(const dg_gemm_desc_t& d, uint64_t sfa_row_stride, uint64_t sfb_row_stride, cudaStream_t stream) {
    FewRowsArgs p{};
    p.a = static_cast<const uint8_t*>(d.a); p.a_stride = d.outer_stride_a;
    p.b = static_cast<const uint8_t*>(d.b); p.b_stride = d.outer_stride_b;
    p.sfa = reinterpret_cast<const uint16_t*>(d.sfa); p.sfa_row = sfa_row_stride; p.sfa_col = d.sfa_stride;
    p.sfb = reinterpret_cast<const uint16_t*>(d.sfb); p.sfb_row = sfb_row_stride; p.sfb_col = d.sfb_stride;
    p.d = d.d; p.d_stride = d.outer_stride_d;
    p.bias = d.epilogue == DG_EPILOGUE_BIAS ? d.bias : nullptr;
    p.has_alpha = d.epilogue == DG_EPILOGUE_ALPHA ? 1u : 0u; p.alpha = d.alpha;
    p.d_is_fp32 = d.d_dtype == DG_F32 ? 1u : 0u;
    p.m = d.m; p.n = d.n; p.k = d.k;
    p.a_pitch = few_a_pitch(d.k);
    const bool fp4 = d.b_dtype == DG_E2M1X2;
    const uint32_t grid = (d.n + kFewTileN - 1) / kFewTileN, pieces = (d.k + kFewPiece - 1) / kFewPiece;
    // one CTA per SM: everything in flight that fits; more: half of that, so that two CTAs share an SM
    p.depth = pieces < kFewMaxDepth ? pieces : kFewMaxDepth;
    while (p.depth > 1 && few_smem(fp4, d.m, d.k, p.depth) > (grid <= 148 ? kFewMaxSmem : kFewMaxSmem / 2)) --p.depth;
    if (int rc = get_status_pointer(&p.status)) return rc;
    static_assert(kFewTileN * 1024 / 64 == kFewThreads && kFewMaxRows * 2 == kFewTileN, "one load a thread for 1024 of K");
    static const void* const kernels[2][3] = {
        {(const void*)few_rows_kernel<false, 2>, (const void*)few_rows_kernel<false, 4>, (const void*)few_rows_kernel<false, 8>},
        {(const void*)few_rows_kernel<true, 2>, (const void*)few_rows_kernel<true, 4>, nullptr},           // (K <= 4096)
    };
    const uint32_t which = d.k <= 2048 ? 0 : d.k <= 4096 ? 1 : 2;
    const void* fn = kernels[fp4][which];
    DG_CHECK_ARG(d.k <= kFewMaxK && fn != nullptr, "not a problem of a few rows: K is too large");
    // (raised once per device and kernel to the most a launch can ask for)
    {
        static std::mutex mu;
        static bool raised[2][3][64] = {};
        int dev = 0;
        DG_CHECK_CUDA(cudaGetDevice(&dev));
        DG_CHECK_ARG(dev >= 0 && dev < 64, "device index out of range");
        std::lock_guard<std::mutex> lock(mu);
        if (!raised[fp4][which][dev]) {
            DG_CHECK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFewMaxSmem));
            raised[fp4][which][dev] = true;
        }
    }
    void* params[] = {&p};
    return launch_overlapped(fn, dim3(grid), dim3(kFewThreads), params, stream, few_smem(fp4, d.m, d.k, p.depth));
}

}  // namespace dg
