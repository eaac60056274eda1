// Dense FP8 x FP8 / FP8 x FP4 GEMM of up to 16 rows on a matrix B of at most 64 MB (few_rows_size has the rule): a decoding step of a few
// sequences through one projection. A CTA takes sixteen rows of B; one CTA has an SM to itself where they all fit, two or more share it where there
// are more (three_share_an_sm), and the rest of a larger B waits for a free place.
//
// The block-scaled tensor-core kernel computes 128 rows whatever M is; to fill the chip it splits K, which costs an exchange
// of partial sums (or a second kernel), and its tensor maps want the scales of A in columns of 16-byte multiples, which M
// rows do not give, so a relayout runs in front. Here sixteen rows of B take the row side of mma.sync, eight rows of A its column side,
// two instructions make one scale block of K = 32, and each block's product is scaled in FP32 and added to FP32
// sums (by the sum of the two exponents where a scale of the CTA's is far from 1, see scale_by_both). Every scale is read where it lies, in any stride. One launch.
//
// Bound by latency: the launch, one round trip to memory, the bytes of a CTA's rows (115 KB at K = 7168) through one SM's port and then through
// its shared memory (eight passes of 128 bytes for a block of 16 x 32, of which B itself is four). So every byte of B is requested as early as
// shared memory allows (two slots or more, but for the sizes that with_few_tile names), in row-wise bulk copies of 1 to 4 KB issued by all warps at once, L2 is asked for the first of them before the wait for the
// kernel in front, and all warps take a part of every piece of K. One row of 2112 x 7168: 9.9 -> 5.4 us back to back (2.8 TB/s), 4096 x 4096 8.0 -> 5.0.
// (One warp that issued every copy needed 8000 cycles for them, and waits, branches between blocks and conversions of the scales made 1000 cycles of a KB of K.)
// Smaller copies are bound by their number; fragments loaded straight to registers touch eight cache lines an instruction and are bound by the tag look-ups.
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

constexpr uint32_t kFewMaxRows = 16;         // rows of A
constexpr uint32_t kFewTileN = 16;           // rows of B per CTA
constexpr uint32_t kFewMaxDepth = 12;
constexpr uint32_t kFewMaxSmem = 208 * 1024;          // (dynamic; the partial sums of 16 warps and 16 rows are 17 KB more)
constexpr uint32_t kFewMaxK = 16384;

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

// What is fixed per instantiation. A CTA's warps split K: warp w takes the K64 units w, w + kWarps, ... of every piece of B.
template <bool kFp4B_, uint32_t kWarps_, uint32_t kPiece_, uint32_t kMaxK_, uint32_t kRows_ = 8>
struct FewTile {
    static constexpr bool kFp4B = kFp4B_;                                          // B is packed E2M1 (expanded to E4M3 in registers, exactly)
    static constexpr uint32_t kWarps = kWarps_, kThreads = kWarps * 32;
    static constexpr uint32_t kPiece = kPiece_;                                    // K per slot of the ring
    static constexpr uint32_t kMaxK = kMaxK_;
    static constexpr uint32_t kRows = kRows_, kColumns = kRows / 8;                // rows of A at most: 8 or 16, one or two column sides of the MMA
    static constexpr uint32_t kRowsPerWarp = kFewTileN / kWarps;                   // of B, whose copies this warp issues
    static constexpr uint32_t kUnits = kPiece / 64 / kWarps;                       // of a warp in a whole piece
    static constexpr uint32_t kUnitBytes = kFp4B ? 32 : 64;
    // The pitch puts the eight-byte (packed E2M1: four-byte) fragments of a half warp (a warp) on distinct banks.
    static constexpr uint32_t kRowBytes = kFp4B ? kPiece / 2 : kPiece;
    static constexpr uint32_t kPitch = kRowBytes + (kFp4B ? 16 : 32);
    static constexpr uint32_t kSlot = kFewTileN * kPitch;
    // scales a thread loads (a fixed number: a branch around the ones it does not need would keep the others from being in flight together)
    static constexpr uint32_t kLoadsB = (kMaxK / 64 * kFewTileN + kThreads - 1) / kThreads, kLoadsA = (kMaxK / 64 * kRows + kThreads - 1) / kThreads;
    static constexpr uint32_t kStaticSmem = kWarps * kRows * (kFewTileN + 1) * 4 + (2 * kFewMaxDepth + 1) * 8 + 8;      // (partial sums, barriers, flag)
};
static uint32_t few_a_pitch(uint32_t k) { return k + (32u + 128u - k % 128u) % 128u; }
// Shared memory: the ring of B, the rows of A, the scales of both (a word for two blocks of a row).
template <class Tile> static uint32_t few_smem(uint32_t m, uint32_t k, uint32_t depth) {
    return depth * Tile::kSlot + m * few_a_pitch(k) + (k + 63) / 64 * (kFewTileN + Tile::kRows) * 4;
}

// Four E4M3 codes -> two pairs of FP16, exactly: elements (0, 1) and (2, 3).
__device__ __forceinline__ uint2 e4m3x4_to_f16x4(uint32_t codes) {
    uint2 v;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(v.x) : "h"((uint16_t)codes));
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(v.y) : "h"((uint16_t)(codes >> 16)));
    return v;
}
// c = A (16 x 32) * B (32 x 8), E4M3 codes multiplied as FP16 (every E4M3 value is an FP16 value), summed in FP32. Which K elements a thread's words
// hold is its own choice as long as A and B agree: thread q of a quad holds elements 8q .. 8q + 7 of the block. (The E4M3 form of the instruction
// takes 2 % longer than this at 2112 x 7168.)
__device__ __forceinline__ void mma_16x8x32(float (&c)[4], uint2 a_row, uint2 a_row8, uint2 b) {
    const uint2 a0 = e4m3x4_to_f16x4(a_row.x), a1 = e4m3x4_to_f16x4(a_row8.x), a2 = e4m3x4_to_f16x4(a_row.y), a3 = e4m3x4_to_f16x4(a_row8.y);
    const uint2 b0 = e4m3x4_to_f16x4(b.x), b1 = e4m3x4_to_f16x4(b.y);
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0.x), "r"(a1.x), "r"(a0.y), "r"(a1.y), "r"(b0.x), "r"(b0.y), "f"(0.f));
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a2.x), "r"(a3.x), "r"(a2.y), "r"(a3.y), "r"(b1.x), "r"(b1.y));
}

// Where a scale is far from 1: s * 2^(ea + eb - 254) for any two scale bytes (255: NaN), as two multiplications by a half of the exponent each: s is a sum of 32
// products, so the first one leaves the range of FP32 only where the result does.
__device__ __forceinline__ float scale_by_both(float s, uint32_t ea, uint32_t eb) {
    if (ea == 255u || eb == 255u) return __uint_as_float(0x7fffffffu);
    const int32_t e = (int32_t)(ea + eb) - 254, e1 = e >> 1, e2 = e - e1;                  // (both in [-127, 127])
    const auto pow2 = [](int32_t x) { return __uint_as_float(x < -126 ? 0x00400000u : (uint32_t)(x + 127) << 23); };
    return s * pow2(e1) * pow2(e2);
}

template <class Tile>
__global__ void __launch_bounds__(Tile::kThreads) few_rows_kernel(const FewRowsArgs p) {
    constexpr bool kFp4B = Tile::kFp4B;
    extern __shared__ __align__(128) uint8_t few_smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kFewMaxDepth + 1];
    __shared__ float partial[Tile::kWarps][Tile::kRows][kFewTileN + 1];
    __shared__ uint32_t aborted;
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, q = lane % 4;
    const uint32_t n0 = blockIdx.x * kFewTileN;
    const uint32_t pieces = (p.k + Tile::kPiece - 1) / Tile::kPiece, units = (p.k + 63) / 64;
    const AbortFlag ab{&aborted, p.status};
    const uint32_t a_bar = smem_u32(&bars[2 * kFewMaxDepth]);
    const auto full_bar = [&](uint32_t s) { return smem_u32(&bars[s]); };
    const auto empty_bar = [&](uint32_t s) { return smem_u32(&bars[kFewMaxDepth + s]); };
    uint8_t* a_rows = few_smem_raw + p.depth * Tile::kSlot;
    uint32_t* sfb_smem = reinterpret_cast<uint32_t*>(a_rows + p.m * p.a_pitch);          // [K64 column][8 pairs of rows g, g + 8]
    uint32_t* sfa_smem = sfb_smem + units * kFewTileN;                                   // [K64 column][rows of A]
    const auto piece_bytes = [&](uint32_t i) { return min(Tile::kPiece, p.k - i * Tile::kPiece) / (kFp4B ? 2 : 1); };
    // (rows beyond N fetch the last one and are not stored)
    const auto row_of_b = [&](uint32_t r) { return p.b + (uint64_t)min(n0 + r, p.n - 1) * p.b_stride; };
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < p.depth; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), Tile::kWarps); }
        mbar_init(a_bar, 1);
        aborted = 0;
        fence_mbar_init();
        fence_proxy_async_smem();
        for (uint32_t s = 0; s < p.depth; ++s) mbar_arrive_expect_tx(full_bar(s), piece_bytes(s) * kFewTileN);
        mbar_arrive_expect_tx(a_bar, p.m * p.k);
    }
    __syncthreads();
    const uint8_t* const src_b = row_of_b(Tile::kRowsPerWarp * warp + lane % Tile::kRowsPerWarp);
    const uint32_t dst_b = smem_u32(few_smem_raw + (Tile::kRowsPerWarp * warp + lane % Tile::kRowsPerWarp) * Tile::kPitch);
    const uint16_t *const sfb = p.sfb + n0 * p.sfb_row, *const sfa = p.sfa;
    const uint32_t rows_b = min(kFewTileN, p.n - n0);
    // While the kernel in front is still finishing, L2 is asked for the first 2 KB of every row of B and for the rows' scales: weights, as a rule, and
    // whatever that kernel still writes to them reaches L2 as well. (2112 x 7168: 6.2 -> 5.9 us for B, 5.4 with the scales; 4 KB and all of a
    // row are slower again where all SMs are busy, 7.0: they hold up the other kernel's last loads.)
    if (lane < Tile::kRowsPerWarp) bulk_prefetch_l2(src_b, min(2048u, kFp4B ? p.k / 2 : p.k));
    for (uint32_t col = threadIdx.x; col < units; col += Tile::kThreads) prefetch_l2(sfb + col * p.sfb_col);
    griddep_wait();
    griddep_launch_dependents();
    // Every load of both operands' scales is issued before the first is used (one after the other they cost a second round
    // trip to memory, 0.7 us). Scales of rows that do not exist are 1.
    uint16_t vb[Tile::kLoadsB], va[Tile::kLoadsA];
    const auto load_scales = [&](auto& v, const uint16_t* src, uint64_t row_stride, uint64_t col_stride, uint32_t rows, auto width) {
        #pragma unroll
        for (uint32_t j = 0; j < sizeof(v) / sizeof(v[0]); ++j) {
            const uint32_t i = threadIdx.x + j * Tile::kThreads, r = i % width.value, col = i / width.value;
            v[j] = 0x7f7f;
            if (col < units && r < rows) v[j] = ld_global_u16(src + r * row_stride + col * col_stride);
        }
    };
    const auto load_all_scales = [&] {
        load_scales(vb, sfb, p.sfb_row, p.sfb_col, rows_b, std::integral_constant<uint32_t, kFewTileN>{});
        load_scales(va, sfa, p.sfa_row, p.sfa_col, p.m, std::integral_constant<uint32_t, Tile::kRows>{});
    };
    // (with sixteen warps a warp has one copy to issue in front and twice as many warps ask for scales: 2112 x 7168 5.4 us with the copies first, 5.6 with
    // the scales first; with eight it is the other way round, 7168 x 2048 5.7 and 5.0)
    if constexpr (Tile::kWarps == 8) load_all_scales();
    // A warp's copies are issued one after the other, about 100 cycles each, so every warp issues those of its own rows, a lane each.
    if (lane < Tile::kRowsPerWarp) bulk_copy_to_smem(dst_b, src_b, piece_bytes(0), full_bar(0));
    else if (const uint32_t r = warp + (lane - Tile::kRowsPerWarp) * Tile::kWarps; lane < Tile::kRowsPerWarp + 2 && r < p.m)
        bulk_copy_to_smem(smem_u32(a_rows + r * p.a_pitch), p.a + r * p.a_stride, p.k, a_bar);
    __syncwarp();
    if constexpr (Tile::kWarps != 8) load_all_scales();
    if (lane < Tile::kRowsPerWarp) {
        for (uint32_t i = 1; i < p.depth; ++i) bulk_copy_to_smem(dst_b + i * Tile::kSlot, src_b + (uint64_t)i * Tile::kRowBytes, piece_bytes(i), full_bar(i));
    }
    __syncwarp();
    // A byte in [64, 191], no farther than 2^64 from 1, has two different top bits: `near` is the AND of that over all bytes. A block's product
    // is between 2^-18 and 2^23, so two such scales can be applied one after the other.
    uint32_t near = 0xffffu;
    const auto store_scales = [&](const auto& v, uint32_t* dst, auto width, auto place) {
        #pragma unroll
        for (uint32_t j = 0; j < sizeof(v) / sizeof(v[0]); ++j) {
            const uint32_t i = threadIdx.x + j * Tile::kThreads;
            // (the second byte of a last, half-used column belongs to no block)
            const uint32_t pair = i < p.k / 64 * width.value ? v[j] : (v[j] & 0xffu) | 0x7f00u;
            near &= pair ^ (pair << 1);
            if (i < units * width.value) dst[place(i)] = ((uint32_t)(v[j] & 0xffu) << 7) | ((uint32_t)(v[j] >> 8) << 23);      // two BF16 powers of two
        }
    };
    store_scales(vb, sfb_smem, std::integral_constant<uint32_t, kFewTileN>{}, [](uint32_t i) { return (i & ~15u) | ((i & 7u) << 1) | ((i >> 3) & 1u); });
    store_scales(va, sfa_smem, std::integral_constant<uint32_t, Tile::kRows>{}, [](uint32_t i) { return i; });
    const bool any_far = __syncthreads_or((near & 0x8080u) != 0x8080u);

    float acc[Tile::kColumns][4] = {};
    uint32_t fetched = p.depth;                        // pieces this warp has requested its rows of
    bool ok = wait_barrier(a_bar, 0, ab, kStatusTimeoutProducer);
    const uint2* const scales_b = reinterpret_cast<const uint2*>(sfb_smem) + g;
    const uint2* const scales_a = reinterpret_cast<const uint2*>(sfa_smem) + q;
    const uint8_t* x_row[Tile::kColumns];                                                 // (columns of rows that do not exist are not stored)
    #pragma unroll
    for (uint32_t c = 0; c < Tile::kColumns; ++c) x_row[c] = a_rows + min(8 * c + g, p.m - 1) * p.a_pitch + q * 8;
    // One K64 unit, two blocks (or the one that is left of it), from the warp's words of B at w.
    const auto multiply = [&](auto far_tag, auto blocks, const uint8_t* w, uint32_t k) {
        const uint2 sw = scales_b[k / 64 * (kFewTileN / 2)];
        uint2 sx[Tile::kColumns];
        #pragma unroll
        for (uint32_t c = 0; c < Tile::kColumns; ++c) sx[c] = scales_a[k / 64 * (Tile::kRows / 2) + 4 * c];
        #pragma unroll
        for (uint32_t h = 0; h < blocks.value; ++h) {
            uint2 lo, hi;
            if constexpr (kFp4B) {
                const uint32_t l = *reinterpret_cast<const uint32_t*>(w + h * 16), u = *reinterpret_cast<const uint32_t*>(w + 8 * Tile::kPitch + h * 16);
                lo = make_uint2(e2m1x4_to_e4m3x4(l), e2m1x4_to_e4m3x4(l >> 16));
                hi = make_uint2(e2m1x4_to_e4m3x4(u), e2m1x4_to_e4m3x4(u >> 16));
            } else {
                lo = *reinterpret_cast<const uint2*>(w + h * 32);
                hi = *reinterpret_cast<const uint2*>(w + 8 * Tile::kPitch + h * 32);
            }
            #pragma unroll
            for (uint32_t c = 0; c < Tile::kColumns; ++c) {
                float s[4];
                mma_16x8x32(s, lo, hi, *reinterpret_cast<const uint2*>(x_row[c] + k + h * 32));
                if constexpr (decltype(far_tag)::value) {
                    const auto byte = [h](uint32_t v) { return (v >> (h ? 23 : 7)) & 0xffu; };
                    acc[c][0] += scale_by_both(s[0], byte(sx[c].x), byte(sw.x));
                    acc[c][1] += scale_by_both(s[1], byte(sx[c].y), byte(sw.x));
                    acc[c][2] += scale_by_both(s[2], byte(sx[c].x), byte(sw.y));
                    acc[c][3] += scale_by_both(s[3], byte(sx[c].y), byte(sw.y));
                } else {
                    const auto pow2 = [h](uint32_t v) { return __uint_as_float(h ? v & 0xffff0000u : v << 16); };
                    acc[c][0] += (s[0] * pow2(sx[c].x)) * pow2(sw.x);
                    acc[c][1] += (s[1] * pow2(sx[c].y)) * pow2(sw.x);
                    acc[c][2] += (s[2] * pow2(sx[c].x)) * pow2(sw.y);
                    acc[c][3] += (s[3] * pow2(sx[c].y)) * pow2(sw.y);
                }
            }
        }
    };
    const std::integral_constant<uint32_t, 1> one_block{};
    const std::integral_constant<uint32_t, 2> two_blocks{};
    // (a loop for each way of scaling, and straight code for whole pieces: a branch between two units keeps their products from overlapping)
    const auto run_pieces = [&](auto far_tag) {
        uint32_t slot = 0, phase = 0;
        for (uint32_t i = 0; ok && i < pieces; ++i) {
            if (!(ok = wait_barrier(full_bar(slot), phase, ab, kStatusTimeoutProducer))) break;
            const uint32_t k0 = i * Tile::kPiece + warp * 64;
            const uint8_t* const w = few_smem_raw + slot * Tile::kSlot + g * Tile::kPitch + warp * Tile::kUnitBytes + q * (kFp4B ? 4 : 8);
            const auto at = [&](uint32_t u) { return w + u * Tile::kWarps * Tile::kUnitBytes; };
            if (!decltype(far_tag)::value && (i + 1) * Tile::kPiece <= p.k) {
                #pragma unroll
                for (uint32_t u = 0; u < Tile::kUnits; ++u) multiply(far_tag, two_blocks, at(u), k0 + u * Tile::kWarps * 64);
            } else {
                #pragma unroll 1
                for (uint32_t u = 0; u < Tile::kUnits; ++u) {
                    const uint32_t k = k0 + u * Tile::kWarps * 64;
                    if (k + 64 <= p.k) multiply(far_tag, two_blocks, at(u), k);
                    else if (k < p.k) multiply(far_tag, one_block, at(u), k);
                }
            }
            if (i + p.depth < pieces) {                                          // the slot is needed again: every warp fetches its rows
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_bar(slot));
                if (!(ok = wait_barrier(empty_bar(slot), phase, ab, kStatusTimeoutProducer))) break;
                __syncwarp();
                const uint32_t len = piece_bytes(i + p.depth);
                if (threadIdx.x == 0) mbar_arrive_expect_tx(full_bar(slot), len * kFewTileN);
                if (lane < Tile::kRowsPerWarp) bulk_copy_to_smem(dst_b + slot * Tile::kSlot, src_b + (uint64_t)(i + p.depth) * Tile::kRowBytes, len, full_bar(slot));
                ++fetched;
            }
            if (++slot == p.depth) { slot = 0; phase ^= 1; }
        }
    };
    if (__builtin_expect(any_far, 0)) run_pieces(std::true_type{});
    else run_pieces(std::false_type{});
    if (!ok) {
        // A wait gave up: what this warp has requested must not land in shared memory that belongs to another CTA by then. (A piece that other warps
        // have not requested never completes: the limit then is longer than any copy takes.)
        const auto landed = [&](uint32_t bar, uint32_t parity, uint64_t t0) {
            while (!mbar_try_wait(bar, parity)) if (global_timer_ns() - t0 > kWaitTimeoutNs) return;
        };
        const uint64_t t0 = global_timer_ns();
        landed(a_bar, 0, t0);
        for (uint32_t s = 0; s < p.depth; ++s) landed(full_bar(s), ((fetched - s + p.depth - 1) / p.depth - 1) & 1u, t0);
    }
    #pragma unroll
    for (uint32_t c = 0; c < Tile::kColumns; ++c) {
        partial[warp][8 * c + 2 * q][g] = acc[c][0];
        partial[warp][8 * c + 2 * q + 1][g] = acc[c][1];
        partial[warp][8 * c + 2 * q][g + 8] = acc[c][2];
        partial[warp][8 * c + 2 * q + 1][g + 8] = acc[c][3];
    }
    __syncthreads();
    const uint32_t row = threadIdx.x / kFewTileN, col = threadIdx.x % kFewTileN;          // (threads beyond the rows have nothing to do)
    if (row < p.m && n0 + col < p.n && !ab.raised()) {
        // (in pairs: one warp's sum after the other, the last additions all round at the size of the result: error 7.5e-8 of the norm for sixteen warps, 5.7e-8 in pairs)
        float part[Tile::kWarps];
        #pragma unroll
        for (uint32_t w = 0; w < Tile::kWarps; ++w) part[w] = partial[w][row][col];
        #pragma unroll
        for (uint32_t half = Tile::kWarps / 2; half > 0; half /= 2)
            #pragma unroll
            for (uint32_t w = 0; w < half; ++w) part[w] += part[w + half];
        float sum = part[0];
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

// E4M3, up to 8 rows, 2048 < K <= 3072, more CTAs than two per SM: three of them share an SM where all pieces of one fit a third of its shared memory (228 KB, 1 KB of
// each CTA's share reserved, allotted in 128 bytes): as two large pieces for one row of K <= 2144, as three pieces of 1024 for up to five rows and most of six to eight.
// Two slots of 2048 leave two CTAs an SM although the second slot holds little more than a remainder: 4 rows of 7104 x 2080 7.5 -> 5.6 us,
// 5 rows of 14336 x 2560 13.6 -> 11.9, 20480 x 2080 17.5 -> 14.1. Fewer slots than pieces are no help (7 rows of 7168 x 2560 8.0, with two slots of 1024 9.2).
using FewWide = FewTile<false, 8, 2048, 4096>;
using FewWide3 = FewTile<false, 8, 1024, 3072>;
template <class Tile> static bool three_share_an_sm(uint32_t m, uint32_t k) {
    return few_smem<Tile>(m, k, (k + Tile::kPiece - 1) / Tile::kPiece) + Tile::kStaticSmem + 1024u + 127u <= 228u * 1024u / 3u;
}

// Where this kernel is the faster one: us of this one / of the block-scaled kernel, packed scales, back to back on rotating operands. (Where the
// rows are not a multiple of 8 the other kernel needs its scales of A relaid, 1.2 us; FP32 scales are relaid in front of either.)
//                       1 row           8 rows          16 rows                          1 row           8 rows          16 rows
//   E4M3  512 x 512     1.8 / 5.6       1.9 / 3.9       2.1 / 4.0       8192 x 4096      9.2 / 14.2     10.3 / 13.8     17.5 / 13.3
//        2112 x 7168    5.4 / 11.9      5.6 / 10.4      7.6 / 10.5     12288 x 4096     13.4 / 15.8     13.9 / 14.3     24 / 13.7
//        4096 x 4096    5.0 / 13.9      5.1 / 12.0      9.0 / 11.9      8192 x 8192     15.5 / 20.7     28 / 19
//       16384 x 512     5.5 / 8.1       5.7 / 6.1       7.1 / 6.1      24576 x 2048     12.7 / 15.2     14.0 / 13.5
//        2112 x 12288   8.4 / 14.7      8.5 / 13.5                     2112 x 16384     9.8 / 15.6 (6 rows 10.7 / 15.7)
//   E2M1 2368 x 4096    4.2 / 13.7      4.4 / 11.6      5.2 / 11.6      8192 x 2048      6.8 / 10.4      7.0 / 8.5       9.8 / 8.4
//        4096 x 7168    9.6 / 13.8     10.2 / 12.9     18.5 / 12.7     16384 x 1024      7.8 / 8.9       8.2 / 7.1
//   E4M3, 5 to 7 rows, K > 4096: 7 rows 8192 x 5120 13.1 / 16.8, 6144 x 7168 15.6 / 17.0, 5120 x 7168 15.4 / 15.7 (5 rows 14.2 / 15.7)
// An SM with one CTA takes its 16 rows of B in no faster however few CTAs there are; with more CTAs than two per SM the rest waits for a place, and the rows of A take
// the shared memory that pieces of B would be in flight in (7168 of K: 7 KB a row). The other kernel's time hardly depends on the rows.
//   Just beyond a limit, most of which are whole waves of CTAs: E4M3 4 rows 24576 x 128 6.7 / 6.4 (22528 5.8 / 6.5), 4 rows 22528 x 2080 15.6 / 15.0 (20480 14.0 / 14.2),
//   7 rows 14336 x 2560 13.7 / 12.9 (12288 11.8 / 11.8), 7 rows 12192 x 4128 16.5 / 16.2 (11456 15.0 / 15.9); E2M1 16 rows 3072 x 128 3.7 / 3.4 (x 96 is 0.93 of the other,
//   3000 x 128 0.84), 8 rows 2560 x 8064 in one slot 12.3 / 11.0 (x 7680 in two 10.8 / 10.9, x 7712 0.78: a K that is no multiple of 128 costs the other kernel a decoder).
//   (Where N is no multiple of 8 the other kernel needs B's scales relaid: 7 rows of 17500 x 2560 0.88 of its time, beyond the limit.)
static bool few_rows_size(uint32_t m, uint32_t n, uint32_t k, bool fp4) {
    constexpr uint32_t kOnePerSm = 148 * kFewTileN;
    if (k > 8192) return k <= kFewMaxK && !fp4 && m <= 8 && m * k <= 96u * 1024 && n >= 512 && n <= kOnePerSm;
    if (m > 8) {
        if (fp4) return k <= 4096 ? n <= (m == 16 && (k == 128 || k == 256) && n % 32 == 0 ? kOnePerSm : 3072) : n >= 1024 && n <= kOnePerSm;
        if (k > 4096) return n >= 512 && n <= kOnePerSm;
        return n <= (k <= 1024 ? 8192 : k <= 3072 ? 6144 : 4096);
    }
    if (m == 8) {
        if (fp4) return n <= (k <= 2048 ? 8192 : k <= 4096 ? 6144 : k <= 7680 || k % 128 != 0 || n % 8 != 0 ? 3072 : kOnePerSm);
        return n <= (k <= 2048 ? 12288 : k <= 4096 ? 8192 : k <= 7168 ? 4096 : 2560);
    }
    if (fp4) return n <= (k <= 2048 ? 16384 : k <= 4096 ? 8192 : 4096);
    if (k > 4096 && m <= 4) return n <= 8192;
    if (k > 7168) return n <= 2560;
    if (n > 24576 || (uint64_t)n * k > (48ull << 20)) return false;
    if (n % 8 != 0 || k <= 64 || (k > 128 && k <= 2048)) return true;
    if (k > 2048 && k <= FewWide3::kMaxK) return n <= (three_share_an_sm<FewWide>(m, k) || three_share_an_sm<FewWide3>(m, k) ? 9 : 6) * kOnePerSm;
    return n <= (k <= 128 ? 10 * kOnePerSm : k <= 4096 ? 24576 : 5 * kOnePerSm);
}

// What is left of them where the scales are relaid right in front (desc.reserved0; FP32 scales): the other kernel then has no launch more than this one, and this one cannot
// begin while the one before it ends. us with both launches, this kernel / the other: E2M1 8 rows 2560 x 8192 16.4 / 14.3, 3072 x 7680 15.4 / 14.3 (2368 x 7680 11.0 / 14.0),
// 1 row 256 x 7680 10.1 / 9.8, 4 rows 10240 x 256 8.9 / 8.7 (a last wave of few CTAs, against whole tiles of 256 columns; 10000 x 256 0.9 of the other); E4M3 4 rows 8192 x 8192
// 25.2 / 23.2, 7 rows 5120 x 7168 19.3 / 18.7 (two large pieces do not fit; 4500 x 7168 0.85 of the other), 6 rows 520 x 16384 13.3 / 12.4. A K that is no multiple of 128
// costs the other kernel more (4 rows 8100 x 7200 0.95 of it, x 7680 1.11).
static bool few_rows_size_relaid(uint32_t m, uint32_t n, uint32_t k, bool fp4) {
    constexpr uint32_t kOnePerSm = 148 * kFewTileN;
    if (k % 128 != 0) return true;
    if (fp4) {
        if (k <= 256) return n <= 4 * kOnePerSm || n > 10752 || n % 256 != 0;
        return k <= (m <= 2 ? 7168u : m <= 5 ? 6656u : 6144u) || (n <= kOnePerSm && (k <= 7168 || n > 256));
    }
    if (k > 14336) return n >= 768;
    return k <= 6144 || n <= 2 * kOnePerSm || m < 4 || (m < 6 && k <= 7168);
}

// The sizes that dg_gemm_few_rows promises (a part of the interface: callers that ask it keep scales of their own strides for exactly these). They take this kernel also
// beyond few_rows_size: 8 rows of 9216 x 2080 7.9 / 9.4 us, 4608 x 4128 6.5 / 12.7, 2816 x 7200 9.8 / 11.9, and in one slot, the one place where the other is faster, 2568 x 7936 12.9 / 11.2.
static bool few_rows_promised_size(uint32_t m, uint32_t n, uint32_t k, bool fp4) {
    if (fp4) return k <= 4096 && n <= 148 * kFewTileN;
    if ((uint64_t)n * k > (20ull << 20)) return false;
    if (k > 4096) return k <= 7168 ? n >= 1024 : k <= 8192 && n >= 2048;
    if (m == 8) return n <= 4 * 148 * kFewTileN;
    return n <= (k <= 512 ? 12288 : k <= 1024 ? 16384 : 10240);
}

bool takes_few_rows(const dg_gemm_desc_t& d) {
    return d.gemm_type == DG_GEMM_NORMAL && d.m >= 1 && d.m <= kFewMaxRows && d.n > 0 && d.k > 0 && d.k % 32 == 0 &&
           d.a_dtype == DG_E4M3 && (d.b_dtype == DG_E4M3 || d.b_dtype == DG_E2M1X2) && d.major_a == DG_MAJOR_K && d.major_b == DG_MAJOR_K &&
           (d.d_dtype == DG_BF16 || d.d_dtype == DG_F32) && !d.accumulate &&
           (d.epilogue == DG_EPILOGUE_IDENTITY || d.epilogue == DG_EPILOGUE_ALPHA || d.epilogue == DG_EPILOGUE_BIAS) &&
           ((few_rows_size(d.m, d.n, d.k, d.b_dtype == DG_E2M1X2) && (d.reserved0 == 0 || few_rows_size_relaid(d.m, d.n, d.k, d.b_dtype == DG_E2M1X2))) ||
            (d.m <= 8 && few_rows_promised_size(d.m, d.n, d.k, d.b_dtype == DG_E2M1X2)));
}
bool promises_few_rows(const dg_gemm_desc_t& d) {
    return takes_few_rows(d) && d.m <= 8 && few_rows_promised_size(d.m, d.n, d.k, d.b_dtype == DG_E2M1X2);
}

// Which tile a problem runs on, and with how many slots: `use(tile, slots)`.
// Large pieces cost fewer copies and waits (2112 x 3168 4.5 -> 3.9 us), where there is room for two of them; E4M3 falls back to pieces of 1024. More CTAs than SMs and
// many rows leave room for one slot all the same: 16 rows from K = 4032 on, 8 rows from 7616 (E4M3) or 7712 (E2M1) on. Such a CTA copies or multiplies, and the
// SM's second one covers for it: 16 x 4096 x 4096 9.0 us, the tensor-core kernel 11.9. Sixteen warps are
// faster where a CTA has an SM and a long K to itself (2112 x 7168 6.0 -> 5.6 us) and slower where CTAs share an SM (4096 x 4096 5.4 -> 5.8).
template <class Use>
static int with_few_tile(const dg_gemm_desc_t& d, Use use) {
    const bool fp4 = d.b_dtype == DG_E2M1X2;
    const uint32_t grid = (d.n + kFewTileN - 1) / kFewTileN;
    // one CTA per SM: everything in flight that fits; more: half of that, so that two CTAs share an SM
    const uint32_t room = grid <= 148 ? kFewMaxSmem : kFewMaxSmem / 2;
    const auto slots_of = [&](auto tile) {
        using Tile = decltype(tile);
        const uint32_t pieces = (d.k + Tile::kPiece - 1) / Tile::kPiece;
        uint32_t slots = pieces < kFewMaxDepth ? pieces : kFewMaxDepth;
        while (slots > 1 && few_smem<Tile>(d.m, d.k, slots) > room) --slots;
        return slots;
    };
    const auto several_slots = [&](auto tile) { return slots_of(tile) > 1 || d.k <= decltype(tile)::kPiece; };
    const auto take = [&](auto tile) -> int { return use(tile, slots_of(tile)); };
    using Rows16 = FewTile<false, 8, 2048, 4096, 16>;
    using LongK = FewTile<false, 8, 2048, 8192>;
    if (fp4) {
        if (d.m > 8) return take(FewTile<true, 8, 2048, 8192, 16>{});
        if (d.k <= 2048) return take(FewTile<true, 8, 2048, 2048>{});
        return take(FewTile<true, 8, 2048, 8192>{});
    }
    if (d.m > 8) {
        if (d.k <= 1024) return take(FewTile<false, 8, 1024, 1024, 16>{});
        if (d.k > 4096) return take(FewTile<false, 16, 1024, 8192, 16>{});
        if (several_slots(Rows16{})) return take(Rows16{});
        return take(FewTile<false, 8, 1024, 4096, 16>{});
    }
    if (d.k <= 1024) return take(FewTile<false, 8, 1024, 1024>{});
    if (d.k <= 2048) return take(FewTile<false, 8, 2048, 2048>{});
    if (d.k <= 4096) {
        if (grid > 2 * 148 && d.k <= FewWide3::kMaxK && !three_share_an_sm<FewWide>(d.m, d.k) && three_share_an_sm<FewWide3>(d.m, d.k)) return take(FewWide3{});
        return take(FewWide{});
    }
    if (d.k > 8192) return take(FewTile<false, 16, 2048, kFewMaxK>{});
    if (grid <= 148) return take(FewTile<false, 16, 4096, 8192>{});
    if (several_slots(LongK{})) return take(LongK{});
    return take(FewTile<false, 8, 1024, 8192>{});
}

// Dynamic shared memory of a CTA. Behind a relayout of the scales (desc.reserved0) a long K of E2M1 asks for so much that no SM takes more than an even share of the
// CTAs: as the kernel in front frees the SMs at different times, two or three of them meet on one and none on another (4 rows of 2368 x 7680 14.3 -> 10.9 us
// with the relayout, 1 row 3072 x 6144 15.4 -> 12.6). On their own, launches overlap better without (4 rows of 1536 x 5120 5.3 us, with it 5.6), and so
// do a few CTAs (1 row 520 x 4128 behind a relayout 5 % longer with it).
template <class Tile> static uint32_t few_dynamic_smem(const dg_gemm_desc_t& d, uint32_t slots) {
    const uint32_t used = few_smem<Tile>(d.m, d.k, slots), share = (d.n + 148 * kFewTileN - 1) / (148 * kFewTileN);
    if (d.reserved0 == 0 || !Tile::kFp4B || d.k <= 4096 || d.n < 1024 || share > 2) return used;
    const uint32_t least = 228u * 1024u / (share + 1) - 1024u - Tile::kStaticSmem + 128u;
    return used < least ? least : used;
}

int few_rows_layout(const dg_gemm_desc_t& d, dg_few_rows_layout_t& out) {
    return with_few_tile(d, [&](auto tile, uint32_t slots) -> int {
        using Tile = decltype(tile);
        out = {Tile::kWarps, Tile::kRows, Tile::kPiece, slots, Tile::kMaxK, few_dynamic_smem<Tile>(d, slots), Tile::kStaticSmem};
        return DG_OK;
    });
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
    const uint32_t grid = (d.n + kFewTileN - 1) / kFewTileN;
    if (int rc = get_status_pointer(&p.status)) return rc;
    return with_few_tile(d, [&](auto tile, uint32_t slots) -> int {
        using Tile = decltype(tile);
        p.depth = slots;
        const uint32_t smem = few_dynamic_smem<Tile>(d, slots);
        DG_CHECK_ARG(d.k <= Tile::kMaxK && smem <= kFewMaxSmem, "not a problem of a few rows: K is too large");
        const void* fn = (const void*)few_rows_kernel<Tile>;
        // (raised once per device and kernel to the most a launch can ask for)
        {
            static std::mutex mu;
            static bool raised[64] = {};
            int dev = 0;
            DG_CHECK_CUDA(cudaGetDevice(&dev));
            DG_CHECK_ARG(dev >= 0 && dev < 64, "device index out of range");
            std::lock_guard<std::mutex> lock(mu);
            if (!raised[dev]) {
                DG_CHECK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFewMaxSmem));
                raised[dev] = true;
            }
        }
        void* params[] = {&p};
        return launch_overlapped(fn, dim3(grid), dim3(Tile::kThreads), params, stream, smem);
    });
}

}  // namespace dg
