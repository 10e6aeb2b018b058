// NVFP4 (e2m1 codes, e4m3 scale per 16 elements of K, f32 global scale) W4A4 linear.
//
//   nvfp4_amax_kernel / nvfp4_scale2_kernel  calibrate-on-the-sample input scale: max(amax, 1e-12) / (6 * 448)
//   quant_nvfp4_act_kernel   static-scale activation quantize, the f32 algebra the reference spells
//                            (emmy/compiler/loader/quant.py:1968-2139, tests/compiler/loader/test_quant.py:1776-1784):
//                            ratio = (amax_blk * f32(1/6)) * f32(1/s2); sbits = e4m3(ratio); fused = dec(sbits) * s2;
//                            codes = e2m1(blk / max(fused, 1e-12)), all round-to-nearest f32.  Bit-exact.
//   nvfp4_tile_scales_kernel re-tiles a plain [rows, K/16] scale matrix into the 512-byte atoms the tensor core's
//                            scale-factor copy reads (load time for weights, inside the quantize for activations)
//   nvfp4_gemm_tc_kernel (128 x 128 tiles for M <= 128; above, 128 x 256 tiles or the 256 x 256 tiles of gemm_pair.cu)
//                            tcgen05.mma kind::mxf4nvf4.block_scale.scale_vec::4X: codes come by TMA (128-byte
//                            swizzle, 256 elements of K per row), scale atoms by bulk copy and then tcgen05.cp into
//                            TMEM, f32 accumulators in TMEM; the epilogue multiplies by the two global scales.
// The hardware applies the raw e4m3 block scale and the global scales are factored out into the epilogue, whereas
// the reference's value path applies f16(block * global) per element: a relative difference of at most 2^-11 per
// operand, far inside the output tolerance; the dequantised-weight export (eq_dequant_nvfp4) stays bit-exact.
#include "gemm_pair.cuh"
#include "quant.cuh"
#include "tc_common.cuh"

namespace eq {

// ------------------------------------------------------------------------------------------------ calibration
template <typename InT>
__global__ void nvfp4_amax_kernel(const InT* __restrict__ x, int64_t n, unsigned int* __restrict__ amax_bits) {
    float m = 0.f;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        m = fmaxf(m, fabsf(to_float(x[i])));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, off));
    if ((threadIdx.x & 31) == 0) atomicMax(amax_bits, __float_as_uint(m));  // non-negative floats order like their bits
}
__global__ void nvfp4_scale2_kernel(const unsigned int* __restrict__ amax_bits, float* __restrict__ scale2) {
    const double amax = fmax(static_cast<double>(__uint_as_float(*amax_bits)), 1e-12);
    *scale2 = static_cast<float>(amax / (6.0 * 448.0));
}

// ------------------------------------------------------------------------------------------------ scale atoms
// Tiled scale layout: [row block of 128][k block of 64 elements][512 B]; inside an atom the scale of (row r, 16-block
// i of the k block) sits at byte (r % 32) * 16 + (r / 32) * 4 + i.  Rows beyond `rows` are zero.
__device__ __forceinline__ size_t sf_tiled_offset(int64_t row, int64_t blk16, int64_t k64_blocks) {
    const int64_t rb = row >> 7, r = row & 127, kb = blk16 >> 2, i = blk16 & 3;
    return static_cast<size_t>((rb * k64_blocks + kb) * 512 + (r & 31) * 16 + (r >> 5) * 4 + i);
}

__global__ void nvfp4_tile_scales_kernel(const uint8_t* __restrict__ plain, int64_t rows, int64_t K, uint8_t* __restrict__ tiled) {
    const int64_t blocks16 = K / 16, k64 = K / 64;
    const int64_t padded_rows = (rows + 127) / 128 * 128;
    const int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (idx >= padded_rows * blocks16) return;
    const int64_t row = idx / blocks16, b = idx % blocks16;
    tiled[sf_tiled_offset(row, b, k64)] = row < rows ? plain[row * blocks16 + b] : 0;
}

// ------------------------------------------------------------------------------------------------ activation quantize
__device__ __forceinline__ uint8_t e4m3_satfinite(float v) {
    uint16_t r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.f), "f"(v));
    return static_cast<uint8_t>(r & 0xFF);
}
// two f32 -> one byte: low nibble = code(lo), high nibble = code(hi)
__device__ __forceinline__ uint8_t e2m1x2_satfinite(float lo, float hi) {
    uint16_t r;
    asm("{ .reg .b8 t; cvt.rn.satfinite.e2m1x2.f32 t, %1, %2; cvt.u16.u8 %0, t; }" : "=h"(r) : "f"(hi), "f"(lo));
    return static_cast<uint8_t>(r);
}

// One thread per 16-element block.  Writes the packed codes [M, K/2], the plain scales [M, K/16] (optional) and the
// tiled scales (optional).  `status`, when given, is cleared for the linear that follows in the stream; that linear
// may be launched as a programmatic dependent and fetch its weights while this kernel runs.
template <typename InT>
__global__ void quant_nvfp4_act_kernel(const InT* __restrict__ x, int64_t M, int64_t K, const float* __restrict__ scale2,
                                       uint8_t* __restrict__ codes, uint8_t* __restrict__ sf_plain, uint8_t* __restrict__ sf_tiled,
                                       int* __restrict__ status) {
    if (status) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // inside a linear, which may start fetching its weights
    // launched as a programmatic dependent itself when it runs inside the linear: the kernel before it (usually the
    // previous linear on this workspace) still reads the codes and the status word this one rewrites
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t blocks16 = K / 16;
    const int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (status && idx == 0) *status = 0;
    if (idx >= M * blocks16) return;
    const int64_t row = idx / blocks16, b = idx % blocks16;
    const InT* src = x + row * K + b * 16;
    float v[16];
    if (sizeof(InT) == 2 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        uint4 raw[2] = {reinterpret_cast<const uint4*>(src)[0], reinterpret_cast<const uint4*>(src)[1]};
        const InT* e = reinterpret_cast<const InT*>(raw);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = to_float(e[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = to_float(src[i]);
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
    const float s2 = scale2[0];
    const float ratio = __fmul_rn(__fmul_rn(amax, __fdiv_rn(1.0f, 6.0f)), __fdiv_rn(1.0f, s2));
    const uint8_t sbits = e4m3_satfinite(ratio);
    const float fused = __fmul_rn(e4m3_to_float(sbits), s2);
    const float div = fmaxf(fused, 1e-12f);
    uint32_t w[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint8_t byte = e2m1x2_satfinite(__fdiv_rn(v[2 * i], div), __fdiv_rn(v[2 * i + 1], div));
        w[i >> 2] |= static_cast<uint32_t>(byte) << (8 * (i & 3));
    }
    *reinterpret_cast<uint2*>(codes + row * (K / 2) + b * 8) = make_uint2(w[0], w[1]);
    if (sf_plain) sf_plain[idx] = sbits;
    if (sf_tiled) sf_tiled[sf_tiled_offset(row, b, K / 64)] = sbits;
}

// The same rule for 16-bit activations at 16-byte aligned addresses, K a multiple of 64, tiled scales only: a CTA takes up to 128
// rows x 64 elements, i.e. one scale atom; four neighbouring threads a row, whose four scale bytes are one word of the atom: no
// division per thread to find its place, no scattered bytes.  Bound by its instructions (336 a warp, 2.8 a cycle and SM, at 24 % of the
// memory rate, before single elements were divided).
// Measured, us a linear, K=5120, N=17408: 1024 rows 54.3 -> 52.9, 4096 rows 175 -> 172 (fewer CTAs that walk over the pieces with the
// next one's loads under way: 177); then, by dividing single elements, 2048 rows of 2048 columns 22.0 -> 20.5.
template <typename InT>
__global__ void __launch_bounds__(512) quant_nvfp4_act_atoms_kernel(const uint4* __restrict__ x, int64_t M, int k64_blocks, const float* __restrict__ scale2,
                                                                    uint8_t* __restrict__ codes, uint8_t* __restrict__ sf_tiled, int* __restrict__ status) {
    // Only inside a linear: on its own this may write the operands of a weight, which a linear behind it would fetch ahead of its wait.
    if (status) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int r = threadIdx.x >> 2, i = threadIdx.x & 3, kb = blockIdx.x;
    if (status && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) *status = 0;
    const float s2 = scale2[0];
    for (int64_t rb = blockIdx.y; rb * 128 < M; rb += gridDim.y) {
        const int64_t row = rb * 128 + r;
        const bool live = row < M;
        const int64_t blk = (live ? row : 0) * (k64_blocks * 4) + kb * 4 + i;  // 16-element block
        const uint4 raw[2] = {__ldg(x + 2 * blk), __ldg(x + 2 * blk + 1)};
        const float amax = fmaxf(quant::abs_max8<InT>(raw[0]), quant::abs_max8<InT>(raw[1]));
        const float ratio = __fmul_rn(__fmul_rn(amax, __fdiv_rn(1.0f, 6.0f)), __fdiv_rn(1.0f, s2));
        const uint8_t sbits = e4m3_satfinite(ratio);
        const float div = fmaxf(__fmul_rn(e4m3_to_float(sbits), s2), 1e-12f);
        uint32_t word = static_cast<uint32_t>(sbits) << (8 * i);
        word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
        word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
        if (live) {
            *reinterpret_cast<uint2*>(codes + blk * 8) = make_uint2(quant::e2m1_codes8<InT>(raw[0], div), quant::e2m1_codes8<InT>(raw[1], div));
            if (i == 0) *reinterpret_cast<uint32_t*>(sf_tiled + (rb * k64_blocks + kb) * 512 + (r & 31) * 16 + (r >> 5) * 4) = word;
        }
    }
}

// RMSNorm in front of the static quantize, in one kernel: h = dtype(dtype(x * rsqrt(mean(x^2) + eps)) * gamma), the model's
// RMSNorm (its normalised value rounded to the activation dtype before the weight multiplies it), then the block rule on h.
// One CTA per row: the sum of squares first, then one thread per 16-element block; the normalised row is never written.
template <typename InT>
__global__ void __launch_bounds__(256) rmsnorm_quant_nvfp4_rows_kernel(const InT* __restrict__ x, const InT* __restrict__ gamma, float eps, int64_t K,
                                                                       const float* __restrict__ scale2, uint8_t* __restrict__ codes,
                                                                       uint8_t* __restrict__ sf_tiled, int* __restrict__ status) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float part[8];
    const int64_t row = blockIdx.x;
    const InT* xr = x + row * K;
    if (status && row == 0 && threadIdx.x == 0) *status = 0;
    float ss = 0.f;
    for (int64_t k = threadIdx.x; k < K; k += blockDim.x) {
        const float v = to_float(xr[k]);
        ss = fmaf(v, v, ss);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) total += part[w];
    const float rstd = rsqrtf(__fdiv_rn(total, static_cast<float>(K)) + eps);
    const float s2 = scale2[0];
    for (int64_t b = threadIdx.x; b < K / 16; b += blockDim.x) {
        float v[16];
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const InT n = from_float<InT>(to_float(xr[b * 16 + i]) * rstd);
            v[i] = to_float(from_float<InT>(to_float(n) * to_float(gamma[b * 16 + i])));
            amax = fmaxf(amax, fabsf(v[i]));
        }
        const float ratio = __fmul_rn(__fmul_rn(amax, __fdiv_rn(1.0f, 6.0f)), __fdiv_rn(1.0f, s2));
        const uint8_t sbits = e4m3_satfinite(ratio);
        const float div = fmaxf(__fmul_rn(e4m3_to_float(sbits), s2), 1e-12f);
        uint32_t w[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint8_t byte = e2m1x2_satfinite(__fdiv_rn(v[2 * i], div), __fdiv_rn(v[2 * i + 1], div));
            w[i >> 2] |= static_cast<uint32_t>(byte) << (8 * (i & 3));
        }
        *reinterpret_cast<uint2*>(codes + row * (K / 2) + b * 8) = make_uint2(w[0], w[1]);
        sf_tiled[sf_tiled_offset(row, b, K / 64)] = sbits;
    }
}

// ------------------------------------------------------------------------------------------------ weight quantize
// The two-level weight quantizer (emmy/compiler/loader/quant.py:206-237), one thread per 16-element block:
// block scale = amax_blk / 6 stored as e4m3 relative to scale_2; the divisor is the FUSED scale f16(dec(bits) * scale_2);
// codes = e2m1(blk / fused) with zero where the fused scale is zero.  Every step an f32 round-to-nearest operation, as
// numpy does them: bit-exact with the reference's output.
template <typename InT>
__global__ void quant_nvfp4_weight_kernel(const InT* __restrict__ w, int64_t N, int64_t K, const float* __restrict__ scale2,
                                          uint8_t* __restrict__ codes, uint8_t* __restrict__ sf_plain) {
    const int64_t blocks16 = K / 16;
    const int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (idx >= N * blocks16) return;
    const InT* src = w + idx * 16;
    float v[16];
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        v[i] = to_float(src[i]);
        amax = fmaxf(amax, fabsf(v[i]));
    }
    const float s2 = scale2[0];
    const uint8_t sbits = e4m3_satfinite(__fdiv_rn(__fdiv_rn(amax, 6.0f), s2));
    const float fused = __half2float(__float2half_rn(__fmul_rn(e4m3_to_float(sbits), s2)));
    uint32_t out[2] = {0, 0};
    if (fused != 0.f) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint8_t byte = e2m1x2_satfinite(__fdiv_rn(v[2 * i], fused), __fdiv_rn(v[2 * i + 1], fused));
            out[i >> 2] |= static_cast<uint32_t>(byte) << (8 * (i & 3));
        }
    }
    *reinterpret_cast<uint2*>(codes + idx * 8) = make_uint2(out[0], out[1]);
    sf_plain[idx] = sbits;
}

// ------------------------------------------------------------------------------------------------ tensor path
constexpr int kBM = 128;
constexpr int kBKBytes = 128;                 // 256 e2m1 elements of K per stage row
constexpr int kTileA = kBM * kBKBytes;
constexpr int kSfA = 4 * 512;                 // four k64 atoms per stage, one row block
constexpr int kGemmThreads = 192;

// BN = 256 for prefill-shaped calls; BN = 128 when there is a single row tile, so that twice as many CTAs stream the weight.
template <int BN>
struct Fp4Cfg {
    static constexpr int kTileB = BN * kBKBytes;
    static constexpr int kSfB = (BN / 128) * 4 * 512;  // one or two row blocks
    static constexpr int kStageBytes = kTileA + kTileB + kSfA + kSfB;
    static constexpr int kStages = BN == 256 ? 4 : 6;
    static constexpr size_t kSmem = static_cast<size_t>(kStages) * kStageBytes + 1024 + 256;
    static constexpr uint32_t kTmemCols = BN == 256 ? 512 : 256;  // accumulator columns + 16 (SFA) + 16 or 32 (SFB), as a power of two
};

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

template <typename OutT, int BN>
__global__ void __launch_bounds__(kGemmThreads, 1)
    nvfp4_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         const uint8_t* __restrict__ sfa, const uint8_t* __restrict__ sfb, const float* __restrict__ gx,
                         const float* __restrict__ gw, OutT* __restrict__ y, int M, int N, int K, int* __restrict__ status) {
    using Cfg = Fp4Cfg<BN>;
    constexpr int kBN = BN, kTileB = Cfg::kTileB, kSfB = Cfg::kSfB, kStages = Cfg::kStages;
    constexpr uint32_t kTmemCols = Cfg::kTmemCols;
    constexpr bool kTwoBlocks = BN == 256;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* tiles_a = smem;
    unsigned char* tiles_b = tiles_a + kStages * kTileA;
    unsigned char* sfs_a = tiles_b + kStages * kTileB;
    unsigned char* sfs_b = sfs_a + kStages * kSfA;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sfs_b + kStages * kSfB);
    uint64_t* full = bars;
    uint64_t* empty = bars + kStages;
    uint64_t* acc_ready = bars + 2 * kStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // row tiles run fastest: the CTAs that share a weight tile are co-resident and the weight comes from DRAM once
    const int n0 = blockIdx.y * kBN, m0 = blockIdx.x * kBM;
    const int k_blocks = K / 256;   // stages of 256 elements
    const int k64_blocks = K / 64;  // scale atoms along K
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            tc::mbar_init(tc::smem_u32(full + s), 1);
            tc::mbar_init(tc::smem_u32(empty + s), 1);
        }
        tc::mbar_init(tc::smem_u32(acc_ready), 1);
        tc::mbar_fence_init();
    }
    if (warp == 1) tc::tmem_alloc(tc::smem_u32(tmem_slot), kTmemCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_sfa = tmem_base + kBN;        // 4 columns per k64 step
    const uint32_t tmem_sfb = tmem_base + kBN + 16;   // 8 columns per k64 step

    // The kernel may have been launched as a programmatic dependent of the activation quantize: the weights and their
    // scales never depend on it, so the first ring of weight stages is requested before the dependency is awaited;
    // every other role waits first, so that its bounded waits count from the moment the codes exist.
    if (warp == 0) {
        if (tc::elect_one()) {
            tc::tma_prefetch_desc(&map_a);
            tc::tma_prefetch_desc(&map_b);
            const int rb_a = m0 / 128, rb_b = n0 / 128;
            const int n_rb = (N + 127) / 128;
            // the second row block of B may lie beyond N (N not a multiple of 256): it is then not copied
            const bool second = kTwoBlocks && rb_b + 1 < n_rb;
            constexpr int kSfBlock = 4 * 512;
            auto weights = [&](int kb, int s, uint32_t bar) {
                tc::mbar_expect_tx(bar, kTileA + kTileB + kSfA + (second ? 2 * kSfBlock : kSfBlock));
                tc::tma_load_2d(tc::smem_u32(tiles_b + s * kTileB), &map_b, kb * kBKBytes, n0, bar);
                bulk_g2s(tc::smem_u32(sfs_b + s * kSfB), sfb + (static_cast<size_t>(rb_b) * k64_blocks + kb * 4) * 512, kSfBlock, bar);
                if (second)
                    bulk_g2s(tc::smem_u32(sfs_b + s * kSfB + kSfBlock),
                             sfb + (static_cast<size_t>(rb_b + 1) * k64_blocks + kb * 4) * 512, kSfBlock, bar);
            };
            auto codes = [&](int kb, int s, uint32_t bar) {
                tc::tma_load_2d(tc::smem_u32(tiles_a + s * kTileA), &map_a, kb * kBKBytes, m0, bar);
                bulk_g2s(tc::smem_u32(sfs_a + s * kSfA), sfa + (static_cast<size_t>(rb_a) * k64_blocks + kb * 4) * 512, kSfA, bar);
            };
            const int ahead = k_blocks < kStages ? k_blocks : kStages;
            for (int kb = 0; kb < ahead; ++kb) weights(kb, kb, tc::smem_u32(full + kb));
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int kb = 0; kb < ahead; ++kb) codes(kb, kb, tc::smem_u32(full + kb));
            for (int kb = ahead; kb < k_blocks; ++kb) {
                const int s = kb % kStages;
                if (!tc::mbar_wait(tc::smem_u32(empty + s), ((kb / kStages) - 1) & 1)) {
                    atomicExch(status, 1);
                    tc::drain_copies(full, kb - kStages, kb, kStages);
                    break;
                }
                const uint32_t bar = tc::smem_u32(full + s);
                weights(kb, s, bar);
                codes(kb, s, bar);
            }
        }
    } else if (warp == 1) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (tc::elect_one()) {
            constexpr uint32_t idesc = tc::instr_desc_nvfp4(kBM, kBN, 0, 0);
            for (int kb = 0; kb < k_blocks; ++kb) {
                const int s = kb % kStages;
                if (!tc::mbar_wait(tc::smem_u32(full + s), (kb / kStages) & 1)) {
                    atomicExch(status, 2);
                    tc::drain_copies(full, kb, min(kb + kStages, k_blocks), kStages);
                    break;
                }
                tc::fence_after_sync();
                const uint32_t a_addr = tc::smem_u32(tiles_a + s * kTileA), b_addr = tc::smem_u32(tiles_b + s * kTileB);
                const uint32_t sfa_addr = tc::smem_u32(sfs_a + s * kSfA), sfb_addr = tc::smem_u32(sfs_b + s * kSfB);
                // scale atoms of the stage's four k64 steps -> TMEM: A rows 0..127 (4 columns per step), B rows 0..127
                // and 128..255 (8 columns per step); all twelve copies are queued before the first MMA
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    tc::tmem_cp_32x128b_warpx4(tmem_sfa + ks * 4, tc::smem_desc_sf(sfa_addr + ks * 512));
                    tc::tmem_cp_32x128b_warpx4(tmem_sfb + ks * 8, tc::smem_desc_sf(sfb_addr + ks * 512));
                    if constexpr (kTwoBlocks) tc::tmem_cp_32x128b_warpx4(tmem_sfb + ks * 8 + 4, tc::smem_desc_sf(sfb_addr + 4 * 512 + ks * 512));
                }
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    const uint64_t da = tc::smem_desc_k_sw128(a_addr + ks * 32), db = tc::smem_desc_k_sw128(b_addr + ks * 32);
                    tc::mma_mxf4nvf4(tmem_base, da, db, idesc, tmem_sfa + ks * 4, tmem_sfb + ks * 8, kb > 0 || ks > 0);
                }
                tc::mma_commit(tc::smem_u32(empty + s));
            }
            tc::mma_commit(tc::smem_u32(acc_ready));
        }
    } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int quarter = warp & 3;
        const int m = m0 + quarter * 32 + lane;
        const bool ok = tc::mbar_wait(tc::smem_u32(acc_ready), 0);
        if (!ok && lane == 0) atomicExch(status, 3);
        tc::fence_after_sync();
        if (ok) {
            const float g = gx[0] * gw[0];
#pragma unroll 1
            for (int c = 0; c < kBN; c += 32) {
                uint32_t r[32];
                tc::tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c, r);
                tc::tmem_ld_wait();
                if (m < M) {
                    OutT* dst = y + static_cast<size_t>(m) * N + n0 + c;
                    if (n0 + c + 32 <= N) {
                        uint32_t packed[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const OutT o0 = from_float<OutT>(__uint_as_float(r[2 * i]) * g), o1 = from_float<OutT>(__uint_as_float(r[2 * i + 1]) * g);
                            packed[i] = static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(&o0)) |
                                        (static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(&o1)) << 16);
                        }
#pragma unroll
                        for (int v = 0; v < 4; ++v)
                            reinterpret_cast<uint4*>(dst)[v] = make_uint4(packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (n0 + c + i < N) dst[i] = from_float<OutT>(__uint_as_float(r[i]) * g);
                    }
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ------------------------------------------------------------------------------------------------ decode tile (M <= 16)
// With a handful of rows the operands swap roles: a 128-channel tile of the WEIGHT is the MMA's A operand (M = 128) and
// the activation rows are B (N = 16), so a K step stages 16 KB of weight codes + 2 KB of activation codes + 2 x 2 KB of
// scale atoms instead of a 16 KB activation tile that is all zeros but its first rows.  Five stages are 110 KB: two
// CTAs fit an SM, and they belong to consecutive launches (programmatic dependent launch: the later one requests its
// weights while the earlier one computes; measured on B200, a launch that streams this matrix alone takes 10.4 us, of
// which 3.5 us are the launch boundary).  The accumulator is [channel (TMEM lane)][row (column)], 16 columns.
constexpr int kDecStages = 5;
constexpr int kDecTileW = 128 * kBKBytes, kDecTileX = 16 * kBKBytes, kDecSf = 4 * 512;
constexpr int kDecStageBytes = kDecTileW + kDecTileX + 2 * kDecSf;
constexpr size_t kDecSmem = static_cast<size_t>(kDecStages) * kDecStageBytes + 1024 + 256;
constexpr uint32_t kDecTmemCols = 64;  // 16 accumulator columns, 16 + 16 scale columns

template <typename OutT>
__global__ void __launch_bounds__(kGemmThreads, 2)
    nvfp4_decode_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                        const uint8_t* __restrict__ sfw, const uint8_t* __restrict__ sfx, const float* __restrict__ gx,
                        const float* __restrict__ gw, OutT* __restrict__ y, int M, int N, int K, int* __restrict__ status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* tiles_w = smem;
    unsigned char* tiles_x = tiles_w + kDecStages * kDecTileW;
    unsigned char* sfs_w = tiles_x + kDecStages * kDecTileX;
    unsigned char* sfs_x = sfs_w + kDecStages * kDecSf;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sfs_x + kDecStages * kDecSf);
    uint64_t* full = bars;
    uint64_t* empty = bars + kDecStages;
    uint64_t* acc_ready = bars + 2 * kDecStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kDecStages + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * 128;
    const int k_blocks = K / 256, k64_blocks = K / 64;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (threadIdx.x == 0) {
        for (int s = 0; s < kDecStages; ++s) {
            tc::mbar_init(tc::smem_u32(full + s), 1);
            tc::mbar_init(tc::smem_u32(empty + s), 1);
        }
        tc::mbar_init(tc::smem_u32(acc_ready), 1);
        tc::mbar_fence_init();
    }
    if (warp == 1) tc::tmem_alloc(tc::smem_u32(tmem_slot), kDecTmemCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_sfw = tmem_base + 16, tmem_sfx = tmem_base + 32;  // 4 columns per k64 step each

    if (warp == 0) {
        if (tc::elect_one()) {
            tc::tma_prefetch_desc(&map_w);
            tc::tma_prefetch_desc(&map_x);
            const int rb_w = n0 / 128;
            auto weights = [&](int kb, int s, uint32_t bar) {
                tc::mbar_expect_tx(bar, kDecStageBytes);
                tc::tma_load_2d(tc::smem_u32(tiles_w + s * kDecTileW), &map_w, kb * kBKBytes, n0, bar);
                bulk_g2s(tc::smem_u32(sfs_w + s * kDecSf), sfw + (static_cast<size_t>(rb_w) * k64_blocks + kb * 4) * 512, kDecSf, bar);
            };
            auto codes = [&](int kb, int s, uint32_t bar) {
                tc::tma_load_2d(tc::smem_u32(tiles_x + s * kDecTileX), &map_x, kb * kBKBytes, 0, bar);
                bulk_g2s(tc::smem_u32(sfs_x + s * kDecSf), sfx + static_cast<size_t>(kb) * 4 * 512, kDecSf, bar);
            };
            // the weights never depend on the kernel before (the activation quantize): request them ahead of the wait
            const int ahead = k_blocks < kDecStages ? k_blocks : kDecStages;
            for (int kb = 0; kb < ahead; ++kb) weights(kb, kb, tc::smem_u32(full + kb));
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int kb = 0; kb < ahead; ++kb) codes(kb, kb, tc::smem_u32(full + kb));
            for (int kb = ahead; kb < k_blocks; ++kb) {
                const int s = kb % kDecStages;
                if (!tc::mbar_wait(tc::smem_u32(empty + s), ((kb / kDecStages) - 1) & 1)) {
                    atomicExch(status, 1);
                    tc::drain_copies(full, kb - kDecStages, kb, kDecStages);
                    break;
                }
                const uint32_t bar = tc::smem_u32(full + s);
                weights(kb, s, bar);
                codes(kb, s, bar);
            }
        }
    } else if (warp == 1) {
        asm volatile("griddepcontrol.wait;" ::: "memory");  // bounded waits count from the moment the codes exist
        if (tc::elect_one()) {
            constexpr uint32_t idesc = tc::instr_desc_nvfp4(128, 16, 0, 0);
            for (int kb = 0; kb < k_blocks; ++kb) {
                const int s = kb % kDecStages;
                if (!tc::mbar_wait(tc::smem_u32(full + s), (kb / kDecStages) & 1)) {
                    atomicExch(status, 2);
                    tc::drain_copies(full, kb, min(kb + kDecStages, k_blocks), kDecStages);
                    break;
                }
                tc::fence_after_sync();
                const uint32_t w_addr = tc::smem_u32(tiles_w + s * kDecTileW), x_addr = tc::smem_u32(tiles_x + s * kDecTileX);
                const uint32_t sfw_addr = tc::smem_u32(sfs_w + s * kDecSf), sfx_addr = tc::smem_u32(sfs_x + s * kDecSf);
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    tc::tmem_cp_32x128b_warpx4(tmem_sfw + ks * 4, tc::smem_desc_sf(sfw_addr + ks * 512));
                    tc::tmem_cp_32x128b_warpx4(tmem_sfx + ks * 4, tc::smem_desc_sf(sfx_addr + ks * 512));
                }
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    const uint64_t da = tc::smem_desc_k_sw128(w_addr + ks * 32), db = tc::smem_desc_k_sw128(x_addr + ks * 32);
                    tc::mma_mxf4nvf4(tmem_base, da, db, idesc, tmem_sfw + ks * 4, tmem_sfx + ks * 4, kb > 0 || ks > 0);
                }
                tc::mma_commit(tc::smem_u32(empty + s));
            }
            tc::mma_commit(tc::smem_u32(acc_ready));
        }
    } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int quarter = warp & 3;
        const int n = n0 + quarter * 32 + lane;  // this thread's output channel
        const bool ok = tc::mbar_wait(tc::smem_u32(acc_ready), 0);
        if (!ok && lane == 0) atomicExch(status, 3);
        tc::fence_after_sync();
        if (ok) {
            const float g = gx[0] * gw[0];
            uint32_t r[16];
            tc::tmem_ld_32x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16), r);
            tc::tmem_ld_wait();
            if (n < N) {
#pragma unroll
                for (int m = 0; m < 16; ++m)
                    if (m < M) y[static_cast<size_t>(m) * N + n] = from_float<OutT>(__uint_as_float(r[m]) * g);
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_base, kDecTmemCols);
    }
}

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
static size_t sf_tiled_bytes(int64_t rows, int64_t K) { return static_cast<size_t>((rows + 127) / 128) * (K / 64) * 512; }

}  // namespace eq

using namespace eq;

extern "C" size_t eq_nvfp4_tiled_scale_bytes(int64_t rows, int64_t K) {
    if (rows <= 0 || K <= 0 || K % 64) return 0;
    return sf_tiled_bytes(rows, K);
}

extern "C" int eq_nvfp4_tile_scales(const uint8_t* scale_bits, int64_t rows, int64_t K, uint8_t* tiled, void* stream) {
    EQ_REQUIRE(scale_bits && tiled, EQ_ERR_BAD_ARG, "eq_nvfp4_tile_scales: null pointer");
    EQ_REQUIRE(rows > 0 && K > 0 && K % 64 == 0, EQ_ERR_UNSUPPORTED, "eq_nvfp4_tile_scales: needs K %% 64 == 0 (K=%lld)", (long long)K);
    const int64_t total = (rows + 127) / 128 * 128 * (K / 16);
    nvfp4_tile_scales_kernel<<<static_cast<unsigned>(ceil_div(total, 256)), 256, 0, static_cast<cudaStream_t>(stream)>>>(scale_bits, rows, K, tiled);
    EQ_LAUNCH_OK("nvfp4_tile_scales_kernel");
    return EQ_OK;
}

extern "C" size_t eq_nvfp4_weight_scale_bytes(int64_t N, int64_t K) {
    if (N <= 0 || K <= 0 || K % 64) return 0;
    return align_up(sf_tiled_bytes(N, K), 256);
}

extern "C" int eq_nvfp4_tile_weight_scales(const uint8_t* scale_bits, int64_t N, int64_t K, uint8_t* tiled, void* stream) {
    EQ_REQUIRE(scale_bits && tiled, EQ_ERR_BAD_ARG, "eq_nvfp4_tile_weight_scales: null pointer");
    EQ_REQUIRE(N > 0 && K > 0 && K % 64 == 0, EQ_ERR_UNSUPPORTED, "eq_nvfp4_tile_weight_scales: needs K %% 64 == 0 (K=%lld)", (long long)K);
    EQ_REQUIRE(aligned(tiled, 256), EQ_ERR_BAD_ALIGN, "eq_nvfp4_tile_weight_scales: the output must be 256-byte aligned");
    return eq_nvfp4_tile_scales(scale_bits, N, K, tiled, stream);
}

extern "C" int eq_nvfp4_global_scale(const void* x, int64_t M, int64_t K, int in_dtype, float* scale2, unsigned int* scratch_u32,
                                     void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    EQ_REQUIRE(x && scale2 && scratch_u32 && M > 0 && K > 0, EQ_ERR_BAD_ARG, "eq_nvfp4_global_scale: bad arguments");
    EQ_CUDA_OK(cudaMemsetAsync(scratch_u32, 0, sizeof(unsigned int), stream));
    const int64_t n = M * K;
    const unsigned grid = static_cast<unsigned>(n / 256 / 8 + 1 < 1184 ? n / 256 / 8 + 1 : 1184);
    switch (in_dtype) {
        case EQ_F16: nvfp4_amax_kernel<__half><<<grid, 256, 0, stream>>>(static_cast<const __half*>(x), n, scratch_u32); break;
        case EQ_BF16: nvfp4_amax_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), n, scratch_u32); break;
        case EQ_F32: nvfp4_amax_kernel<float><<<grid, 256, 0, stream>>>(static_cast<const float*>(x), n, scratch_u32); break;
        default: return fail(EQ_ERR_BAD_ARG, "eq_nvfp4_global_scale: unknown dtype %d", in_dtype);
    }
    EQ_LAUNCH_OK("nvfp4_amax_kernel");
    nvfp4_scale2_kernel<<<1, 1, 0, stream>>>(scratch_u32, scale2);
    EQ_LAUNCH_OK("nvfp4_scale2_kernel");
    return EQ_OK;
}

extern "C" int eq_quant_nvfp4_weight(const void* values, int64_t N, int64_t K, int in_dtype, uint8_t* packed, uint8_t* scale_bits,
                                     float* scale_2, unsigned int* scratch_u32, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    EQ_REQUIRE(values && packed && scale_bits && scale_2 && scratch_u32, EQ_ERR_BAD_ARG, "eq_quant_nvfp4_weight: null pointer");
    EQ_REQUIRE(N > 0 && K > 0, EQ_ERR_BAD_ARG, "eq_quant_nvfp4_weight: bad extents");
    EQ_REQUIRE(K % 16 == 0, EQ_ERR_UNSUPPORTED, "eq_quant_nvfp4_weight: K must be a multiple of 16");
    EQ_REQUIRE(aligned(packed, 8), EQ_ERR_BAD_ALIGN, "eq_quant_nvfp4_weight: packed must be 8-byte aligned");
    int st = eq_nvfp4_global_scale(values, N, K, in_dtype, scale_2, scratch_u32, stream_);  // the same max(amax, 1e-12) / (6 * 448)
    if (st != EQ_OK) return st;
    const int64_t total = N * (K / 16);
    const unsigned grid = static_cast<unsigned>(ceil_div(total, 128));
    switch (in_dtype) {
        case EQ_F16: quant_nvfp4_weight_kernel<__half><<<grid, 128, 0, stream>>>(static_cast<const __half*>(values), N, K, scale_2, packed, scale_bits); break;
        case EQ_BF16: quant_nvfp4_weight_kernel<__nv_bfloat16><<<grid, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(values), N, K, scale_2, packed, scale_bits); break;
        case EQ_F32: quant_nvfp4_weight_kernel<float><<<grid, 128, 0, stream>>>(static_cast<const float*>(values), N, K, scale_2, packed, scale_bits); break;
        default: return fail(EQ_ERR_BAD_ARG, "eq_quant_nvfp4_weight: unknown dtype %d", in_dtype);
    }
    EQ_LAUNCH_OK("quant_nvfp4_weight_kernel");
    return EQ_OK;
}

// `pad_rows`: zero the tiled scales of the rows between M and the end of its 128-row block (what a caller that reads the
// tiled layout expects).  The linear passes false: those rows of A arrive as zeros from the tensor map and the output
// rows they produce are never stored.  `status`: cleared by the kernel for the linear behind it.
static int quant_nvfp4_act(const void* x, int64_t M, int64_t K, int in_dtype, const float* input_scale, uint8_t* codes, uint8_t* scale_bits,
                           uint8_t* scale_tiled, bool pad_rows, int* status, cudaStream_t stream) {
    EQ_REQUIRE(M >= 0 && K > 0, EQ_ERR_BAD_ARG, "eq_quant_nvfp4_act: bad extents");
    if (M == 0) return EQ_OK;
    EQ_REQUIRE(x && input_scale && codes, EQ_ERR_BAD_ARG, "eq_quant_nvfp4_act: null pointer");
    EQ_REQUIRE(K % 16 == 0 && (!scale_tiled || K % 64 == 0), EQ_ERR_UNSUPPORTED, "eq_quant_nvfp4_act: K must be a multiple of 16 (64 with tiled scales)");
    EQ_REQUIRE(aligned(codes, 8), EQ_ERR_BAD_ALIGN, "eq_quant_nvfp4_act: codes must be 8-byte aligned");
    EQ_REQUIRE(in_dtype == EQ_F16 || in_dtype == EQ_BF16 || in_dtype == EQ_F32, EQ_ERR_BAD_ARG, "eq_quant_nvfp4_act: unknown dtype %d", in_dtype);
    if (scale_tiled && pad_rows) EQ_CUDA_OK(cudaMemsetAsync(scale_tiled, 0, sf_tiled_bytes(M, K), stream));
    const int64_t total = M * (K / 16);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ceil_div(total, 128)));
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = status ? 1 : 0;  // inside the linear: resident, and past its launch latency, when the kernel before it ends
    // (up to 64 rows the kernel of one thread per block has the shorter chain: a linear of 16 rows 12.9 against 13.5 us)
    if (M > 64 && in_dtype != EQ_F32 && scale_tiled && !scale_bits && aligned(x, 16) && aligned(scale_tiled, 4)) {
        const int64_t row_blocks = ceil_div(M, 128);
        cfg.gridDim = dim3(static_cast<unsigned>(K / 64), static_cast<unsigned>(row_blocks < 65535 ? row_blocks : 65535));
        cfg.blockDim = dim3(512);
        const uint4* xv = static_cast<const uint4*>(x);
        const int k64 = static_cast<int>(K / 64);
        if (in_dtype == EQ_F16) EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, quant_nvfp4_act_atoms_kernel<__half>, xv, M, k64, input_scale, codes, scale_tiled, status));
        else EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, quant_nvfp4_act_atoms_kernel<__nv_bfloat16>, xv, M, k64, input_scale, codes, scale_tiled, status));
        return EQ_OK;
    }
    switch (in_dtype) {
        case EQ_F16: EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, quant_nvfp4_act_kernel<__half>, static_cast<const __half*>(x), M, K, input_scale, codes, scale_bits, scale_tiled, status)); break;
        case EQ_BF16: EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, quant_nvfp4_act_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(x), M, K, input_scale, codes, scale_bits, scale_tiled, status)); break;
        default: EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, quant_nvfp4_act_kernel<float>, static_cast<const float*>(x), M, K, input_scale, codes, scale_bits, scale_tiled, status)); break;
    }
    return EQ_OK;
}

extern "C" int eq_quant_nvfp4_act(const void* x, int64_t M, int64_t K, int in_dtype, const float* input_scale, uint8_t* codes,
                                  uint8_t* scale_bits, uint8_t* scale_tiled, void* stream_) {
    return quant_nvfp4_act(x, M, K, in_dtype, input_scale, codes, scale_bits, scale_tiled, true, nullptr, static_cast<cudaStream_t>(stream_));
}

extern "C" size_t eq_nvfp4_workspace_bytes(int64_t M, int64_t K) {
    if (M <= 0 || K <= 0) return 0;
    return align_up(static_cast<size_t>(M) * K / 2, 256) + align_up(sf_tiled_bytes(M, K), 256) + 256;
}

static int nvfp4_linear_any(const uint8_t* weight, const uint8_t* weight_scale_tiled, const float* weight_scale_2, int64_t N, int64_t K,
                            const void* x, const float* input_scale, int64_t M, int act_dtype, void* y, void* workspace, size_t workspace_bytes,
                            void* stream_, const void* gamma, float eps);

extern "C" int eq_nvfp4_linear(const uint8_t* weight, const uint8_t* weight_scale_tiled, const float* weight_scale_2, int64_t N,
                               int64_t K, const void* x, const float* input_scale, int64_t M, int act_dtype, void* y, void* workspace,
                               size_t workspace_bytes, void* stream_) {
    return nvfp4_linear_any(weight, weight_scale_tiled, weight_scale_2, N, K, x, input_scale, M, act_dtype, y, workspace, workspace_bytes, stream_,
                            nullptr, 0.f);
}

extern "C" int eq_nvfp4_linear_rmsnorm(const uint8_t* weight, const uint8_t* weight_scale_tiled, const float* weight_scale_2, int64_t N, int64_t K,
                                       const void* x, const void* gamma, float eps, const float* input_scale, int64_t M, int act_dtype, void* y,
                                       void* workspace, size_t workspace_bytes, void* stream_) {
    EQ_REQUIRE(gamma, EQ_ERR_BAD_ARG, "eq_nvfp4_linear_rmsnorm: null norm weight");
    return nvfp4_linear_any(weight, weight_scale_tiled, weight_scale_2, N, K, x, input_scale, M, act_dtype, y, workspace, workspace_bytes, stream_, gamma,
                            eps);
}

static int nvfp4_linear_any(const uint8_t* weight, const uint8_t* weight_scale_tiled, const float* weight_scale_2, int64_t N, int64_t K,
                            const void* x, const float* input_scale, int64_t M, int act_dtype, void* y, void* workspace, size_t workspace_bytes,
                            void* stream_, const void* gamma, float eps) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    EQ_REQUIRE(N > 0 && K > 0 && M >= 0, EQ_ERR_BAD_ARG, "eq_nvfp4_linear: bad extents M=%lld K=%lld N=%lld", (long long)M, (long long)K, (long long)N);
    if (M == 0) return EQ_OK;
    EQ_REQUIRE(weight && weight_scale_tiled && weight_scale_2 && x && input_scale && y, EQ_ERR_BAD_ARG, "eq_nvfp4_linear: null pointer");
    EQ_REQUIRE(act_dtype == EQ_F16 || act_dtype == EQ_BF16, EQ_ERR_BAD_ARG, "eq_nvfp4_linear: activations must be f16 or bf16");
    EQ_REQUIRE(K % 256 == 0 && N % 8 == 0, EQ_ERR_UNSUPPORTED, "eq_nvfp4_linear: needs K %% 256 == 0 and N %% 8 == 0 (K=%lld N=%lld)", (long long)K, (long long)N);
    EQ_REQUIRE(aligned(weight, 16) && aligned(weight_scale_tiled, 256) && aligned(y, 16), EQ_ERR_BAD_ALIGN, "eq_nvfp4_linear: weight and scales must be 16-byte aligned");
    EQ_REQUIRE(workspace && workspace_bytes >= eq_nvfp4_workspace_bytes(M, K), EQ_ERR_WORKSPACE, "eq_nvfp4_linear: workspace of %zu bytes needed, %zu given",
               eq_nvfp4_workspace_bytes(M, K), workspace_bytes);
    EQ_REQUIRE(aligned(workspace, 256), EQ_ERR_BAD_ALIGN, "eq_nvfp4_linear: workspace must be 256-byte aligned");
    uint8_t* codes = static_cast<uint8_t*>(workspace);
    uint8_t* sfa = codes + align_up(static_cast<size_t>(M) * K / 2, 256);
    int* status = reinterpret_cast<int*>(sfa + align_up(sf_tiled_bytes(M, K), 256));
    int st = EQ_OK;
    if (gamma) {
        // the model's RMSNorm inside the quantize kernel (a programmatic dependent, like the plain quantize)
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(M));
        cfg.blockDim = dim3(256);
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (act_dtype == EQ_F16)
            EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, rmsnorm_quant_nvfp4_rows_kernel<__half>, static_cast<const __half*>(x), static_cast<const __half*>(gamma), eps,
                                          K, input_scale, codes, sfa, status));
        else
            EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, rmsnorm_quant_nvfp4_rows_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(x),
                                          static_cast<const __nv_bfloat16*>(gamma), eps, K, input_scale, codes, sfa, status));
    } else {
        st = quant_nvfp4_act(x, M, K, act_dtype, input_scale, codes, nullptr, sfa, false, status, stream);
    }
    if (st != EQ_OK) return st;
    CUtensorMap map_a, map_b;
    if (M <= 16) {
        // decode-shaped: weight tiles as the MMA's A operand, the rows as B
        st = make_tensor_map_2d(&map_a, weight, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K / 2, K / 2, 128, kBKBytes, CU_TENSOR_MAP_SWIZZLE_128B);
        if (st != EQ_OK) return st;
        st = make_tensor_map_2d(&map_b, codes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, M, K / 2, K / 2, 16, kBKBytes, CU_TENSOR_MAP_SWIZZLE_128B);
        if (st != EQ_OK) return st;
        auto run = [&](auto kernel, auto* yt) -> int {
            EQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kDecSmem)));
            EQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(static_cast<unsigned>(ceil_div(N, 128)));
            cfg.blockDim = dim3(kGemmThreads);
            cfg.dynamicSmemBytes = kDecSmem;
            cfg.stream = stream;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            const uint8_t* sfx = sfa;
            EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, weight_scale_tiled, sfx, input_scale, weight_scale_2, yt, static_cast<int>(M),
                                          static_cast<int>(N), static_cast<int>(K), status));
            return EQ_OK;
        };
        return act_dtype == EQ_F16 ? run(nvfp4_decode_kernel<__half>, static_cast<__half*>(y))
                                   : run(nvfp4_decode_kernel<__nv_bfloat16>, static_cast<__nv_bfloat16*>(y));
    }
    // codes are bytes holding two e2m1 values: the maps move bytes; 128 bytes = 256 elements of K per tile row
    st = make_tensor_map_2d(&map_a, codes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, M, K / 2, K / 2, kBM, kBKBytes, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != EQ_OK) return st;
    // More than 128 rows: 256 x 256 tiles on CTA pairs (figures in gemm_pair.cu).  128 x 256 tiles of one CTA, where they fit one wave, stay
    // - for an odd number of 128-row tiles where the pairs, half of the last row of tiles empty, take two waves (N=12288, 300 rows: K=5120
    //   19.9 us against 24.9, K=1024 10.4 against 14.9);
    // - for a short K, where the pairs' cluster barriers and second operand hand-over are not hidden (one-CTA : pairs, us; K=512 N=2048,
    //   256 rows 7.7 : 8.2; K=1024 N=4096, 129 rows 8.2 : 8.7, 1000 rows 9.2 : 10.2; K=2048 N=6144, 257 rows 11.3 : 12.3; K=2560 2.6 % and
    //   K=3072 1.5 % on the mean of 50 shapes; K=4096 even, K=8192 N=4096, 200 rows 19.8 : 17.9).
    // Linears with the quantize, graph replays over four weights, both forms forced.
    const int64_t col_tiles = ceil_div(N, 256);
    const bool one_wave = ceil_div(M, 128) * col_tiles <= sm_count();
    const bool pairs = M > 128 && !(one_wave && (K < 4096 || ceil_div(M, 256) * col_tiles > sm_count() / 2));
    if (pairs) return nvfp4_pair_launch(codes, sfa, input_scale, weight, weight_scale_tiled, weight_scale_2, y, M, N, K, act_dtype, status, stream);
    // the 128-row-block scale layout at the front of the blob
    const int bn = M <= 128 ? 128 : 256;
    st = make_tensor_map_2d(&map_b, weight, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K / 2, K / 2, bn, kBKBytes, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != EQ_OK) return st;
    dim3 grid(static_cast<unsigned>(ceil_div(M, kBM)), static_cast<unsigned>(ceil_div(N, bn)));
    auto run = [&](auto kernel, size_t smem, auto* yt) -> int {
        EQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        EQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(kGemmThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // may start (and fetch weights) while the quantize runs
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const uint8_t* sfa_c = sfa;
        EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, sfa_c, weight_scale_tiled, input_scale, weight_scale_2, yt, static_cast<int>(M),
                                      static_cast<int>(N), static_cast<int>(K), status));
        return EQ_OK;
    };
    if (act_dtype == EQ_F16)
        return bn == 128 ? run(nvfp4_gemm_tc_kernel<__half, 128>, Fp4Cfg<128>::kSmem, static_cast<__half*>(y))
                         : run(nvfp4_gemm_tc_kernel<__half, 256>, Fp4Cfg<256>::kSmem, static_cast<__half*>(y));
    return bn == 128 ? run(nvfp4_gemm_tc_kernel<__nv_bfloat16, 128>, Fp4Cfg<128>::kSmem, static_cast<__nv_bfloat16*>(y))
                     : run(nvfp4_gemm_tc_kernel<__nv_bfloat16, 256>, Fp4Cfg<256>::kSmem, static_cast<__nv_bfloat16*>(y));
}

extern "C" int eq_nvfp4_status(const void* workspace, int64_t M, int64_t K, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    EQ_REQUIRE(workspace && M > 0 && K > 0, EQ_ERR_BAD_ARG, "eq_nvfp4_status: bad arguments");
    const unsigned char* base = static_cast<const unsigned char*>(workspace);
    const int* status = reinterpret_cast<const int*>(base + align_up(static_cast<size_t>(M) * K / 2, 256) + align_up(sf_tiled_bytes(M, K), 256));
    int host = 0;
    EQ_CUDA_OK(cudaMemcpyAsync(&host, status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    EQ_CUDA_OK(cudaStreamSynchronize(stream));
    EQ_REQUIRE(host == 0, EQ_ERR_TIMEOUT, "eq_nvfp4_status: a bounded pipeline wait ran out (code %d)", host);
    return EQ_OK;
}
