// FP8 W8A8 (per-channel) and NVFP4 W4A4 GEMMs on CTA pairs (tcgen05 cta_group::2), for more than 128 rows.
//
// A pair owns a 256 x 256 output tile: 128 rows of it in each CTA's TMEM.  Each CTA fetches its own 128 activation rows and
// HALF of the 256 weight rows; the pair's MMA (256 x 256 x 32 bytes of K, issued by the even CTA) reads both halves.
//   warp 0      TMA of this CTA's operands, completing on the even CTA's barrier; weights of the first tile are requested
//               before the grid ahead (the activation quantize) has ended
//   warp 1      MMA issuer (even CTA)
//   warps 2..9  epilogue: two warps per TMEM lane quarter, alternating 32-column chunks
// Persistent over tiles with the epilogue of one under the main loop of the next.  FP8: two accumulators of 256 columns fill
// TMEM.  NVFP4 needs 48 columns for its scale factors, so its two accumulators share columns 208..255: the epilogue reads the
// shared columns first (from the top in the lower accumulator, from the bottom in the upper one) and the next tile's MMAs start
// as soon as those are in registers.
//
// Why pairs: a lone CTA's tile is bound by shared memory (fills and operand reads of a 256 x 256 FP8 tile, 160 KB a K step, are 1250
// cycles at 128 B/clock beside 1024 of MMA; of a 256 x 224 NVFP4 tile 164 KB, 1280 beside 950); here an SM moves 64 KB for
// 128 x 256 x 128 bytes, 512 cycles beside 512.
// Measured (us a linear, quantize included; K=5120 N=17408; graph replays over several weights).  One-CTA tiles -> here, both with the
// two-pass quantizers of that time: NVFP4 512 rows 36.7 -> 29.3, 1024 rows 70 -> 50, 4096 rows 235 -> 162; FP8 200 rows 47 -> 35, 1024
// rows 103 -> 87, 2048 rows 198 -> 158, 8192 rows 761 -> 559.  With the quantizers of quant.cuh: NVFP4 512 rows 27.5, 1024 rows 47,
// 4096 rows 158 to 168 (the GEMM alone 135: 5.4 PFLOP/s); FP8 200 rows 27.3, 1024 rows 76, 2048 rows 141, 8192 rows 550 to 626 (power cap).
#include "gemm_pair.cuh"
#include "tc_common.cuh"

namespace eq {
namespace {

constexpr int kBKBytes = 128;                  // K per stage: 128 e4m3 or 256 e2m1 elements
constexpr int kTile = 128 * kBKBytes;          // a CTA's 128 rows of either operand
constexpr int kAtoms = 4 * 512;                // scale atoms of 128 rows and one stage (NVFP4)
constexpr int kEpiWarps = 8;
constexpr int kThreads = (2 + kEpiWarps) * 32;

template <bool FP4>
struct PairCfg {
    static constexpr int kStageBytes = 2 * kTile + (FP4 ? 3 * kAtoms : 0);  // scales: this CTA's rows, both halves of the weight
    static constexpr int kStages = FP4 ? 5 : 6;
    static constexpr int kAcc1 = FP4 ? 208 : 256;  // first column of the second accumulator
    static constexpr int kAhead = FP4 ? 1 : 2;     // tiles between an accumulator's release and its next use
    static constexpr int kScaleBytes = FP4 ? 0 : 2 * 256 * 4;
    static constexpr size_t kSmem = static_cast<size_t>(kStages) * kStageBytes + 1024 + 256 + kScaleBytes;
    static_assert(kSmem <= 227 * 1024, "one CTA per SM");
    static_assert(kAcc1 + 256 + (FP4 ? 48 : 0) <= 512, "both accumulators and the scales fit TMEM");
};

__device__ __forceinline__ void mma_pair_fp8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
    const uint32_t acc = accumulate ? 1u : 0u;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_pair_fp4(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t tsfa, uint32_t tsfb, bool accumulate) {
    const uint32_t acc = accumulate ? 1u : 0u;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc), "r"(tsfa), "r"(tsfb)
        : "memory");
}
// In both CTAs of the pair, each from its own shared memory into its own TMEM.
__device__ __forceinline__ void tmem_cp_pair(uint32_t taddr, uint64_t smem_desc) {
    asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(smem_desc) : "memory");
}

struct PairArgs {
    const float* sx;  // FP8: [M]; NVFP4: the activations' global scale
    const float* sw;  // FP8: [N]; NVFP4: the weight's global scale
    void* y;
    int M, N, k_blocks, row_tiles, units;
    int* status;
};

template <typename OutT, bool FP4>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_sfa,
                     const __grid_constant__ CUtensorMap map_sfb, const PairArgs p) {
    using Cfg = PairCfg<FP4>;
    constexpr int S = Cfg::kStages;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t tiles_a = tc::smem_u32(smem), tiles_b = tiles_a + S * kTile, sfs_a = tiles_b + S * kTile, sfs_b = sfs_a + S * kAtoms;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S * Cfg::kStageBytes);
    const uint32_t full = tc::smem_u32(bars);  // [S] the even CTA's: both CTAs' copies
    const uint32_t empty = full + 8 * S;       // [S] MMA -> TMA, in each CTA
    const uint32_t acc_full = empty + 8 * S;   // [2] MMA -> epilogue, in each CTA
    const uint32_t acc_free = acc_full + 16;   // [2] the even CTA's: both CTAs' epilogue warps
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
    float* sw_tile = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(bars) + 256);  // FP8: [2][256] scales of the tile's columns

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = static_cast<int>(tc::cluster_rank());
    const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            tc::mbar_init(full + 8 * s, 1);
            tc::mbar_init(empty + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(acc_full + 8 * b, 1);
            tc::mbar_init(acc_free + 8 * b, 2 * kEpiWarps);
        }
        tc::mbar_fence_init();
    }
    __syncthreads();
    tc::cluster_sync();  // both CTAs run, the peer's barriers exist
    // Not before: an allocation for the pair that one CTA asks for while the other has not started can wait for ever.
    if (warp == 1) tc::tmem_alloc_pair(tc::smem_u32(tmem_slot), 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();
    tc::fence_after_sync();
    // With the TMEM columns in hand: a dependent grid that took them first and then waited for this one would never give them back.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t lead_full = tc::map_to_rank(full, 0), lead_free = tc::map_to_rank(acc_free, 0);
    // row tiles fastest: the pairs that share a weight tile run together and the weight comes from DRAM once
    auto row_of = [&](int u) { return (u % p.row_tiles) * 256; };
    auto col_of = [&](int u) { return (u / p.row_tiles) * 256; };

    if (warp == 0) {
        if (tc::elect_one()) {
            tc::tma_prefetch_desc(&map_a);
            tc::tma_prefetch_desc(&map_b);
            auto weights = [&](int u, int kb, int s) {
                if (rank == 0) tc::mbar_expect_tx(full + 8 * s, 2 * Cfg::kStageBytes);
                const uint32_t bar = lead_full + 8 * s;
                const int n0 = col_of(u);
                tc::tma_load_2d_pair(tiles_b + s * kTile, &map_b, kb * kBKBytes, n0 + rank * 128, bar);
                if constexpr (FP4) {  // both CTAs hold the scales of all 256 columns
                    const int atom = (n0 >> 7) * 4 * p.k_blocks + 4 * kb;
                    tc::tma_load_2d_pair(sfs_b + s * 2 * kAtoms, &map_sfb, 0, atom, bar);
                    tc::tma_load_2d_pair(sfs_b + s * 2 * kAtoms + kAtoms, &map_sfb, 0, atom + 4 * p.k_blocks, bar);
                }
            };
            auto rows = [&](int u, int kb, int s) {
                const uint32_t bar = lead_full + 8 * s;
                const int m0 = row_of(u) + rank * 128;
                tc::tma_load_2d_pair(tiles_a + s * kTile, &map_a, kb * kBKBytes, m0, bar);
                if constexpr (FP4) tc::tma_load_2d_pair(sfs_a + s * kAtoms, &map_sfa, 0, (m0 >> 7) * 4 * p.k_blocks + 4 * kb, bar);
            };
            const int ahead = p.k_blocks < S ? p.k_blocks : S;
            for (int kb = 0; kb < ahead; ++kb) weights(cluster, kb, kb);
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int kb = 0; kb < ahead; ++kb) rows(cluster, kb, kb);
            int seq = 0;
            bool broken = false;
            for (int u = cluster; u < p.units && !broken; u += clusters) {
                for (int kb = 0; kb < p.k_blocks; ++kb, ++seq) {
                    if (seq < ahead) continue;
                    const int s = seq % S;
                    if (seq >= S && !tc::mbar_wait(empty + 8 * s, ((seq / S) - 1) & 1)) {
                        atomicExch(p.status, 1);
                        broken = true;
                        break;
                    }
                    weights(u, kb, s);
                    rows(u, kb, s);
                }
            }
            // nobody else waits for these: the pair does not end with a copy under way into either CTA (the even CTA's barriers count both)
            if (broken && rank == 0)
                for (int i = seq < S ? 0 : seq - S; i < seq; ++i) tc::mbar_wait(full + 8 * (i % S), (i / S) & 1);
        }
    } else if (warp == 1) {
        asm volatile("griddepcontrol.wait;" ::: "memory");  // bounded waits count from the moment the codes exist
        if (rank == 0 && tc::elect_one()) {
            constexpr uint32_t idesc = FP4 ? tc::instr_desc_nvfp4(256, 256, 0, 0) : tc::instr_desc(0, 0, 256, 256);
            const uint32_t tmem_sfa = tmem_base + 464, tmem_sfb = tmem_base + 480;  // NVFP4: 4 and 8 columns per 64 of K
            int seq = 0, t = 0;
            bool broken = false;
            for (int u = cluster; u < p.units && !broken; u += clusters, ++t) {
                const int b = t & 1, before = t - Cfg::kAhead;
                if (before >= 0) broken = !tc::mbar_wait(acc_free + 8 * (before & 1), (before >> 1) & 1);
                const uint32_t d = tmem_base + b * Cfg::kAcc1;
                for (int kb = 0; kb < p.k_blocks && !broken; ++kb, ++seq) {
                    const int s = seq % S;
                    if (!tc::mbar_wait(full + 8 * s, (seq / S) & 1)) {
                        broken = true;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint32_t a_addr = tiles_a + s * kTile, b_addr = tiles_b + s * kTile;
                    if constexpr (FP4) {  // all scale copies of the stage are queued before its first MMA
                        const uint32_t sfa_addr = sfs_a + s * kAtoms, sfb_addr = sfs_b + s * 2 * kAtoms;
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            tmem_cp_pair(tmem_sfa + ks * 4, tc::smem_desc_sf(sfa_addr + ks * 512));
                            tmem_cp_pair(tmem_sfb + ks * 8, tc::smem_desc_sf(sfb_addr + ks * 512));
                            tmem_cp_pair(tmem_sfb + ks * 8 + 4, tc::smem_desc_sf(sfb_addr + kAtoms + ks * 512));
                        }
                    }
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                        const uint64_t da = tc::smem_desc_k_sw128(a_addr + ks * 32), db = tc::smem_desc_k_sw128(b_addr + ks * 32);
                        if constexpr (FP4)
                            mma_pair_fp4(d, da, db, idesc, tmem_sfa + ks * 4, tmem_sfb + ks * 8, kb > 0 || ks > 0);
                        else
                            mma_pair_fp8(d, da, db, idesc, kb > 0 || ks > 0);
                    }
                    tc::commit_pair(empty + 8 * s);
                }
                tc::commit_pair(acc_full + 8 * b);
                if (broken) {
                    atomicExch(p.status, 2);
                    // neither shared memory nor TMEM goes back with a copy (one that was never issued runs out) or an MMA under way
                    for (int i = seq; i < seq + S; ++i) tc::mbar_wait(full + 8 * (i % S), (i / S) & 1);
                    tc::mbar_wait(acc_full + 8 * b, (t >> 1) & 1);
                }
            }
        }
    } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        OutT* const y = static_cast<OutT*>(p.y);
        const float g = FP4 ? p.sx[0] * p.sw[0] : 0.f;
        int t = 0;
        bool broken = false;
        for (int u = cluster; u < p.units; u += clusters, ++t) {
            const int b = t & 1, n0 = col_of(u), m = row_of(u) + rank * 128 + quarter * 32 + lane;
            float row_scale = 0.f;
            if constexpr (!FP4) {
                if (m < p.M) row_scale = p.sx[m];
                const int i = threadIdx.x - 64;
                sw_tile[b * 256 + i] = n0 + i < p.N ? p.sw[n0 + i] : 0.f;
                asm volatile("bar.sync 1, 256;" ::: "memory");  // the epilogue warps; the other half of sw_tile is free again too
            }
            // A warp that gives up meets the others at the barrier above until its tiles end, and does nothing else: their waits, each with
            // its own clock, may have been met a moment later.
            if (!broken && !__all_sync(0xFFFFFFFFu, tc::mbar_wait(acc_full + 8 * b, (t >> 1) & 1))) {
                if (lane == 0) atomicExch(p.status, 3);
                broken = true;
            }
            if (broken) continue;
            tc::fence_after_sync();
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
                // NVFP4: chunks 6 and 7 of the lower accumulator, 0 and 1 of the upper one hold the shared columns
                const int c = 32 * (b == 0 ? 7 - half - 2 * i : half + 2 * i);
                uint32_t r[32];
                tc::tmem_ld_32x32(t_lane + b * Cfg::kAcc1 + c, r);
                tc::tmem_ld_wait();
                if (i == (FP4 ? 0 : 3)) {
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::arrive_pair(lead_free + 8 * b);
                }
                if (m < p.M && n0 + c < p.N) {
                    OutT* dst = y + static_cast<size_t>(m) * p.N + n0 + c;
                    auto out = [&](int k) {
                        if constexpr (FP4) return from_float<OutT>(__uint_as_float(r[k]) * g);
                        return from_float<OutT>(__uint_as_float(r[k]) * row_scale * sw_tile[b * 256 + c + k]);  // a broadcast
                    };
                    if (n0 + c + 32 <= p.N) {
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            uint32_t pk[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const OutT lo = out(8 * v + 2 * k), hi = out(8 * v + 2 * k + 1);
                                pk[k] = static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(&lo)) | (static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(&hi)) << 16);
                            }
                            reinterpret_cast<uint4*>(dst)[v] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 32; ++k)
                            if (n0 + c + k < p.N) dst[k] = out(k);
                    }
                }
            }
        }
    }
    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();  // neither CTA leaves while the other may still signal it or read its operands
    tc::fence_after_sync();
    if (warp == 1) tc::tmem_dealloc_pair(tmem_base, 512);
    __syncwarp();
    tc::cluster_sync();  // nor before the other has given its columns back
}

template <typename OutT, bool FP4>
int launch(const CUtensorMap& map_a, const CUtensorMap& map_b, const CUtensorMap& map_sfa, const CUtensorMap& map_sfb, const PairArgs& args, cudaStream_t stream) {
    auto kernel = gemm_pair_kernel<OutT, FP4>;
    EQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(PairCfg<FP4>::kSmem)));
    const int pairs = sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(2 * (args.units > pairs ? pairs : args.units)));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = PairCfg<FP4>::kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, map_sfa, map_sfb, args));
    return EQ_OK;
}

PairArgs make_args(const float* sx, const float* sw, void* y, int64_t M, int64_t N, int64_t row_bytes, int* status) {
    PairArgs a = {};
    a.sx = sx;
    a.sw = sw;
    a.y = y;
    a.M = static_cast<int>(M);
    a.N = static_cast<int>(N);
    a.k_blocks = static_cast<int>(row_bytes / kBKBytes);
    a.row_tiles = static_cast<int>(ceil_div(M, 256));
    a.units = static_cast<int>(a.row_tiles * ceil_div(N, 256));
    a.status = status;
    return a;
}

int map_rows(CUtensorMap* map, const uint8_t* base, int64_t rows, int64_t row_bytes) {
    return make_tensor_map_2d(map, base, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, rows, row_bytes, row_bytes, 128, kBKBytes, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace

int fp8_pair_launch(const uint8_t* qx, const float* sx, const uint8_t* w, const float* sw, void* y, int64_t M, int64_t N, int64_t K, int act_dtype,
                    int* status, cudaStream_t stream) {
    CUtensorMap map_a, map_b;
    int st = map_rows(&map_a, qx, M, K);
    if (st != EQ_OK) return st;
    st = map_rows(&map_b, w, N, K);
    if (st != EQ_OK) return st;
    const PairArgs args = make_args(sx, sw, y, M, N, K, status);
    return act_dtype == EQ_F16 ? launch<__half, false>(map_a, map_b, map_a, map_b, args, stream) : launch<__nv_bfloat16, false>(map_a, map_b, map_a, map_b, args, stream);
}

int nvfp4_pair_launch(const uint8_t* codes, const uint8_t* sfa, const float* gx, const uint8_t* w, const uint8_t* sfw, const float* gw, void* y, int64_t M,
                      int64_t N, int64_t K, int act_dtype, int* status, cudaStream_t stream) {
    CUtensorMap map_a, map_b, map_sfa, map_sfb;
    int st = map_rows(&map_a, codes, M, K / 2);
    if (st != EQ_OK) return st;
    st = map_rows(&map_b, w, N, K / 2);
    if (st != EQ_OK) return st;
    // scale atoms: rows of 512 bytes (as 128 words), [row block][k64]; four of them are a stage's.  Row blocks beyond the matrix read as zeros.
    st = make_tensor_map_2d(&map_sfa, sfa, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, ceil_div(M, 128) * (K / 64), 128, 512, 4, 128, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (st != EQ_OK) return st;
    st = make_tensor_map_2d(&map_sfb, sfw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, ceil_div(N, 128) * (K / 64), 128, 512, 4, 128, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (st != EQ_OK) return st;
    const PairArgs args = make_args(gx, gw, y, M, N, K / 2, status);
    return act_dtype == EQ_F16 ? launch<__half, true>(map_a, map_b, map_sfa, map_sfb, args, stream) : launch<__nv_bfloat16, true>(map_a, map_b, map_sfa, map_sfb, args, stream);
}

}  // namespace eq
