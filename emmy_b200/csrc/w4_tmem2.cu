// W4A16 linear for prefill (w4_tmem_pairs: when): the weights-in-TMEM form of w4_tmem.cu on CTA pairs (tcgen05 cta_group::2).
//
// A pair owns 256 output channels (128 TMEM lanes in each CTA) by up to NB activation rows.  Each CTA expands its own
// channels' int4 into its own TMEM (A operand) and fetches HALF of the activation rows; the pair's MMA (256 x rows x 16,
// issued by the even CTA) reads both halves.  So per multiply-add a CTA moves half the activation bytes of a lone CTA
// through L2 and shared memory, nothing of the weight but its packed bytes touches shared memory, and an SM expands 128
// channels per K step where the one-CTA 256 x 256 tile (w4_gemm.cu) expands 256.
//   warps 0..15   dequant (cp.async ring per warp, tcgen05.st), as in w4_tmem.cu: four warps per item, four items at a time,
//                 one TMEM stage each; then the unit's epilogue
//   warp 16       TMA of this CTA's half of the rows, completing on the even CTA's barrier
//   warp 17       MMA issuer (even CTA)
// TMEM: 256 accumulator columns + 4 stages of 64 columns of A = 512.  (Two accumulators of 192 columns and two stages,
// with the epilogue under the next unit's main loop, measured slower: the stages are what hides the expansion's latency.)
// Measured (us, one-CTA 256 x 256 tiles with the dequant through shared memory -> here): K=4096 N=14336, 2048 rows 232.6 ->
// 182.4; [gate | up] of hidden 4096, intermediate 14336: 300 rows 111 -> 82, 1024 rows 242 -> 190, 4096 rows 841 -> 724.
// Persistent over units (column tile of 256, row tile); A holds (q - z) * scale in the activation dtype, f32 accumulation
// over all of K.
#include "tc_common.cuh"
#include "w4_tile.cuh"
#include "w4_tmem.cuh"

namespace eq {
namespace {

using namespace tm;

constexpr int kGK = 64;
constexpr int kDW = 16, kGroups = kDW / 4;  // dequant warps; groups of four, each with its own stage
constexpr int kNB = 256;                    // rows per unit at most
constexpr int kHalfRows = kNB / 2;          // rows a CTA fetches
constexpr int kStagesA = kGroups, kStagesB = 3, kDepth = 3;
constexpr int kTileB = kHalfRows * 256;  // an item's rows: two 64-wide pieces
constexpr int kRing = kDW * kDepth * 2 * kItemBytes;
constexpr int kBoxRows = 32;
constexpr int kWarps = kDW + 2, kThreads = kWarps * 32;
constexpr size_t kSmem = 1024 + static_cast<size_t>(kStagesB) * kTileB + kRing + 256;
constexpr uint32_t kTmemCols = 512;
// Of the choice of row tiles: cycles of an SM for one item of 128 channels, for a unit's prologue and epilogue.  Weights of a model, not
// measured cycles: at 1965 MHz an item takes 0.32 us (620 cycles) with 32 or 48 rows, 0.40 with 80, 0.42 with 112, 0.51 with 128, 0.60
// with 144, 0.81 with 256 (K=4096 against 12288, N=18944), a unit 2.5 to 5 us.  900 cycles an item in their place: 300 rows equal, K=4096
// I=3584 at 600 rows 59.7 -> 69.9 us.
constexpr int64_t kExpandCycles = 480, kUnitCycles = 3500;
static_assert(kNB + 64 * kStagesA <= 512, "accumulator and A stages fill TMEM");
static_assert(kSmem <= 227 * 1024, "one CTA per SM");

__device__ __forceinline__ void mma_f16_ts_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
    const uint32_t acc = accumulate ? 1u : 0u;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc)
        : "memory");
}
template <typename ActT, bool CVT, bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    w4a16_tmem_pair_kernel(const __grid_constant__ CUtensorMap map_x, const W4TmemArgs a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t tiles_b = tc::smem_u32(smem);
    unsigned char* ring = smem + kStagesB * kTileB;
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring + kRing);
    constexpr int kBars = 2 * kStagesA + 2 * kStagesB + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars);
    const uint32_t full_a = tc::smem_u32(bars), empty_a = full_a + 8 * kStagesA, full_b = empty_a + 8 * kStagesA, empty_b = full_b + 8 * kStagesB,
                   acc_full = empty_b + 8 * kStagesB, acc_empty = acc_full + 8;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_rank();
    const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;
    const int items = a.K / 128, n_tiles = a.N / 16;  // SWIGLU: a CTA's channels are four gate and four up tiles
    const int units = a.units;

    auto locate = [&](int u, int& col, int& row0, int& rows) {
        const int rt = u % a.row_tiles;  // row tiles fastest: the pairs that share a weight tile run together
        col = u / a.row_tiles;
        row0 = rt * a.rows_per_tile;
        rows = min(a.rows_per_tile, a.M - row0);
    };
    auto first_tile = [&](int col, int q) { return SWIGLU ? (col * 2 + static_cast<int>(rank)) * 4 + q : (col * 2 + static_cast<int>(rank)) * 8 + 2 * q; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStagesA; ++s) {
            tc::mbar_init(full_a + 8 * s, 8);  // four warps of each CTA
            tc::mbar_init(empty_a + 8 * s, 1);
        }
        for (int s = 0; s < kStagesB; ++s) {
            tc::mbar_init(full_b + 8 * s, 1);
            tc::mbar_init(empty_b + 8 * s, 1);
        }
        tc::mbar_init(acc_full, 1);
        tc::mbar_init(acc_empty, 2 * kDW);
        tc::mbar_fence_init();
    }
    __syncthreads();
    tc::cluster_sync();  // both CTAs run, the peer's barriers exist
    // Not before: an allocation for the pair that one CTA asks for while the other has not started can wait for ever.
    if (warp == kWarps - 1) tc::tmem_alloc_pair(tc::smem_u32(tmem_slot), kTmemCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();
    tc::fence_after_sync();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // with the TMEM columns in hand (w4_tmem.cu)
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_a = tmem_base + kNB;
    const uint32_t lead_full_a = tc::map_to_rank(full_a, 0), lead_full_b = tc::map_to_rank(full_b, 0), lead_acc_empty = tc::map_to_rank(acc_empty, 0);

    if (warp < kDW) {
        const int q = warp & 3, wg = warp >> 2;
        const uint32_t my_ring = tc::smem_u32(ring) + warp * (kDepth * 2 * kItemBytes);
        const LaneOffsets lo;
        int pf_unit = cluster, pf_item = wg;
        uint32_t pf_slot = my_ring;
        const unsigned char *pf0 = nullptr, *pf1 = nullptr;  // the warp's two tiles: item pf_item of unit pf_unit, at this lane
        auto pf_locate = [&]() {
            int col, row0, rows;
            locate(pf_unit, col, row0, rows);
            const unsigned char* base = a.wq + static_cast<size_t>(pf_item) * kItemBytes + lane * 16;
            // tiles beyond the weight read tile 0: their channels are never stored
            int t0 = first_tile(col, q), t1 = SWIGLU ? t0 + n_tiles / 2 : t0 + 1;
            if (SWIGLU && t0 >= n_tiles / 2) t0 = 0;
            if (t0 >= n_tiles) t0 = 0;
            if (t1 >= n_tiles) t1 = 0;
            pf0 = base + static_cast<size_t>(t0) * items * kItemBytes;
            pf1 = base + static_cast<size_t>(t1) * items * kItemBytes;
        };
        auto prefetch = [&]() {
            if (pf_item >= items && pf_unit < units) {
                do {
                    pf_item -= items;
                    pf_unit += clusters;
                } while (pf_unit < units && pf_item >= items);
                if (pf_unit < units) pf_locate();
            }
            if (pf_unit < units) {
                fetch_items(pf_slot, lo, pf0, pf1);
                pf0 += kGroups * kItemBytes;
                pf1 += kGroups * kItemBytes;
                pf_item += kGroups;
            }
            cp_commit();
            pf_slot += 2 * kItemBytes;
            if (pf_slot == my_ring + kDepth * 2 * kItemBytes) pf_slot = my_ring;
        };
        if (pf_item < items) pf_locate();
#pragma unroll 1
        for (int d = 0; d < kDepth; ++d) prefetch();

        int next = wg;  // this warp's next item (every fourth of the pair's sequence), from the start of the current unit
        uint32_t phase = 1;
        bool first = true, broken = false, waited = false;
        int n_unit = 0;
        const uint32_t a_dst = tmem_a + (static_cast<uint32_t>(32 * q) << 16) + 64 * wg;
        const uint32_t my_full = lead_full_a + 8 * wg, my_empty = empty_a + 8 * wg;
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(32 * q) << 16);
        for (int u = cluster; u < units && !broken; u += clusters, ++n_unit) {
            for (; next < items; next += kGroups) {
                cp_wait<kDepth - 1>();
                __syncwarp();
                ItemWords w;
                load_item(pf_slot, lo, w);  // the oldest of the ring, and the next to be refilled
                __syncwarp();
                prefetch();  // refills it
                if (!first && !__all_sync(0xFFFFFFFFu, wait_asleep<true>(my_empty, phase))) {
                    if (lane == 0) atomicExch(a.status, 4);
                    broken = true;
                    break;
                }
                first = false;
                phase ^= 1;
                tc::fence_after_sync();
                expand_item<ActT, CVT, false>(w, a_dst);
                tmem_st_wait();
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::arrive_pair(my_full);
            }
            next -= items;
            // ---- epilogue: group wg takes the 16-row chunks wg, wg + 4, ...
            int col, row0, rows;
            locate(u, col, row0, rows);
            if (!waited) {
                asm volatile("griddepcontrol.wait;" ::: "memory");  // y may be in use by the previous grid
                waited = true;
            }
            if (!__all_sync(0xFFFFFFFFu, wait_asleep(acc_full, n_unit & 1))) {
                if (lane == 0) atomicExch(a.status, 3);
                break;
            }
            tc::fence_after_sync();
            const int tile_lo = first_tile(col, q);
#pragma unroll 1
            for (int c = 16 * wg; c < rows; c += 16 * kGroups) {
                uint32_t r[16];
                tc::tmem_ld_32x16(t_row + c, r);
                tc::tmem_ld_wait();
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
                emit16<ActT, SWIGLU, false>(a, v, tile_lo, row0, rows, c);
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::arrive_pair(lead_acc_empty);
        }
        cp_wait<0>();  // (left with copies under way only where a wait ran out)
    } else if (warp == kWarps - 2) {
        if (tc::elect_one()) {
            tc::tma_prefetch_desc(&map_x);
            asm volatile("griddepcontrol.wait;" ::: "memory");  // x may be the previous grid's output
            int seq = 0;
            bool broken = false;
            for (int u = cluster; u < units && !broken; u += clusters) {
                int col, row0, rows;
                locate(u, col, row0, rows);
                const int half_rows = ((rows + 15) & ~15) / 2;  // this CTA's rows of the MMA
                const int boxes = (half_rows + kBoxRows - 1) / kBoxRows;
                const int first = row0 + static_cast<int>(rank) * half_rows;
                for (int it = 0; it < items; ++it, ++seq) {
                    const int stage = seq % kStagesB, use = seq / kStagesB;
                    if (use > 0 && !wait_asleep(empty_b + 8 * stage, (use - 1) & 1)) {
                        atomicExch(a.status, 1);
                        broken = true;
                        break;
                    }
                    if (rank == 0) tc::mbar_expect_tx(full_b + 8 * stage, 2 * 2 * boxes * kBoxRows * 128);  // both CTAs' copies
                    const uint32_t dst = tiles_b + stage * kTileB;
                    for (int piece = 0; piece < 2; ++piece)
                        for (int bx = 0; bx < boxes; ++bx)
                            tc::tma_load_2d_pair(dst + piece * (kHalfRows * 128) + bx * (kBoxRows * 128), &map_x, it * 128 + piece * kGK, first + bx * kBoxRows,
                                             lead_full_b + 8 * stage);
                }
            }
            // nobody else waits for these: the pair does not end with a copy under way into either CTA's rows (the even CTA's
            // barriers count both)
            if (broken && rank == 0)
                for (int i = seq < kStagesB ? 0 : seq - kStagesB; i < seq; ++i) wait_asleep(full_b + 8 * (i % kStagesB), (i / kStagesB) & 1);
        }
    } else if (rank == 0) {
        if (tc::elect_one()) {
            int seq = 0, n_unit = 0;
            bool broken = false;
            for (int u = cluster; u < units && !broken; u += clusters, ++n_unit) {
                int col, row0, rows;
                locate(u, col, row0, rows);
                const uint32_t idesc = tc::instr_desc(Mul<ActT>::kFmt, Mul<ActT>::kFmt, 256, static_cast<uint32_t>((rows + 15) & ~15));
                if (n_unit > 0) broken = !wait_asleep<true>(acc_empty, (n_unit - 1) & 1);
                for (int it = 0; it < items && !broken; ++it, ++seq) {
                    const int sa = seq % kStagesA, sb = seq % kStagesB;
                    if (!wait_asleep<true>(full_b + 8 * sb, (seq / kStagesB) & 1) || !wait_asleep<true>(full_a + 8 * sa, (seq / kStagesA) & 1)) {
                        broken = true;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint64_t b_desc = tc::smem_desc_k_sw128(tiles_b + sb * kTileB);  // further steps: + bytes / 16
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)
                        mma_f16_ts_pair(tmem_base, tmem_a + 64 * sa + 8 * ks, b_desc + ((ks >> 2) * (kHalfRows * 128) + (ks & 3) * 32) / 16, idesc, ks > 0 || it > 0);
                    tc::commit_pair(empty_a + 8 * sa);
                    tc::commit_pair(empty_b + 8 * sb);
                }
                tc::commit_pair(acc_full);
                if (broken) {
                    atomicExch(a.status, 2);
                    // neither shared memory nor TMEM goes back with a copy (one that was never issued runs out) or an MMA under way
                    for (int i = seq; i < seq + kStagesB; ++i) wait_asleep(full_b + 8 * (i % kStagesB), (i / kStagesB) & 1);
                    wait_asleep(acc_full, n_unit & 1);
                }
            }
        }
    }
    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();  // neither CTA leaves while the other may still signal it or read its rows
    tc::fence_after_sync();
    if (warp == kWarps - 1) tc::tmem_dealloc_pair(tmem_base, kTmemCols);
    __syncwarp();
    tc::cluster_sync();  // nor before the other has given its columns back
}

template <typename ActT, bool SWIGLU>
int launch(const W4TmemArgs& a, const void* x, int scale_dtype, cudaStream_t stream) {
    CUtensorMap map_x;
    const CUtensorMapDataType elem = Mul<ActT>::kFmt == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int st = make_tensor_map_2d(&map_x, x, elem, 2, a.M, a.K, static_cast<uint64_t>(a.K) * 2, kBoxRows, kGK, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != EQ_OK) return st;
    const bool cvt = scale_dtype != (Mul<ActT>::kFmt == 0 ? EQ_F16 : EQ_BF16);
    auto kernel = cvt ? w4a16_tmem_pair_kernel<ActT, true, SWIGLU> : w4a16_tmem_pair_kernel<ActT, false, SWIGLU>;
    EQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem)));
    const int pairs = sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(2 * (a.units > pairs ? pairs : a.units)));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, map_x, a));
    return EQ_OK;
}

}  // namespace

int w4_tmem_pair_dense_launch(const unsigned char* wq, int scale_dtype, const void* x, void* y, int64_t M, int64_t N, int64_t K, int act_dtype, bool swiglu,
                              int* status, cudaStream_t stream) {
    W4TmemArgs a = {};
    a.wq = wq;
    a.y = y;
    a.M = static_cast<int>(M);
    a.N = static_cast<int>(N);
    a.K = static_cast<int>(K);
    a.status = status;
    // Row tiles of equal height, in the MMA's steps of 16; of the heights up to 256 the one whose last wave of units wastes
    // least: an item costs a pair 4 cycles a row, at least the expansion's, and a unit its epilogue.
    const int64_t items = K / 128, col_tiles = swiglu ? ceil_div(N / 32, 8) : ceil_div(N / 16, 16), pairs = sm_count() / 2;
    int64_t best = -1;
    for (int64_t tiles = ceil_div(M, kNB); tiles <= ceil_div(M, kNB) + 3; ++tiles) {
        const int64_t rows = ceil_div(ceil_div(M, tiles), 16) * 16, used = ceil_div(M, rows);
        const int64_t item = 4 * rows > kExpandCycles ? 4 * rows : kExpandCycles;
        const int64_t cost = ceil_div(col_tiles * used, pairs) * (items * item + kUnitCycles);
        if (best < 0 || cost < best) {
            best = cost;
            a.rows_per_tile = static_cast<int>(rows);
            a.row_tiles = static_cast<int>(used);
        }
    }
    a.units = static_cast<int>(swiglu ? ceil_div(N / 32, 8) : ceil_div(N / 16, 16)) * a.row_tiles;
    if (act_dtype == EQ_F16)
        return swiglu ? launch<__half, true>(a, x, scale_dtype, stream) : launch<__half, false>(a, x, scale_dtype, stream);
    return swiglu ? launch<__nv_bfloat16, true>(a, x, scale_dtype, stream) : launch<__nv_bfloat16, false>(a, x, scale_dtype, stream);
}

}  // namespace eq
