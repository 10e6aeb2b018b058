// W4A16 linear with the weights as the tensor core's A operand in tensor memory: y[M,N] = x[M,K] @ W.
//
// A CTA owns 128 output channels (TMEM lane = channel) by up to NB activation rows (accumulator column = row) and walks K
// in items of 128.  Nothing of the weight touches shared memory but its packed bytes:
//   warps 0..7    dequant.  A warp owns two 16-channel weight tiles, the 32 TMEM lanes it may write; warps 0-3 take the
//                 even items of the CTA's sequence, warps 4-7 the odd ones.  Packed records come by cp.async into a ring
//                 private to the warp (16-byte pieces placed so that the 4-byte reads below hit 32 different banks).
//                 The repack deals a lane eight consecutive k of one channel as nibble pairs of four words; read one word
//                 per lane instead, lane j of a quad holds pair j of such a run for channel g: exactly the fragment that
//                 tcgen05.st.16x128b wants (register i of lane 4 g + j = row g, 32-bit column 4 i + j), with K in natural
//                 order.  One item of a tile is 64 TMEM columns.
//   warp T        TMA of the activation rows (K-major, 128-byte swizzle): the MMA's B operand
//   warp T + 1    MMA issuer: tcgen05.mma kind::f16, A from TMEM, 128 x rows x 16, rows rounded up to 16
// The kernel is persistent over units (column tile, row block): weight copies of the next unit are under way while the
// current one ends.  Where the tiles leave CTA slots idle (SPLIT) the K slices of a tile are the CTAs of a cluster and their
// f32 partial tiles meet in distributed shared memory, in a fixed order.  (Meeting in a global workspace by atomic adds cost
// 8 us a call: K=N=4096, 64 rows 15.1 us against 11.1; K=14336 N=4096 22.0 against 17.3.)
//
// Two accumulations.  PROMOTE: A holds the integers q - z, every item gets a fresh accumulator (two alternate) and four
// more warps add scale * accumulator to f32 sums in registers, which is the rounding of the decode kernel (w4_stream.cu).
// Otherwise A holds (q - z) * scale rounded to the activation dtype, what the dequantize-then-matmul path feeds its matmul
// (emmy/compiler/loader/quant.py:402-470), and the accumulator runs over all of K.
//
// Why the roles are this way round: with rows as the MMA's M a 64-row call pads every MMA to 128 rows and pushes each
// dequantised byte through shared memory twice (store, operand read).  Measured against that form (us, rows as M, dequant
// through shared memory -> here; K=4096 N=14336 | K=14336 N=4096 | K=N=4096): 64 rows 33.0 -> 17.1 | 31.3 -> 17.2 | 18.2 ->
// 11.1; 128 rows 35.6 -> 21.5 | 39.7 -> 22.6; 256 rows of K=N=4096 50.2 -> 16.5; an MLP of hidden 4096, intermediate 14336,
// 64 rows, over more layers than the L2 holds: 81 -> 47 to 49.
//
// What bounds it: issue slots.  An item costs an SM about 1600 warp instructions (eight nibbles: five integer and eight half
// instructions and one shared read) against the 380 cycles HBM needs for its bytes; two CTAs of ten or fourteen warps are what
// keeps the slots busy (at one CTA an item takes 0.45 us, at two each 0.65).
#include "tc_common.cuh"
#include "w4_tile.cuh"
#include "w4_tmem.cuh"

namespace eq {
namespace {

using namespace tm;

constexpr int kGK = 64;         // K per 128-byte activation row piece
constexpr int kDW = 8;          // dequant warps
constexpr int kScaleRing = 8;   // items whose scales are kept for the promoting warps: more than stages + accumulators

template <int NB, bool PROMOTE>
struct TmemCfg {
    static constexpr int kAccs = PROMOTE ? 2 : 1;
    static constexpr int kAccCols = NB < 32 ? 32 : NB;
    static constexpr int kTmemCols = 256;
    // one stage: 64 columns of A and the item's activation rows; an even split of TMEM between two resident CTAs
    static constexpr int kFit = (kTmemCols - kAccs * kAccCols) / 64;
    static constexpr int kStages = kFit < 3 ? kFit : 3;
    static constexpr int kDepth = NB >= 128 ? 2 : 3;  // items in flight per dequant warp
    static constexpr int kStageBytes = NB * 256;
    static constexpr int kRing = kDW * kDepth * 2 * kItemBytes;
    static constexpr int kBoxRows = NB < 64 ? NB : 64;
    static constexpr int kWarps = kDW + (PROMOTE ? 4 : 0) + 2;
    static constexpr int kThreads = 32 * kWarps;
    static constexpr size_t kSmem = 1024 + static_cast<size_t>(kStages) * kStageBytes + kRing + kScaleRing * 128 * 4 + 256;
    static_assert(kStages >= 2, "two stages at least");
    static_assert(kSmem <= 113 * 1024, "two CTAs per SM");
};

template <typename ActT, int NB, bool CVT, bool PROMOTE, bool SWIGLU, bool GROUPED, bool SPLIT>
__global__ void __launch_bounds__(TmemCfg<NB, PROMOTE>::kThreads, 2)
    w4a16_tmem_kernel(const __grid_constant__ CUtensorMap map_x, const W4TmemArgs a) {
    using Cfg = TmemCfg<NB, PROMOTE>;
    constexpr int S = Cfg::kStages, D = Cfg::kDepth;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* tiles_b = smem;
    unsigned char* ring = smem + S * Cfg::kStageBytes;
    float* scales = reinterpret_cast<float*>(ring + Cfg::kRing);
    uint64_t* bars = reinterpret_cast<uint64_t*>(scales + kScaleRing * 128);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * S + 4);
    const uint32_t full_a = tc::smem_u32(bars), full_b = full_a + 8 * S, empty = full_b + 8 * S, acc_full = empty + 8 * S, acc_empty = acc_full + 16;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int items = a.K / 128, n_tiles = a.N / 16;
    const int col_tiles = SWIGLU ? (a.N / 32 + 3) / 4 : (n_tiles + 7) / 8;  // SWIGLU: four gate and four up tiles per CTA
    int units = a.units;
    if constexpr (GROUPED) asm volatile("griddepcontrol.wait;" ::: "memory");  // the block list and the rows are of the grids before
    if constexpr (GROUPED) units = *a.n_blocks * col_tiles;
    if (static_cast<int>(blockIdx.x) >= units) return;  // the whole CTA, before any barrier exists

    // unit u -> column tile, first row and row count, first item and item count
    auto locate = [&](int u, int& col, int& row0, int& rows, int& item0, int& n_items, int& expert) {
        item0 = 0;
        n_items = items;
        expert = 0;
        if constexpr (GROUPED) {
            const int b = u / col_tiles;
            col = u - b * col_tiles;
            const RowBlock rb = a.blocks[b];
            row0 = rb.row0;
            rows = rb.rows;
            expert = rb.expert;
        } else {
            int rest = u;
            if constexpr (SPLIT) {
                const int z = rest % a.splits;
                rest /= a.splits;
                item0 = static_cast<int>(static_cast<long long>(items) * z / a.splits);
                n_items = static_cast<int>(static_cast<long long>(items) * (z + 1) / a.splits) - item0;
            }
            const int rt = rest % a.row_tiles;  // row tiles fastest: the CTAs that share a weight tile run together
            col = rest / a.row_tiles;
            row0 = rt * a.rows_per_tile;
            rows = min(a.rows_per_tile, a.M - row0);
        }
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            tc::mbar_init(full_a + 8 * s, 4);
            tc::mbar_init(full_b + 8 * s, 1);
            tc::mbar_init(empty + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(acc_full + 8 * b, 1);
            tc::mbar_init(acc_empty + 8 * b, PROMOTE ? 4 : kDW);
        }
        tc::mbar_fence_init();
    }
    constexpr int kTmaWarp = Cfg::kWarps - 2, kMmaWarp = Cfg::kWarps - 1;
    if (warp == kMmaWarp) tc::tmem_alloc(tc::smem_u32(tmem_slot), Cfg::kTmemCols);

    // ---- dequant warps: the prefetch cursor runs D items (of this warp's parity) ahead of use
    const int q = warp & 3, wg = warp >> 2;
    const uint32_t my_ring = tc::smem_u32(ring) + warp * (D * 2 * kItemBytes);
    const LaneOffsets lo;
    int pf_unit = blockIdx.x, pf_item = wg, pf_items = 0;
    uint32_t pf_slot = my_ring;
    const unsigned char *pf0 = nullptr, *pf1 = nullptr;  // the warp's two tiles: item pf_item of unit pf_unit, at this lane
    auto pf_locate = [&]() {
        int col, row0, rows, item0, expert;
        locate(pf_unit, col, row0, rows, item0, pf_items, expert);
        const unsigned char* base = a.wq + static_cast<size_t>(item0 + pf_item) * kItemBytes + lane * 16;
        if constexpr (GROUPED) base += static_cast<size_t>(expert) * a.expert_stride;
        // tiles beyond the weight read tile 0: their channels are never stored
        int t0 = SWIGLU ? col * 4 + q : col * 8 + 2 * q, t1 = SWIGLU ? t0 + n_tiles / 2 : t0 + 1;
        if (SWIGLU && t0 >= n_tiles / 2) t0 = 0;
        if (t0 >= n_tiles) t0 = 0;
        if (t1 >= n_tiles) t1 = 0;
        pf0 = base + static_cast<size_t>(t0) * items * kItemBytes;
        pf1 = base + static_cast<size_t>(t1) * items * kItemBytes;
    };
    auto prefetch = [&]() {
        if (pf_item >= pf_items && pf_unit < units) {
            do {
                pf_item -= pf_items;
                pf_unit += gridDim.x;
                if (pf_unit < units) pf_locate();
            } while (pf_unit < units && pf_item >= pf_items);
        }
        if (pf_unit < units) {
            fetch_items(pf_slot, lo, pf0, pf1);
            pf0 += 2 * kItemBytes;
            pf1 += 2 * kItemBytes;
            pf_item += 2;
        }
        cp_commit();
        pf_slot += 2 * kItemBytes;
        if (pf_slot == my_ring + D * 2 * kItemBytes) pf_slot = my_ring;
    };
    if (warp < kDW) {
        pf_locate();
#pragma unroll 1
        for (int d = 0; d < D; ++d) prefetch();
    }

    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    // Only now, with this CTA's TMEM in hand: a dependent grid that took the columns first and then waited for this grid
    // would never give them back.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_a = tmem_base + Cfg::kAccs * Cfg::kAccCols;  // stages of 64 columns behind the accumulators

    // Sixteen accumulator columns to their place: y, or (SPLIT) this CTA's f32 partial tile [row][channel] in shared memory,
    // over the activation stages, which are idle once the accumulator is complete.
    float* const part = reinterpret_cast<float*>(tiles_b);
    auto emit = [&](const float (&v)[16], int col, int row0, int rows, int c) {
        if constexpr (SPLIT) {
#pragma unroll
            for (int i = 0; i < 16; ++i) part[(c + i) * 128 + 32 * q + lane] = v[i];
        } else {
            emit16<ActT, SWIGLU, GROUPED>(a, v, SWIGLU ? col * 4 + q : col * 8 + 2 * q, row0, rows, c);
        }
    };

    if (warp < kDW) {
        // this warp's items: every second one of the CTA's sequence over all units
        int next = wg;       // its next item, counted from the start of the current unit
        int stage = wg, phase = 1, ring_at = wg;  // stage and (inverted) use parity of that item; its scales' slot
        bool first = true, broken = false;
        bool waited = false;  // behind griddepcontrol.wait
        int n_unit = 0;
        const int g = lane >> 2, j = lane & 3;
        const uint32_t a_lane = tmem_a + (static_cast<uint32_t>(32 * q) << 16);
        for (int u = blockIdx.x; u < units && !broken; u += gridDim.x, ++n_unit) {
            int col, row0, rows, item0, n_items, expert;
            locate(u, col, row0, rows, item0, n_items, expert);
            for (; next < n_items; next += 2) {
                cp_wait<D - 1>();
                __syncwarp();
                ItemWords w;
                load_item(pf_slot, lo, w);  // the oldest of the ring, and the next to be refilled
                __syncwarp();
                prefetch();  // refills it
                if (!first && !__all_sync(0xFFFFFFFFu, wait_asleep<!GROUPED>(empty + 8 * stage, phase))) {
                    if (lane == 0) atomicExch(a.status, 4);
                    broken = true;
                    break;
                }
                tc::fence_after_sync();
                if constexpr (PROMOTE) {
                    if (j < 2) {
#pragma unroll
                        for (int t = 0; t < 2; ++t) {
                            const uint32_t raw = j == 0 ? (w.mt[t].x & 0xFFFFu) : (w.mt[t].x >> 16);
                            scales[ring_at * 128 + 32 * q + 16 * t + 8 * j + g] = scale16_to_float(static_cast<uint16_t>(raw), a.scale_dtype);
                        }
                    }
                    ring_at = (ring_at + 2) % kScaleRing;
                }
                expand_item<ActT, CVT, PROMOTE>(w, a_lane + 64 * stage);
                tmem_st_wait();
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(full_a + 8 * stage);
                stage += 2;
                if (stage >= S) {
                    stage -= S;
                    phase ^= 1;
                    first = false;
                }
            }
            next -= n_items;
            if constexpr (!PROMOTE) {
                if (!GROUPED && !waited) {
                    asm volatile("griddepcontrol.wait;" ::: "memory");  // y may be in use by the previous grid
                    waited = true;
                }
                const bool ok = __all_sync(0xFFFFFFFFu, wait_asleep(acc_full, n_unit & 1));
                if (!ok && lane == 0) atomicExch(a.status, 3);
                broken |= !ok;
                tc::fence_after_sync();
                const uint32_t t_row = tmem_base + (static_cast<uint32_t>(32 * q) << 16);
#pragma unroll 1
                for (int c = 16 * wg; ok && c < rows; c += 32) {
                    uint32_t r[16];
                    tc::tmem_ld_32x16(t_row + c, r);
                    tc::tmem_ld_wait();
                    float v[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
                    emit(v, col, row0, rows, c);
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(acc_empty);
            }
        }
        cp_wait<0>();  // (left with copies under way only where a wait ran out)
    } else if (PROMOTE && warp < kDW + 4) {
        // ---- promotion: sums[r] += scale * accumulator, then the epilogue
        int seq = 0;
        bool broken = false, waited = false;
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(32 * q) << 16);
        for (int u = blockIdx.x; u < units && !broken; u += gridDim.x) {
            int col, row0, rows, item0, n_items, expert;
            locate(u, col, row0, rows, item0, n_items, expert);
            float sum[NB];
#pragma unroll
            for (int i = 0; i < NB; ++i) sum[i] = 0.f;
            for (int it = 0; it < n_items; ++it, ++seq) {
                const int b = seq & 1;
                if (!__all_sync(0xFFFFFFFFu, wait_asleep<!GROUPED>(acc_full + 8 * b, (seq >> 1) & 1))) {
                    if (lane == 0) atomicExch(a.status, 3);
                    broken = true;
                    break;
                }
                tc::fence_after_sync();
                const float s = scales[(seq % kScaleRing) * 128 + 32 * q + lane];
#pragma unroll
                for (int c = 0; c < NB; c += 16) {
                    uint32_t r[16];
                    tc::tmem_ld_32x16(t_row + b * Cfg::kAccCols + c, r);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum[c + i] = fmaf(s, __uint_as_float(r[i]), sum[c + i]);
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(acc_empty + 8 * b);
            }
            if (!GROUPED && !waited) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                waited = true;
            }
#pragma unroll
            for (int c = 0; c < NB; c += 16) {
                if (c < rows && !broken) {
                    float v[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = sum[c + i];
                    emit(v, col, row0, rows, c);
                }
            }
        }
    } else if (warp == kTmaWarp) {
        if (tc::elect_one()) {
            tc::tma_prefetch_desc(&map_x);
            if constexpr (!GROUPED) asm volatile("griddepcontrol.wait;" ::: "memory");  // x may be the previous grid's output
            int seq = 0;
            bool broken = false;
            for (int u = blockIdx.x; u < units && !broken; u += gridDim.x) {
                int col, row0, rows, item0, n_items, expert;
                locate(u, col, row0, rows, item0, n_items, expert);
                const int boxes = (rows + Cfg::kBoxRows - 1) / Cfg::kBoxRows;
                for (int it = 0; it < n_items; ++it, ++seq) {
                    const int stage = seq % S, use = seq / S;
                    if (use > 0 && !wait_asleep(empty + 8 * stage, (use - 1) & 1)) {
                        atomicExch(a.status, 1);
                        broken = true;
                        break;
                    }
                    const uint32_t bar = full_b + 8 * stage, dst = tc::smem_u32(tiles_b) + stage * Cfg::kStageBytes;
                    tc::mbar_expect_tx(bar, 2 * boxes * Cfg::kBoxRows * 128);
                    for (int half = 0; half < 2; ++half)
                        for (int bx = 0; bx < boxes; ++bx)
                            tc::tma_load_2d(dst + half * (NB * 128) + bx * (Cfg::kBoxRows * 128), &map_x, (item0 + it) * 128 + half * kGK, row0 + bx * Cfg::kBoxRows, bar);
                }
            }
            if (broken)  // nobody else waits for these: the CTA does not end with a copy under way into its shared memory
                for (int i = seq < S ? 0 : seq - S; i < seq; ++i) wait_asleep(full_b + 8 * (i % S), (i / S) & 1);
        }
    } else {
        if (tc::elect_one()) {
            int seq = 0, n_unit = 0;
            bool broken = false;
            for (int u = blockIdx.x; u < units && !broken; u += gridDim.x, ++n_unit) {
                int col, row0, rows, item0, n_items, expert;
                locate(u, col, row0, rows, item0, n_items, expert);
                const uint32_t idesc = tc::instr_desc(Mul<ActT>::kFmt, Mul<ActT>::kFmt, 128, static_cast<uint32_t>((rows + 15) & ~15));
                if (!PROMOTE && n_unit > 0) broken = !wait_asleep<!GROUPED>(acc_empty, (n_unit - 1) & 1);
                for (int it = 0; it < n_items && !broken; ++it, ++seq) {
                    const int stage = seq % S, b = PROMOTE ? (seq & 1) : 0;
                    const uint32_t parity = (seq / S) & 1;
                    bool ok = !PROMOTE || seq < 2 || wait_asleep<!GROUPED>(acc_empty + 8 * b, ((seq >> 1) - 1) & 1);
                    ok = ok && wait_asleep<!GROUPED>(full_b + 8 * stage, parity);
                    ok = ok && wait_asleep<!GROUPED>(full_a + 8 * stage, parity);
                    if (!ok) {
                        broken = true;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint64_t b_desc = tc::smem_desc_k_sw128(tc::smem_u32(tiles_b) + stage * Cfg::kStageBytes);  // further steps: + bytes / 16
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)
                        mma_f16_ts(tmem_base + b * Cfg::kAccCols, tmem_a + 64 * stage + 8 * ks, b_desc + ((ks >> 2) * (NB * 128) + (ks & 3) * 32) / 16, idesc,
                                   ks > 0 || (!PROMOTE && it > 0));
                    tc::mma_commit(empty + 8 * stage);
                    if (PROMOTE) tc::mma_commit(acc_full + 8 * b);
                }
                if (!PROMOTE) tc::mma_commit(acc_full);
                if (broken) {
                    atomicExch(a.status, 2);
                    // neither shared memory nor TMEM goes back with a copy (one that was never issued runs out) or an MMA under way
                    for (int i = seq; i < seq + S; ++i) wait_asleep(full_b + 8 * (i % S), (i / S) & 1);
                    if (!PROMOTE) wait_asleep(acc_full, n_unit & 1);
                    if (PROMOTE && seq > 0) wait_asleep(acc_full + 8 * ((seq - 1) & 1), ((seq - 1) >> 1) & 1);
                }
            }
        }
    }
    __syncwarp();
    if constexpr (SPLIT) {
        // The K slices of a tile are the CTAs of one cluster (one unit each): every CTA adds up and stores its share of the
        // rows from all partial tiles, in the slices' order.
        tc::cluster_sync();
        int col, row0, rows, item0, n_items, expert;
        locate(blockIdx.x, col, row0, rows, item0, n_items, expert);
        const int rank = static_cast<int>(tc::cluster_rank());
        const int r_lo = rows * rank / a.splits, r_hi = rows * (rank + 1) / a.splits;
        const uint32_t part_addr = tc::smem_u32(part);
        constexpr int kPerRow = SWIGLU ? 16 : 32;  // threads of a row: four channels each
        const int t = threadIdx.x % kPerRow;
        const int at = SWIGLU ? 32 * (t >> 2) + 4 * (t & 3) : 4 * t;  // the thread's channels in the tile (gate's, for SWIGLU)
        const int out_n = SWIGLU ? a.N / 2 : a.N, ch = (SWIGLU ? col * 64 : col * 128) + 4 * t;
        asm volatile("griddepcontrol.wait;" ::: "memory");  // y may be in use by the previous grid
        for (int r = r_lo + static_cast<int>(threadIdx.x) / kPerRow; r < r_hi; r += Cfg::kThreads / kPerRow) {
            float s[4] = {0.f, 0.f, 0.f, 0.f}, up[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int z = 0; z < a.splits; ++z) {
                const uint32_t src = tc::map_to_rank(part_addr, z) + static_cast<uint32_t>(r * 128 + at) * 4;
                const float4 v = ld_cluster_v4(src);
                s[0] += v.x, s[1] += v.y, s[2] += v.z, s[3] += v.w;
                if constexpr (SWIGLU) {
                    const float4 w = ld_cluster_v4(src + 64);
                    up[0] += w.x, up[1] += w.y, up[2] += w.z, up[3] += w.w;
                }
            }
            if constexpr (SWIGLU) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float g = to_float(from_float<ActT>(s[i]));
                    s[i] = to_float(from_float<ActT>(g / (1.f + expf(-g)))) * to_float(from_float<ActT>(up[i]));
                }
            }
            if (ch < out_n)
                *reinterpret_cast<uint2*>(static_cast<ActT*>(a.y) + static_cast<size_t>(row0 + r) * out_n + ch) =
                    make_uint2(bits16<ActT>(s[0]) | (bits16<ActT>(s[1]) << 16), bits16<ActT>(s[2]) | (bits16<ActT>(s[3]) << 16));
        }
        __syncwarp();
        tc::cluster_sync();  // nobody leaves while its partial tile may still be read
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

template <typename ActT, int NB, bool PROMOTE, bool SWIGLU, bool GROUPED, bool SPLIT>
int launch(W4TmemArgs a, const void* x, int64_t x_rows, int scale_dtype, cudaStream_t stream) {
    using Cfg = TmemCfg<NB, PROMOTE>;
    CUtensorMap map_x;
    const CUtensorMapDataType elem = Mul<ActT>::kFmt == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int st = make_tensor_map_2d(&map_x, x, elem, 2, x_rows, a.K, static_cast<uint64_t>(a.K) * 2, Cfg::kBoxRows, kGK, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != EQ_OK) return st;
    a.scale_dtype = scale_dtype;
    const bool cvt = !PROMOTE && scale_dtype != (Mul<ActT>::kFmt == 0 ? EQ_F16 : EQ_BF16);
    auto kernel = cvt ? w4a16_tmem_kernel<ActT, NB, !PROMOTE, PROMOTE, SWIGLU, GROUPED, SPLIT> : w4a16_tmem_kernel<ActT, NB, false, PROMOTE, SWIGLU, GROUPED, SPLIT>;
    EQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Cfg::kSmem)));
    const int slots = 2 * sm_count();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(GROUPED || a.units > slots ? slots : a.units));
    cfg.blockDim = dim3(Cfg::kThreads);
    cfg.dynamicSmemBytes = Cfg::kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(SPLIT ? a.splits : 1);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = SPLIT ? 2 : 1;
    EQ_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, map_x, a));
    return EQ_OK;
}

template <typename ActT, int NB, bool PROMOTE, bool SWIGLU>
int launch_dense(W4TmemArgs a, const void* x, int scale_dtype, cudaStream_t stream) {
    const int items = a.K / 128;
    const int col_tiles = static_cast<int>(SWIGLU ? ceil_div(a.N / 32, 4) : ceil_div(a.N / 16, 8));
    a.row_tiles = static_cast<int>(ceil_div(a.M, NB));
    a.rows_per_tile = static_cast<int>(ceil_div(ceil_div(a.M, a.row_tiles), 8) * 8);
    if (a.rows_per_tile > NB) a.rows_per_tile = NB;
    a.row_tiles = static_cast<int>(ceil_div(a.M, a.rows_per_tile));
    const int tiles = col_tiles * a.row_tiles, slots = 2 * sm_count();
    // K slices (a cluster's CTAs, eight at most) where the tiles leave CTA slots idle; at least two items a slice.  A cluster
    // lives in one GPC, so not every slot can be filled: with 288 of the 296 asked for (K=14336 N=4096, 300 rows, clusters of
    // three) a second wave ran and the call took 72 us.
    // A meeting costs about what three items do, so a short K is not cut, nor one into two slices only (promoted: 9 items)
    // (plain linears; us, cut against whole.  32 rows: 512 x 14336 6.7 : 4.2, 1024 x 14336 8.1 : 6.7, 1536 x 14336 10.4 : 9.3;
    // 128 rows: 512 x 14336 9.6 : 7.2; 20 rows: 512 x 14336 6.4 : 4.7, 1280 x 14336 even).  The SwiGLU epilogue gains from being
    // shared out: K=768, 20 rows, cutting is 4 to 39 % faster.
    int splits = (slots - slots / 8) / tiles;
    if (splits > items / 2) splits = items / 2;
    if (splits > 8) splits = 8;
    if (!SWIGLU && (items <= 6 || (splits == 2 && items < (PROMOTE ? 9 : 14)))) splits = 1;
    if (splits < 1) splits = 1;
    a.splits = splits;
    a.units = tiles * splits;
    return splits > 1 ? launch<ActT, NB, PROMOTE, SWIGLU, false, true>(a, x, a.M, scale_dtype, stream)
                      : launch<ActT, NB, PROMOTE, SWIGLU, false, false>(a, x, a.M, scale_dtype, stream);
}

template <typename ActT>
int dense_typed(const W4TmemArgs& a, const void* x, int scale_dtype, bool swiglu, bool promote, cudaStream_t stream) {
    if (promote) return swiglu ? launch_dense<ActT, 32, true, true>(a, x, scale_dtype, stream) : launch_dense<ActT, 32, true, false>(a, x, scale_dtype, stream);
    // 65 to 128 rows of a short K, where the epilogue is the larger part, run as two row tiles of 64 on twice as many CTAs (128
    // rows: 512 x 4096 5.8 -> 4.3 us, 512 x 14336 7.4 -> 5.8, 896 x 11136 9.2 -> 6.7; at K=1024 the second expansion costs more)
    if (a.M <= 64 || (!swiglu && a.M <= 128 && a.K <= 896)) return swiglu ? launch_dense<ActT, 64, false, true>(a, x, scale_dtype, stream) : launch_dense<ActT, 64, false, false>(a, x, scale_dtype, stream);
    return swiglu ? launch_dense<ActT, 128, false, true>(a, x, scale_dtype, stream) : launch_dense<ActT, 128, false, false>(a, x, scale_dtype, stream);
}

}  // namespace

int w4_tmem_dense_launch(const unsigned char* wq, int scale_dtype, const void* x, void* y, int64_t M, int64_t N, int64_t K, int act_dtype, bool swiglu,
                         bool promote, int* status, cudaStream_t stream) {
    W4TmemArgs a = {};
    a.wq = wq;
    a.y = y;
    a.M = static_cast<int>(M);
    a.N = static_cast<int>(N);
    a.K = static_cast<int>(K);
    a.status = status;
    return act_dtype == EQ_F16 ? dense_typed<__half>(a, x, scale_dtype, swiglu, promote, stream) : dense_typed<__nv_bfloat16>(a, x, scale_dtype, swiglu, promote, stream);
}

namespace {

template <typename ActT>
int grouped_typed(const W4TmemArgs& a, const void* x, int64_t R, int scale_dtype, bool swiglu, int block_rows, cudaStream_t stream) {
    if (block_rows <= 16)
        return swiglu ? launch<ActT, 16, true, true, true, false>(a, x, R, scale_dtype, stream) : launch<ActT, 16, true, false, true, false>(a, x, R, scale_dtype, stream);
    return swiglu ? launch<ActT, 128, false, true, true, false>(a, x, R, scale_dtype, stream) : launch<ActT, 128, false, false, true, false>(a, x, R, scale_dtype, stream);
}

}  // namespace

int w4_tmem_grouped_launch(const unsigned char* wq, size_t expert_stride, int scale_dtype, const void* x, void* y, int64_t R, int64_t N, int64_t K,
                           int act_dtype, const RowBlock* blocks, const int32_t* n_blocks, int block_rows, const int32_t* y_rows, bool swiglu, int* status,
                           cudaStream_t stream) {
    W4TmemArgs a = {};
    a.wq = wq;
    a.y = y;
    a.M = static_cast<int>(R);
    a.N = static_cast<int>(N);
    a.K = static_cast<int>(K);
    a.status = status;
    a.blocks = blocks;
    a.n_blocks = n_blocks;
    a.y_rows = y_rows;
    a.expert_stride = expert_stride;
    return act_dtype == EQ_F16 ? grouped_typed<__half>(a, x, R, scale_dtype, swiglu, block_rows, stream)
                               : grouped_typed<__nv_bfloat16>(a, x, R, scale_dtype, swiglu, block_rows, stream);
}

}  // namespace eq
