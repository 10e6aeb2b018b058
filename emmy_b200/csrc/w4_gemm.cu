// Grouped W4A16 GEMM of the expert-parallel MoE layer: 256-row blocks of one expert each, weights dequantised into shared
// memory, on the tcgen05 tensor cores; and the dense prefill entry, which picks between w4_tmem.cu and w4_tmem2.cu.
//
// The int4 weight never exists as a 16-bit matrix in global memory.  A CTA owns a tile of 256 activation rows by 256 weight
// columns and walks K in steps of 64:
//   warp 0        TMA producer: the 64-wide slice of the x rows, 128-byte swizzle, into the stage's A tile
//   warp 1        MMA issuer: tcgen05.mma kind::f16, 128 x 256 x 16 per instruction, f32 accumulators in TMEM (one
//                 accumulator per 128 activation rows; both read the same B tile)
//   warps 2..     dequant producers, then the epilogue.  A producer warp reads the packed nibbles of one 16-column
//                 weight tile straight from global memory into registers (one 16-byte load per lane and K step,
//                 issued kAhead steps early), expands them exactly as the decode kernel does (lop3 to 1024 + q, one
//                 subtract / fma removes 1024 and the zero point), multiplies by the group scale in the activation
//                 dtype, which is the value the reference's dequantize-then-matmul path feeds its matmul
//                 (emmy/compiler/loader/quant.py:402-470), and writes the stage's B tile in the same 128-byte-swizzled
//                 K-major layout TMA would have produced.  fence.proxy.async makes the writes visible to the tensor
//                 core; one arrive per warp completes the stage.
// The repack (w4_repack.cu) deals the 128 input rows of an item to lanes so that a lane's four words of one half-tile
// hold, for columns g and g + 8, two runs of eight consecutive rows: exactly two 16-byte chunks of a swizzled row per
// column.  Lanes (g, h, jj) of a warp take the pieces of rows 64 t + 32 jj + 8 h (+16) of K step t of the item, so one
// K step of the MMA is 64 consecutive input rows and x needs no reordering.  Act-order weights (a row permutation)
// gather the columns of x into the workspace first.
#include "tc_common.cuh"
#include "w4_tile.cuh"
#include "w4_tmem.cuh"

namespace eq {

namespace {

constexpr int kGK = 64;             // K per stage: 128 bytes of 16-bit elements
constexpr int kRowBytes = 128;

constexpr int kHalves = 2;              // 128-row activation blocks per CTA
constexpr int kBN = 256;                // weight columns per CTA
constexpr int kTileA = kHalves * 128 * kRowBytes, kTileB = kBN * kRowBytes;
constexpr int kStages = 3;
constexpr int kDequantWarps = kBN / 16; // one 16-column weight tile each; and epilogue warps, in quartets (one warp per TMEM lane quarter)
constexpr int kQuartets = kDequantWarps / 4;
constexpr int kAhead = 2;               // items (two K steps each) whose packed bytes are in a warp's registers ahead of use
constexpr int kThreads = 64 + 32 * kDequantWarps;
constexpr size_t kSmem = static_cast<size_t>(kStages) * (kTileA + kTileB) + 1024 + 256;
constexpr uint32_t kTmemCols = kHalves * kBN;
static_assert(kTmemCols == 512 && kSmem <= 227 * 1024, "all of TMEM, one CTA per SM");

// 8-byte read-only load that stays where it is written (issued kAhead steps before its use).
__device__ __forceinline__ uint2 ld_pinned_v2(const void* p) {
    uint2 r;
    asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// xg[m][k'] = x[m][perm[k']]
template <typename ActT>
__global__ void gather_cols_kernel(const ActT* __restrict__ x, const int32_t* __restrict__ perm, int64_t M, int64_t K,
                                   ActT* __restrict__ xg) {
    const int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (idx >= M * K) return;
    const int64_t m = idx / K, k = idx - m * K;
    xg[idx] = x[m * K + perm[k]];
}

// blockIdx.y walks a device-side list of row blocks, each a run of rows of ONE expert in an expert-ordered activation matrix; the
// weight is that expert's slice of a stacked tensor.  SWIGLU: the first 128 columns of the CTA's B tile are taken from the gate
// half and the last 128 from the up half of a [gate | up] weight, and the epilogue writes act(silu(gate)) * up
// (emmy/compiler/trace/huggingface.py:1663-1669) into y, a matrix of N / 2 columns.  Otherwise every row has a destination of
// its own.
struct GroupArgs {
    const RowBlock* blocks;
    const int32_t* n_blocks;
    const uint64_t* y_ptrs;  // output row m starts at address y_ptrs[m] (0 = drop the row); may be a peer GPU's memory
    size_t expert_stride;    // bytes between the experts' repacked weights
};

template <typename ActT, bool CVT, bool SWIGLU>
__global__ void __launch_bounds__(kThreads)
    w4a16_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_x, const unsigned char* __restrict__ wq, ActT* __restrict__ y,
                         int N, int K, int* __restrict__ status, const GroupArgs grp) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* tiles_a = smem;
    unsigned char* tiles_b = smem + kStages * kTileA;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * (kTileA + kTileB));
    uint64_t* full_a = bars;                  // [kStages] TMA -> MMA
    uint64_t* full_b = bars + kStages;        // [kStages] dequant warps -> MMA
    uint64_t* empty = bars + 2 * kStages;     // [kStages] MMA -> producers
    uint64_t* acc_ready = bars + 3 * kStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * kStages + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * kBN;
    if (static_cast<int>(blockIdx.y) >= *grp.n_blocks) return;  // the whole CTA, before any barrier exists
    const RowBlock rb = grp.blocks[blockIdx.y];
    const int m0 = rb.row0, m_end = rb.row0 + rb.rows;
    wq += static_cast<size_t>(rb.expert) * grp.expert_stride;
    const int items = K / 128;
    const int k_blocks = 2 * items;
    const int live_halves = min(kHalves, (m_end - m0 + 127) / 128);  // 128-row blocks of this tile that hold rows

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            tc::mbar_init(tc::smem_u32(full_a + s), 1);
            tc::mbar_init(tc::smem_u32(full_b + s), kDequantWarps);
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
    // shared-window addresses, computed once: barrier s of a ring sits 8 s bytes on
    const uint32_t full_a_addr = tc::smem_u32(full_a), full_b_addr = tc::smem_u32(full_b), empty_addr = tc::smem_u32(empty);
    const uint32_t a_base = tc::smem_u32(tiles_a), b_base = tc::smem_u32(tiles_b);

    if (warp == 0) {
        // ---- TMA producer of the activation tiles
        if (tc::elect_one()) {
            tc::tma_prefetch_desc(&map_x);
            int stage = 0;
            uint32_t phase = 0;
            bool first = true;
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!first && !tc::mbar_wait(empty_addr + 8 * stage, phase ^ 1)) {
                    atomicExch(status, 1);
                    tc::drain_copies(full_a, kb - kStages, kb, kStages);
                    break;
                }
                const uint32_t bar = full_a_addr + 8 * stage;
                tc::mbar_expect_tx(bar, kTileA);
                tc::tma_load_2d(a_base + stage * kTileA, &map_x, kb * kGK, m0, bar);
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1;
                    first = false;
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        if (tc::elect_one()) {
            constexpr uint32_t idesc = tc::instr_desc(tm::Mul<ActT>::kFmt, tm::Mul<ActT>::kFmt, 128, kBN);
            int stage = 0;
            uint32_t phase = 0;
            for (int kb = 0; kb < k_blocks; ++kb) {
                const bool got_a = tc::mbar_wait(full_a_addr + 8 * stage, phase);
                const bool got_b = got_a && tc::mbar_wait(full_b_addr + 8 * stage, phase);
                if (!got_b) {
                    atomicExch(status, 2);
                    tc::drain_copies(full_a, kb, min(kb + kStages, k_blocks), kStages);
                    break;
                }
                tc::fence_after_sync();
                const uint32_t a_addr = a_base + stage * kTileA, b_addr = b_base + stage * kTileB;
#pragma unroll
                for (int ks = 0; ks < kGK / 16; ++ks) {
                    const uint64_t db = tc::smem_desc_k_sw128(b_addr + ks * 32);
#pragma unroll
                    for (int hh = 0; hh < kHalves; ++hh)
                        if (hh < live_halves)
                            tc::mma_f16(tmem_base + hh * kBN, tc::smem_desc_k_sw128(a_addr + hh * 128 * kRowBytes + ks * 32), db, idesc, kb > 0 || ks > 0);
                }
                tc::mma_commit(empty_addr + 8 * stage);
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            tc::mma_commit(tc::smem_u32(acc_ready));  // on a broken pipeline too: the epilogue must not sit out its wait
        }
    } else {
        // ---- dequant producers
        const int dw = warp - 2;
        const int g = lane & 7, h = (lane >> 3) & 1, jj = lane >> 4;
        // Shared-memory byte offsets of the lane's four 16-byte chunks inside a B tile: row r = 16 tile + g (+8) is an
        // output column, chunk q = 4 jj + 2 high + h of its 128 bytes is swizzled with r & 7 = g.
        int tile = n0 / 16 + dw;
        if constexpr (SWIGLU) {
            constexpr int kHalfTiles = kBN / 32;  // gate tiles of this CTA, then as many up tiles
            const int col_tile = n0 / 32 + dw % kHalfTiles;
            tile = col_tile < N / 32 ? col_tile + (dw / kHalfTiles) * (N / 32) : N / 16;
        }
        const bool live = tile < N / 16;
        const unsigned char* rec = wq + static_cast<size_t>(live ? tile : 0) * items * kItemBytes;
        const unsigned char* wp = rec + h * 512 + (4 * g + jj) * 16;  // the lane's 16 bytes of K step 0 of item 0; K step 1 is 32 bytes on
        const unsigned char* mp = rec + 1024 + g * 8;                 // its scale / zero record of item 0
        const uint32_t off_lo = static_cast<uint32_t>((dw * 16 + g) * kRowBytes + (((4 * jj + h) ^ g) << 4));
        // register ring of whole items (two K steps each)
        uint4 w0[kAhead], w1[kAhead];
        uint2 meta[kAhead];
#pragma unroll
        for (int d = 0; d < kAhead; ++d) {
            if (d < items) {
                w0[d] = ld_stream_v4(wp + static_cast<size_t>(d) * kItemBytes);
                w1[d] = ld_stream_v4(wp + static_cast<size_t>(d) * kItemBytes + 32);
                meta[d] = ld_pinned_v2(mp + static_cast<size_t>(d) * kItemBytes);
            }
        }
        bool broken = false, first = true;
        int stage = 0;
        uint32_t phase = 0;
        for (int it0 = 0; it0 < items && !broken; it0 += kAhead) {
#pragma unroll
            for (int d = 0; d < kAhead; ++d) {
                const int it = it0 + d;
                if (it >= items || broken) continue;
                // the item's constants: exact-dequant zero terms and the scale pair of columns g and g + 8
                const typename Frag<ActT>::Zero z_lo = Frag<ActT>::zero(__byte_perm(meta[d].y, 0, 0x1010));
                const typename Frag<ActT>::Zero z_hi = Frag<ActT>::zero(__byte_perm(meta[d].y, 0, 0x3232));
                const uint32_t s_lo = tm::Mul<ActT>::template pair<CVT>(meta[d].x & 0xFFFFu), s_hi = tm::Mul<ActT>::template pair<CVT>(meta[d].x >> 16);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (broken) continue;
                    if (!first && !tc::mbar_wait(empty_addr + 8 * stage, phase ^ 1)) {
                        if (lane == 0) atomicExch(status, 4);
                        broken = true;
                        continue;
                    }
                    const uint4 w = t == 0 ? w0[d] : w1[d];
                    const uint32_t wv[4] = {w.x, w.y, w.z, w.w};
                    uint32_t a[4][4];
#pragma unroll
                    for (int wi = 0; wi < 4; ++wi) Frag<ActT>::expand(wv[wi], z_lo, z_hi, a[wi]);
                    // a[wi][0]: column g, low run; [2]: column g, high run; [1] / [3]: the same for column g + 8
                    if (live) {
                        const uint32_t addr = b_base + stage * kTileB + off_lo;
                        auto put = [&](uint32_t at, int run, uint32_t sc) {
                            st_shared_v4(at, tm::Mul<ActT>::mul(a[0][run], sc), tm::Mul<ActT>::mul(a[1][run], sc), tm::Mul<ActT>::mul(a[2][run], sc),
                                         tm::Mul<ActT>::mul(a[3][run], sc));
                        };
                        put(addr, 0, s_lo);
                        put(addr ^ 32u, 2, s_lo);
                        put(addr + 8 * kRowBytes, 1, s_hi);
                        put((addr ^ 32u) + 8 * kRowBytes, 3, s_hi);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(full_b_addr + 8 * stage);
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1;
                        first = false;
                    }
                }
                if (it + kAhead < items) {  // refill this ring slot
                    const size_t off = static_cast<size_t>(it + kAhead) * kItemBytes;
                    w0[d] = ld_stream_v4(wp + off);
                    w1[d] = ld_stream_v4(wp + off + 32);
                    meta[d] = ld_pinned_v2(mp + off);
                }
            }
        }

        // ---- epilogue: warp w may touch TMEM lanes 32 (w % 4) .. +31
        const int quarter = warp & 3;
        const int quartet = dw >> 2;
        const bool ok = __all_sync(0xFFFFFFFFu, tc::mbar_wait(tc::smem_u32(acc_ready), 0));
        if (!ok && lane == 0) atomicExch(status, 3);
        tc::fence_after_sync();
        // Work units: (128-row half, chunk of columns), dealt round-robin to the warp quartets.  Everything that decides whether
        // a unit runs is warp-uniform: the TMEM loads are warp-wide instructions.
        if constexpr (SWIGLU) {
            // gate columns [0, 128) and up columns [128, 256) of the accumulator -> 128 columns of the output
            constexpr int kChunks = kBN / 64;
            const int out_n = N / 2, out0 = n0 / 2;
#pragma unroll 1
            for (int unit = quartet; ok && unit < kHalves * kChunks; unit += kQuartets) {
                const int half = unit / kChunks, c = (unit - half * kChunks) * 32;
                if (half >= live_halves) break;
                const int m = m0 + half * 128 + quarter * 32 + lane;
                const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * kBN;
                uint32_t rg[32], ru[32];
                tc::tmem_ld_32x32(t_row + c, rg);
                tc::tmem_ld_32x32(t_row + kBN / 2 + c, ru);
                tc::tmem_ld_wait();
                if (m < m_end && out0 + c < out_n) {
                    ActT* dst = y + static_cast<size_t>(m) * out_n + out0 + c;
                    uint32_t packed[16];
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float g = to_float(from_float<ActT>(__uint_as_float(rg[i])));
                        const float u = to_float(from_float<ActT>(__uint_as_float(ru[i])));
                        const float sg = to_float(from_float<ActT>(g / (1.f + expf(-g))));
                        const uint32_t bits = tm::bits16<ActT>(sg * u);
                        if (i & 1)
                            packed[i >> 1] |= bits << 16;
                        else
                            packed[i >> 1] = bits;
                    }
                    // (a chunk is whole: the expert's intermediate size is a multiple of 128)
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        reinterpret_cast<uint4*>(dst)[v] = make_uint4(packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
                }
            }
        } else {
            // Rows leave for their own addresses (possibly on a peer GPU): a thread's 64 bytes of its own row would make every
            // warp-wide store 32 separate 16-byte pieces, which NVLink carries at a fraction of its rate (measured: the
            // expert-parallel down projection took 480 us against 195 us with local stores).  The warp turns its 32 rows x 64
            // columns in shared memory (the stages are idle once the accumulator is complete) and stores 128 contiguous bytes
            // of one row with every eight lanes.
            constexpr int kChunks = kBN / 64;
            unsigned char* stg = smem + dw * 4096;  // [32 rows][8 x 16 B], chunk v of row r at v ^ (r & 7)
            const uint32_t stg_w = tc::smem_u32(stg) + lane * 128;
#pragma unroll 1
            for (int unit = quartet; ok && unit < kHalves * kChunks; unit += kQuartets) {
                const int half = unit / kChunks, c = (unit - half * kChunks) * 64;
                if (half >= live_halves) break;
                const int m = m0 + half * 128 + quarter * 32 + lane;
                const uint64_t mine = m < m_end ? grp.y_ptrs[m] : 0ull;  // lane r holds row r's destination
                const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * kBN;
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    uint32_t r[32];
                    tc::tmem_ld_32x32(t_row + c + 32 * part, r);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        uint32_t pk[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            pk[i] = tm::bits16<ActT>(__uint_as_float(r[8 * v + 2 * i])) | (tm::bits16<ActT>(__uint_as_float(r[8 * v + 2 * i + 1])) << 16);
                        st_shared_v4(stg_w + (((4 * part + v) ^ (lane & 7)) << 4), pk[0], pk[1], pk[2], pk[3]);
                    }
                }
                __syncwarp();
                const int v = lane & 7;
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    const int rr = it * 4 + (lane >> 3);
                    const uint64_t dst = __shfl_sync(0xFFFFFFFFu, mine, rr);
                    const uint4 val = *reinterpret_cast<const uint4*>(stg + rr * 128 + ((v ^ (rr & 7)) << 4));
                    if (dst != 0ull && n0 + c + 8 * v < N)
                        *reinterpret_cast<uint4*>(dst + static_cast<size_t>(n0 + c + 8 * v) * sizeof(ActT)) = val;
                }
                __syncwarp();
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

template <typename ActT, bool SWIGLU>
int launch_grouped(const unsigned char* wq, int scale_dtype, const void* x, void* y, int64_t R, int64_t N, int64_t K, int* status, const GroupArgs& grp,
                   int max_blocks, cudaStream_t stream) {
    CUtensorMap map_x;
    const CUtensorMapDataType elem = tm::Mul<ActT>::kFmt == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int st = make_tensor_map_2d(&map_x, x, elem, 2, R, K, K * 2, 128 * kHalves, kGK, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != EQ_OK) return st;
    const bool cvt = scale_dtype != (tm::Mul<ActT>::kFmt == 0 ? EQ_F16 : EQ_BF16);
    auto kernel = cvt ? w4a16_gemm_tc_kernel<ActT, true, SWIGLU> : w4a16_gemm_tc_kernel<ActT, false, SWIGLU>;
    EQ_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem)));
    const dim3 grid(static_cast<unsigned>(ceil_div(N, kBN)), static_cast<unsigned>(max_blocks));
    kernel<<<grid, kThreads, kSmem, stream>>>(map_x, wq, static_cast<ActT*>(y), static_cast<int>(N), static_cast<int>(K), status, grp);
    EQ_LAUNCH_OK("w4a16_gemm_tc_kernel");
    return EQ_OK;
}

template <typename ActT>
int launch_typed(const unsigned char* wq, int scale_dtype, const int32_t* perm, const ActT* x, ActT* y, int64_t M, int64_t N,
                 int64_t K, ActT* gathered, int* status, cudaStream_t stream) {
    if (perm) {
        const int64_t total = M * K;
        gather_cols_kernel<ActT><<<static_cast<unsigned>(ceil_div(total, 256)), 256, 0, stream>>>(x, perm, M, K, gathered);
        EQ_LAUNCH_OK("gather_cols_kernel");
        x = gathered;
    }
    const int act = tm::Mul<ActT>::kFmt == 0 ? EQ_F16 : EQ_BF16;
    if (!w4_tmem_pairs(M, N, K)) return w4_tmem_dense_launch(wq, scale_dtype, x, y, M, N, K, act, false, false, status, stream);
    return w4_tmem_pair_dense_launch(wq, scale_dtype, x, y, M, N, K, act, false, status, stream);
}

}  // namespace

// gathered: M * K elements of scratch when perm is given.  status: one word, set by a bounded wait that ran out.
int w4_gemm_tc_launch(const unsigned char* wq, int scale_dtype, const int32_t* perm, const void* x, void* y, int64_t M, int64_t N,
                      int64_t K, int act_dtype, void* gathered, int* status, cudaStream_t stream) {
    if (act_dtype == EQ_F16)
        return launch_typed<__half>(wq, scale_dtype, perm, static_cast<const __half*>(x), static_cast<__half*>(y), M, N, K,
                                    static_cast<__half*>(gathered), status, stream);
    return launch_typed<__nv_bfloat16>(wq, scale_dtype, perm, static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), M,
                                       N, K, static_cast<__nv_bfloat16*>(gathered), status, stream);
}

// Grouped expert GEMM of the expert-parallel layer.  x: [R][K] activations in expert order; blocks / n_blocks: device-side list
// of row blocks of at most 256 rows; wq: E stacked repacked weights expert_stride bytes apart, each [N][K] logical, N and K
// multiples of 128.  swiglu: N is the width of the [gate | up] weight, y has N / 2 columns and y_ptrs is not read; otherwise the
// rows go to y_ptrs and y is not used.  max_blocks bounds the grid.
int w4_gemm_tc_grouped_launch(const unsigned char* wq, size_t expert_stride, int scale_dtype, const void* x, void* y, int64_t R, int64_t N,
                              int64_t K, int act_dtype, const RowBlock* blocks, const int32_t* n_blocks, int max_blocks, const uint64_t* y_ptrs,
                              bool swiglu, int* status, cudaStream_t stream) {
    const GroupArgs grp = {blocks, n_blocks, y_ptrs, expert_stride};
    if (act_dtype == EQ_F16)
        return swiglu ? launch_grouped<__half, true>(wq, scale_dtype, x, y, R, N, K, status, grp, max_blocks, stream)
                      : launch_grouped<__half, false>(wq, scale_dtype, x, y, R, N, K, status, grp, max_blocks, stream);
    return swiglu ? launch_grouped<__nv_bfloat16, true>(wq, scale_dtype, x, y, R, N, K, status, grp, max_blocks, stream)
                  : launch_grouped<__nv_bfloat16, false>(wq, scale_dtype, x, y, R, N, K, status, grp, max_blocks, stream);
}

}  // namespace eq
