// W4A16 with the weights in tensor memory (w4_tmem.cu, w4_tmem2.cu): which calls, launch functions, shared device code.
#pragma once
#include "tc_common.cuh"
#include "w4_tile.cuh"

namespace eq {

// Row counts at which the weights-in-TMEM kernels take over (us in graph replays, both kernels forced, streamed : in TMEM).
// From 17 rows: 17 rows K=4096 N=14336 23.6 : 15.8, K=14336 N=4096 21.2 : 15.8, K=N=4096 11.5 : 9.0.  At 16 rows w4_stream.cu, which
// then stages all rows in shared memory at once, is the faster one for K=4096 (14.4 : 15.4, K=N=4096 8.6 : 8.9), and for the
// [gate | up] + down MLP of hidden 4096, intermediate 14336 (f16 42.2 : 45.5, bf16 43.4 : 47.8; 12 rows 40.4 : 45.1, 8 rows 33.2 : 44.5),
// but not for every shape: from 12 rows on a K that has to be cut to fit is the slower one streamed (K=14336 N=4096, 8 rows 13.9 :
// 15.4, 12 rows 17.2 : 15.5, 16 rows 18.3 : 15.8; MLP of hidden 5120, intermediate 17408, 8 rows 43.1 : 51.6, 12 rows 64.8 : 51.3, 16 rows
// 70.5 : 50.6).  The rule does not look at that yet.
// 17 to 24 rows keep the stream's arithmetic, integers in the MMA and scales applied to f32 sums (PROMOTE); above, the weights are
// scaled before the MMA (28 rows, K=4096 N=14336: 15.8 against 20.0 promoted, measured when the kernel was new).
constexpr int64_t kTmemPromoteRows = 24;

// 17 to 24 rows of a small matrix stay with w4_stream.cu: with little of K per slice the tensor path's prologue, hand-overs
// and cluster meeting are not hidden, and one wave of the stream's column tiles (16 channels a CTA) takes no longer for a
// wider matrix.  So the limits on K are: short whatever the width (K=512 N=4096, 17 rows: 3.8 us streamed against 4.9);
// about 1280 for one or one and a half waves (1280 x 2048: 4.3 | 5.2, 24 rows 4.8 | 5.3; 1280 x 512: even; 1792 x 2048, 24
// rows: 6.0 | 5.7); above that a limit on K x rows, the staged x, and on K x N x rows (1792 x 4096, 17 rows 6.1 | 7.2, 24 rows
// 6.7 | 7.4; 2560 x 4096, 17 rows 7.3 | 7.9, 24 rows even; 3072 x 4096: 8.3 | 8.1; 1792 x 8192, 24 rows even).  A long K with a
// handful of column tiles leaves the tensor path fewer CTAs than the stream's K slices (14336 x 256: 7.3 | 9.1; 5120 x 256:
// 5.2 | 5.5; 5120 x 512: 6.3 | 5.7).
inline bool w4_few_rows_stream(int64_t M, int64_t N, int64_t K) {
    if (K <= 896) return N <= 8192;
    if (K >= 5120) return K >= 20 * N;
    if (N <= 3072) return N >= 1024 && K <= 1280;
    return N <= 8192 && K * M <= 43520 && K * N * M <= int64_t(1) << 28;
}

// More than 256 rows (128 from K=2048 on, where a pair's longer prologue and epilogue are hidden) whose 256 x 256 tiles occupy
// at least half of the CTA pairs run on pairs (w4_tmem2.cu), the rest on one-CTA tiles of at most 128 rows with K slices where
// CTAs would idle.  Measured, us, one-CTA against pairs: MLP of hidden 4096, intermediate 14336, both linears forced: 300 rows
// 158 : 134, 1024 rows 317 : 277, 4096 rows 1266 : 1076; K=N=4096, 512 rows (32 tiles) 21.2 : 28.0, K=14336 N=4096, 300 rows
// (32 tiles) 48 : 50; K=4096 N=1792, 2048 rows (56 tiles) 33.5 : 28.8.  [gate | up] of hidden 5120, intermediate 17408: 160
// rows 66 : 50, 256 rows 80 : 68; linears of 136 to 256 rows, pairs over one-CTA: K=4096 N=14336 0.78 to 0.91, K=2048 N=9472
// 1.00 to 0.93, K=1024 N=9472 1.14 to 1.10.
inline bool w4_tmem_pairs(int64_t M, int64_t N, int64_t K) {
    return M > (K >= 2048 ? 128 : 256) && ceil_div(N, 256) * ceil_div(M, 256) * 4 >= sm_count();
}

// The kernel of a call of more than 16 rows with a 16-byte aligned output.  perm: the weight carries a row permutation (the
// stream kernel gathers x while it stages it, the tensor path needs a pass of its own).  swiglu: N is the width of [gate | up].
enum class W4Route { kStream, kPromoted, kScaled, kPairs };
inline W4Route w4_route(int64_t M, int64_t N, int64_t K, bool perm, bool swiglu) {
    if (M <= kTmemPromoteRows) return perm || (!swiglu && w4_few_rows_stream(M, N, K)) ? W4Route::kStream : W4Route::kPromoted;
    return w4_tmem_pairs(M, N, K) ? W4Route::kPairs : W4Route::kScaled;
}

// w4_tmem.cu.  Dense: y[M, N] = x W, or with swiglu act(silu(gate)) * up of a [gate | up] weight of N columns; promote: scales on
// f32 sums (at most 32 rows).  status: one word, set by a bounded wait that ran out.
int w4_tmem_dense_launch(const unsigned char* wq, int scale_dtype, const void* x, void* y, int64_t M, int64_t N, int64_t K, int act_dtype, bool swiglu,
                         bool promote, int* status, cudaStream_t stream);
// Grouped: x [R][K] in expert order; blocks / n_blocks: device-side list of row blocks of at most block_rows (16 or 128) rows of
// one expert each; wq: stacked repacked weights expert_stride bytes apart; y_rows (optional): output row m goes to row y_rows[m].
int w4_tmem_grouped_launch(const unsigned char* wq, size_t expert_stride, int scale_dtype, const void* x, void* y, int64_t R, int64_t N, int64_t K,
                           int act_dtype, const RowBlock* blocks, const int32_t* n_blocks, int block_rows, const int32_t* y_rows, bool swiglu, int* status,
                           cudaStream_t stream);
// w4_tmem2.cu
int w4_tmem_pair_dense_launch(const unsigned char* wq, int scale_dtype, const void* x, void* y, int64_t M, int64_t N, int64_t K, int act_dtype, bool swiglu,
                              int* status, cudaStream_t stream);

struct W4TmemArgs {
    const unsigned char* wq;   // repacked weight (of expert 0)
    void* y;
    int M, N, K;               // N: columns of the weight; the SwiGLU form writes N / 2
    int row_tiles, rows_per_tile, splits, units;  // dense form
    int scale_dtype;
    int* status;
    // grouped form
    const RowBlock* blocks;
    const int32_t* n_blocks;
    const int32_t* y_rows;     // optional: output row m goes to row y_rows[m]
    size_t expert_stride;
};

// ---- device code shared by w4_tmem.cu and w4_tmem2.cu ----------------------------------------------------------
namespace tm {

// Bounded wait as tc::mbar_wait, but the thread sleeps in the barrier unit between looks: with dequantisation bound by issue
// slots, spinning TMA and MMA threads would take theirs.
// DEPENDENT: in a programmatic dependent the warps wait for each other while the grid before it may still run, for as long as
// it likes: a wait that runs out is taken once more from the end of that grid.  (griddepcontrol.wait ahead of the first wait
// does that too, but costs 0.3 to 0.6 us of a 16 us launch where launches follow each other.)
__device__ __forceinline__ bool try_asleep(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity), "r"(1000000u)
                 : "memory");
    return ok != 0;
}
template <bool DEPENDENT = false>
__device__ __forceinline__ bool wait_asleep(uint32_t bar, uint32_t parity) {
    if (try_asleep(bar, parity)) return true;  // the usual case, without a look at the clock
    bool again = DEPENDENT;
    long long start = clock64();
#pragma unroll 1
    while (!try_asleep(bar, parity)) {
        if (clock64() - start > tc::kWaitCycles) {
            if (!again) return false;
            again = false;
            asm volatile("griddepcontrol.wait;" ::: "memory");
            start = clock64();
        }
    }
    return true;
}

// ---- distributed shared memory
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

template <typename ActT>
struct Mul;
template <>
struct Mul<__half> {
    static constexpr uint32_t kFmt = 0;
    template <bool CVT>
    static __device__ __forceinline__ uint32_t pair(uint32_t raw) {
        if constexpr (CVT) raw = __half_as_ushort(__float2half_rn(__uint_as_float(raw << 16)));
        return __byte_perm(raw, 0, 0x1010);
    }
    static __device__ __forceinline__ uint32_t mul(uint32_t v, uint32_t s) {
        uint32_t r;
        asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(s));
        return r;
    }
};
template <>
struct Mul<__nv_bfloat16> {
    static constexpr uint32_t kFmt = 1;
    template <bool CVT>
    static __device__ __forceinline__ uint32_t pair(uint32_t raw) {
        if constexpr (CVT) raw = __bfloat16_as_ushort(__float2bfloat16_rn(__half2float(__ushort_as_half(static_cast<unsigned short>(raw)))));
        return __byte_perm(raw, 0, 0x1010);
    }
    static __device__ __forceinline__ uint32_t mul(uint32_t v, uint32_t s) {
        uint32_t r;
        asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(s));
        return r;
    }
};

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// 16 lanes x 32 columns: lane 4 g + j of the warp gives rows g and g + 8 of column 4 i + j in registers 2 i, 2 i + 1.
__device__ __forceinline__ void tmem_st_16x128b_x8(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
    const uint32_t acc = accumulate ? 1u : 0u;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc)
        : "memory");
}

template <typename ActT>
__device__ __forceinline__ uint32_t bits16(float v) {
    const ActT o = from_float<ActT>(v);
    return *reinterpret_cast<const uint16_t*>(&o);
}
// Two values rounded by one instruction, and back.  (The epilogue of an expert's [gate | up] tile is a quarter of its instructions:
// with pairs rounded and exchanged together the routed layer of 4096 tokens takes 509 us for 525.)
template <typename ActT>
__device__ __forceinline__ uint32_t pack16(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack16<__half>(float lo, float hi) {
    const __half2 p = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}
template <>
__device__ __forceinline__ uint32_t pack16<__nv_bfloat16>(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}
template <typename ActT>
__device__ __forceinline__ float2 unpack16(uint32_t p);
template <>
__device__ __forceinline__ float2 unpack16<__half>(uint32_t p) { return __half22float2(*reinterpret_cast<const __half2*>(&p)); }
template <>
__device__ __forceinline__ float2 unpack16<__nv_bfloat16>(uint32_t p) { return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xFFFF0000u)); }

// Sixteen accumulator columns (rows c .. c + 15 of a unit) of one warp's 32 channels -> y.  tile_lo: weight tile of lanes
// 0-15; lanes 16-31 hold the next one, or (SWIGLU) the up tile that belongs to it.
template <typename ActT, bool SWIGLU, bool GROUPED>
__device__ __forceinline__ void emit16(const W4TmemArgs& a, const float (&v)[16], int tile_lo, int row0, int rows, int c) {
    const int lane = threadIdx.x & 31, n_tiles = a.N / 16;
    if constexpr (SWIGLU) {
        // lanes 0-15 hold gate, 16-31 up of the same channels: of two rows, the low lanes finish the first
        const int out_n = a.N / 2;
        const bool live = tile_lo < n_tiles / 2;
        ActT* dst = static_cast<ActT*>(a.y) + tile_lo * 16 + (lane & 14);
        const uint32_t mine_first = lane < 16 ? 0x5410u : 0x3276u;  // {gate, up} of the row this lane finishes, from (own, other) pairs
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
            float o[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t own = pack16<ActT>(v[i + 2 * h], v[i + 2 * h + 1]), other = __shfl_xor_sync(0xFFFFFFFFu, own, 16);
                const float2 gu = unpack16<ActT>(__byte_perm(own, other, mine_first));
                const float sg = to_float(from_float<ActT>(gu.x / (1.f + expf(-gu.x))));
                o[h] = sg * gu.y;
            }
            // neighbours swap so that a lane holds two channels of one row
            const uint32_t p = pack16<ActT>(o[0], o[1]), pn = __shfl_xor_sync(0xFFFFFFFFu, p, 1);
            const uint32_t w = (lane & 1) ? __byte_perm(p, pn, 0x3276) : __byte_perm(p, pn, 0x5410);
            const int r = c + i + 2 * (lane & 1) + (lane >> 4);
            if (live && r < rows) *reinterpret_cast<uint32_t*>(dst + static_cast<size_t>(row0 + r) * out_n) = w;
        }
    } else {
        const bool live = tile_lo + (lane >> 4) < n_tiles;
        const int ch = tile_lo * 16 + (lane & 30);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const uint32_t p = pack16<ActT>(v[i], v[i + 1]), pn = __shfl_xor_sync(0xFFFFFFFFu, p, 1);
            const uint32_t w = (lane & 1) ? __byte_perm(p, pn, 0x3276) : __byte_perm(p, pn, 0x5410);
            const int r = c + i + (lane & 1);
            if (live && r < rows) {
                const size_t row = GROUPED && a.y_rows ? static_cast<size_t>(a.y_rows[row0 + r]) : static_cast<size_t>(row0 + r);
                *reinterpret_cast<uint32_t*>(static_cast<ActT*>(a.y) + row * a.N + ch) = w;
            }
        }
    }
}

// A dequant warp's view of one item: two weight tiles of 16 channels, read from the warp's ring slot.
struct ItemWords {
    uint32_t wd[2][8];
    uint2 mt[2];
};
// A lane's byte offsets inside a ring slot.  The 16-byte piece of lane 4 g + r of a half tile is put at place
// (r + g / 2) % 4 of its channel's four, so that the 32 lanes reading word j of piece r of their channels hit 32 banks.
struct LaneOffsets {
    uint32_t put, put_meta, get[4], get_meta;
    __device__ __forceinline__ LaneOffsets() {
        const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
        put = ((lane & ~3) + ((lane + (lane >> 3)) & 3)) * 16;
        put_meta = 1024 + lane * 16;
#pragma unroll
        for (int r = 0; r < 4; ++r) get[r] = (4 * g + ((r + (g >> 1)) & 3)) * 16 + 4 * j;
        get_meta = 1024 + 8 * g;
    }
};
// (Offsets as immediates: with an address computed for each of them the reads and copies cost thirty more instructions an item.)
template <int OFF>
__device__ __forceinline__ uint32_t lds32_at(uint32_t a) {
    uint32_t r;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(r) : "r"(a), "n"(OFF) : "memory");
    return r;
}
__device__ __forceinline__ void load_item(uint32_t slot_addr, const LaneOffsets& o, ItemWords& w) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint32_t at = slot_addr + o.get[r];
        w.wd[0][2 * r] = lds32_at<0>(at);
        w.wd[0][2 * r + 1] = lds32_at<512>(at);
        w.wd[1][2 * r] = lds32_at<kItemBytes>(at);
        w.wd[1][2 * r + 1] = lds32_at<kItemBytes + 512>(at);
    }
    const uint32_t meta = slot_addr + o.get_meta;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w.mt[0].x), "=r"(w.mt[0].y) : "r"(meta) : "memory");
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(w.mt[1].x), "=r"(w.mt[1].y) : "r"(meta), "n"(kItemBytes) : "memory");
}
// The records (1088 bytes) of a warp's two tiles into its ring slot; src0, src1: the records + 16 * lane.
__device__ __forceinline__ void fetch_items(uint32_t slot_addr, const LaneOffsets& o, const unsigned char* src0, const unsigned char* src1) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.lt.u32 p, %4, 4;\n"
        "cp.async.cg.shared.global [%0], [%2], 16;\n"
        "cp.async.cg.shared.global [%0+512], [%2+512], 16;\n"
        "@p cp.async.cg.shared.global [%1], [%2+1024], 16;\n"
        "cp.async.cg.shared.global [%0+%5], [%3], 16;\n"
        "cp.async.cg.shared.global [%0+%6], [%3+512], 16;\n"
        "@p cp.async.cg.shared.global [%1+%5], [%3+1024], 16;\n"
        "}\n" ::"r"(slot_addr + o.put),
        "r"(slot_addr + o.put_meta), "l"(src0), "l"(src1), "r"(threadIdx.x & 31), "n"(kItemBytes), "n"(kItemBytes + 512)
        : "memory");
}
// Zero point pair -> constants of the exact dequant (Frag<ActT>::expand), fewer instructions than Frag<ActT>::zero: the
// zero points are the integers 0..16.
template <typename ActT>
__device__ __forceinline__ typename Frag<ActT>::Zero zero_of(uint32_t z_pair);
template <>
__device__ __forceinline__ Frag<__half>::Zero zero_of<__half>(uint32_t z_pair) {
    Frag<__half>::Zero r;
    asm("add.f16x2 %0, %1, %2;" : "=r"(r.sub) : "r"(z_pair), "r"(0x64006400u));                              // 1024 + z
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r.fma) : "r"(z_pair), "r"(0xBC00BC00u), "r"(0xD400D400u));  // -(64 + z)
    return r;
}
template <>
__device__ __forceinline__ Frag<__nv_bfloat16>::Zero zero_of<__nv_bfloat16>(uint32_t z_pair) {
    Frag<__nv_bfloat16>::Zero r;
    uint32_t t;
    asm("add.f16x2 %0, %1, %2;" : "=r"(t) : "r"(z_pair), "r"(0x64006400u));  // low mantissa bits of 1024 + z: the integer z
    r.sub = lop3<0xEA>(t, 0x001F001Fu, 0x43004300u);                           // bf16 128 + z
    r.fma = 0;
    return r;
}
// Expands the item into 64 columns of TMEM at taddr (lanes of this warp's quarter): q - z, times the scale unless PROMOTE.
template <typename ActT, bool CVT, bool PROMOTE>
__device__ __forceinline__ void expand_item(const ItemWords& w, uint32_t taddr) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const typename Frag<ActT>::Zero z_lo = zero_of<ActT>(__byte_perm(w.mt[t].y, 0, 0x1010)), z_hi = zero_of<ActT>(__byte_perm(w.mt[t].y, 0, 0x3232));
        uint32_t s_lo = 0, s_hi = 0;
        if constexpr (!PROMOTE) {
            s_lo = Mul<ActT>::template pair<CVT>(w.mt[t].x & 0xFFFFu);
            s_hi = Mul<ActT>::template pair<CVT>(w.mt[t].x >> 16);
        }
        const uint32_t dst = taddr + (static_cast<uint32_t>(16 * t) << 16);
#pragma unroll
        for (int half = 0; half < 2; ++half) {  // 64 k = 32 columns
            uint32_t r[16];
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // k run 32 (2 half + i / 2) + 8 (i & 1), and the one 16 further on
                uint32_t f[4];
                Frag<ActT>::expand(w.wd[t][4 * half + i], z_lo, z_hi, f);
                const int c = 4 * (i >> 1) + (i & 1);
                if constexpr (PROMOTE) {
                    r[2 * c] = f[0];
                    r[2 * c + 1] = f[1];
                    r[2 * (c + 2)] = f[2];
                    r[2 * (c + 2) + 1] = f[3];
                } else {
                    r[2 * c] = Mul<ActT>::mul(f[0], s_lo);
                    r[2 * c + 1] = Mul<ActT>::mul(f[1], s_hi);
                    r[2 * (c + 2)] = Mul<ActT>::mul(f[2], s_lo);
                    r[2 * (c + 2) + 1] = Mul<ActT>::mul(f[3], s_hi);
                }
            }
            tmem_st_16x128b_x8(dst + 32 * half, r);
        }
    }
}

}  // namespace tm
}  // namespace eq
