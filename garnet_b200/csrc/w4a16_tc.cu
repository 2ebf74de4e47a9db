// Tensor-core (tcgen05 / TMEM) tile kernel of the int4 linear, for batches above
// the streaming kernel's 16 rows.
//
// The weights are the A operand and live in tensor memory: a CTA owns a panel of 128 weight rows (8 strips) and a tile of up to
// 192 batch rows (the UMMA N dimension).  Per 64 columns of K:
//   pack producer   TMA of the packed strip-chunks (codes + scales) of 128 columns, L2 prefetch ahead of it;
//   x producer      TMA of the activation tile (128-byte swizzle), the only operand that the MMAs read from shared memory;
//   dequant warps   a lane owns a weight row: 64 codes -> bf16 x group scale -> tcgen05.st into one of four A tiles; four
//                   groups of four warps, so that a warp has four steps' time for its chain, or two groups when a CTA has one
//                   item (and half of the registers, so that two CTAs share an SM: the next launch's weights are on their way);
//   MMA warp        one thread issues 4 tcgen05.mma (A in tensor memory, K = 16);
//   4 epilogue      read the accumulator with tcgen05.ld, round to bf16 and store y[m, n]; accumulators are double
//   warps           buffered so that the next tile's main loop overlaps the epilogue.
// Small matrices are cut along K over a cluster of up to 8 CTAs, whose fp32 partial tiles meet in distributed shared memory
// and are added in slice order: no partial sums in global memory and no second launch.
// Bound: an MMA of N columns takes N / 2 clocks and reads N x 32 bytes; expanding through shared memory instead (the form
// before: 32 KiB written and 48 KiB read per 128 x 256 x 64 step, a proxy fence per warp and step) took 1535 clocks per step
// against 512 of MMAs.  Batch tiles are even shares of the batch in multiples of 16 rows, so little of them is padding.
//   rows x K -> N             before      now (called from Python; x [1000, 2048]: 829 TFLOP/s)
//   1000 x 2048 -> 12288      74.3 us     60.7 us
//     77 x 2048 -> 4096       15.6 us     9.5 us
//     16 x 6144 -> 2048       17.6 us     8.0 us
// Numerics: w = bf16(q * s) (one rounding of the dequantised weight), products
// exact, fp32 accumulation in TMEM, bf16 output.
#include <algorithm>
#include <cooperative_groups.h>

#include "layout.h"
#include "tc_common.cuh"
#include "w4a16.h"

namespace gb200 {

namespace cg = cooperative_groups;

constexpr int kTcAStages = 4;             // A tiles of 64 columns of K in tensor memory, 32 columns each
constexpr int kTcBStages = 6;             // activation tiles of 64 columns of K
constexpr int kTcPackStages = 4;          // packed chunks of 128 columns of K
constexpr int kTcPrefetchChunks = 8;      // packed chunks prefetched into L2 ahead of the ring
constexpr int kTcFirstDequant = 4, kTcEpilogueWarps = 4;
__host__ __device__ constexpr int tc_threads(int groups) { return (kTcFirstDequant + 4 * groups + kTcEpilogueWarps) * 32; }
constexpr int kTcChunkBytes = 1024 + 32;  // int4 strip-chunk
constexpr int kTcPackBytes = 8 * kTcChunkBytes;
constexpr uint32_t kTcACols = 32;
// Tensor memory: two accumulators and the A tiles, or, when a CTA has one item of at most 128 rows, one accumulator and the A
// tiles in half of it, so that the next launch's CTA can move in (its weights are on their way while this one finishes).
constexpr int kTcHalfRows = 128;
static_assert(2 * kTcMaxRows + kTcAStages * kTcACols <= 512 && kTcHalfRows + kTcAStages * kTcACols <= 256, "tensor memory");

struct TcParams {
    __nv_bfloat16* y;
    int* fault;
    int m, n;
    int ldy;
    int chunks;
    int panels, row_tiles, tile_rows;
    int kslices;                     // the K dimension of a tile may be cut into slices handled by the CTAs of a cluster
    int scale_dtype;
    int tmem_cols, col_a;            // tensor memory: columns, and where the A tiles start
};

// Work item -> (panel, batch tile, K slice) and the slice's chunk range.
struct TcItem {
    int panel, tt, c0, c1;
};
__device__ __forceinline__ TcItem tc_decode(const TcParams& p, int item)
{
    TcItem it;
    const int per_panel = p.row_tiles * p.kslices;
    it.panel = item / per_panel;
    const int rem = item - it.panel * per_panel;
    it.tt = rem / p.kslices;
    const int slice = rem - it.tt * p.kslices;
    it.c0 = tc_first_chunk(p.chunks, p.kslices, slice);
    it.c1 = tc_first_chunk(p.chunks, p.kslices, slice + 1);
    return it;
}

// Shared memory: packed ring, barriers, activation ring (a stage is tile_rows x 128 bytes).  The partial tile of a K slice,
// [batch row][128 weight rows] fp32, takes the activation ring's place.
struct TcSmem {
    static constexpr int pk = 0;
    static constexpr int bars = pk + kTcPackStages * kTcPackBytes;
    static constexpr int b = (bars + 512 + 1023) / 1024 * 1024;
    static constexpr int total(int tile_rows) { return b + kTcBStages * tile_rows * 128 + 1024; }   // slack for 1024-byte alignment
};
static_assert(128 * 4 <= kTcBStages * 128, "partial tile");
static_assert(2 * (TcSmem::total(kTcSharedRows) + 1024) <= 228 * 1024 && 2 * (TcSmem::total(kTcSharedRows + 16) + 1024) > 228 * 1024,
              "tiles with which two CTAs share an SM");

// One int4 word (8 codes of one row, pair-interleaved) times a scale -> 8 bf16.
__device__ __forceinline__ uint4 int4_word_to_bf16x8(uint32_t w, uint32_t scale_bf16x2)
{
    uint4 r;
    const uint32_t p0 = int4x2_to_bf16x2(w), p1 = int4x2_to_bf16x2(w >> 4), p2 = int4x2_to_bf16x2(w >> 8),
                   p3 = int4x2_to_bf16x2(w >> 12);
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r.x) : "r"(p0), "r"(scale_bf16x2));
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r.y) : "r"(p1), "r"(scale_bf16x2));
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r.z) : "r"(p2), "r"(scale_bf16x2));
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r.w) : "r"(p3), "r"(scale_bf16x2));
    return r;
}
// Same with an fp32 scale (fp16-scaled artifacts): q * s rounded once to bf16.
__device__ __forceinline__ uint4 int4_word_to_bf16x8_f32(uint32_t w, float s)
{
    uint32_t out[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t p = int4x2_to_bf16x2(w >> (4 * j));
        const float lo = __uint_as_float(p << 16) * s, hi = __uint_as_float(p & 0xffff0000u) * s;
        const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        out[j] = *reinterpret_cast<const uint32_t*>(&v);
    }
    return make_uint4(out[0], out[1], out[2], out[3]);
}

__device__ __forceinline__ void tc_st_32x32(uint32_t taddr, const uint4 (&v)[8])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w), "r"(v[2].x), "r"(v[2].y),
        "r"(v[2].z), "r"(v[2].w), "r"(v[3].x), "r"(v[3].y), "r"(v[3].z), "r"(v[3].w), "r"(v[4].x), "r"(v[4].y), "r"(v[4].z), "r"(v[4].w),
        "r"(v[5].x), "r"(v[5].y), "r"(v[5].z), "r"(v[5].w), "r"(v[6].x), "r"(v[6].y), "r"(v[6].z), "r"(v[6].w), "r"(v[7].x), "r"(v[7].y),
        "r"(v[7].z), "r"(v[7].w)
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// y[row, n], y[row, n + 1] of a pair of neighbouring outputs.
__device__ __forceinline__ void tc_store_pair(const TcParams& p, int row, int n, float a, float b, bool wide)
{
    __nv_bfloat16* at = p.y + size_t(row) * p.ldy + n;
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    if (wide && n + 1 < p.n) *reinterpret_cast<__nv_bfloat162*>(at) = v;
    else {
        if (n < p.n) at[0] = v.x;
        if (n + 1 < p.n) at[1] = v.y;
    }
}

template <int kGroups>
__global__ void __launch_bounds__(tc_threads(kGroups), 4 / kGroups)
w4a16_tc_kernel(const TcParams p, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map)
{
    constexpr int kTcThreads = tc_threads(kGroups), kTcFirstEpilogue = kTcFirstDequant + 4 * kGroups;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* b_ring = smem + TcSmem::b;
    uint8_t* pk_ring = smem + TcSmem::pk;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TcSmem::bars);
    uint64_t* pk_full = bars;                          // [kTcPackStages]
    uint64_t* pk_empty = pk_full + kTcPackStages;      // [kTcPackStages]
    uint64_t* a_full = pk_empty + kTcPackStages;       // [kTcAStages]
    uint64_t* a_empty = a_full + kTcAStages;           // [kTcAStages]
    uint64_t* b_full = a_empty + kTcAStages;           // [kTcBStages]
    uint64_t* b_empty = b_full + kTcBStages;           // [kTcBStages]
    uint64_t* acc_full = b_empty + kTcBStages;         // [2]
    uint64_t* acc_empty = acc_full + 2;                // [2]
    uint64_t* drained = acc_empty + 2;                 // every MMA done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kTcPackStages; ++s) {
            mbar_init(&pk_full[s], 1);
            mbar_init(&pk_empty[s], 8);   // four warps per half of the chunk
        }
        for (int s = 0; s < kTcAStages; ++s) {
            mbar_init(&a_full[s], 4);
            mbar_init(&a_empty[s], 1);
        }
        for (int s = 0; s < kTcBStages; ++s) {
            mbar_init(&b_full[s], 1);
            mbar_init(&b_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], kTcEpilogueWarps);
        }
        mbar_init(drained, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    pdl_launch_dependents();

    const int items = p.panels * p.row_tiles * p.kslices;

    if (warp == 0) {
        // ------------------------------------- producer of packed codes + scales
        // Weights are constants: this stream starts before the previous kernel in the
        // stream has finished, and runs as far ahead as its ring allows.
        if (elect_one()) {
            // One thread feeds the ring, so its loop carries no divisions: the stage index, the
            // ring's wrap count and the prefetch cursor advance by increments.
            uint32_t ps = 0, round = 0, issued = 0, prefetched = 0;
            int pf_item = blockIdx.x;
            TcItem pf = pf_item < items ? tc_decode(p, pf_item) : TcItem{};
            int pf_c = pf.c0;
            for (int item = blockIdx.x; item < items && !*abort_flag; item += gridDim.x) {
                const TcItem it = tc_decode(p, item);
                for (int c = it.c0; c < it.c1; ++c, ++issued) {
                    // keep the L2 prefetch kTcPrefetchChunks ahead of the ring, across items
                    while (pf_item < items && prefetched < issued + kTcPrefetchChunks) {
                        tma_prefetch_2d(&w_map, pf_c * (kTcChunkBytes / 8), pf.panel * 8);
                        ++prefetched;
                        if (++pf_c == pf.c1) {
                            pf_item += gridDim.x;
                            if (pf_item < items) {
                                pf = tc_decode(p, pf_item);
                                pf_c = pf.c0;
                            }
                        }
                    }
                    if (round > 0 && !mbar_wait_suspended(&pk_empty[ps], (round - 1) & 1)) {
                        atomicExch(p.fault, 11);
                        *abort_flag = 1;
                        break;
                    }
                    // one TMA operation fetches chunk c of all the panel's strips
                    mbar_expect_tx(&pk_full[ps], kTcPackBytes);
                    tma_load_2d(pk_ring + ps * kTcPackBytes, &w_map, c * (kTcChunkBytes / 8), it.panel * 8, &pk_full[ps]);
                    if (++ps == kTcPackStages) {
                        ps = 0;
                        ++round;
                    }
                }
            }
            ring_wait_landed(pk_full, kTcPackStages, ps, round);
        }
    } else if (warp == 2) {
        // ------------------------------------------ producer of activation tiles
        if (elect_one()) {
            uint32_t s = 0, round = 0;
            const uint32_t bytes = p.tile_rows * 128;
            pdl_wait();   // activations come from the previous kernel in the stream
            for (int item = blockIdx.x; item < items && !*abort_flag; item += gridDim.x) {
                const TcItem it = tc_decode(p, item);
                for (int kt = 2 * it.c0; kt < 2 * it.c1; ++kt) {
                    if (round > 0 && !mbar_wait_suspended(&b_empty[s], (round - 1) & 1)) {
                        atomicExch(p.fault, 12);
                        *abort_flag = 1;
                        break;
                    }
                    mbar_expect_tx(&b_full[s], bytes);
                    tma_load_2d(b_ring + s * bytes, &x_map, kt * 64, it.tt * p.tile_rows, &b_full[s]);
                    if (++s == kTcBStages) s = 0, ++round;
                }
            }
            ring_wait_landed(b_full, kTcBStages, s, round);
        }
    } else if (warp == 1) {
        // ----------------------------------------------------------- MMA issuer
        if (elect_one()) {
            uint32_t s = 0, a_phase = 0, sb = 0, b_phase = 0, it_n = 0;
            bool good = true;
            // UMMA M = 128 weight rows (TMEM lanes), N = the tile's batch rows (TMEM columns)
            const uint32_t idesc = umma_idesc_f16(1, 128, p.tile_rows);
            const uint32_t b0 = umma_desc_lo(smem_u32(b_ring));
            for (int item = blockIdx.x; item < items && good; item += gridDim.x, ++it_n) {
                const uint32_t buf = it_n & 1;
                if (it_n >= 2 && !mbar_wait_suspended(&acc_empty[buf], ((it_n >> 1) - 1) & 1)) {
                    atomicExch(p.fault, 13);
                    good = false;
                    break;
                }
                tc_fence_after();
                const TcItem it = tc_decode(p, item);
                const int ktiles = 2 * (it.c1 - it.c0);
                const uint32_t d = tmem_base + buf * kTcMaxRows;
                for (int kt = 0; kt < ktiles; ++kt) {
                    if (!mbar_wait_suspended(&b_full[sb], b_phase) || !mbar_wait_suspended(&a_full[s], a_phase)) {
                        atomicExch(p.fault, 14);
                        good = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a = tmem_base + p.col_a + s * kTcACols, b = b0 + sb * (p.tile_rows * 128 >> 4);
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16) umma_f16_ts(d, a + k16 * 8, b + k16 * 2, idesc, kt > 0 || k16 > 0);
                    umma_commit(&a_empty[s]);    // stages reusable once these MMAs have read them
                    umma_commit(&b_empty[sb]);
                    if (++s == kTcAStages) s = 0, a_phase ^= 1;
                    if (++sb == kTcBStages) sb = 0, b_phase ^= 1;
                }
                if (good) umma_commit(&acc_full[buf]);
            }
            if (!good) *abort_flag = 1;
            // no MMA is in flight when the CTA gives its memory back, also after a wait that gave up
            umma_commit(drained);
            mbar_wait_suspended(drained, 0);
        }
    } else if (warp >= kTcFirstDequant && warp < kTcFirstEpilogue) {
        // -------------------------------------------------------------- dequant
        // A group of four warps expands every kGroups-th 64 columns (half of every chunk or of every other chunk) into A tile
        // 2 (chunk % 2) + half.  Warp w writes the 32-lane quarter w % 4 (the only one it may), lane = weight row: two strips of
        // 16 rows per warp.  Rows r and r + 8 of a strip share their 16-byte units (words x, z and y, w), which their two lanes
        // read together.
        const int quarter = warp & 3, group = (warp - kTcFirstDequant) >> 2, half = group & 1;
        const int strip = 2 * quarter + (lane >> 4), r = lane & 15, g = ((r & 3) << 1) | ((r >> 2) & 1);   // row_of_g(g) == r & 7
        const bool upper = r >= 8;
        const uint8_t* units = pk_ring + strip * kTcChunkBytes + half * 512 + g * 64;
        const uint8_t* scales = pk_ring + strip * kTcChunkBytes + 1024 + g * 4 + (upper ? 2 : 0);
        const uint32_t a_tiles = tmem_base + (uint32_t(quarter * 32) << 16) + p.col_a;
        uint32_t n = 0;   // chunks that have gone by
        bool good = true;
        for (int item = blockIdx.x; item < items && good; item += gridDim.x) {
            const TcItem it = tc_decode(p, item);
            for (int c = it.c0; c < it.c1; ++c, ++n) {
                if (kGroups == 4 && int(n & 1) != group >> 1) continue;
                const uint32_t tile = 2 * (n & 1) + half;
                const uint32_t ps = n % kTcPackStages;
                good = mbar_wait_warp(&pk_full[ps], (n / kTcPackStages) & 1, abort_flag);
                if (!good) {
                    atomicCAS(p.fault, 0, 15);
                    break;
                }
                uint32_t w[8];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const uint4 u = *reinterpret_cast<const uint4*>(units + ps * kTcPackBytes + t * 16);
                    w[t] = upper ? u.y : u.x;
                    w[4 + t] = upper ? u.w : u.z;
                }
                const uint32_t sw = *reinterpret_cast<const uint16_t*>(scales + ps * kTcPackBytes);
                uint4 v[8];
                if (p.scale_dtype == GARNET_B200_BF16) {
#pragma unroll
                    for (int t = 0; t < 8; ++t) v[t] = int4_word_to_bf16x8(w[t], sw * 0x10001u);
                } else {
                    const float f = __half2float(__ushort_as_half(uint16_t(sw)));
#pragma unroll
                    for (int t = 0; t < 8; ++t) v[t] = int4_word_to_bf16x8_f32(w[t], f);
                }
                good = n < 2 || mbar_wait_warp(&a_empty[tile], ((n >> 1) - 1) & 1, abort_flag);
                if (!good) {
                    atomicCAS(p.fault, 0, 16);
                    break;
                }
                tc_fence_after();
                tc_st_32x32(a_tiles + tile * kTcACols, v);
                tc_fence_before();
                __syncwarp();
                // The packed stage is given back only here, where the loaded values have been used: right after the loads the
                // arrival can overtake them in the shared-memory queue, and the next TMA then overwrites what they read.
                if (lane == 0) mbar_arrive(&pk_empty[ps]), mbar_arrive(&a_full[tile]);
            }
        }
    } else if (warp >= kTcFirstEpilogue) {
        // ------------------------------------------------------------- epilogue
        const int quarter = warp & 3;   // TMEM lanes 32*quarter .. +31 belong to this warp
        const bool wide = (p.ldy & 1) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 3) == 0, odd = lane & 1;
        uint32_t it_n = 0;
        for (int item = blockIdx.x; item < items; item += gridDim.x, ++it_n) {
            const TcItem it = tc_decode(p, item);
            const uint32_t buf = it_n & 1;
            if (!mbar_wait_warp(&acc_full[buf], (it_n >> 1) & 1, abort_flag)) {
                atomicCAS(p.fault, 0, 17);
                break;
            }
            tc_fence_after();
            if (it_n == 0) pdl_wait();   // y may still be read by the previous kernel in the stream
            // TMEM lane = weight row of the panel, column = batch row of the tile
            const int row0 = it.tt * p.tile_rows, rows = min(p.tile_rows, p.m - row0), n = it.panel * 128 + quarter * 32 + lane;
            const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + buf * kTcMaxRows;
            for (int c0 = 0; c0 < rows; c0 += 16) {
                uint32_t v[16];
                tmem_ld_32x16(taddr + c0, v);
                tmem_ld_wait();
                if (p.kslices > 1) {
                    float* part = reinterpret_cast<float*>(b_ring) + size_t(c0) * 128 + quarter * 32 + lane;
#pragma unroll
                    for (int j = 0; j < 16; ++j) part[j * 128] = __uint_as_float(v[j]);
                    continue;
                }
                // neighbouring lanes hold neighbouring outputs of a row: each finishes one row of a pair of rows
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const float other = __uint_as_float(__shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1));
                    const float mine = __uint_as_float(odd ? v[j + 1] : v[j]);
                    const int c = c0 + j + int(odd);
                    if (c < rows) tc_store_pair(p, row0 + c, n & ~1, odd ? other : mine, odd ? mine : other, wide);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncwarp();
    if (p.kslices > 1) {
        // One item per CTA; the cluster's CTAs hold the K slices of one tile.  The batch rows go round the CTAs, each of which
        // adds the slices of its rows in slice order.
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        const TcItem it = tc_decode(p, blockIdx.x);
        const int row0 = it.tt * p.tile_rows, rows = min(p.tile_rows, p.m - row0), rank = int(cluster.block_rank());
        const bool wide = (p.ldy & 1) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 3) == 0;
        const int pair = (threadIdx.x & 63) * 2;
        if (!*abort_flag) {
            pdl_wait();
            for (int c = rank + int(threadIdx.x >> 6) * p.kslices; c < rows; c += (kTcThreads / 64) * p.kslices) {
                float2 part[kTcMaxSlices], sum = make_float2(0.f, 0.f);
#pragma unroll
                for (int s = 0; s < kTcMaxSlices; ++s)
                    part[s] = s < p.kslices ? *reinterpret_cast<const float2*>(cluster.map_shared_rank(reinterpret_cast<float*>(b_ring), s) + size_t(c) * 128 + pair)
                                            : make_float2(0.f, 0.f);
#pragma unroll
                for (int s = 0; s < kTcMaxSlices; ++s)
                    if (s < p.kslices) sum.x += part[s].x, sum.y += part[s].y;
                tc_store_pair(p, row0 + c, it.panel * 128 + pair, sum.x, sum.y, wide);
            }
        }
        cluster.sync();   // peers may still read this CTA's partial tile
    }

    // ---- teardown: every role arrives here, also after a wait that gave up
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, p.tmem_cols);
    }
}

// ------------------------------------------------------------------ host side

// The size that garnet_b200_w4a16_workspace reports: the fp32 partial sums of the plan that once met in global memory.  Nothing
// uses such a workspace; the reported size is part of the interface.
size_t tc_workspace(const PackGeom& geo, int m)
{
    const int row_tiles = (m + 127) / 128, panels256 = (geo.strips_padded + 15) / 16;
    const int tiles = (panels256 * row_tiles >= 2 * kSmCount ? panels256 : geo.strips_padded / 8) * row_tiles;
    int want = tiles >= kSmCount ? 1 : (kSmCount + tiles - 1) / tiles;
    want = std::min(want, std::min(geo.chunks, 16));
    const size_t plane = size_t(m) * geo.rows * sizeof(float);
    want = int(std::max<size_t>(1, std::min<size_t>(size_t(want), (size_t(6) << 20) / std::max<size_t>(plane, 1))));
    const int per_slice = (geo.chunks + want - 1) / want, slices = (geo.chunks + per_slice - 1) / per_slice;
    return slices > 1 ? slices * plane : 0;
}

TensorMapEncodeFn tensor_map_encoder()
{
    static TensorMapEncodeFn fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            ptr = nullptr;
        return reinterpret_cast<TensorMapEncodeFn>(ptr);
    }();
    return fn;
}

int make_tensor_map_2d_16bit(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows)
{
    TensorMapEncodeFn enc = tensor_map_encoder();
    if (!enc) return fail(GARNET_B200_NOT_SUPPORTED, "cuTensorMapEncodeTiled is not available from this driver");
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GARNET_B200_CUDA_ERROR, "cuTensorMapEncodeTiled failed with code %d", int(r));
    return GARNET_B200_OK;
}

int make_tensor_map_2d_bytes(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes,
                             uint64_t stride_bytes, uint32_t box_bytes, uint32_t box_rows)
{
    TensorMapEncodeFn enc = tensor_map_encoder();
    if (!enc) return fail(GARNET_B200_NOT_SUPPORTED, "cuTensorMapEncodeTiled is not available from this driver");
    const cuuint64_t dims[2] = {row_bytes / 8, rows};
    const cuuint64_t strides[1] = {stride_bytes};
    const cuuint32_t box[2] = {box_bytes / 8, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GARNET_B200_CUDA_ERROR, "cuTensorMapEncodeTiled (bytes) failed with code %d", int(r));
    return GARNET_B200_OK;
}

int W4A16::init_tc()
{
    static_assert(sizeof(tc_packed_map) == sizeof(CUtensorMap), "tensor map storage size");
    if (int rc = make_tensor_map_2d_bytes(reinterpret_cast<CUtensorMap*>(&tc_packed_map), packed, uint64_t(geo.strips_padded),
                                          geo.strip_bytes(), geo.strip_bytes(), kTcChunkBytes, 8))
        return rc;
    GB_CUDA(cudaFuncSetAttribute(w4a16_tc_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcSmem::total(kTcMaxRows)));
    GB_CUDA(cudaFuncSetAttribute(w4a16_tc_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcSmem::total(kTcHalfRows)));
    return GARNET_B200_OK;
}

int W4A16::launch_tc(const __nv_bfloat16* x, __nv_bfloat16* y, int m, unsigned flags, cudaStream_t stream)
{
    const TcPlan plan = tc_plan(geo.strips_padded, geo.chunks, m);
    CUtensorMap map;
    if (int rc = make_tensor_map_2d_16bit(&map, x, uint64_t(m), uint64_t(geo.cols), uint32_t(plan.tile_rows))) return rc;
    TcParams p;
    p.y = y;
    p.fault = fault_dev;
    p.m = m;
    p.n = geo.rows;
    p.ldy = geo.rows;
    p.chunks = geo.chunks;
    p.panels = plan.panels;
    p.row_tiles = plan.row_tiles;
    p.tile_rows = plan.tile_rows;
    p.kslices = plan.kslices;
    p.scale_dtype = scale_dtype;
    const long long items = (long long)p.panels * p.row_tiles * p.kslices;
    const bool half = items <= kSmCount && p.tile_rows <= kTcHalfRows;
    p.tmem_cols = half ? 256 : 512;
    p.col_a = half ? kTcHalfRows : 2 * kTcMaxRows;
    cudaLaunchConfig_t cfg = {};
    // with K slices every CTA has one item (tc_plan keeps them below the SM count), else the CTAs are persistent
    cfg.gridDim = dim3(unsigned(std::min<long long>(items, kSmCount)));
    const auto kernel = half ? w4a16_tc_kernel<2> : w4a16_tc_kernel<4>;
    cfg.blockDim = dim3(half ? tc_threads(2) : tc_threads(4));
    cfg.dynamicSmemBytes = unsigned(TcSmem::total(p.tile_rows));
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int attrs = 0;
    if (p.kslices > 1) {
        attr[attrs].id = cudaLaunchAttributeClusterDimension;
        attr[attrs++].val.clusterDim = {unsigned(p.kslices), 1, 1};
    }
    if (flags & 1u) {
        attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = unsigned(attrs);
    GB_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, map, *reinterpret_cast<const CUtensorMap*>(&tc_packed_map)));
    return GARNET_B200_OK;
}

}  // namespace gb200
