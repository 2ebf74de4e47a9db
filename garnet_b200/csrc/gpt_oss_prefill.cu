// gpt-oss attention of many query rows (prefill, or any call that the one-token kernel does not take) on the tensor
// cores, for 64-wide heads: S = Q K^T and O += P V as tcgen05 MMAs over the paged bf16 cache, softmax in fp32 with the
// head's sink in the denominator only (the arithmetic of RunGptOssAttention, plugins/gpt_oss/cuda/gpt_oss_kernels.cu:125-160).
//
// A CTA owns one kv head and one or two tiles of 128 query rows; a tile's rows are (token, q head of the group), so the
// K and V rows that a tile stages serve all the q heads of the group, and a causal tile of 16 tokens x 8 heads ends
// within 16 positions of its last key.  Per 64 keys:
//   2 loader warps    look up the cache pages and copy 64 K and V rows of 128 bytes (cp.async) into the 128-byte-swizzled
//                     tile that serves as the K-major operand of Q K^T and as the MN-major operand of P V; a ring of 8,
//                     whose first 3 steps are requested before the queries are converted;
//   MMA warp          one thread: P V of these keys when their P is there, then Q K^T of the keys two steps on into the
//                     columns that P leaves, tile by tile: scores are ready before the softmax wants them;
//   2 x 4 softmax     one thread per query row: 64 scores into registers, running maximum (the sink is its first value),
//   warps             p = 2^(s c - m c), the row's sum in fp32, P over the scores in tensor memory; the P V of the step before
//                     is added to O, which stays in registers and is rescaled only when a row's maximum has grown by more than
//                     2^8 since the last time (the final division makes that exact; the conditional rescaling of
//                     FlashAttention-4).  The fp32 work runs two values per instruction (f32x2).
// Numerics: the queries are bf16-valued fp32, so Q K^T has exact products; the queries of a CTA that holds others enter as three
// bf16 numbers each.  P is fp32 and enters the MMA as three bf16 numbers, which hold eight of its 24 bits each.  The tensor core
// truncates what it accumulates, so a sum that stays in it loses about half a unit of its last place per MMA: each step starts a
// new one, smallest pieces first, and the steps are added in fp32.  Share of the results that are not the bf16 rounding of the
// float64 result, 2048 tokens / 64 tokens after 4000: 4.2e-4 / 8.5e-4 by the fp32 row loop, 2.7e-3 / 5.2e-3 with two pieces and O
// in tensor memory, 1.9e-3 / 6.8e-3 with three, 1.6e-4 / 2.0e-4 as it is now.  A row that comes out NaN (infinities in the cache
// meet a zero piece) is computed again by the row loop.
//
// Bound: per 128 x 64 scores the tensor pipe needs about 600 clocks (12 P V MMAs at 33, 4 Q K^T MMAs at 50) and the exponentials
// 512 (16 per clock and SM).  Neither is what it waits for: at 2048 tokens the tensor pipe is 23 % busy and the issue slots 44 %
// (ncu), and a warp spends its time on fixed latencies and on tensor memory and barriers: the chain of a tile's step (scores ->
// maximum -> exponentials -> pieces -> P V) with one other tile on the SM to hide it.
// 2048 tokens, 64 / 8 heads (events, append included): 131 us; 110 us with two pieces of P and O in tensor memory, whose sums
// were worse than the row loop's; pieces rounded instead of cut off 135 us, stored 32 keys at a time 141 us.
#include <algorithm>
#include <cfloat>

#include "gpt_oss_attn.cuh"
#include "tc_common.cuh"

namespace gb200 {

namespace {

constexpr int kPfRows = 128;          // query rows of a tile (UMMA M, one softmax thread each)
constexpr int kPfKeys = 64;           // keys of a step (UMMA N of Q K^T, K of P V)
constexpr int kPfStages = 8, kPfAhead = 3;
constexpr int kPfTileBytes = 128 * 128;          // a tile of queries
constexpr int kPfKvBytes = kPfKeys * 128;        // a step's K rows, and its V rows
// 8 softmax warps, MMA, 2 loaders: 11 warps leave a thread 168 registers, which the softmax needs (13 would leave 128)
constexpr int kPfMmaWarp = 8, kPfFirstLoader = 9, kPfLoaders = 2;
constexpr int kPfThreads = (kPfFirstLoader + kPfLoaders) * 32;
// Tensor memory of a tile: two sets of 64 scores (the first two pieces of P replace them), P V of a step, the third pieces of P.
constexpr uint32_t kPfColMid = 32, kPfColPv = 128, kPfColLow = 192, kPfCols = 256;

struct PfSmem {
    static constexpr int q = 0;                                    // [3 pieces][2 tiles]; the first piece alone when it says it all
    static constexpr int kv = q + 6 * kPfTileBytes;                // [stages] K tile, V tile
    static constexpr int ok = kv + kPfStages * 2 * kPfKvBytes;     // [stages][2] bits of the keys that exist
    static constexpr int bars = ok + kPfStages * 8;
    static constexpr int total = bars + 256 + 1024;                // barriers, and slack for 1024-byte alignment
};
static_assert(PfSmem::total <= 227 * 1024, "shared memory budget");

__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// The upper halves of two fp32 numbers: their first eight bits, as bf16.
__device__ __forceinline__ uint32_t upper_halves(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Two fp32 values per instruction.
__device__ __forceinline__ uint64_t f32x2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f32x2_split(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Bits [lo, hi) of a 32-bit word, for any lo and hi.
__device__ __forceinline__ uint32_t bit_range(int lo, int hi)
{
    lo = max(lo, 0), hi = min(hi, 32);
    if (lo >= hi) return 0u;
    return (hi == 32 ? 0xffffffffu : (1u << hi) - 1u) & ~((1u << lo) - 1u);
}

template <int qtiles>
__global__ void __launch_bounds__(kPfThreads, 1) oss_attention_prefill_kernel(const OssAttn p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_tiles = smem + PfSmem::q;
    uint8_t* kv_ring = smem + PfSmem::kv;
    uint32_t* ok_bits = reinterpret_cast<uint32_t*>(smem + PfSmem::ok);
    uint64_t* kv_full = reinterpret_cast<uint64_t*>(smem + PfSmem::bars);   // [stages]
    uint64_t* kv_empty = kv_full + kPfStages;                               // [stages]
    uint64_t* s_full = kv_empty + kPfStages;                                // [2 tiles][2 sets] scores written
    uint64_t* p_full = s_full + 4;                                          // [2 tiles][2 sets] P written
    uint64_t* pv_full = p_full + 4;                                         // [2 tiles] P V of a step done
    uint64_t* drained = pv_full + 2;                                        // every MMA done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int kv = blockIdx.x, b = blockIdx.z, group = p.q_heads / p.kv_heads;
    const int tile_tokens = kPfRows / group;   // the launch makes sure of group <= 128
    // the tiles with the most keys first, so that the short ones fill the gaps at the end
    const int t0 = int(gridDim.y - 1 - blockIdx.y) * tile_tokens * qtiles, t1 = min(p.tokens, t0 + tile_tokens * qtiles);
    const int tiles = t0 + tile_tokens < t1 ? qtiles : 1;   // the last block of a sequence may have rows for one tile only
    const int limit = p.logical_pages * p.page_size;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPfStages; ++s) {
            mbar_init(&kv_full[s], kPfLoaders);
            mbar_init(&kv_empty[s], 1);
        }
        for (int s = 0; s < 4; ++s) {
            mbar_init(&s_full[s], 1);
            mbar_init(&p_full[s], 4);
            if (s < 2) mbar_init(&pv_full[s], 1);
        }
        mbar_init(drained, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    const uint32_t tmem_cols = kPfCols * qtiles;
    if (warp == kPfMmaWarp) {
        tmem_alloc(tmem_slot, tmem_cols);
        tmem_relinquish();
    }
    pdl_wait();   // the cache rows and the queries come from the kernels before this one

    // keys that some row of the CTA sees
    const int start = p.starts[b];
    const bool active = p.active[b] != 0;
    int first_end, last_end;
    if (p.prefill) first_end = max(1, start + t0 + 1), last_end = min(limit, start + t1);
    else first_end = last_end = p.lengths[b];
    if (!active || first_end <= 0 || last_end > limit || first_end > last_end) first_end = last_end = 0;
    const int key0 = p.window ? max(0, first_end - p.window) : 0, key1 = last_end;
    const int steps = (key1 - key0 + kPfKeys - 1) / kPfKeys;

    // ---- loaders: the row of a key (one per lane), and the copies of a step
    const int lw = warp - kPfFirstLoader;
    const auto look_up = [&](int j) -> unsigned long long {
        const int pos = key0 + j * kPfKeys + lw * 32 + lane;
        return pos < key1 ? oss_cache_offset(p, b, pos, kv) : SIZE_MAX;
    };
    const auto request = [&](int j, unsigned long long off) {
        if (j < steps) {
            const int st = j % kPfStages, piece = lane & 7;
            const uint32_t exists = __ballot_sync(0xffffffffu, off != SIZE_MAX);
            if (lane == 0) ok_bits[st * 2 + lw] = exists;
            const uint32_t kt = smem_u32(kv_ring + st * 2 * kPfKvBytes) + lw * 32 * 128, vt = kt + kPfKvBytes;
#pragma unroll
            for (int it = 0; it < 8; ++it) {
                const int row = it * 4 + (lane >> 3);
                const unsigned long long o = __shfl_sync(0xffffffffu, off, row);
                const bool valid = o != SIZE_MAX;   // rows that do not exist are filled with zeros
                const size_t at = (valid ? o : 0) + piece * 8;
                const uint32_t to = row * 128 + ((piece ^ (row & 7)) << 4);
                cp_async16(kt + to, p.keys + at, valid);
                cp_async16(vt + to, p.values + at, valid);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // ---- queries: 8 values of a row (zeros where there is none), and their place in a tile
    const auto load_queries = [&](int i, float (&f)[8]) {
        const int row = i >> 3, r = row & (kPfRows - 1), in_tile = r / group, t = t0 + (row >> 7) * tile_tokens + in_tile;
        float4 f0 = make_float4(0.f, 0.f, 0.f, 0.f), f1 = f0;
        if (steps && in_tile < tile_tokens && t < t1) {
            const size_t packed = size_t(p.q_heads + 2 * p.kv_heads) * kOssDim;
            const float4* src = reinterpret_cast<const float4*>(p.qkv + (size_t(b) * p.tokens + t) * packed + (kv * group + r % group) * kOssDim + (i & 7) * 8);
            f0 = __ldg(src), f1 = __ldg(src + 1);
        }
        f[0] = f0.x, f[1] = f0.y, f[2] = f0.z, f[3] = f0.w, f[4] = f1.x, f[5] = f1.y, f[6] = f1.z, f[7] = f1.w;
    };
    const auto store_queries = [&](int i, int piece, const float (&f)[8]) {
        const int row = i >> 3;
        *reinterpret_cast<uint4*>(q_tiles + piece * 2 * kPfTileBytes + row * 128 + (((i & 7) ^ (row & 7)) << 4)) =
            make_uint4(bf16x2_of(f[0], f[1]), bf16x2_of(f[2], f[3]), bf16x2_of(f[4], f[5]), bf16x2_of(f[6], f[7]));
    };
    unsigned long long ahead = SIZE_MAX;   // rows of the next step to request
    int inexact = 0;
    if (warp >= kPfFirstLoader) {
        const unsigned long long first[kPfAhead] = {look_up(0), look_up(1), look_up(2)};
#pragma unroll
        for (int j = 0; j < kPfAhead; ++j) request(j, first[j]);
        ahead = look_up(kPfAhead);
    } else {
        // ---- queries: fp32 to bf16, 128-byte-swizzled K-major tiles
#pragma unroll 4
        for (int i = threadIdx.x; i < qtiles * kPfRows * 8; i += kPfFirstLoader * 32) {
            float f[8];
            load_queries(i, f);
#pragma unroll
            for (int j = 0; j < 8; ++j) inexact |= int(__float_as_uint(f[j]) & 0xffffu);
            store_queries(i, 0, f);
        }
        fence_proxy_async_smem();
    }
    tc_fence_before();
    const int q_pieces = __syncthreads_or(inexact) ? 3 : 1;
    if (q_pieces > 1) {
        // some query is not a bf16 value: the second and third pieces of them all
        if (warp < kPfFirstLoader) {
            for (int i = threadIdx.x; i < qtiles * kPfRows * 8; i += kPfFirstLoader * 32) {
                float f[8];
                load_queries(i, f);
#pragma unroll
                for (int piece = 1; piece < 3; ++piece) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) f[j] -= bf16_round_f(f[j]);
                    store_queries(i, piece, f);
                }
            }
            fence_proxy_async_smem();
        }
        __syncthreads();
    }
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    if (steps == 0) {
        // no visible key
        const int rows = (t1 - t0) * group;
        for (int i = warp; i < rows; i += kPfThreads / 32)
            oss_attention_row(p, b * p.tokens + t0 + i / group, kv * group + i % group, lane);
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (warp == kPfMmaWarp) tmem_dealloc(tmem_base, tmem_cols);
        return;
    }

    if (warp >= kPfFirstLoader) {
        // -------------------------------------------------------------- loaders
        // a step is announced as soon as it is there, before the wait for the stage of the next request
        for (int j = 0; j < steps; ++j) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kPfAhead - 1) : "memory");
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&kv_full[j % kPfStages]);
            const int next = j + kPfAhead;
            if (next >= kPfStages && next < steps && !mbar_wait_warp(&kv_empty[next % kPfStages], ((next / kPfStages) - 1) & 1, abort_flag)) break;
            request(next, ahead);
            ahead = look_up(next + 1);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == kPfMmaWarp) {
        // ----------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc_qk = umma_idesc_f16(1, kPfRows, kPfKeys);
            constexpr uint32_t idesc_pv = umma_idesc_f16(1, kPfRows, kOssDim) | (1u << 16);   // V: MN-major
            const uint32_t q_lo = umma_desc_lo(smem_u32(q_tiles)), k_lo = umma_desc_lo(smem_u32(kv_ring)), v_lo = umma_desc_lo(smem_u32(kv_ring + kPfKvBytes));
            constexpr uint32_t kStage = 2 * kPfKvBytes >> 4;
            // scores of step j of tile q, into set j & 1
            const auto scores = [&](int j, int q) {
                const uint32_t d = tmem_base + q * kPfCols + (j & 1) * kPfKeys;
                const uint32_t a = q_lo + q * (kPfTileBytes >> 4), k = k_lo + (j % kPfStages) * kStage;
#pragma unroll 1
                for (int piece = q_pieces - 1; piece >= 0; --piece) {
#pragma unroll
                    for (int k16 = 0; k16 < kOssDim / 16; ++k16)
                        umma_f16_ss(d, a + piece * (2 * kPfTileBytes >> 4) + k16 * 2, k + k16 * 2, idesc_qk, piece + 1 < q_pieces || k16 > 0);
                }
                umma_commit(&s_full[q * 2 + (j & 1)]);
            };
            bool good = true;
            for (int j = 0; j < 2 && j < steps && good; ++j) {
                good = mbar_wait_suspended(&kv_full[j], 0);
                tc_fence_after();
#pragma unroll
                for (int q = 0; q < qtiles; ++q)
                    if (q < tiles) scores(j, q);
            }
            for (int j = 0; j < steps && good; ++j) {
                const uint32_t v = v_lo + (j % kPfStages) * kStage;
#pragma unroll
                for (int q = 0; q < qtiles; ++q) {
                    if (q >= tiles) break;
                    good = good && mbar_wait_suspended(&p_full[q * 2 + (j & 1)], (j >> 1) & 1);
                    if (good && q == 0 && j + 2 < steps) good = mbar_wait_suspended(&kv_full[(j + 2) % kPfStages], ((j + 2) / kPfStages) & 1);
                    if (!good) break;
                    tc_fence_after();
                    const uint32_t tile = tmem_base + q * kPfCols, set = (j & 1) * kPfKeys;
                    const uint32_t pieces[3] = {tile + kPfColLow + set / 2, tile + set + kPfColMid, tile + set};
#pragma unroll
                    for (int piece = 0; piece < 3; ++piece)
#pragma unroll
                        for (int k16 = 0; k16 < kPfKeys / 16; ++k16)
                            umma_f16_ts(tile + kPfColPv, pieces[piece] + k16 * 8, v + k16 * (2048 >> 4), idesc_pv, piece > 0 || k16 > 0);
                    umma_commit(&pv_full[q]);
                    if (j + 2 < steps) scores(j + 2, q);
                }
                umma_commit(&kv_empty[j % kPfStages]);
            }
            if (!good) *abort_flag = 1;
            // no MMA is in flight when the CTA gives its memory back, also after a wait that gave up
            umma_commit(drained);
            mbar_wait_suspended(drained, 0);
        }
        __syncwarp();
    } else if ((warp >> 2) < tiles) {
        // -------------------------------------------------------------- softmax
        const int q = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t tm = tmem_base + q * kPfCols + (uint32_t((warp & 3) * 32) << 16);
        const int in_tile = r / group, t = t0 + q * tile_tokens + in_tile, head = kv * group + r % group;
        const bool mine = in_tile < tile_tokens && t < t1;
        int end = p.prefill ? start + t + 1 : p.lengths[b];
        int begin = p.window ? max(0, end - p.window) : 0;
        if (!mine || end <= 0 || end > limit) begin = end = 0;
        constexpr float kLog2e = 1.4426950408889634f;
        const float c = 0.125f * kLog2e;                       // 1 / sqrt(64), in powers of two
        float ref = mine ? p.sinks[head] * kLog2e : 0.f;       // what the exponents are taken against
        float sum = 1.f;                                       // the sink's own term
        uint64_t o2[kOssDim / 2];                              // O, two values each
#pragma unroll
        for (int i = 0; i < kOssDim / 2; ++i) o2[i] = 0;
        // adds P V of step j
        const auto add_pv = [&](int j) -> bool {
            if (!mbar_wait_warp(&pv_full[q], j & 1, abort_flag)) return false;
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t pv[32];
                tmem_ld_32x32(tm + kPfColPv + 32 * h, pv);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    o2[16 * h + i] = add2(o2[16 * h + i], f32x2(__uint_as_float(pv[2 * i]), __uint_as_float(pv[2 * i + 1])));
            }
            return true;
        };
        bool good = true;
        for (int j = 0; j < steps; ++j) {
            const int st = j % kPfStages, kb = key0 + j * kPfKeys;
            const uint32_t ts = tm + (j & 1) * kPfKeys;
            good = mbar_wait_warp(&kv_full[st], (j / kPfStages) & 1, abort_flag) && mbar_wait_warp(&s_full[q * 2 + (j & 1)], (j >> 1) & 1, abort_flag);
            if (!good) break;
            tc_fence_after();
            uint32_t s[2][32];
            tmem_ld_32x32(ts, s[0]);
            tmem_ld_32x32(ts + 32, s[1]);
            const uint32_t there[2] = {ok_bits[st * 2], ok_bits[st * 2 + 1]};
            tmem_ld_wait();
            if (!__all_sync(0xffffffffu, begin <= kb && end >= kb + kPfKeys && (there[0] & there[1]) == 0xffffffffu)) {
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const uint32_t vis = there[w] & bit_range(begin - kb - 32 * w, end - kb - 32 * w);
#pragma unroll
                    for (int i = 0; i < 32; ++i) s[w][i] = (vis >> i) & 1 ? s[w][i] : 0xff800000u;   // -inf
                }
            }
            float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 32; ++i) m[i & 3] = max3(m[i & 3], __uint_as_float(s[0][i]), __uint_as_float(s[1][i]));
            const float top = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])) * c;
            const bool grow = j == 0 ? top > ref : top > ref + 8.f;
            const bool rescale = __any_sync(0xffffffffu, grow);
            const float f = grow ? ex2(ref - top) : 1.f;
            if (grow) ref = top;
            sum *= f;
            const float base = ref == -INFINITY ? 0.f : ref;
            const uint64_t scale2 = f32x2(c, c), base2 = f32x2(-base, -base), minus1 = f32x2(-1.f, -1.f);
            uint64_t part2[2] = {0, 0};
#pragma unroll
            for (int w = 0; w < 4; ++w) {   // 16 keys at a time
                uint64_t e2[8];
                uint32_t b[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t* two = s[w >> 1] + (w & 1) * 16 + 2 * i;
                    float a, d;
                    f32x2_split(fma2(f32x2(__uint_as_float(two[0]), __uint_as_float(two[1])), scale2, base2), a, d);
                    a = ex2(a), d = ex2(d);
                    e2[i] = f32x2(a, d);
                    part2[i & 1] = add2(part2[i & 1], e2[i]);
                    b[i] = upper_halves(a, d);
                }
                tmem_st_32x8(ts + 8 * w, b);
#pragma unroll
                for (int piece = 1; piece < 3; ++piece) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        float a, d;
                        f32x2_split(e2[i], a, d);
                        e2[i] = fma2(f32x2(__uint_as_float(__float_as_uint(a) & 0xffff0000u), __uint_as_float(__float_as_uint(d) & 0xffff0000u)), minus1, e2[i]);
                        f32x2_split(e2[i], a, d);
                        b[i] = upper_halves(a, d);
                    }
                    tmem_st_32x8(piece == 1 ? ts + kPfColMid + 8 * w : tm + kPfColLow + (j & 1) * (kPfKeys / 2) + 8 * w, b);
                }
            }
            float part[2];
            f32x2_split(add2(part2[0], part2[1]), part[0], part[1]);
            sum += part[0] + part[1];
            good = j == 0 || add_pv(j - 1);   // before this step's P V takes its place
            if (!good) break;
            if (rescale) {
                const uint64_t f2 = f32x2(f, f);
#pragma unroll
                for (int i = 0; i < kOssDim / 2; ++i) o2[i] = mul2(o2[i], f2);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[q * 2 + (j & 1)]);
        }
        good = good && add_pv(steps - 1);
        // a wait that gave up leaves NaNs, which no caller can take for a result
        if (!good) sum = NAN;
        float* out = p.out + (size_t(b) * p.tokens + t) * p.q_heads * kOssDim + head * kOssDim;
        bool bad = mine && ref == INFINITY;   // an infinite sink: the row loop says what comes of it
        if (mine) {
#pragma unroll
            for (int i = 0; i < kOssDim / 4; ++i) {
                float v[4];
                f32x2_split(o2[2 * i], v[0], v[1]);
                f32x2_split(o2[2 * i + 1], v[2], v[3]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    v[e] = end > begin ? bf16_round_f(v[e] / sum) : 0.f;
                    bad = bad || isnan(v[e]);
                }
                *reinterpret_cast<float4*>(out + 4 * i) = make_float4(v[0], v[1], v[2], v[3]);
            }
        }
        __syncwarp();
        for (uint32_t redo = __ballot_sync(0xffffffffu, bad && good); redo; redo &= redo - 1) {
            const int from = __ffs(redo) - 1;
            oss_attention_row(p, __shfl_sync(0xffffffffu, b * p.tokens + t, from), __shfl_sync(0xffffffffu, head, from), lane);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kPfMmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem_base, tmem_cols);
    }
}

}  // namespace

bool oss_prefill_takes(const OssAttn& p)
{
    const uintptr_t bits = reinterpret_cast<uintptr_t>(p.keys) | reinterpret_cast<uintptr_t>(p.values) |
                           reinterpret_cast<uintptr_t>(p.qkv) | reinterpret_cast<uintptr_t>(p.out);
    const int group = p.q_heads / p.kv_heads;
    return p.head_dim == kOssDim && group <= kPfRows && (bits & 15) == 0 && p.batch <= 65535 && p.tokens / (kPfRows / group) < 65535;
}

int oss_prefill_launch(const OssAttn& p, cudaStream_t stream)
{
    const int tile_tokens = kPfRows / (p.q_heads / p.kv_heads);
    const int qtiles = oss_prefill_tiles(p.batch, p.kv_heads, p.tokens, tile_tokens);
    const auto kernel = qtiles == 2 ? oss_attention_prefill_kernel<2> : oss_attention_prefill_kernel<1>;
    GB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PfSmem::total));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(p.kv_heads), unsigned((p.tokens + tile_tokens * qtiles - 1) / (tile_tokens * qtiles)), unsigned(p.batch));
    cfg.blockDim = dim3(kPfThreads);
    cfg.dynamicSmemBytes = PfSmem::total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GB_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    return GARNET_B200_OK;
}

}  // namespace gb200
