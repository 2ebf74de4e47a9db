// gpt-oss attention of many query rows (prefill, or any call that the one-token kernel does not take) on the tensor
// cores, for 64-wide heads: S = Q K^T and O += P V as tcgen05 MMAs over the paged bf16 cache, softmax in fp32 with the
// head's sink in the denominator only (the arithmetic of RunGptOssAttention, plugins/gpt_oss/cuda/gpt_oss_kernels.cu:125-160).
//
// A CTA owns one kv head and one or two tiles of 128 query rows; a tile's rows are (token, q head of the group), so the
// K and V rows that a tile stages serve all the q heads of the group, and a causal tile of 16 tokens x 8 heads ends
// within 16 positions of its last key.  Per 128 keys:
//   4 loader warps    look up the cache pages and copy 128 K and V rows of 128 bytes (cp.async) into the 128-byte-swizzled
//                     tile that serves as the K-major operand of Q K^T and as the MN-major operand of P V; a ring of 3;
//   MMA warp          one thread: P V of the previous keys, then Q K^T of these, tile by tile, so that one tile's MMAs
//                     run under the other tile's softmax;
//   2 x 4 softmax     one thread per query row: running maximum (the sink is its first value), p = 2^(s c - m c), the
//   warps             row's sum in fp32, P back into tensor memory; O in tensor memory is rescaled only when a row's
//                     maximum has grown by more than 2^8 since the last time (the final division makes that exact).
// Numerics: the queries are bf16-valued fp32 (a tile that holds others takes the fp32 row loop instead), so Q K^T has exact
// products.  P is fp32: it enters the MMA as two bf16 numbers, hi = bf16(p) and lo = bf16(p - hi), which leaves at most
// 2^-18 p - less than the rounding errors of an fp32 sum over some hundreds of positions, and 2^-9 of the step of the
// bf16 result.
//
// Bound: 16 exponentials per clock and SM, 1024 clocks per tile of 128 x 128 scores, against 768 clocks of MMAs (hi and lo).
#include <algorithm>
#include <cfloat>

#include "gpt_oss_attn.cuh"
#include "mx_common.cuh"
#include "tc_common.cuh"

namespace gb200 {

namespace {

constexpr int kPfRows = 128;          // query rows of a tile (UMMA M, one softmax thread each)
constexpr int kPfKeys = 128;          // keys of a step (UMMA N of Q K^T, K of P V)
constexpr int kPfStages = 3;
constexpr int kPfTileBytes = 128 * 128;
constexpr int kPfMmaWarp = 8, kPfFirstLoader = 9, kPfLoaders = 4;
constexpr int kPfThreads = (kPfFirstLoader + kPfLoaders) * 32;
// Tensor memory of a tile: scores (the hi half of P replaces them), the lo half of P, the output.
constexpr uint32_t kPfColLo = 128, kPfColO = 192, kPfCols = 256;

struct PfSmem {
    static constexpr int q = 0;                                    // [2] tiles
    static constexpr int kv = q + 2 * kPfTileBytes;                // [stages] K tile, V tile
    static constexpr int ok = kv + kPfStages * 2 * kPfTileBytes;   // [stages][4] bits of the keys that exist
    static constexpr int bars = ok + kPfStages * 16;
    static constexpr int total = bars + 128 + 1024;                // barriers, and slack for 1024-byte alignment
};

__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// D[tmem] (+)= A[tmem] * B[smem]; issued by one thread.
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(uint32_t(accumulate))
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Bits [lo, hi) of a 32-bit word, for any lo and hi.
__device__ __forceinline__ uint32_t bit_range(int lo, int hi)
{
    lo = max(lo, 0), hi = min(hi, 32);
    if (lo >= hi) return 0u;
    return (hi == 32 ? 0xffffffffu : (1u << hi) - 1u) & ~((1u << lo) - 1u);
}

__global__ void __launch_bounds__(kPfThreads, 1) oss_attention_prefill_kernel(const OssAttn p, const int qtiles)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_tiles = smem + PfSmem::q;
    uint8_t* kv_ring = smem + PfSmem::kv;
    uint32_t* ok_bits = reinterpret_cast<uint32_t*>(smem + PfSmem::ok);
    uint64_t* kv_full = reinterpret_cast<uint64_t*>(smem + PfSmem::bars);   // [stages]
    uint64_t* kv_empty = kv_full + kPfStages;                               // [stages]
    uint64_t* s_full = kv_empty + kPfStages;                                // [2] scores written (and the P V before them done)
    uint64_t* p_full = s_full + 2;                                          // [2] P written
    uint64_t* o_full = p_full + 2;                                          // [2] last P V done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kv = blockIdx.x, b = blockIdx.z, group = p.q_heads / p.kv_heads;
    const int tile_tokens = kPfRows / group;   // the launch makes sure of group <= 128
    // the tiles with the most keys first, so that the short ones fill the gaps at the end
    const int t0 = int(gridDim.y - 1 - blockIdx.y) * tile_tokens * qtiles, t1 = min(p.tokens, t0 + tile_tokens * qtiles);
    const int limit = p.logical_pages * p.page_size;
    const int start = p.starts[b];
    const bool active = p.active[b] != 0;

    // keys that some row of the CTA sees
    int first_end, last_end;
    if (p.prefill) first_end = max(1, start + t0 + 1), last_end = min(limit, start + t1);
    else first_end = last_end = p.lengths[b];
    if (!active || first_end <= 0 || last_end > limit || first_end > last_end) first_end = last_end = 0;
    const int key0 = p.window ? max(0, first_end - p.window) : 0, key1 = last_end;
    const int steps = (key1 - key0 + kPfKeys - 1) / kPfKeys;

    // ---- queries: fp32 to bf16, 128-byte-swizzled K-major tiles
    const int packed = (p.q_heads + 2 * p.kv_heads) * kOssDim;
    int inexact = 0;
    for (int i = threadIdx.x; i < qtiles * kPfRows * 8; i += kPfThreads) {
        const int row = i >> 3, piece = i & 7, r = row & (kPfRows - 1), in_tile = r / group;
        const int t = t0 + (row >> 7) * tile_tokens + in_tile, head = kv * group + r % group;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (steps && in_tile < tile_tokens && t < t1) {
            const float4* src = reinterpret_cast<const float4*>(p.qkv + (size_t(b) * p.tokens + t) * packed + head * kOssDim + piece * 8);
            const float4 f0 = __ldg(src), f1 = __ldg(src + 1);
            const float f[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) inexact |= int(__float_as_uint(f[j]) & 0xffffu);
            v = make_uint4(bf16x2_of(f0.x, f0.y), bf16x2_of(f0.z, f0.w), bf16x2_of(f1.x, f1.y), bf16x2_of(f1.z, f1.w));
        }
        *reinterpret_cast<uint4*>(q_tiles + row * 128 + ((piece ^ (row & 7)) << 4)) = v;
    }
    fence_proxy_async_smem();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kPfStages; ++s) {
            mbar_init(&kv_full[s], kPfLoaders);
            mbar_init(&kv_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&s_full[s], 1);
            mbar_init(&p_full[s], 4);
            mbar_init(&o_full[s], 1);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (__syncthreads_or(inexact) || steps == 0) {
        // queries that are not bf16 values (outside the operand's contract), or no visible key at all
        const int rows = (t1 - t0) * group;
        for (int i = warp; i < rows; i += kPfThreads / 32)
            oss_attention_row(p, b * p.tokens + t0 + i / group, kv * group + i % group, lane);
        return;
    }
    const uint32_t tmem_cols = kPfCols * qtiles;
    if (warp == kPfMmaWarp) {
        tmem_alloc(tmem_slot, tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp >= kPfFirstLoader) {
        // -------------------------------------------------------------- loaders
        const int lw = warp - kPfFirstLoader;
        for (int j = 0; j < steps && !*abort_flag; ++j) {
            const int st = j % kPfStages;
            if (j >= kPfStages && !mbar_wait_bounded(&kv_empty[st], ((j / kPfStages) - 1) & 1)) {
                *abort_flag = 1;
                break;
            }
            const int pos = key0 + j * kPfKeys + lw * 32 + lane;
            const size_t off = pos < key1 ? oss_cache_offset(p, b, pos, kv) : SIZE_MAX;
            const uint32_t exists = __ballot_sync(0xffffffffu, off != SIZE_MAX);
            if (lane == 0) ok_bits[st * 4 + lw] = exists;
            const uint32_t kt = smem_u32(kv_ring + st * 2 * kPfTileBytes) + lw * 32 * 128, vt = kt + kPfTileBytes;
            const int piece = lane & 7;
#pragma unroll
            for (int it = 0; it < 8; ++it) {
                const int row = it * 4 + (lane >> 3);
                const unsigned long long o = __shfl_sync(0xffffffffu, static_cast<unsigned long long>(off), row);
                const bool valid = o != SIZE_MAX;   // rows that do not exist are filled with zeros
                const size_t at = (valid ? o : 0) + piece * 8;
                const uint32_t to = row * 128 + ((piece ^ (row & 7)) << 4);
                cp_async16(kt + to, p.keys + at, valid);
                cp_async16(vt + to, p.values + at, valid);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (j > 0) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&kv_full[(j - 1) % kPfStages]);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && !*abort_flag) mbar_arrive(&kv_full[(steps - 1) % kPfStages]);
    } else if (warp == kPfMmaWarp) {
        // ----------------------------------------------------------- MMA issuer
        if (lane == 0) {
            const uint32_t idesc_qk = umma_idesc_f16(1, kPfRows, kPfKeys);
            const uint32_t idesc_pv = umma_idesc_f16(1, kPfRows, kOssDim) | (1u << 16);   // V: MN-major
            for (int j = 0; j <= steps && !*abort_flag; ++j) {
                const int st = j % kPfStages;
                if (j < steps && !mbar_wait_bounded(&kv_full[st], (j / kPfStages) & 1)) {
                    *abort_flag = 1;
                    break;
                }
                for (int q = 0; q < qtiles; ++q) {
                    const uint32_t tm = tmem_base + q * kPfCols;
                    if (j > 0) {
                        if (!mbar_wait_bounded(&p_full[q], (j - 1) & 1)) {
                            *abort_flag = 1;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t v_addr = smem_u32(kv_ring + ((j - 1) % kPfStages) * 2 * kPfTileBytes) + kPfTileBytes;
#pragma unroll
                        for (int half = 0; half < 2; ++half)
#pragma unroll
                            for (int k16 = 0; k16 < kPfKeys / 16; ++k16)
                                umma_f16_ts(tm + kPfColO, tm + half * kPfColLo + k16 * 8, umma_desc_k_sw128(v_addr + k16 * 2048), idesc_pv,
                                            j > 1 || half > 0 || k16 > 0);
                    }
                    if (j < steps) {
                        tc_fence_after();
                        const uint32_t q_addr = smem_u32(q_tiles + q * kPfTileBytes), k_addr = smem_u32(kv_ring + st * 2 * kPfTileBytes);
#pragma unroll
                        for (int k16 = 0; k16 < kOssDim / 16; ++k16)
                            umma_f16(tm, umma_desc_k_sw128(q_addr + k16 * 32), umma_desc_k_sw128(k_addr + k16 * 32), idesc_qk, k16 > 0);
                        umma_commit(&s_full[q]);
                    } else {
                        umma_commit(&o_full[q]);
                    }
                }
                if (j > 0) umma_commit(&kv_empty[(j - 1) % kPfStages]);
            }
        }
    } else if ((warp >> 2) < qtiles) {
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
        for (int j = 0; j < steps && !*abort_flag; ++j) {
            const int st = j % kPfStages, kb = key0 + j * kPfKeys;
            if (!mbar_wait_bounded(&kv_full[st], (j / kPfStages) & 1) || !mbar_wait_bounded(&s_full[q], j & 1)) {
                *abort_flag = 1;
                break;
            }
            tc_fence_after();
            uint32_t vis[4];
            bool all = true;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                vis[w] = ok_bits[st * 4 + w] & bit_range(begin - kb - 32 * w, end - kb - 32 * w);
                all = all && vis[w] == 0xffffffffu;
            }
            all = __all_sync(0xffffffffu, all);
            float top = -INFINITY;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                uint32_t s[32];
                tmem_ld_32x32(tm + 32 * w, s);
                tmem_ld_wait();
                if (all) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) top = fmaxf(top, __uint_as_float(s[i]));
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) top = fmaxf(top, (vis[w] >> i) & 1 ? __uint_as_float(s[i]) : -INFINITY);
                }
            }
            top *= c;
            const bool grow = j == 0 ? top > ref : top > ref + 8.f;
            if (__any_sync(0xffffffffu, grow)) {
                const float f = grow ? ex2(ref - top) : 1.f;
                if (grow) ref = top;
                sum *= f;
                if (j > 0) {
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        uint32_t o[16];
                        tmem_ld_32x16(tm + kPfColO + 16 * h, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                        tmem_st_32x16(tm + kPfColO + 16 * h, o);
                    }
                }
            }
            const float base = ref == -INFINITY ? 0.f : ref;
            float part[2] = {0.f, 0.f};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                uint32_t s[32], hi[16], lo[16];
                tmem_ld_32x32(tm + 32 * w, s);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float a = ex2(fmaf(__uint_as_float(s[2 * i]), c, -base)), d = ex2(fmaf(__uint_as_float(s[2 * i + 1]), c, -base));
                    if (!all) {
                        a = (vis[w] >> (2 * i)) & 1 ? a : 0.f;
                        d = (vis[w] >> (2 * i + 1)) & 1 ? d : 0.f;
                    }
                    part[0] += a;
                    part[1] += d;
                    hi[i] = bf16x2_of(a, d);
                    lo[i] = bf16x2_of(a - __uint_as_float(hi[i] << 16), d - __uint_as_float(hi[i] & 0xffff0000u));
                }
                tmem_st_32x16(tm + 16 * w, hi);
                tmem_st_32x16(tm + kPfColLo + 16 * w, lo);
            }
            sum += part[0] + part[1];
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[q]);
        }
        if (!*abort_flag && !mbar_wait_bounded(&o_full[q], 0)) *abort_flag = 1;
        tc_fence_after();
        // a wait that gave up leaves NaNs, which no caller can take for a result
        if (*abort_flag) sum = NAN;
        float* out = p.out + (size_t(b) * p.tokens + t) * p.q_heads * kOssDim + head * kOssDim;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            uint32_t o[16];
            tmem_ld_32x16(tm + kPfColO + 16 * h, o);
            tmem_ld_wait();
            if (mine) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = end > begin ? bf16_round_f(__uint_as_float(o[4 * i + e]) / sum) : 0.f;
                    *reinterpret_cast<float4*>(out + 16 * h + 4 * i) = make_float4(v[0], v[1], v[2], v[3]);
                }
            }
            __syncwarp();
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
    auto blocks = [&](int qtiles) { return (p.tokens + tile_tokens * qtiles - 1) / (tile_tokens * qtiles); };
    // Two tiles per CTA keep the exponential unit busy while the other tile's MMAs run; with fewer CTAs than SMs one tile each
    // uses twice the SMs.
    const int qtiles = (long long)p.batch * p.kv_heads * blocks(2) >= kSmCount ? 2 : 1;
    GB_CUDA(cudaFuncSetAttribute(oss_attention_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PfSmem::total));
    oss_attention_prefill_kernel<<<dim3(unsigned(p.kv_heads), unsigned(blocks(qtiles)), unsigned(p.batch)), kPfThreads, PfSmem::total,
                                   stream>>>(p, qtiles);
    GB_CUDA(cudaGetLastError());
    return GARNET_B200_OK;
}

}  // namespace gb200
