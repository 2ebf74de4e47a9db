// gpt-oss decode attention: one new token per sequence, 64-wide heads, paged bf16 cache, learned sinks, sliding window
// (the arithmetic of decodeAttentionPartial / Merge, plugins/gpt_oss/cuda/gpt_oss_kernels.cu:376-428,513-535).
//
// A cluster of up to 8 CTAs serves one (sequence, kv head).  Its visible positions are cut into tiles of 16, which go round
// the cluster's warps; a warp works alone: page lookup of a tile's 16 rows (one per lane), K and V rows by cp.async into the
// warp's own ring of 4 tiles, S = Q K^T and O += P V by mma.sync with the q heads of the group as the 16 MMA rows, running
// maximum and sum in fp32.  The warps of a CTA meet in shared memory, the CTAs of the cluster through distributed shared
// memory, where each CTA finishes some of the heads: no partial results in global memory, no counter, no last CTA.
// Numerics: K is bf16 and the queries are bf16-valued (products exact); queries that are not enter as three bf16 numbers.
// P is fp32 and enters as three bf16 numbers (24 bits).  The tensor core truncates what it accumulates, so sums run over the
// smallest pieces first and P V over one tile only, the tiles being added in fp32.  Share of the results that are not the bf16
// rounding of the float64 result, 16 sequences of 8191 positions: 2.9e-4 by scalar fp32 products over splits of 64, 6.4e-4 with O
// in the MMAs' accumulators, 1.8e-4 as it is now; queries that are not bf16 values, 3000 positions: 4.2e-4, 5.4e-4, 2.1e-4.
// A row whose result is NaN (infinities in the cache meet the zero pieces) is computed again by the general row loop.
//
// Bound: the latency of its chain (lengths -> page -> rows -> softmax -> merge) at one sequence, HBM for a batch: 8 sequences
// of 8192 positions read 134 MB.  Against scalar fp32 products over shared-memory rows with the splits merged by a last CTA:
// 4 sequences of 2250-3000 positions 38.6 -> 15.5 us (ncu, cold caches).
#include <algorithm>
#include <cooperative_groups.h>

#include "gpt_oss_attn.cuh"

namespace gb200 {

namespace {

namespace cg = cooperative_groups;

constexpr int kDecMaxWarps = 8, kDecStages = 4, kDecTile = 16, kDecHeads = 16;
constexpr int kDecStageBytes = 2 * kDecTile * kOssDim * 2;      // K rows, V rows
constexpr int kDecWarpBytes = kDecStages * kDecStageBytes;      // a warp's ring; after the main loop its results:
constexpr int kDecOut = 0, kDecTop = kDecHeads * kOssDim * 4, kDecSum = kDecTop + kDecHeads * 4;   // [head][64], [head], [head]
static_assert(kDecSum + kDecHeads * 4 <= kDecWarpBytes, "the ring holds the warp's results");
constexpr int kDecMaxSplits = 8;

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// One bf16 piece of two fp32 numbers; what it leaves stays in (a, b).
__device__ __forceinline__ uint32_t take_piece(float& a, float& b)
{
    const uint32_t r = bf16x2_of(a, b);
    a -= __uint_as_float(r << 16);
    b -= __uint_as_float(r & 0xffff0000u);
    return r;
}

// 168 registers: three CTAs of four warps on an SM.
__global__ void __maxnreg__(168) oss_attention_decode_kernel(const OssAttn p)
{
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float cta_max[kDecHeads], cta_sum[kDecHeads];
    __shared__ __align__(16) float cta_out[kDecHeads][kOssDim];
    cg::cluster_group cluster = cg::this_cluster();
    const int splits = int(cluster.num_blocks()), split = int(cluster.block_rank());
    const int kv = int(blockIdx.x) / splits, b = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int group = p.q_heads / p.kv_heads;
    pdl_launch_dependents();
    pdl_wait();   // the cache rows and the queries come from the kernels before this one

    const int end = p.lengths[b];
    const bool live = p.active[b] && end > 0 && end <= p.logical_pages * p.page_size;
    const int begin = p.window ? max(0, end - p.window) : 0;
    const int rows = live ? end - begin : 0;
    const int tiles = (rows + kDecTile - 1) / kDecTile;
    const int warps = int(blockDim.x) >> 5, stride = splits * warps, first = split * warps + warp;

    uint8_t* ring = smem + warp * kDecWarpBytes;
    uint64_t there = 0;   // 16 bits per stage: which of its rows exist
    // Rows of two tiles (one per half warp), then a tile's copies from the row offsets of its half.
    const auto look_up = [&](int tile) -> unsigned long long {
        const int r = (tile + (lane >> 4) * stride) * kDecTile + (lane & 15);
        return r < rows ? oss_cache_offset(p, b, begin + r, kv) : SIZE_MAX;
    };
    const auto request = [&](int tile, int stage, unsigned long long offs, int half) {
        if (tile < tiles) {
            const uint64_t bits = (__ballot_sync(0xffffffffu, offs != SIZE_MAX) >> (16 * half)) & 0xffffu;
            there = (there & ~(uint64_t(0xffff) << (16 * stage))) | (bits << (16 * stage));
            const uint32_t kt = smem_u32(ring + stage * kDecStageBytes), vt = kt + kDecStageBytes / 2;
            const int piece = lane & 7;
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int row = it * 4 + (lane >> 3);
                const unsigned long long o = __shfl_sync(0xffffffffu, offs, half * 16 + row);
                const bool valid = o != SIZE_MAX;   // rows that do not exist are filled with zeros
                const size_t at = (valid ? o : 0) + piece * 8;
                const uint32_t to = row * 128 + ((piece ^ (row & 7)) << 4);
                cp_async16(kt + to, p.keys + at, valid);
                cp_async16(vt + to, p.values + at, valid);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    {
        const unsigned long long a = look_up(first), c = look_up(first + 2 * stride);   // both requested at once
#pragma unroll 1   // code that runs once per CTA is fetched cold
        for (int s = 0; s < kDecStages; ++s) request(first + s * stride, s, s < 2 ? a : c, s & 1);
    }
    // the tiles after those: looked up a round of two ahead of their requests
    unsigned long long next = look_up(first + kDecStages * stride);

    // ---- queries: MMA row = head of the group, in bf16 pieces (one when all are bf16 values)
    uint32_t qa[3][4][4];
    uint32_t inexact = 0;
    const bool q_pairs = (reinterpret_cast<uintptr_t>(p.qkv) & 7) == 0, out_wide = (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int head = g + 8 * (r & 1), d = ks * 16 + 2 * t + 8 * (r >> 1);
            float2 f = make_float2(0.f, 0.f);
            if (head < group) {
                const float* from = p.qkv + size_t(b) * (p.q_heads + 2 * p.kv_heads) * kOssDim + (kv * group + head) * kOssDim + d;
                f = q_pairs ? *reinterpret_cast<const float2*>(from) : make_float2(from[0], from[1]);
            }
            inexact |= (__float_as_uint(f.x) | __float_as_uint(f.y)) & 0xffffu;
#pragma unroll
            for (int piece = 0; piece < 3; ++piece) qa[piece][ks][r] = take_piece(f.x, f.y);
        }
    const bool whole = __any_sync(0xffffffffu, inexact != 0);   // all three pieces

    float top[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f}, acc[8][4] = {};
    const float scale = rsqrtf(float(kOssDim));
    int stage = 0;
    for (int tile = first; tile < tiles; tile += stride) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kDecStages - 1) : "memory");
        __syncwarp();
        const uint32_t kt = smem_u32(ring + stage * kDecStageBytes), vt = kt + kDecStageBytes / 2;
        const uint32_t ok = uint32_t(there >> (16 * stage));
        float s[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
            for (int i = 0; i < 4; ++i) s[nt][i] = 0.f;
            const int row = nt * 8 + (lane & 7);
            uint32_t kb[2][4];
#pragma unroll
            for (int half = 0; half < 2; ++half) ldmatrix_x4(kt + row * 128 + (((half * 4 + (lane >> 3)) ^ (row & 7)) << 4), kb[half]);
#pragma unroll
            for (int piece = 2; piece >= 0; --piece) {
                if (piece > 0 && !whole) continue;
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16) mma_bf16_16816(s[nt], qa[piece][k16], kb[k16 >> 1][(k16 & 1) * 2], kb[k16 >> 1][(k16 & 1) * 2 + 1], s[nt]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) s[nt][i] = (ok >> (nt * 8 + 2 * t + (i & 1))) & 1 ? s[nt][i] * scale : -INFINITY;
        }
        // ---- running maximum and sum of head g (values 0, 1) and head g + 8 (values 2, 3)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float m = fmaxf(fmaxf(s[0][2 * h], s[0][2 * h + 1]), fmaxf(s[1][2 * h], s[1][2 * h + 1]));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            m = fmaxf(m, top[h]);
            const float base = m == -INFINITY ? 0.f : m;
            const float f = __expf(top[h] - base);
            top[h] = m;
            sum[h] *= f;
#pragma unroll
            for (int n = 0; n < 8; ++n) acc[n][2 * h] *= f, acc[n][2 * h + 1] *= f;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    s[nt][2 * h + e] = __expf(s[nt][2 * h + e] - base);
                    sum[h] += s[nt][2 * h + e];
                }
        }
        uint32_t pa[3][4];
#pragma unroll
        for (int piece = 0; piece < 3; ++piece)
#pragma unroll
            for (int r = 0; r < 4; ++r) pa[piece][r] = take_piece(s[r >> 1][2 * (r & 1)], s[r >> 1][2 * (r & 1) + 1]);
#pragma unroll
        for (int d = 0; d < 8; d += 2) {
            const int row = lane & 15;
            uint32_t vb[4];
            ldmatrix_x4_trans(vt + row * 128 + (((d + (lane >> 4)) ^ (row & 7)) << 4), vb);
            float pv[2][4] = {};
#pragma unroll
            for (int piece = 2; piece >= 0; --piece) {
                mma_bf16_16816(pv[0], pa[piece], vb[0], vb[1], pv[0]);
                mma_bf16_16816(pv[1], pa[piece], vb[2], vb[3], pv[1]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[d][i] += pv[0][i], acc[d + 1][i] += pv[1][i];
        }
        __syncwarp();   // the stage is read: its next tile may come in
        request(tile + kDecStages * stride, stage, next, stage & 1);
        if (stage & 1) next = look_up(tile + (kDecStages + 1) * stride);
        stage = (stage + 1) & (kDecStages - 1);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // every ring is free

    // ---- the CTA's result of each head
    float* w_out = reinterpret_cast<float*>(ring + kDecOut);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
        sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
        const int head = g + 8 * h;
        if (head >= group) continue;
        if (t == 0) *reinterpret_cast<float*>(ring + kDecTop + head * 4) = top[h], *reinterpret_cast<float*>(ring + kDecSum + head * 4) = sum[h];
#pragma unroll
        for (int n = 0; n < 8; ++n)
            *reinterpret_cast<float2*>(w_out + head * kOssDim + n * 8 + 2 * t) = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
    }
    __syncthreads();
    const int d4 = (threadIdx.x & 15) * 4;   // 16 threads per head, four values each
    for (int head = threadIdx.x >> 4; head < group; head += warps * 2) {
        float m = -INFINITY;
        for (int w = 0; w < warps; ++w) m = fmaxf(m, *reinterpret_cast<const float*>(smem + w * kDecWarpBytes + kDecTop + head * 4));
        const float base = m == -INFINITY ? 0.f : m;
        float total = 0.f;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int w = 0; w < warps; ++w) {
            const uint8_t* from = smem + w * kDecWarpBytes;
            const float f = __expf(*reinterpret_cast<const float*>(from + kDecTop + head * 4) - base);
            const float4 v = *reinterpret_cast<const float4*>(from + kDecOut + (head * kOssDim + d4) * 4);
            total += f * *reinterpret_cast<const float*>(from + kDecSum + head * 4);
            o.x += f * v.x, o.y += f * v.y, o.z += f * v.z, o.w += f * v.w;
        }
        if ((threadIdx.x & 15) == 0) cta_max[head] = m, cta_sum[head] = total;
        *reinterpret_cast<float4*>(&cta_out[head][d4]) = o;
    }
    cluster.sync();
    // ---- the CTAs' results and the sink (denominator only); the heads go round the cluster, two per warp and round
    for (int h0 = warp * 2; h0 * splits < group; h0 += warps * 2) {
        const int head = (h0 + (lane >> 4)) * splits + split;
        bool bad = false;
        if (head < group) {
            const float sink = p.sinks[kv * group + head];
            float pm[kDecMaxSplits], ps[kDecMaxSplits];
            float4 po[kDecMaxSplits];
#pragma unroll
            for (int c = 0; c < kDecMaxSplits; ++c) {
                const int from = c < splits ? c : 0;
                pm[c] = *cluster.map_shared_rank(&cta_max[head], from);
                ps[c] = c < splits ? *cluster.map_shared_rank(&cta_sum[head], from) : 0.f;
                po[c] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&cta_out[head][d4], from));
            }
            float m = sink;
#pragma unroll
            for (int c = 0; c < kDecMaxSplits; ++c) m = fmaxf(m, pm[c]);
            float total = __expf(sink - m);
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int c = 0; c < kDecMaxSplits; ++c) {
                if (ps[c] == 0.f) continue;   // nothing visible there
                const float f = __expf(pm[c] - m);
                total += f * ps[c];
                o.x += f * po[c].x, o.y += f * po[c].y, o.z += f * po[c].z, o.w += f * po[c].w;
            }
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live)
                r = make_float4(bf16_round_f(o.x / total), bf16_round_f(o.y / total), bf16_round_f(o.z / total), bf16_round_f(o.w / total));
            bad = isnan(r.x) || isnan(r.y) || isnan(r.z) || isnan(r.w);
            float* to = p.out + (size_t(b) * p.q_heads + kv * group + head) * kOssDim + d4;
            if (out_wide) *reinterpret_cast<float4*>(to) = r;
            else to[0] = r.x, to[1] = r.y, to[2] = r.z, to[3] = r.w;
        }
        __syncwarp();   // the row loop writes over what these lanes have written
        const uint32_t redo = __ballot_sync(0xffffffffu, bad);
        for (int h = 0; h < 2; ++h)
            if ((redo >> (16 * h)) & 0xffffu) oss_attention_row(p, b, kv * group + (h0 + h) * splits + split, lane);
    }
    cluster.sync();   // peers may still read this CTA's results
}

}  // namespace

bool oss_decode_takes(const OssAttn& p)
{
    const uintptr_t bits = reinterpret_cast<uintptr_t>(p.keys) | reinterpret_cast<uintptr_t>(p.values);
    return p.tokens == 1 && !p.prefill && p.head_dim == kOssDim && p.q_heads / p.kv_heads <= kDecHeads && (bits & 15) == 0 && p.batch <= 65535;
}

int oss_decode_launch(const OssAttn& p, cudaStream_t stream)
{
    // As many CTAs per (sequence, kv head) as have a tile for each of their warps; a grid of more than eight CTAs per SM, which is
    // well over two waves, gets smaller clusters.  With more CTAs than SMs a CTA has four warps, so that three fit an SM (64 KiB of
    // rings, 168 registers); else eight.
    const long long span = (long long)p.logical_pages * p.page_size, seen = p.window ? std::min<long long>(p.window, span) : span;
    const long long pairs = (long long)p.batch * p.kv_heads;
    int splits = kDecMaxSplits;
    while (splits > 1 && ((seen + splits - 1) / splits < kDecMaxWarps * kDecTile || pairs * splits > 8 * kSmCount)) splits /= 2;
    GB_CUDA(cudaFuncSetAttribute(oss_attention_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kDecMaxWarps * kDecWarpBytes));
    const int warps = pairs * splits > kSmCount ? kDecMaxWarps / 2 : kDecMaxWarps;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(splits * p.kv_heads), unsigned(p.batch));
    cfg.blockDim = dim3(unsigned(warps * 32));
    cfg.dynamicSmemBytes = warps * kDecWarpBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim = {unsigned(splits), 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    GB_CUDA(cudaLaunchKernelEx(&cfg, oss_attention_decode_kernel, p));
    return GARNET_B200_OK;
}

}  // namespace gb200
